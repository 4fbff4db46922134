// dem_mixed.cu -- mixed-precision force path (DEM_PREC_MIXED).
//
// Same sweep, same pair sets, same history semantics and summation order as
// the FP64 kernel; what changes is the arithmetic of a contact:
//  - the candidate test DeltaDijSq = MinDijSq - DijSq stays FP64 (from FP64
//    positions), so the contact-pair set equals the FP64 one;
//  - the overlap is formed as delta = DeltaDijSq / (MinDij + Dij), which
//    keeps its relative digits in FP32 (MinDij - Dij itself would cancel);
//  - everything downstream (normal, relative velocity, spring-dashpot,
//    tangential spring, Coulomb cap, torques, per-particle sums) is FP32;
//  - the tangential spring is carried as an FP32 pair (hi, lo) and each
//    increment is added with a compensated (Kahan/TwoSum) sum;
//  - velocities are gathered as FP32 copies; positions, the ABM ring and
//    the predictor/corrector stay FP64.
// This translation unit is compiled without multiply-add contraction (every
// kernel that inlines the same code then rounds alike), with the hardware's
// approximate FP32 division and square root.
#include "dem_mixed.cuh"
#include "dem_test.cuh"

namespace dem {

namespace {

struct F3 {
  float x, y, z;
};
__device__ __forceinline__ F3 mk(float x, float y, float z) { return F3{x, y, z}; }
__device__ __forceinline__ F3 operator+(F3 a, F3 b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ F3 operator-(F3 a, F3 b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ F3 operator*(float s, F3 a) { return mk(s * a.x, s * a.y, s * a.z); }
// (dot and cross products and the two-term combinations below use explicit
// fused multiply-adds: one rounding per term, whatever kernel inlines them)
__device__ __forceinline__ float dot(F3 a, F3 b) {
  return __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)));
}
__device__ __forceinline__ F3 cross(F3 a, F3 b) {
  return mk(__fmaf_rn(a.y, b.z, -__fmul_rn(a.z, b.y)), __fmaf_rn(a.z, b.x, -__fmul_rn(a.x, b.z)),
            __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x)));
}
// s*a + t*b
__device__ __forceinline__ F3 comb(float s, F3 a, float t, F3 b) {
  return mk(__fmaf_rn(s, a.x, __fmul_rn(t, b.x)), __fmaf_rn(s, a.y, __fmul_rn(t, b.y)),
            __fmaf_rn(s, a.z, __fmul_rn(t, b.z)));
}
// a - s*b
__device__ __forceinline__ F3 sub_scaled(F3 a, float s, F3 b) {
  return mk(__fmaf_rn(-s, b.x, a.x), __fmaf_rn(-s, b.y, a.y), __fmaf_rn(-s, b.z, a.z));
}
// FP64 sums of a particle's FP32 contributions (exact terms, one rounding
// per addition at FP64: the net force of a packing, where contact forces
// nearly cancel, keeps the contact forces' own accuracy)
struct D3 {
  double x, y, z;
};
__device__ __forceinline__ D3 operator+(D3 a, F3 b) {
  return D3{a.x + (double)b.x, a.y + (double)b.y, a.z + (double)b.z};
}
__device__ __forceinline__ D3 operator-(D3 a, F3 b) {
  return D3{a.x - (double)b.x, a.y - (double)b.y, a.z - (double)b.z};
}

struct MPair {
  float min_dij, kn, yn, kt, yt, mu_sq;
};

template <bool PP>
struct MMat;

template <>
struct MMat<false> {
  __device__ __forceinline__ static double min_dij_sq(const DevParams& P, int ca, double, int cb,
                                                      double) {
    return P.min_dij_sq[ca * NCM + cb];
  }
  __device__ __forceinline__ static void pair(const DevParams& P, int ca, float, int cb, float,
                                              MPair& m) {
    int k = ca * NCM + cb;
    m.min_dij = (float)P.min_dij[k];
    m.kn = (float)P.kn[k];
    m.yn = (float)P.yn[k];
    m.kt = (float)P.kt[k];
    m.yt = (float)P.yt[k];
    m.mu_sq = (float)P.mu_sq[k];
  }
  __device__ __forceinline__ static void wall(const DevParams& P, int ca, float, int w, MPair& m) {
    int k = ca * NWM + w;
    m.kn = (float)P.knw[k];
    m.yn = (float)P.ynw[k];
    m.kt = (float)P.ktw[k];
    m.yt = (float)P.ytw[k];
    m.mu_sq = (float)P.muw_sq[k];
  }
  __device__ __forceinline__ static void self(const DevParams& P, int ca, float, float& im,
                                              float& ii, float& em) {
    im = (float)P.comp_inv_mass[ca];
    ii = (float)P.comp_inv_inertia[ca];
    em = (float)P.comp_eff_mass[ca];
  }
};

template <>
struct MMat<true> {
  __device__ __forceinline__ static double min_dij_sq(const DevParams&, int, double Ra, int,
                                                      double Rb) {
    double d = Ra + Rb;
    return d * d;
  }
  __device__ __forceinline__ static float mass(const DevParams& P, float R) {
    return (float)P.pp_mass_coef * (R * R * R);
  }
  __device__ __forceinline__ static void pair(const DevParams& P, int, float Ra, int, float Rb,
                                              MPair& m) {
    float ma = mass(P, Ra), mb = mass(P, Rb);
    float meff = ma * mb / (ma + mb);
    m.min_dij = Ra + Rb;
    m.kn = (float)P.pp_kn;
    m.kt = (float)P.pp_kt;
    m.yn = (float)P.pp_gamma_n * sqrtf(meff * m.kn);
    m.yt = (float)P.pp_gamma_t * sqrtf(meff * m.kt);
    m.mu_sq = (float)P.pp_mu_sq;
  }
  __device__ __forceinline__ static void wall(const DevParams& P, int, float Ra, int w, MPair& m) {
    float ma = mass(P, Ra);
    m.kn = (float)P.pp_knw[w];
    m.kt = (float)P.pp_ktw[w];
    m.yn = (float)P.pp_gamma_nw[w] * sqrtf(ma * m.kn);
    m.yt = (float)P.pp_gamma_tw[w] * sqrtf(ma * m.kt);
    m.mu_sq = (float)P.pp_muw_sq[w];
  }
  __device__ __forceinline__ static void self(const DevParams& P, int, float R, float& im,
                                              float& ii, float& em) {
    float m = mass(P, R);
    im = 1.0f / m;
    ii = 1.0f / (0.4f * m * (R * R));
    em = (float)((double)m * (P.pp_density - P.pp_fluid_density) / P.pp_density);
  }
};

__device__ __forceinline__ F3 change_plane_f(F3 V, F3 N) {
  F3 P = sub_scaled(V, dot(V, N), N);
  float ns = dot(P, P);
  if (ns != 0.0f) return sqrtf(dot(V, V) / ns) * P;
  return mk(0.f, 0.f, 0.f);
}

// TwoSum: s + e == a + b exactly
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  float bp = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

struct MOut {
  F3 FN, FT, FTlo, VT, N, NxFT;
};

// CommonCalculations (src/MForces.f90:339-387) in FP32 given the geometry.
__device__ __forceinline__ void common_mixed(F3 Rij, F3 N, F3 DispN, F3 Vij, F3 VijC,
                                             float DeltaDijSq, float half_dt, bool contacting,
                                             F3 ft0, F3 ft0lo, F3 vt0, const MPair& m, MOut& o) {
  F3 VijN = dot(VijC, N) * N;
  o.VT = VijC - VijN;
  o.FN = comb(m.kn, DispN, m.yn, VijN);
  if (contacting) {
    F3 VT0 = change_plane_f(vt0, N);
    F3 dD = half_dt * (VT0 + o.VT);
    F3 dV = o.VT - VT0;
    // rotate the compensated spring (hi + lo) onto the new contact plane
    F3 ph = sub_scaled(ft0, dot(ft0, N), N);
    F3 pl = sub_scaled(ft0lo, dot(ft0lo, N), N);
    float ns = dot(ph, ph);
    F3 hi = mk(0.f, 0.f, 0.f), lo = mk(0.f, 0.f, 0.f);
    if (ns != 0.0f) {
      float f = sqrtf(dot(ft0, ft0) / ns);
      hi = f * ph;
      lo = f * pl;
    }
    F3 inc = comb(m.kt, dD, m.yt, dV);
    float e;
    two_sum(hi.x, inc.x, o.FT.x, e);
    o.FTlo.x = lo.x + e;
    two_sum(hi.y, inc.y, o.FT.y, e);
    o.FTlo.y = lo.y + e;
    two_sum(hi.z, inc.z, o.FT.z, e);
    o.FTlo.z = lo.z + e;
  } else {
    float PartialDt;
    float VijSq = dot(Vij, Vij);
    if (VijSq > 0.0f) {
      // (R.V + sqrt((R.V)^2 + |V|^2 dD2)) / |V|^2; for approaching particles
      // (R.V < 0) the sum cancels, so use the equal form dD2 / (sqrt(..) - R.V)
      float RijVij = dot(Rij, Vij);
      float a = 2.0f * half_dt;
      float root = sqrtf(RijVij * RijVij + VijSq * DeltaDijSq);
      float b = RijVij >= 0.0f ? (RijVij + root) / VijSq : DeltaDijSq / (root - RijVij);
      PartialDt = b < a ? b : a;
    } else {
      PartialDt = 0.0f;
    }
    o.FT = (m.kt * PartialDt + m.yt) * o.VT;
    o.FTlo = mk(0.f, 0.f, 0.f);
  }
  float mun = m.mu_sq * dot(o.FN, o.FN);
  float nt = dot(o.FT, o.FT);
  if (nt > mun) {
    float g = sqrtf(mun / nt);
    o.FT = g * o.FT;
    o.FTlo = g * o.FTlo;
  }
  o.N = N;
  o.NxFT = cross(N, o.FT);
}

// pair branch (src/MForces.f90:230-252), "i" = a, "j" = b, Rij = xb - xa
__device__ __forceinline__ void mixed_pair(const double Rd[3], double DijSq, double Delta,
                                           const MPair& m, float Ra, F3 va, F3 wa, float Rb,
                                           F3 vb, F3 wb, float half_dt, bool contacting, F3 ft0,
                                           F3 ft0lo, F3 vt0, MOut& o) {
  const float D = sqrtf((float)DijSq);
  const float fDelta = (float)Delta;
  const float delta = fDelta / (m.min_dij + D);  // = MinDij - Dij, without cancellation
  const float rD = 1.0f / D;
  F3 Rij = mk((float)Rd[0], (float)Rd[1], (float)Rd[2]);
  F3 N = rD * Rij;
  F3 DispN = (-delta) * N;
  F3 Vij = vb - va;
  F3 ws = Ra * wa + Rb * wb;
  F3 VijC = Vij - cross(ws, N);
  common_mixed(Rij, N, DispN, Vij, VijC, fDelta, half_dt, contacting, ft0, ft0lo, vt0, m, o);
}

__device__ __forceinline__ void rec_read(const float4* a, const float4* b, const float* c,
                                         size_t i, F3& ft, F3& lo, F3& vt) {
  float4 x = a[i], y = b[i];
  ft = mk(x.x, x.y, x.z);
  vt = mk(x.w, y.x, y.y);
  lo = mk(y.z, y.w, c[i]);
}
__device__ __forceinline__ void rec_write(float4* a, float4* b, float* c, size_t i, F3 ft, F3 lo,
                                          F3 vt) {
  a[i] = make_float4(ft.x, ft.y, ft.z, vt.x);
  b[i] = make_float4(vt.y, vt.z, lo.x, lo.y);
  c[i] = lo.z;
}

// a pair record: one 32-byte piece and the last remainder
__device__ __forceinline__ void pair_rec_read(const F8* a, const float* c, size_t i, F3& ft, F3& lo,
                                              F3& vt) {
  const F8 x = ld32(a + i);
  ft = mk(x.v[0], x.v[1], x.v[2]);
  vt = mk(x.v[3], x.v[4], x.v[5]);
  lo = mk(x.v[6], x.v[7], c[i]);
}
__device__ __forceinline__ void pair_rec_write(F8* a, float* c, size_t i, F3 ft, F3 lo, F3 vt) {
  st32(a + i, F8{{ft.x, ft.y, ft.z, vt.x, vt.y, vt.z, lo.x, lo.y}});
  c[i] = lo.z;
}

// The mixed-precision force pass: the FP64 pass's structure (the same test
// kernel and contact list, exact FP64 overlap test, orientation, history
// semantics, each contact evaluated once, summation order), FP32 contact
// arithmetic, FP64 integrator epilogue.

// The pair kernel: one thread per contact (pair_sweep).  (Body for block
// `vblock` of a grid of `vgrid` blocks.)
template <bool PP>
__device__ __forceinline__ void pair_mixed_body(const PassArgs<float4, float2>& A,
                                                const MixedView& V, int vblock, int vgrid,
                                                int nseg) {
  __shared__ int s_abort;
  if (threadIdx.x == 0) s_abort = A.cnt->abort;
  __syncthreads();
  if (s_abort) return;
  const int total = A.cnt->n_contacts;
  if (vblock == 0 && threadIdx.x == 0) {
    // the pass's pair contacts: the length of its contact list
    atomicAdd(&A.cnt->pair_contacts, (unsigned long long)total);
    atomicMax(&A.cnt->need_cl, total);
  }
  const bool update = A.update != 0;
  const float half_dt = (float)A.half_dt;
  const History& Hr = A.Hr;
  const History& Hw = A.Hw;
  unsigned n_col = 0;
  int need = 0, need_in = 0;
  bool overflow = false, in_over = false;
  // A contact's pair record is nearly always at the contact's own number
  // among i's (the table is written in that order and contacts last for many
  // passes), so that slot is read together with the particles' data; the
  // next contact's list entry is read a turn ahead, and its partner's data
  // requested into L2 before this one's results are written.
  const PairSweep w = pair_sweep(total, vblock, vgrid, nseg);
  const int stride = w.stride, end = w.end;
  int s = w.first + threadIdx.x;
  int2 e = make_int2(0, 0);
  int ord = 0;
  if (s < end) {
    e = A.clist[s];
    ord = A.cord[s];
  }
  while (s < end) {
    const int p = e.x, q = e.y;
    const int s_in = atomicAdd(&A.in_cnt[q], 1);  // q's "j" record (returns early)
    int2 e2 = e;
    int ord2 = 0;
    if (s + stride < end) {
      e2 = A.clist[s + stride];
      ord2 = A.cord[s + stride];
    }
    if (ord == ORD_MAX) ord = s - A.cstart[p];
    const int hc = Hr.cnt[p];
    const bool room = ord < Hr.cap;
    const size_t hg = hslot(Hr, p, room ? ord : 0);
    const int kg = Hr.key[hg];
    F3 ft0, ft0lo, vt0;
    pair_rec_read(V.r8, V.rc, hg, ft0, ft0lo, vt0);
    const DevParams& P = sys_params(A.P, A.sysid, p);
    const double4 p4 = ld32(A.X + p), q4 = ld32(A.X + q);
    const float4 pv4 = A.v4[p], qv4 = A.v4[q];
    const float2 pw2 = A.w2[p], qw2 = A.w2[q];
    const int cp = PP ? 0 : A.comp[p], cq = PP ? 0 : A.comp[q];
    double Rij[3] = {q4.x - p4.x, q4.y - p4.y, q4.z - p4.z};
#pragma unroll
    for (int k = 0; k < 3; k++) Rij[k] = min_image_exact(Rij[k], P.box, k);
    const double DijSq = sumsq3(Rij);
    const double Delta = MMat<PP>::min_dij_sq(P, cp, p4.w, cq, q4.w) - DijSq;
    const float Ra = (float)p4.w, Rb = (float)q4.w;
    MPair m;
    MMat<PP>::pair(P, cp, Ra, cq, Rb, m);
    const F3 vo = mk(pv4.x, pv4.y, pv4.z), wo = mk(pv4.w, pw2.x, pw2.y);
    const F3 vq = mk(qv4.x, qv4.y, qv4.z), wq = mk(qv4.w, qw2.x, qw2.y);
    // i's records, then j's
    int r = room && ord < hc && kg == q ? ord : -1;
    bool contacting = r >= 0;
    if (!contacting) {
      r = find_record(Hr, p, q);
      contacting = r >= 0;
      if (contacting) {
        pair_rec_read(V.r8, V.rc, hslot(Hr, p, r), ft0, ft0lo, vt0);
      } else {
        const int r2 = find_record(Hr, q, p);
        contacting = r2 >= 0;
        if (contacting) pair_rec_read(V.r8, V.rc, hslot(Hr, q, r2), ft0, ft0lo, vt0);
      }
    }
    // (the fold reads the matched bits of history-updating passes only)
    if (update && r >= 0 && r < 32) atomicOr(&A.matched[p], 1u << r);
    if (!contacting) n_col++;
    MOut out;
    mixed_pair(Rij, DijSq, Delta, m, Ra, vo, wo, Rb, vq, wq, half_dt, contacting, ft0, ft0lo,
               vt0, out);
    const F3 FTs = out.FT + out.FTlo;
    if (s + stride < end) {
      prefetch_l2(A.X + e2.y);
      prefetch_l2(A.v4 + e2.y);
      prefetch_l2(A.w2 + e2.y);
      prefetch_l2(A.in_cnt + e2.y);
    }
    // "j" half into q's incoming records
    if (s_in < A.in_cap) {
      const unsigned long long key = sweep_key(A.cell_cur[p], A.rank[p]);
      char* const in = (char*)A.in_rec;
      st32((F8*)(in + in_head(IN_BYTES32, A.in_stride, s_in, q)),
           F8{{out.FN.x, out.FN.y, out.FN.z, FTs.x, FTs.y, FTs.z, out.NxFT.x, out.NxFT.y}});
      *(float4*)(in + in_tail(IN_BYTES32, A.in_stride, s_in, q)) =
          make_float4(out.NxFT.z, 0.f, __uint_as_float((unsigned)key),
                      __uint_as_float((unsigned)(key >> 32)));
    } else {
      in_over = true;
    }
    need_in = need_in > s_in + 1 ? need_in : s_in + 1;
    // "i" half at the contact's place
    const F3 tq = cross(Ra * out.N, out.FT);
    st32((F8*)A.irec + s,
         F8{{out.FN.x, out.FN.y, out.FN.z, FTs.x, FTs.y, FTs.z, tq.x, tq.y}});
    ((float*)A.irec9)[s] = tq.z;
    if (update) {
      if (ord < Hw.cap) {
        const size_t i = hslot(Hw, p, ord);
        Hw.key[i] = q;
        pair_rec_write(V.w8, V.wc, i, out.FT, out.FTlo, out.VT);
      } else {
        overflow = true;
      }
      need = need > ord + 1 ? need : ord + 1;
    }
    s += stride;
    e = e2;
    ord = ord2;
  }
  if (overflow) {
    atomicExch(&A.cnt->overflow, 1);
    set_abort(A.cnt, A.tag);
  }
  if (in_over) {
    atomicExch(&A.cnt->in_overflow, 1);
    set_abort(A.cnt, A.tag);
  }
  publish_pair_block(A.cnt, update, n_col, (unsigned)need, (unsigned)need_in);
}

template <bool PP, int MINB>
__global__ void __launch_bounds__(128, MINB) k_pair_mixed(PassArgs<float4, float2> A,
                                                          MixedView V, int nseg) {
  pass_kernel_entry();
  pair_mixed_body<PP>(A, V, blockIdx.x, gridDim.x, nseg);
}

// The fold kernel: p's block of the sweep, Force and Torque in sweep order
// (FP32), a = F/m, alpha = T/I, then the FP64 integrator epilogue.  WALLS:
// some system has walls; CONE: some wall is a cone.  (Body for block
// `vblock` of particles.)
template <bool PP, int EPI, bool WALLS, bool CONE>
__device__ __forceinline__ void fold_mixed_body(const PassArgs<float4, float2>& A,
                                                const MixedView& V, int vblock, double* stage) {
  __shared__ float s_w[WALLS ? NWM : 1][128];  // |FN| of each wall contact
  __shared__ int s_abort;
  const int p0 = vblock * blockDim.x + threadIdx.x;
  const int p = p0 < A.n ? p0 : 0;
  // requested together: the abort word (one decision for the warp; with walls,
  // for the block, which meets block barriers later), what the contact results
  // hang on, the particle's own data, then the integrator's columns.  (The
  // columns first: 119.7 us per launch at 1M spheres with 0.8 contacts each
  // instead of 116.7, 416 instead of 398 at 4M.  The FP64 fold has them first
  // and loses the other way round, 131.5 instead of 128.4.)
  int stop = 0;
  if (threadIdx.x == 0 || (!WALLS && (threadIdx.x & 31) == 0)) stop = A.cnt->abort;
  const int ni = A.in_cnt[p];
  const unsigned matched = A.matched[p];
  const int c = A.cell_cur[p];
  const int rank = A.rank[p];
  const int nc = A.ccount[p];
  const int st0 = A.cstart[p];
  const double4 p4 = ld32(A.X + p);
  stage_epilogue<EPI, true>(A, vblock * blockDim.x, stage);
  if (WALLS) {
    if (threadIdx.x == 0) s_abort = stop;
    __syncthreads();
    stop = s_abort;
  } else {
    stop = __shfl_sync(0xffffffffu, stop, 0);
  }
  if (stop) {
    stage_wait();
    return;
  }
  if (WALLS)
    for (int w = 0; w < A.nw_max; w++) s_w[w][threadIdx.x] = 0.f;
  if (vblock == 0 && threadIdx.x == 0) atomicAdd(&A.cnt->pass_id, 1);  // this pass is done
  // (a slab of a decomposition advances only its own particles)
  const bool valid = p0 < A.n && in_slab(sys_params(A.P, A.sysid, p), c);
  const int most = __reduce_max_sync(0xffffffffu, valid ? ni : 0);
  const bool update = A.update != 0;
  const History& Hr = A.Hr;
  const History& Hw = A.Hw;
  unsigned n_wc = 0;
  int need = 0;
  bool overflow = false;
  double d2 = 0.0, acc[3] = {0.0, 0.0, 0.0}, alp[3] = {0.0, 0.0, 0.0};
  if (valid) {
    const DevParams& P = sys_params(A.P, A.sysid, p);
    const unsigned long long key_p = sweep_key(c, rank);
    if (ni) A.in_cnt[p] = 0;  // for the next pass's pair kernel
    if (matched) A.matched[p] = 0u;
    const double xp[3] = {p4.x, p4.y, p4.z};
    const double Rpd = p4.w;
    const float Rp = (float)Rpd;
    const int cp = PP ? 0 : A.comp[p];
    float inv_m, inv_i, eff_m;
    MMat<PP>::self(P, cp, Rp, inv_m, inv_i, eff_m);
    // ---- p's block: gravity, its contacts as "i" in row order
    F3 iF = mk(eff_m * (float)P.gravity[0], eff_m * (float)P.gravity[1],
               eff_m * (float)P.gravity[2]);
    F3 iT = mk(0.f, 0.f, 0.f);
    // (two records in flight at a time)
    auto load_ir = [&](int k) {
      return IRec32{ld32((const F8*)A.irec + (st0 + k)), ((const float*)A.irec9)[st0 + k]};
    };
    auto add_ir = [&](const IRec32& r) {
      iF = iF + mk(r.a.v[0], r.a.v[1], r.a.v[2]) + mk(r.a.v[3], r.a.v[4], r.a.v[5]);
      iT = iT + mk(r.a.v[6], r.a.v[7], r.z);
    };
    const char* const in = (const char*)A.in_rec;
    const SweepOrder ord = sweep_order(ni, most, key_p, in, IN_BYTES32, A.in_stride, p);
    for (int k = 0; k < nc; k += 2) {
      const IRec32 r0 = load_ir(k);
      IRec32 r1;
      if (k + 1 < nc) r1 = load_ir(k + 1);
      add_ir(r0);
      if (k + 1 < nc) add_ir(r1);
    }
    int hw_n = nc;  // the pair kernel wrote the records of the contacts
    if (WALLS) {
      const float4 pv4 = A.v4[p];
      const float2 pw2 = A.w2[p];
      const F3 vp = mk(pv4.x, pv4.y, pv4.z);
      const F3 wp = mk(pv4.w, pw2.x, pw2.y);
      const float half_dt = (float)A.half_dt;
      for (int w = 0; w < P.nw; w++) {
        const dem_wall& W = P.walls[w];
        const size_t wi = (size_t)p * P.nw + w;
        const bool contacting = Hr.wflag[wi] != 0;
        F3 ft0 = mk(0.f, 0.f, 0.f), ft0lo = ft0, vt0 = ft0;
        if (contacting) rec_read(V.rwa, V.rwb, V.rwc, wi, ft0, ft0lo, vt0);
        double Dij, Nij[3], Qji[3];
        const bool ov = overlap_wall<CONE>(P, W, xp, Rpd, Dij, Nij, Qji);
        if (ov) {
          n_wc++;
          const double Delta = Rpd * Rpd - Dij * Dij;
          const float delta = (float)(Rpd - Dij);
          F3 N = mk((float)Nij[0], (float)Nij[1], (float)Nij[2]);
          F3 Q = mk((float)Qji[0], (float)Qji[1], (float)Qji[2]);
          F3 wv = mk((float)W.velocity[0], (float)W.velocity[1], (float)W.velocity[2]);
          F3 ww = mk((float)W.omega[0], (float)W.omega[1], (float)W.omega[2]);
          F3 Vij = (wv + cross(ww, Q)) - vp;
          F3 VijC = Vij - cross(Rp * wp, N);
          F3 Rw = mk((float)(W.position[0] + Qji[0] - xp[0]),
                     (float)(W.position[1] + Qji[1] - xp[1]),
                     (float)(W.position[2] + Qji[2] - xp[2]));
          MPair m;
          MMat<PP>::wall(P, cp, Rp, w, m);
          MOut o;
          common_mixed(Rw, N, (-delta) * N, Vij, VijC, (float)Delta, half_dt, contacting, ft0,
                       ft0lo, vt0, m, o);
          iF = iF + o.FN + (o.FT + o.FTlo);
          iT = iT + cross(Rp * o.N, o.FT);
          s_w[w][threadIdx.x] = sqrtf(dot(o.FN, o.FN));
          if (update) {
            Hw.wflag[wi] = 1;
            rec_write(V.wwa, V.wwb, V.wwc, wi, o.FT, o.FTlo, o.VT);
          }
        } else if (update) {
          Hw.wflag[wi] = 0;
        }
      }
    }
    if (A.drag)  // iForce = iForce + DragForce(iPart) (src/MForces.f90:316)
      iF = iF + mk((float)A.drag[(size_t)3 * p], (float)A.drag[(size_t)3 * p + 1],
                   (float)A.drag[(size_t)3 * p + 2]);
    if (update) {
      const int hc = Hr.cnt[p];
      for (int r = 0; r < hc; r++) {
        if (r < 32 && ((matched >> r) & 1u)) continue;
        const size_t i = hslot(Hr, p, r);
        const int q2 = Hr.key[i];
        if (q2 >= A.n || !partner_adjacent(A, P, c, q2)) {
          if (hw_n < Hw.cap) {
            F3 ft, lo, vt;
            pair_rec_read(V.r8, V.rc, i, ft, lo, vt);
            const size_t o = hslot(Hw, p, hw_n);
            Hw.key[o] = q2;
            pair_rec_write(V.w8, V.wc, o, ft, lo, vt);
          } else {
            overflow = true;
          }
          hw_n++;
        }
      }
      Hw.cnt[p] = hw_n < Hw.cap ? hw_n : Hw.cap;
      if (hw_n > Hw.cap) overflow = true;
      need = hw_n;
    }
    // ---- Force and Torque in sweep order
    D3 F = D3{0.0, 0.0, 0.0}, T = D3{0.0, 0.0, 0.0};
    fold_in_order(
        ni, key_p, ord, in, IN_BYTES32, A.in_stride, p,
        [&](int e) {
          return InRec32{ld32((const F8*)(in + in_head(IN_BYTES32, A.in_stride, e, p))),
                         *(const float*)(in + in_tail(IN_BYTES32, A.in_stride, e, p))};
        },
        [&]() {
          F = F + iF;
          T = T + iT;
        },
        [&](const InRec32& r) {
          const F3 FN = mk(r.a.v[0], r.a.v[1], r.a.v[2]), FTs = mk(r.a.v[3], r.a.v[4], r.a.v[5]);
          const F3 NxFT = mk(r.a.v[6], r.a.v[7], r.z);
          F = F - FN - FTs;
          T = T + Rp * NxFT;
        });
    if (EPI == EPI_STORE && A.amsum) {
      const size_t n3 = (size_t)3 * A.n, q = (size_t)3 * p;
      A.amsum[q] = F.x; A.amsum[q + 1] = F.y; A.amsum[q + 2] = F.z;
      A.amsum[n3 + q] = T.x; A.amsum[n3 + q + 1] = T.y; A.amsum[n3 + q + 2] = T.z;
    }
    acc[0] = F.x * (double)inv_m;
    acc[1] = F.y * (double)inv_m;
    acc[2] = F.z * (double)inv_m;
    alp[0] = T.x * (double)inv_i;
    alp[1] = T.y * (double)inv_i;
    alp[2] = T.z * (double)inv_i;
  }
  stage_wait();
  if (valid) {
    // the integrator runs on FP64 velocities: Particle's for the predictor,
    // Predicted's for the corrector (the pass copies are FP32)
    const DevParams& P = sys_params(A.P, A.sysid, p);
    const double* const cols = stage + threadIdx.x;
    const double xp[3] = {p4.x, p4.y, p4.z};
    double vd[3] = {0.0, 0.0, 0.0}, wd[3] = {0.0, 0.0, 0.0};
    if (EPI == EPI_PREDICT) {
#pragma unroll
      for (int d = 0; d < 3; d++) vd[d] = cols[(27 + d) * 128];
#pragma unroll
      for (int d = 0; d < 3; d++) wd[d] = cols[(30 + d) * 128];
    } else if (EPI == EPI_CORRECT) {
#pragma unroll
      for (int d = 0; d < 3; d++) vd[d] = cols[(18 + d) * 128];
    }
    epilogue<EPI>(A, P, p, xp, p4.w, vd, wd, acc, alp, c, cols, d2);
  }
  if (WALLS && A.nw_max > 0) wall_partials(s_w, A.nw_max, A.wall_part, vblock);
  if (overflow) {
    atomicExch(&A.cnt->overflow, 1);
    set_abort(A.cnt, A.tag);
  }
  publish_fold(A.cnt, n_wc, (unsigned)need, d2);
}

// (STRIDE: grid-stride over blocks of 128 particles.  The kernel is bound by
// the latency of the contact results it gathers and by instruction issue,
// not by its streams: the staged columns alone move at 6.2 TB/s.  Register
// budget: 5 blocks of 128 per SM, 96 registers, no spills without cones; the
// corrector without walls, which needs fewer, 7 blocks, 72 registers (1M
// spheres, mean of the two kernels: 127 -> 119 us per launch with 0.8
// contacts each, 198 -> 189 with 6.6, both 2 less since its requests are in
// today's order; with walls it would spill, 61 -> 65 us).
// The predictor at 6 blocks loses on the dense packing (210 against 196) what
// it gains on the thin one; one record in flight instead of two: 134 against
// 127.  Before the columns were staged, the records read in 32-byte pieces
// and the block barriers dropped: 142 and 212 us.)
template <bool PP, int EPI, bool WALLS, bool CONE, bool STRIDE>
__global__ void __launch_bounds__(128, EPI == EPI_CORRECT && !WALLS ? 7 : 5)
    k_fold_mixed(PassArgs<float4, float2> A, MixedView V) {
  pass_kernel_entry();
  __shared__ __align__(16) double stage[EpiStage<EPI, true>::SIZE];
  if (!STRIDE) {
    fold_mixed_body<PP, EPI, WALLS, CONE>(A, V, blockIdx.x, stage);
    return;
  }
  const int nvb = (A.n + 127) / 128;
  for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
    fold_mixed_body<PP, EPI, WALLS, CONE>(A, V, vb, stage);
    __syncthreads();  // the block's shared arrays are reused by the next block of particles
  }
}

// The persistent chunk kernel (mixed): k_chunk_fp64's structure with the
// mixed pair and fold bodies.  The relink and test bodies are the FP64
// unit's code, written with explicitly rounded operations, so this unit's
// approximate division and square root do not reach them; this unit is
// compiled without contraction, so the inlined pair and fold bodies round
// exactly as in k_pair_mixed / k_fold_mixed.
using ChunkPassMx = ChunkPass<float4, float2, MixedView>;

// the fold phase of this block
template <bool PP, int EPI, bool WALLS, bool CONE>
__device__ __forceinline__ void fold_blocks_mixed(const ChunkPassMx& sp, double* stage) {
  const int nvb = (sp.t.n + 127) / 128;
  for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
    fold_mixed_body<PP, EPI, WALLS, CONE>(sp.a, sp.v, vb, stage);
    __syncthreads();
  }
}
// MINB: blocks an SM holds.  1: the launch is one cluster instead (ClusterRun),
// for systems so
// small that a pass is a chain of latencies: no launch boundaries, a hardware
// barrier between the phases, npass passes of a program that repeats, and
// the whole register file of an SM for each block.
// A cooperative launch takes 3 or 4 (chunk_blocks_per_sm).
template <bool PP, bool WALLS, bool CONE, int MINB>
__global__ void __launch_bounds__(128, MINB)
    k_chunk_mixed(const ChunkPassMx* __restrict__ prog, int npass, GridSync g, ClusterRun cr) {
  constexpr bool CLUSTER = MINB == 1;
  __shared__ ChunkPassMx sp;
  // (the larger of the two epilogues')
  __shared__ __align__(16) double stage[EpiStage<EPI_PREDICT, true>::SIZE];
  // (the relink's and the test's shared arrays lie in the fold's columns)
  int(*const sh)[RELINK_ROOM] = reinterpret_cast<int(*)[RELINK_ROOM]>(stage);
  TestWarp* const warps = reinterpret_cast<TestWarp*>(stage);
  static_assert(sizeof(stage) >= 4 * sizeof(TestWarp) && sizeof(stage) >= 4 * RELINK_ROOM * 4,
                "shared arrays of the phases");
  const int gwarp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int nwarps = gridDim.x * (blockDim.x >> 5);
  auto sync = [&]() -> bool {
    if (!CLUSTER) return grid_sync(g);
    cluster_sync();
    return true;
  };
  for (int k = 0; k < npass; k++) {
    load_pass(sp, prog + (CLUSTER ? k % cr.period : k));
    if (CLUSTER) cluster_pass(sp, cr, k);
    chunk_relink(sp, gwarp, nwarps, sh[threadIdx.x >> 5]);
    if (!sync()) return;
    chunk_rows<PP>(sp, gwarp, nwarps);
    if (!sync()) return;
    chunk_test<PP>(sp, warps);
    if (!sync()) return;
    pair_mixed_body<PP>(sp.a, sp.v, blockIdx.x, gridDim.x, 1);
    if (!sync()) return;
    if (sp.epi == EPI_PREDICT) fold_blocks_mixed<PP, EPI_PREDICT, WALLS, CONE>(sp, stage);
    else fold_blocks_mixed<PP, EPI_CORRECT, WALLS, CONE>(sp, stage);
    if (!sync()) return;  // (also: every block is done with sp)
  }
}

// FP64 records <-> FP32 records
__global__ void k_hist_to_mixed(int n, History H, float4* a, float* c, int nw, float4* wa,
                                float4* wb, float* wc) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int r = 0; r < H.cnt[i]; r++) {
    const size_t k = hslot(H, i, r);
    double2 x = H.val[2 * k], y = H.val[2 * k + 1], z = H.val2[k];
    a[2 * k] = make_float4((float)x.x, (float)x.y, (float)y.x, (float)y.y);
    a[2 * k + 1] = make_float4((float)z.x, (float)z.y, 0.f, 0.f);
    c[k] = 0.f;
  }
  for (int w = 0; w < nw; w++) {
    size_t k = (size_t)i * nw + w;
    double2 x = H.wval[3 * k], y = H.wval[3 * k + 1], z = H.wval[3 * k + 2];
    wa[k] = make_float4((float)x.x, (float)x.y, (float)y.x, (float)y.y);
    wb[k] = make_float4((float)z.x, (float)z.y, 0.f, 0.f);
    wc[k] = 0.f;
  }
}

__global__ void k_hist_from_mixed(int n, History H, const float4* a, const float* c, int nw,
                                  const float4* wa, const float4* wb, const float* wc) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int r = 0; r < H.cnt[i]; r++) {
    const size_t k = hslot(H, i, r);
    float4 x = a[2 * k], y = a[2 * k + 1];
    H.val[2 * k] = make_double2((double)x.x + y.z, (double)x.y + y.w);
    H.val[2 * k + 1] = make_double2((double)x.z + c[k], (double)x.w);
    H.val2[k] = make_double2((double)y.x, (double)y.y);
  }
  for (int w = 0; w < nw; w++) {
    size_t k = (size_t)i * nw + w;
    float4 x = wa[k], y = wb[k];
    H.wval[3 * k] = make_double2((double)x.x + y.z, (double)x.y + y.w);
    H.wval[3 * k + 1] = make_double2((double)x.z + wc[k], (double)x.w);
    H.wval[3 * k + 2] = make_double2((double)y.x, (double)y.y);
  }
}

__global__ void k_mixed_regrow(int n, int ns, int nd, const int* cnt, const float4* a,
                               const float* c, float4* na, float* nc) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int r = 0; r < cnt[i]; r++) {
    // slot-major: record r of particle i at r*stride + i, the old tables laid
    // out for ns rows, the new ones for nd
    const size_t s = (size_t)r * ns + i, d = (size_t)r * nd + i;
    na[2 * d] = a[2 * s];
    na[2 * d + 1] = a[2 * s + 1];
    nc[d] = c[s];
  }
}

unsigned blocks(long long n, int b) { return (unsigned)((n + b - 1) / b); }

// blocks of a cooperative launch of `k`: as many as fit on the device at
// once (occupancy x SMs), at most `want`
template <class K>
int coop_blocks(K k, int want) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, 128, 0);
  const int most = per * sms;
  return want < most ? want : most;
}

template <class K>
cudaError_t launch_chunk(K k, const ChunkPassMx* prog, int npass, GridSync g, int want,
                         cudaStream_t st, int* blocks_out) {
  const int nb = coop_blocks(k, want);
  if (nb <= 0) return cudaErrorLaunchOutOfResources;
  g.expected += (unsigned)nb;  // (on entry: the blocks a test adds to every barrier)
  ClusterRun cr{};
  void* args[] = {(void*)&prog, (void*)&npass, (void*)&g, (void*)&cr};
  if (blocks_out) *blocks_out = nb;
  return cudaLaunchCooperativeKernel((const void*)k, dim3(nb), dim3(128), args, 0, st);
}

}  // namespace

bool mixed_available() { return true; }

bool mixed_alloc(MixedBuffers& M, int n, int nw, int cap) {
  mixed_free(M);
  size_t N = (size_t)(n > 0 ? n : 1);
  size_t W = N * (size_t)(nw > 0 ? nw : 1);
  M.n = n;
  M.nw = nw;
  M.cap = cap;
  bool ok = true;
  for (int b = 0; b < 2 && ok; b++) {
    ok = cudaMalloc(&M.h[b], N * cap * 2 * sizeof(float4)) == cudaSuccess &&
         cudaMalloc(&M.hc[b], N * cap * sizeof(float)) == cudaSuccess &&
         cudaMalloc(&M.wa[b], W * sizeof(float4)) == cudaSuccess &&
         cudaMalloc(&M.wb[b], W * sizeof(float4)) == cudaSuccess &&
         cudaMalloc(&M.wc[b], W * sizeof(float)) == cudaSuccess;
  }
  M.ready = ok;
  return ok;
}

void mixed_free(MixedBuffers& M) {
  for (int b = 0; b < 2; b++) {
    cudaFree(M.h[b]);
    cudaFree(M.hc[b]);
    cudaFree(M.wa[b]);
    cudaFree(M.wb[b]);
    cudaFree(M.wc[b]);
  }
  M = MixedBuffers{};
}

bool mixed_regrow(MixedBuffers& M, int n, int stride, int newcap, int cur, const History& old,
                  cudaStream_t st) {
  size_t N = (size_t)(stride > 0 ? stride : 1);
  float4* na[2];
  float* nc[2];
  for (int b = 0; b < 2; b++) {
    if (cudaMalloc(&na[b], N * newcap * 2 * sizeof(float4)) != cudaSuccess ||
        cudaMalloc(&nc[b], N * newcap * sizeof(float)) != cudaSuccess)
      return false;
  }
  if (n > 0)
    k_mixed_regrow<<<blocks(n, 256), 256, 0, st>>>(n, old.n, (int)N, old.cnt, M.h[cur], M.hc[cur],
                                                    na[cur], nc[cur]);
  cudaStreamSynchronize(st);
  for (int b = 0; b < 2; b++) {
    cudaFree(M.h[b]);
    cudaFree(M.hc[b]);
    M.h[b] = na[b];
    M.hc[b] = nc[b];
  }
  M.cap = newcap;
  return true;
}

bool mixed_grow_walls(MixedBuffers& M, int n, int stride, int cur, cudaStream_t st) {
  const size_t W = (size_t)(stride > 0 ? stride : 1) * (size_t)(M.nw > 0 ? M.nw : 1);
  const size_t keep = (size_t)n * (size_t)(M.nw > 0 ? M.nw : 1);
  float4 *na[2], *nb[2];
  float* nc[2];
  for (int b = 0; b < 2; b++)
    if (cudaMalloc(&na[b], W * sizeof(float4)) != cudaSuccess ||
        cudaMalloc(&nb[b], W * sizeof(float4)) != cudaSuccess ||
        cudaMalloc(&nc[b], W * sizeof(float)) != cudaSuccess)
      return false;
  if (keep) {
    cudaMemcpyAsync(na[cur], M.wa[cur], keep * sizeof(float4), cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(nb[cur], M.wb[cur], keep * sizeof(float4), cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(nc[cur], M.wc[cur], keep * sizeof(float), cudaMemcpyDeviceToDevice, st);
  }
  cudaStreamSynchronize(st);
  for (int b = 0; b < 2; b++) {
    cudaFree(M.wa[b]);
    cudaFree(M.wb[b]);
    cudaFree(M.wc[b]);
    M.wa[b] = na[b];
    M.wb[b] = nb[b];
    M.wc[b] = nc[b];
  }
  M.n = stride;
  return true;
}

MixedView mixed_view(const MixedBuffers& M, int cur) {
  MixedView V;
  V.r8 = (const F8*)M.h[cur];
  V.rc = M.hc[cur];
  V.w8 = (F8*)M.h[cur ^ 1];
  V.wc = M.hc[cur ^ 1];
  V.rwa = M.wa[cur];
  V.rwb = M.wb[cur];
  V.rwc = M.wc[cur];
  V.wwa = M.wa[cur ^ 1];
  V.wwb = M.wb[cur ^ 1];
  V.wwc = M.wc[cur ^ 1];
  return V;
}

void mixed_pass(MixedBuffers& M, bool pp, int epi, int variant, bool walls, bool cone,
                const PassArgs<float4, float2>& A, int cur, cudaStream_t st, int part,
                int pair_waves, int ppt, bool early) {
  if (A.n == 0) return;
  const MixedView V = mixed_view(M, cur);
  if (part == 0) {
#define PCASE(PPV, MB)                                                                    \
  launch_pass(early, k_pair_mixed<PPV, MB>, pair_grid(A.n, MB, pair_waves), 128, st, A, V, \
              pair_waves)
    if (variant == 1) {
      if (pp) PCASE(true, 4);
      else PCASE(false, 4);
    } else if (variant == 2) {
      if (pp) PCASE(true, 8);
      else PCASE(false, 8);
    } else {
      if (pp) PCASE(true, 6);
      else PCASE(false, 6);
    }
#undef PCASE
    return;
  }
  const unsigned nvb = blocks(A.n, 128);
  const bool stride = ppt > 1 && epi != EPI_STORE;
  const unsigned g = stride ? (nvb + ppt - 1) / ppt : nvb;
#define FK(PPV, E, W, CN, S) launch_pass(early, k_fold_mixed<PPV, E, W, CN, S>, g, 128, st, A, V)
#define FCASE(PPV, W, CN)                          \
  do {                                             \
    if (epi == EPI_PREDICT) {                      \
      if (stride) FK(PPV, EPI_PREDICT, W, CN, true); \
      else FK(PPV, EPI_PREDICT, W, CN, false);     \
    } else if (epi == EPI_CORRECT) {               \
      if (stride) FK(PPV, EPI_CORRECT, W, CN, true); \
      else FK(PPV, EPI_CORRECT, W, CN, false);     \
    } else {                                       \
      FK(PPV, EPI_STORE, W, CN, false);            \
    }                                              \
  } while (0)
  if (!walls) {
    if (pp) FCASE(true, false, false);
    else FCASE(false, false, false);
  } else if (cone) {
    if (pp) FCASE(true, true, true);
    else FCASE(false, true, true);
  } else {
    if (pp) FCASE(true, true, false);
    else FCASE(false, true, false);
  }
#undef FCASE
#undef FK
}

cudaError_t mixed_chunk(bool pp, bool walls, bool cone,
                        const ChunkPass<float4, float2, MixedView>* prog, int npass, GridSync g,
                        int want_blocks, cudaStream_t st, int* blocks_out,
                        const ClusterRun* cluster) {
  const int mb = chunk_blocks_per_sm(want_blocks);
#define CCASE(PPV, W, CN)                                                                      \
  return cluster ? launch_cluster(k_chunk_mixed<PPV, W, CN, 1>, prog, npass, *cluster, st)      \
         : mb == 3 ? launch_chunk(k_chunk_mixed<PPV, W, CN, 3>, prog, npass, g, want_blocks, st, \
                                  blocks_out)                                                    \
                   : launch_chunk(k_chunk_mixed<PPV, W, CN, 4>, prog, npass, g, want_blocks, st, \
                                  blocks_out)
  if (!walls) {
    if (pp) CCASE(true, false, false);
    CCASE(false, false, false);
  }
  if (cone) {
    if (pp) CCASE(true, true, true);
    CCASE(false, true, true);
  }
  if (pp) CCASE(true, true, false);
  CCASE(false, true, false);
#undef CCASE
}

void mixed_import_history(MixedBuffers& M, const History& H, int n, int nw, int cur,
                          cudaStream_t st) {
  if (n == 0) return;
  k_hist_to_mixed<<<blocks(n, 256), 256, 0, st>>>(n, H, M.h[cur], M.hc[cur], nw,
                                                  M.wa[cur], M.wb[cur], M.wc[cur]);
}

void mixed_export_history(MixedBuffers& M, const History& H, int n, int nw, int cur,
                          cudaStream_t st) {
  if (n == 0) return;
  k_hist_from_mixed<<<blocks(n, 256), 256, 0, st>>>(n, H, M.h[cur], M.hc[cur], nw,
                                                    M.wa[cur], M.wb[cur], M.wc[cur]);
}

}  // namespace dem
