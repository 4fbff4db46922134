// dem_pass.cuh -- device helpers shared by the FP64 and the mixed force
// passes: the per-block counters, the ordered fold, the AB/AM epilogues and the
// cell transition (RedistributeParticles3D's bookkeeping) for the next pass.
//
// A force pass is three kernels.  The test kernel (one thread per particle,
// in original index order) applies the reference's overlap test to the
// particle's candidate row (the partners it meets as "i") and lists its
// contacts; the pair kernel evaluates every listed contact once and hands its
// "i" half to the contact's place in the list and its "j" half to the
// partner; the fold kernel (one thread per particle) builds the particle's
// block of the sweep, adds the received halves and the block in the sweep's
// order and finishes with the integrator step of the pass (AB predictor or
// AM corrector).  Its epilogue also hashes the particle's next
// position into its cell and, when the cell changes, records the move for
// the next relink: the arrival list of the new cell and the dirty list of
// both cells.  Every such side effect is idempotent, so a pass that was
// stopped by a table overflow can be launched again after the tables grow.
#pragma once
#include <cstring>

#include "dem_device.cuh"

namespace dem {

__device__ __forceinline__ void mark_dirty(const CellLists& L, Counters* cnt, int par, int c) {
  if (atomicExch(&L.dflag[c], 1) == 0) {
    const int k = atomicAdd(&cnt->n_dirty[par], 1);
    L.dlist[par][k] = c;
  }
}

// Cell of particle p under the next assignment; a particle that changes cell
// is pushed once onto its new cell's arrival list.
__device__ __forceinline__ void note_cell(const CellLists& L, Counters* cnt, int par, int p,
                                          int c_old, int c_new) {
  L.cell[par][p] = c_new;
  if (c_new != c_old) {
    if (atomicExch(&L.mflag[p], 1) == 0) {
      L.mnext[p] = L.next[p];  // the relink walks the old list past p with it
      L.arr_next[p] = atomicExch(&L.arr_head[c_new], p);
      atomicAdd(&cnt->movers_pending, 1ull);
    }
    mark_dirty(L, cnt, par, c_old);
    mark_dirty(L, cnt, par, c_new);
  }
}

// squared minimum-image displacement between two positions of a particle
template <class BoxT>
__device__ __forceinline__ double disp2(const BoxT& P, const double a[3], const double b[3]) {
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double d = a[k] - b[k];
    if (P.pbc[k]) d = d - P.lbox[k] * rint(d * P.inv_lbox[k]);
    s = s + d * d;
  }
  return s;
}

// Largest displacement of the warp into the pass maximum (FP32 rounded up;
// non-negative floats order like their bit patterns).
__device__ __forceinline__ void publish_disp(Counters* cnt, double d2) {
  const unsigned bits = __float_as_uint(__double2float_ru(sqrt(d2)));
  const unsigned m = __reduce_max_sync(0xffffffffu, bits);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(&cnt->disp_max, m);
}

// The pair kernel's statistics over the block (one atomic per counter per
// block of at most 256 threads): new records, the most records and the most
// "j" results a particle needs.  All threads of the block call.
__device__ __forceinline__ void publish_pair_block(Counters* cnt, bool update, unsigned n_col,
                                                   unsigned need, unsigned need_in) {
  const unsigned FULL = 0xffffffffu;
  __shared__ unsigned s_c[8][3];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned v[3] = {__reduce_add_sync(FULL, n_col), __reduce_max_sync(FULL, need),
                         __reduce_max_sync(FULL, need_in)};
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < 3; k++) s_c[wid][k] = v[k];
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned t[3] = {0u, 0u, 0u};
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
      t[0] += s_c[w][0];
      t[1] = t[1] > s_c[w][1] ? t[1] : s_c[w][1];
      t[2] = t[2] > s_c[w][2] ? t[2] : s_c[w][2];
    }
    if (t[0]) atomicAdd(update ? &cnt->ncol_pending : &cnt->ncol, (unsigned long long)t[0]);
    if (t[1]) atomicMax(&cnt->need_capacity, (int)t[1]);
    if (t[2]) atomicMax(&cnt->need_in, (int)t[2]);
  }
}

// The fold kernel's statistics per warp: wall contacts, the most records a
// particle needs and the largest displacement (rounded up twice in FP32: it
// is a bound).  The two maxima only grow
// during a pass, so a warp whose value is not above the current one sends
// nothing (a stale read only costs an atomic); no block barrier.
__device__ __forceinline__ void publish_fold(Counters* cnt, unsigned n_wc, unsigned need,
                                             double d2) {
  const unsigned FULL = 0xffffffffu;
  n_wc = __reduce_add_sync(FULL, n_wc);
  need = __reduce_max_sync(FULL, need);
  const unsigned d =
      __reduce_max_sync(FULL, __float_as_uint(__fsqrt_ru(__double2float_ru(d2))));
  if ((threadIdx.x & 31) == 0) {
    if (n_wc) atomicAdd(&cnt->wall_contacts, (unsigned long long)n_wc);
    if ((int)need > *(volatile int*)&cnt->need_capacity) atomicMax(&cnt->need_capacity, (int)need);
    if (d > *(volatile unsigned*)&cnt->disp_max) atomicMax(&cnt->disp_max, d);
  }
}

// The contacts of one block of the pair kernel: first + k*stride (+ thread)
// below end.  The list is cut into nseg segments, one for each wave of
// resident blocks, and a wave sweeps its segment front to back with all its
// blocks side by side: the contacts in work at any time are neighbours in the
// list, so the partners' data and the half-written sectors of their results
// meet in L2 (a sweep of the whole list per wave passes every place once
// more: 260 against 219 us per launch at 1M spheres with 6.6 contacts each).
struct PairSweep {
  int first, stride, end;
};
// Blocks of a wave: what an SM holds at the kernel's register budget (mb), on
// 148 SMs; a small system takes no more than four contacts per sphere fill
// (blocks without contacts still cost their launch).
inline unsigned pair_grid(int n, int mb, int waves) {
  const long long want = ((long long)4 * n + 128 * waves - 1) / (128 * waves);
  const long long most = 148 * mb;
  return (unsigned)((want < most ? (want > 1 ? want : 1) : most) * waves);
}
__device__ __forceinline__ PairSweep pair_sweep(int total, int vblock, int vgrid, int nseg) {
  const int per = vgrid / nseg, seg = vblock / per;  // (vgrid: a multiple of nseg)
  const int lo = (int)((long long)total * seg / nseg);
  PairSweep w;
  w.first = lo + (vblock - seg * per) * (int)blockDim.x;
  w.stride = per * (int)blockDim.x;
  w.end = (int)((long long)total * (seg + 1) / nseg);
  return w;
}

// Slot of partner `hi` among the records of `lo`; -1: no record.
__device__ __forceinline__ int find_record(const History& H, int lo, int hi) {
  const int c = H.cnt[lo];
  for (int r = 0; r < c; r++)
    if (H.key[hslot(H, lo, r)] == hi) return r;
  return -1;
}

// The "j" results a particle received in this pass, in the order of the
// givers' blocks in the sweep (their keys), with the particle's own block
// (key_p) at its place: the order in which ComputeAccelerations adds them to
// Force(p) and Torque(p) (src/MForces.f90:254-259, 319-320).
//
// SweepOrder: turn t of the first 8 records in 4 bits each (the record's
// number), and the turns before the particle's own block.  The keys of one
// particle's records differ (a giver evaluates a pair once), so a record's
// turn is the number of smaller keys; with the order in one register the
// keys need none while the records are read and added.  More than 8 records
// (rare): the keys are searched turn by turn.
struct SweepOrder {
  unsigned perm;
  int own;
};
__device__ __forceinline__ unsigned long long in_key(const char* in, int rec, int stride, int e,
                                                     int p) {
  return *(const unsigned long long*)(in + in_tail(rec, stride, e, p) + 8);
}
// (at most M records per particle of the warp)
template <int M>
__device__ __forceinline__ SweepOrder order_of(int ni, unsigned long long key_p, const char* in,
                                               int rec, int stride, int p) {
  SweepOrder o{0u, 0};
  unsigned long long kr[M];
  int t[M];
#pragma unroll
  for (int e = 0; e < M; e++) kr[e] = e < ni ? in_key(in, rec, stride, e, p) : ~0ull;
#pragma unroll
  for (int e = 0; e < M; e++) t[e] = e;  // (every earlier one smaller, as far as is known)
#pragma unroll
  for (int e = 0; e < M; e++)
#pragma unroll
    for (int f = e + 1; f < M; f++)
      if (kr[f] < kr[e]) {
        t[e]++;
        t[f]--;
      }
#pragma unroll
  for (int e = 0; e < M; e++) {
    o.perm |= (unsigned)e << (4 * t[e]);
    if (kr[e] < key_p) o.own++;
  }
  return o;
}
// All threads of the warp that hold a particle call (`most`: the largest
// count of them): the order is formed for 2, 4 or 8 records.
__device__ __forceinline__ SweepOrder sweep_order(int ni, int most, unsigned long long key_p,
                                                  const char* in, int rec, int stride, int p) {
  if (most == 0) return SweepOrder{0u, 0};
  if (most <= 2) return order_of<2>(ni, key_p, in, rec, stride, p);
  if (most <= 4) return order_of<4>(ni, key_p, in, rec, stride, p);
  return order_of<8>(ni, key_p, in, rec, stride, p);
}

// load(e) reads a record, own() and add(record) fold; two records are in
// flight at a time.
template <class Load, class Own, class Add>
__device__ __forceinline__ void fold_in_order(int ni, unsigned long long key_p, SweepOrder o,
                                              const char* in, int rec, int stride, int p,
                                              Load&& load, Own&& own, Add&& add) {
  if (ni <= 8) {
    for (int t = 0; t < ni; t += 2) {
      auto r0 = load((int)(o.perm & 15u));
      decltype(r0) r1;
      if (t + 1 < ni) r1 = load((int)((o.perm >> 4) & 15u));
      o.perm >>= 8;
      if (t == o.own) own();
      add(r0);
      if (t + 1 < ni) {
        if (t + 1 == o.own) own();
        add(r1);
      }
    }
    if (o.own >= ni) own();
    return;
  }
  bool own_done = false;
  unsigned long long lo = 0ull;  // every key >= lo is still to be folded
  for (int t = 0; t < ni; t++) {
    int best = 0;
    unsigned long long km = ~0ull;
    for (int e = 0; e < ni; e++) {
      const unsigned long long k = in_key(in, rec, stride, e, p);
      if (k >= lo && k < km) {
        km = k;
        best = e;
      }
    }
    if (!own_done && key_p < km) {
      own();
      own_done = true;
    }
    add(load(best));
    lo = km + 1ull;
  }
  if (!own_done) own();
}

template <class T>
__device__ __forceinline__ T mk_v4(double a, double b, double c, double d);
template <>
__device__ __forceinline__ double4 mk_v4<double4>(double a, double b, double c, double d) {
  return make_double4(a, b, c, d);
}
template <>
__device__ __forceinline__ float4 mk_v4<float4>(double a, double b, double c, double d) {
  return make_float4((float)a, (float)b, (float)c, (float)d);
}
template <class T>
__device__ __forceinline__ T mk_w2(double a, double b);
template <>
__device__ __forceinline__ double2 mk_w2<double2>(double a, double b) {
  return make_double2(a, b);
}
template <>
__device__ __forceinline__ float2 mk_w2<float2>(double a, double b) {
  return make_float2((float)a, (float)b);
}

__device__ __forceinline__ void prefetch_l2(const void* ptr) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr));
}

// The state the integrator epilogues of a warp's 32 particles will read,
// copied into the block's shared memory with cp.async: column c of the
// block's 128 particles at [c*128 + thread].  The copies are requested as the
// first thing of the fold kernel and hold no registers while they are in
// flight; in 16-byte pieces they pass by the L1, which the contact results
// read in between need (8-byte pieces go through it).  A half-warp copies the
// 32 particles of one column, so an instruction moves two columns; every
// column starts on 16 bytes and the block's first particle is a multiple of
// 128.  Predictor: the ring slots (9 columns each), then (mixed) Particle
// v, w; corrector: the ring sums, Particle x, v, w, then (mixed) Predicted v.
template <int EPI, bool MIXED>
struct EpiStage {
  static constexpr int COLS = EPI == EPI_STORE     ? 0
                              : EPI == EPI_PREDICT ? 27 + (MIXED ? 6 : 0)
                                                   : 18 + (MIXED ? 3 : 0);
  static constexpr int SIZE = COLS > 0 ? COLS * 128 : 1;  // doubles of a block
};

__device__ __forceinline__ void async_copy16(double* dst, const double* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// p0: the block's first particle; stage: the block's columns.  All threads
// of the warp call.
template <int EPI, bool MIXED, class V4, class W2>
__device__ __forceinline__ void stage_epilogue(const PassArgs<V4, W2>& A, int p0, double* stage) {
  if (EPI == EPI_STORE) return;
  const int lane = threadIdx.x & 31;
  const int at = (threadIdx.x & ~31) + 2 * (lane & 15);  // place in the block
  const int p = p0 + at;
  if (p >= A.n) return;  // (a piece may end one particle past the last: padding)
  const int half = lane >> 4;
  const size_t n = ring_stride(A.n);
  if (EPI == EPI_PREDICT) {
    const int nc = 9 * A.nprev;
#pragma unroll
    for (int k = 0; k < 28; k += 2) {
      const int c = k + half;
      const int slot = c / 9;
      if (c < nc)
        async_copy16(stage + c * 128 + at,
                     A.ring + ((size_t)A.rm.phys[slot] * 9 + (c - 9 * slot)) * n + p);
    }
    if (MIXED) {
      const double* v[6] = {A.part.vx, A.part.vy, A.part.vz, A.part.wx, A.part.wy, A.part.wz};
#pragma unroll
      for (int d = 0; d < 6; d += 2)
        async_copy16(stage + (27 + d + half) * 128 + at, (half ? v[d + 1] : v[d]) + p);
    }
  } else {
    if (A.amsum)
#pragma unroll
      for (int d = 0; d < 10; d += 2)
        if (d + half < 9) async_copy16(stage + (d + half) * 128 + at, A.amsum + (d + half) * n + p);
    const double* q[12] = {A.part.px, A.part.py, A.part.pz, A.part.vx, A.part.vy, A.part.vz,
                           A.part.wx, A.part.wy, A.part.wz, A.pred.vx, A.pred.vy, A.pred.vz};
#pragma unroll
    for (int d = 0; d < (MIXED ? 12 : 10); d += 2)
      if (d + half < (MIXED ? 12 : 9))
        async_copy16(stage + (9 + d + half) * 128 + at, (half ? q[d + 1] : q[d]) + p);
  }
}
// the warp's columns have arrived (all threads of the warp call)
__device__ __forceinline__ void stage_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}

// The integrator part of a pass, after a = F/m and alpha = T/I
// (src/MForces.f90:330-333):
//  EPI_STORE   a, alpha -> tgt;
//  EPI_PREDICT the AB predictor of MoveParticles (src/MDEM.f90:296-331) from
//              x(t) = xp, v(t) = vp, w(t) = wp and the ring, (v,a,alpha)(t)
//              into the spare ring slot; the prediction is the next pass's
//              position;
//  EPI_CORRECT the AM corrector (src/MDEM.f90:340-367) with v~ = vp; the new
//              x(t+dt) is the next pass's position.
// d2 receives the squared displacement from this pass's position to the next.
// s: the thread's staged columns (stage_epilogue; the caller has waited).
template <int EPI, class V4, class W2>
__device__ __forceinline__ void epilogue(const PassArgs<V4, W2>& A, const DevParams& P, int p,
                                         const double xp[3], double Rp, const double vp[3],
                                         const double wp[3], const double acc[3],
                                         const double alp[3], int c_cur, const double* s,
                                         double& d2) {
  const Box& B = P.box;
  const size_t n = ring_stride(A.n);
  if (EPI == EPI_STORE) {
    A.tgt.ax[p] = acc[0]; A.tgt.ay[p] = acc[1]; A.tgt.az[p] = acc[2];
    A.tgt.lx[p] = alp[0]; A.tgt.ly[p] = alp[1]; A.tgt.lz[p] = alp[2];
    return;
  }
  double x[3], v[3], w[3];
  if (EPI == EPI_PREDICT) {
    const StateArrays& Q = A.part;
    const StateArrays& R = A.pred;
    // (with A.lazy, a and alpha stay in the new ring slot only)
    if (!A.lazy || A.nprev == 0) {
      Q.ax[p] = acc[0]; Q.ay[p] = acc[1]; Q.az[p] = acc[2];
      Q.lx[p] = alp[0]; Q.ly[p] = alp[1]; Q.lz[p] = alp[2];
    }
    // the predictor also forms the corrector's sums: after the ring rotation
    // its slot k is this pass's (v, a, alpha) for k = 0, else the slot k-1
    // read here
    const bool am = A.amsum && A.nprev > 0;
    double* rg = A.ring + (size_t)A.rm.phys[A.nprev] * 9 * n + p;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      double sv = 0.0, sa = 0.0, sl = 0.0;
      double mv = 0.0 + P.am[0] * vp[d], ma = 0.0 + P.am[0] * acc[d],
             ml = 0.0 + P.am[0] * alp[d];
#pragma unroll
      for (int k = 0; k < 3; k++)
        if (k < A.nprev) {
          const double C = P.ab[k];
          const double tv = s[(9 * k + d) * 128], ta = s[(9 * k + 3 + d) * 128],
                       tl = s[(9 * k + 6 + d) * 128];
          sv = sv + C * tv;
          sa = sa + C * ta;
          sl = sl + C * tl;
          if (k + 1 < 3 && k + 1 < A.nprev) {
            const double M = P.am[k + 1 < 3 ? k + 1 : 0];
            mv = mv + M * tv;
            ma = ma + M * ta;
            ml = ml + M * tl;
          }
        }
      if (am) {
        A.amsum[d * n + p] = mv;
        A.amsum[(3 + d) * n + p] = ma;
        A.amsum[(6 + d) * n + p] = ml;
      }
      x[d] = xp[d] + P.ab0 * vp[d] + sv;
      v[d] = vp[d] + P.ab0 * acc[d] + sa;
      w[d] = wp[d] + P.ab0 * alp[d] + sl;
      if (B.pbc[d]) x[d] = x[d] - B.lbox[d] * fnint(x[d] * B.inv_lbox[d]);
      if (A.nprev > 0) {
        rg[d * n] = vp[d];
        rg[(3 + d) * n] = acc[d];
        rg[(6 + d) * n] = alp[d];
      }
    }
    // (with A.lazy, Predicted x stays in the position copy Xn, and with
    // FP64 copies Predicted v, w stay in v4n, w2n; the mixed corrector reads
    // Predicted v, and its FP32 copies do not hold v, w exactly)
    if (!A.lazy) {
      R.px[p] = x[0]; R.py[p] = x[1]; R.pz[p] = x[2];
    }
    if (!A.lazy || sizeof(V4) != sizeof(double4)) {
      R.vx[p] = v[0]; R.vy[p] = v[1]; R.vz[p] = v[2];
      R.wx[p] = w[0]; R.wy[p] = w[1]; R.wz[p] = w[2];
    }
  } else {
    const StateArrays& Q = A.part;
    const StateArrays& R = A.pred;
    R.ax[p] = acc[0]; R.ay[p] = acc[1]; R.az[p] = acc[2];
    R.lx[p] = alp[0]; R.ly[p] = alp[1]; R.lz[p] = alp[2];
    double* q[9] = {Q.px, Q.py, Q.pz, Q.vx, Q.vy, Q.vz, Q.wx, Q.wy, Q.wz};
    bool out = false;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      // sum_k AM(k)*Previous(ipc(k)) over the rotated ring, as the predictor
      // pass formed it (no ring: empty sums)
      const double sv = A.amsum ? s[d * 128] : 0.0, sa = A.amsum ? s[(3 + d) * 128] : 0.0,
                   sl = A.amsum ? s[(6 + d) * 128] : 0.0;
      x[d] = s[(9 + d) * 128] + P.am0 * vp[d] + sv;
      v[d] = s[(12 + d) * 128] + P.am0 * acc[d] + sa;
      w[d] = s[(15 + d) * 128] + P.am0 * alp[d] + sl;
      if (B.pbc[d]) x[d] = x[d] - B.lbox[d] * fnint(x[d] * B.inv_lbox[d]);
      q[d][p] = x[d];
      q[3 + d][p] = v[d];
      q[6 + d][p] = w[d];
      const double h = 0.5 * B.lbox[d];
      out = out || (x[d] > h) || (x[d] < -h);
    }
    if (out) atomicAdd(&A.cnt->escaped, 1ull);
  }
  // the next pass's copies, cell and displacement
  st32(A.Xn + p, make_double4(x[0], x[1], x[2], Rp));
  stv(A.v4n + p, mk_v4<V4>(v[0], v[1], v[2], w[0]));
  A.w2n[p] = mk_w2<W2>(w[1], w[2]);
  note_cell(A.L, A.cnt, A.par_nxt, p, c_cur, current_cell(P, x[0], x[1], x[2]));
  d2 = disp2(B, x, xp);
  if (!isfinite(x[0] + x[1] + x[2])) {
    // a diverged state would put every particle into one cell; stop here
    atomicExch(&A.cnt->nonfinite, 1);
    set_abort(A.cnt, A.tag);
  }
}

// First statement of every kernel of a force pass (relink, rows, lists, test,
// pair, fold).  A kernel launched with programmatic stream serialization may
// be scheduled while the kernel before it in the stream is still running; it
// waits here until that kernel has completed and its writes are visible, and
// then allows the next kernel of the pass to be scheduled (whose blocks take
// the SM slots this kernel's last blocks free, and wait in turn).  Without
// that launch attribute both instructions return at once.  Nothing is read
// before the wait, not even what kernels further ahead wrote: those have
// completed by then (a kernel allows its successor only after its own wait),
// but their writes are promised to be visible only to threads that have
// waited, and a block may start on an SM whose L1 holds older values.
__device__ __forceinline__ void pass_kernel_entry() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Host side: launch a pass kernel on `st`, with programmatic stream
// serialization when `early` (the kernel must begin with pass_kernel_entry).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pass(bool early, void (*kernel)(KArgs...), unsigned grid, unsigned block,
                               cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

__device__ __forceinline__ void set_abort(Counters* cnt, int tag) {
  atomicCAS(&cnt->abort_tag, 0, tag + 1);
  atomicExch(&cnt->abort, 1);
}

}  // namespace dem
