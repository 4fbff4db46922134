// dem_test.cuh -- the precision-independent parts of a force pass: the
// relink of the cell lists, the candidate rows and the exact overlap test.
// Both translation units include them (the FP64 one, compiled with IEEE
// square root, and the mixed one, compiled with approximate division and
// square root), so every floating-point operation here is written with an
// explicitly rounded intrinsic (__dadd_rn, __dsub_rn, __dmul_rn,
// __dsqrt_rn), which no compiler flag changes: the candidate rows and the
// contact lists are the same bits in either unit, and equal to the
// reference's (src/MForces.f90:218-224 tests DeltaDijSq = MinDijSq - DijSq
// > 0 in FP64).
#pragma once
#include "dem_pass.cuh"

namespace dem {

// min_image_exact, sumsq3 and the pair's MinDijSq with every operation
// rounded on its own (no contraction into fused multiply-adds)
__device__ __forceinline__ double min_image_rn(double r, const Box& B, int k) {
  if (B.pbc[k] && !(fabs(r) < B.half_lim[k]))
    r = __dsub_rn(r, __dmul_rn(B.lbox[k], (double)(int)round(__dmul_rn(r, B.inv_lbox[k]))));
  return r;
}
// the image itself, for a component known to be beyond the shortcut's bound
__device__ __forceinline__ double image_rn(double r, const Box& B, int k) {
  return __dsub_rn(r, __dmul_rn(B.lbox[k], (double)(int)round(__dmul_rn(r, B.inv_lbox[k]))));
}
__device__ __forceinline__ double sumsq3_rn(const double a[3]) {
  double c = __dmul_rn(a[0], a[0]);  // (0.0 + a square: the square itself)
  c = __dadd_rn(c, __dmul_rn(a[1], a[1]));
  c = __dadd_rn(c, __dmul_rn(a[2], a[2]));
  return c;
}
// MinDijSq of a pair: the material table (components ca, cb), or (Ra + Rb)^2
// for per-particle radii (PP)
template <bool PP>
__device__ __forceinline__ double min_dij_sq_rn(const DevParams& P, int ca, double Ra, int cb,
                                                double Rb) {
  if (PP) {
    const double d = __dadd_rn(Ra, Rb);
    return __dmul_rn(d, d);
  }
  return P.min_dij_sq[ca * NCM + cb];
}

// Copy cell c's list into its slots (the first scap entries) and record
// its length; a walk longer than n (corrupt links) records -1.
__device__ __forceinline__ void copy_slots(const CellLists& L, int c, int first, int n) {
  int k = 0;
  for (int q = first; q != -1; q = L.next[q]) {
    if (k >= n) {
      k = -1;
      break;
    }
    if (k < L.scap) L.slot[(size_t)c * L.scap + k] = q;
    k++;
  }
  L.slot_n[c] = k;
}

// The o-th (0 <= o < 14) of the cells whose particles' rows read cell c: c
// itself (o = 13) and c + o' for the 13 offsets with kx + Nx*(ky + Ny*kz) < 0;
// -1: off the grid.
__device__ __forceinline__ int reading_cell(const DevParams& P, int c, int o) {
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  int cx, cy, cz;
  cell_coords(P, c, cx, cy, cz);
  const int jx = cx + o % 3 - 1, jy = cy + (o / 3) % 3 - 1, jz = cz + o / 9 - 1;
  const bool ok = (P.pbc[0] || (jx >= 0 && jx < nx)) && (P.pbc[1] || (jy >= 0 && jy < ny)) &&
                  (P.pbc[2] || (jz >= 0 && jz < nz));
  if (!ok) return -1;
  return P.coff + axis_wrap(jx, nx, P.pbc[0]) +
         nx * (axis_wrap(jy, ny, P.pbc[1]) + ny * axis_wrap(jz, nz, P.pbc[2]));
}

// The rewrite of a cell whose list does not fit the slots, by one thread: the
// old list is walked link by link (a leaver's successor was saved when it
// moved, mnext: its own link may be rewritten by the warp of the cell it
// entered), the leavers dropped, the arrivals prepended in decreasing index.
template <class Rec, class Gid>
__device__ __forceinline__ bool relink_links(const CellLists& L, const int* cell_new, int c,
                                             int n, Rec&& record, Gid&& G) {
  int prev = -1, first = -1, guard = 0;
  int q = L.head[c];
  while (q != -1) {
    if (++guard > n) return false;
    const bool stays = cell_new[q] == c;
    const int nq = stays ? L.next[q] : L.mnext[q];
    if (!stays) {
      record(q);
    } else {
      if (prev == -1) first = q;
      else L.next[prev] = q;
      prev = q;
    }
    q = nq;
  }
  if (prev != -1) L.next[prev] = -1;
  int sh = -1, tail = -1, a = L.arr_head[c];
  guard = 0;
  while (a != -1) {
    if (++guard > n) return false;
    const int an = L.arr_next[a];  // (guard: arrivals so far)
    L.mflag[a] = 0;
    record(a);
    if (sh == -1) {
      sh = tail = a;
      L.next[a] = -1;
    } else if (G(a) > G(sh)) {
      L.next[a] = sh;
      sh = a;
    } else {
      int q2 = sh;
      for (int g2 = 0; L.next[q2] != -1 && G(L.next[q2]) > G(a) && g2 < guard; g2++)
        q2 = L.next[q2];
      L.next[a] = L.next[q2];
      L.next[q2] = a;
      if (L.next[a] == -1) tail = a;
    }
    a = an;
  }
  if (sh != -1) {
    L.next[tail] = first;
    first = sh;
  }
  L.head[c] = first;
  copy_slots(L, c, first, n);
  return true;
}

// Relink (RedistributeParticles3D's list updates, src/MCells.f90:607-643):
// one warp per dirty cell of list `par` drops the particles that left it
// (TransferParticle's unlink, :747-774) and prepends its arrivals in
// decreasing index (AddParticle, :684-698, applied in increasing index
// order), records the movers with the cell, and stamps the 14 cells whose
// rows read it.  The lanes hold the old list (from the cell's slots) and the
// arrivals side by side, so a cell costs four round trips to memory and not
// one per element; the kernel is bound by those round trips (14 us per launch
// at 1M spheres with one thread per cell and its list in local memory).
// Thread 0 also closes the previous pass's bookkeeping and decides whether
// this pass rebuilds every candidate row.
// (The body of k_relink; warp / nwarps: this warp's index among the warps
// that share the work, `sh` RELINK_ROOM ints of shared memory of its own.)
constexpr int RELINK_ROOM = SLOT_MAX + 32;
__device__ __forceinline__ void relink_body(const DevParams* __restrict__ PT,
                                            const int* __restrict__ cellsys, const CellLists& L,
                                            int par, int n, int update, int stop_tag,
                                            Counters* cnt, int warp, int nwarps, int* sh) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool first_thread = warp == 0 && lane == 0;
  // (the status words, the dirty-cell count and the pass number requested
  // together; the abort word may be set meanwhile, so one lane's reading
  // decides for the warp, whose lanes meet in the loops below)
  const int abort1 = lane == 0 ? cnt->abort : 0;
  const unsigned long long escaped = cnt->escaped;
  const int m = cnt->n_dirty[par];
  const int stamp = cnt->pass_id + 1;  // fold kernels advance pass_id, not this one
  if (__shfl_sync(FULL, abort1, 0)) return;
  // inside a captured chunk, particles that left the box in the last step
  // stop the chunk before this step (the host runs UpdateParticleList); the
  // count is final here (written by the previous kernel), so every block
  // takes the same branch
  if (stop_tag >= 0 && escaped != 0ull) {
    if (first_thread) {
      cnt->escape_stop = 1;
      set_abort(cnt, stop_tag);
    }
    return;
  }
  if (first_thread) {
    const DevParams& P = PT[0];  // the integrator settings are shared
    cnt->n_mlist[(stamp & 1) ^ 1] = 0;  // for the next pass's relink
    cnt->n_dirty[par ^ 1] = 0;
    cnt->movers = cnt->movers_pending;
    cnt->movers_pending = 0ull;
    if (cnt->ncol_pending) {  // the previous history-updating pass completed
      cnt->ncol += cnt->ncol_pending;
      cnt->ncol_pending = 0ull;
    }
    cnt->pair_contacts = 0ull;
    cnt->wall_contacts = 0ull;
    cnt->n_contacts = 0;  // the contact list of this pass starts empty
    if (update) {
      cnt->need_capacity = 0;
      cnt->need_in = 0;
      cnt->need_cl = 0;
    } else {
      cnt->escaped = 0ull;  // escapes are counted by the current step's corrector
    }
    const double d = (double)__uint_as_float(cnt->disp_max);
    cnt->disp_max = 0u;
    const double acc = cnt->disp_acc + d;
    const int full = cnt->force_full != 0 || !(acc <= P.vl_thr);
    cnt->full_due = full;
    cnt->disp_acc = full ? 0.0 : acc;
    if (full) cnt->force_full = 0;
  }
  const int* cell_new = L.cell[par];
  // the reference's index (gid when the storage is in cell order)
  auto G = [&](int x) { return L.gid ? L.gid[x] : x; };
  for (int i = warp; i < m; i += nwarps) {
    const int c = L.dlist[par][i];
    const int len = L.slot_n[c];
    const int ah = L.arr_head[c];
    const int* sl = L.slot + (size_t)c * L.scap;
    const int e0 = lane < len && len <= L.scap ? sl[lane] : -1;
    const int e1 = lane + 32 < len && len <= L.scap ? sl[lane + 32] : -1;
    const DevParams& P = sys_params(PT, cellsys, c);
    if (!in_slab(P, c)) {
      // a cell another slab advances (a particle of this slab left for it):
      // its list here is not kept; only the transition is forgotten
      if (lane == 0) {
        for (int a = ah, g2 = 0; a != -1 && g2 < n; a = L.arr_next[a], g2++) L.mflag[a] = 0;
        L.arr_head[c] = -1;
        L.dflag[c] = 0;
      }
      continue;
    }
    // a particle that leaves or enters the cell, for the row kernel
    auto record = [&](int x) {
      const int k = atomicAdd(&cnt->n_mlist[stamp & 1], 1);
      if (k < L.mcap) L.mlist[(size_t)(stamp & 1) * L.mcap + k] = make_int2(x, c);
    };
    // the arrivals, one per lane (every lane walks their list)
    int arr = -1, na = 0;
    for (int a = ah; a != -1 && na <= 32; a = L.arr_next[a]) {
      if (lane == na) arr = a;
      na++;
    }
    if (len >= 0 && len <= L.scap && na <= 32) {
      const bool s0 = e0 >= 0 && cell_new[e0] == c;
      const bool s1 = e1 >= 0 && cell_new[e1] == c;
      const unsigned b0 = __ballot_sync(FULL, s0), b1 = __ballot_sync(FULL, s1);
      if (e0 >= 0 && !s0) record(e0);
      if (e1 >= 0 && !s1) record(e1);
      if (arr >= 0) {
        L.mflag[arr] = 0;
        record(arr);
      }
      // the new list: the arrivals in decreasing index, then the stayers in
      // their old order
      int at = 0;
      const int ga = arr >= 0 ? G(arr) : -1;
      for (int j = 0; j < na; j++) at += __shfl_sync(FULL, ga, j) > ga ? 1 : 0;
      const unsigned lt = (1u << lane) - 1u;
      if (arr >= 0) sh[at] = arr;
      if (s0) sh[na + __popc(b0 & lt)] = e0;
      if (s1) sh[na + __popc(b0) + __popc(b1 & lt)] = e1;
      const int len2 = na + __popc(b0) + __popc(b1);
      __syncwarp();
      for (int k = lane; k < len2; k += 32) {
        const int x = sh[k];
        L.next[x] = k + 1 < len2 ? sh[k + 1] : -1;
        if (k < L.scap) L.slot[(size_t)c * L.scap + k] = x;
      }
      if (lane == 0) {
        L.head[c] = len2 > 0 ? sh[0] : -1;
        L.slot_n[c] = len2;
      }
      __syncwarp();  // (sh is used again)
    } else {
      int ok = 1;
      if (lane == 0) ok = relink_links(L, cell_new, c, n, record, G) ? 1 : 0;
      if (!__shfl_sync(FULL, ok, 0)) {
        if (lane == 0) {
          atomicExch(&cnt->list_error, 1);
          atomicExch(&cnt->abort, 1);
        }
        return;
      }
    }
    if (lane == 0) {
      L.arr_head[c] = -1;
      L.dflag[c] = 0;
    }
    // the rows that read c: a row of a particle in cell b holds the rest of
    // b's list and the half-shell cells b + o, kx + Nx*(ky + Ny*kz) > 0, so c
    // is read by the rows of c itself and of c + o' for the 13 offsets o' with
    // kx + Nx*(ky + Ny*kz) < 0; those 14 cells are stamped with the pass
    const int b = lane < 14 ? reading_cell(P, c, lane) : -1;
    if (b >= 0) L.rflag[b] = stamp;
  }
}

// Arguments of a relink
struct RelinkArgs {
  const DevParams* PT;
  const int* cellsys;
  CellLists L;
  int par, n, update, stop_tag;
  Counters* cnt;
};

// ---------------------------------------------------------------------------
// K2: candidate rows

// The row of particle p (cell c) when a list it reads does not fit the slots,
// built by one warp.  Lane L < 27 owns the neighbour cell at offset (L%3-1, L/3%3-1, L/9-1); lane 13 (own cell) walks
// the part of the list after p, lane 27 the part before p (p's rank).  The
// row holds the partners the sweep meets with p as "i": the own cell after p,
// then the half-shell cells (offset index kx + Nx*(ky + Ny*kz) > 0,
// AddAllNeighbours3D src/MCells.f90:456) in FirstNeighbour order, i.e.
// descending (kz, ky, kx) -- NeighbourParticles' list (src/MCells.f90:
// 793-829) from p on.
template <bool PP>
__device__ __noinline__ void build_row_links(const DevParams& P, int n, int p, int c,
                                             const double4* __restrict__ X,
                                             const int* __restrict__ comp, const CellLists& L,
                                             const Rows& R, Counters* cnt, int tag) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  const int cl = c - P.coff;
  const int cx = cl % nx, cy = (cl / nx) % ny, cz = cl / (nx * ny);
  const double4 p4 = ld32(X + p);
  const int cp = PP ? 0 : comp[p];
  int cw = -1, order = 1 << 20;  // the lane's cell, its place in the row
  bool walk = false;
  if (lane < 27) {
    const int d[3] = {lane % 3 - 1, (lane / 3) % 3 - 1, lane / 9 - 1};
    const int cc[3] = {cx, cy, cz};
    const int N[3] = {nx, ny, nz};
    bool ok = true;
    int w[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      int j = cc[k] + d[k];
      if (P.pbc[k]) {
        if (j == N[k]) j = 0;
        if (j == -1) j = N[k] - 1;
      } else if (j < 0 || j >= N[k]) {
        ok = false;
      }
      w[k] = j;
    }
    const int lex = d[0] + 3 * d[1] + 9 * d[2];
    if (lane == 13) {
      cw = c;
      order = 0;
      walk = true;
    } else if (ok && lex > 0) {
      cw = P.coff + w[0] + nx * (w[1] + ny * w[2]);
      order = 1 + (13 - lex);
      walk = true;
    }
  } else if (lane == 27) {
    cw = c;
  }
  const double skin = P.vl_skin;
  auto is_cand = [&](int q) -> bool {
    const double4 q4 = ld32(X + q);
    double Rij[3] = {__dsub_rn(q4.x, p4.x), __dsub_rn(q4.y, p4.y), __dsub_rn(q4.z, p4.z)};
#pragma unroll
    for (int k = 0; k < 3; k++) Rij[k] = min_image_rn(Rij[k], P.box, k);
    const double DijSq = sumsq3_rn(Rij);
    double md;
    if (PP) md = __dadd_rn(p4.w, q4.w);
    else md = __dsqrt_rn(min_dij_sq_rn<PP>(P, cp, p4.w, comp[q], q4.w));
    md = __dadd_rn(md, skin);
    return __dsub_rn(__dmul_rn(md, md), DijSq) > 0.0;
  };
  // pass 1: count the candidates; lane 13 (own cell after p) starts behind p,
  // lane 27 counts the list before p (p's rank).  The first 8 elements and
  // their test results stay in registers for pass 2.
  unsigned hits = 0u;
  int count = 0, walked = 0;
  int cache[8];
  bool bad = false;
  int q = -1;
#pragma unroll
  for (int i = 0; i < 8; i++) cache[i] = -1;
  if (cw >= 0) {
    q = lane == 13 ? L.next[p] : L.head[cw];
    if (walk) {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if (q != -1) {
          cache[i] = q;
          walked = i + 1;
          if (is_cand(q)) {
            hits |= 1u << i;
            count++;
          }
          q = L.next[q];
        }
      }
    }
  }
  const int resume = q;  // first element not cached (-1: none)
  if (cw >= 0) {
    int guard = 0;
    if (walk) {
      while (q != -1) {
        if (++guard > n) {
          bad = true;
          break;
        }
        if (is_cand(q)) count++;
        q = L.next[q];
      }
    } else if (lane == 27) {
      while (q != p) {
        if (q == -1 || ++guard > n) {
          bad = true;
          break;
        }
        count++;
        q = L.next[q];
      }
    }
  }
  if (__any_sync(FULL, bad)) {
    if (lane == 0) {
      atomicExch(&cnt->list_error, 1);
      set_abort(cnt, tag);
    }
    return;
  }
  int off = 0, m = 0;
  for (int l = 0; l < 27; l++) {
    const int ol = __shfl_sync(FULL, order, l);
    const int cl2 = __shfl_sync(FULL, walk ? count : 0, l);
    if (ol < order) off += cl2;
    m += cl2;
  }
  const int rank = __shfl_sync(FULL, count, 27);
  if (m > R.kc) {
    if (lane == 0) {
      atomicMax(&cnt->need_kc, m);
      atomicExch(&cnt->row_overflow, 1);
      set_abort(cnt, tag);
      R.meta[p] = 0;
    }
    return;
  }
  // pass 2: write the cached part, then the rest
  if (walk) {
    int k = off;
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (i < walked && ((hits >> i) & 1u)) R.cand[(size_t)(k++) * n + p] = cache[i];
    int q2 = resume;
    while (q2 != -1) {
      if (is_cand(q2)) R.cand[(size_t)(k++) * n + p] = q2;
      q2 = L.next[q2];
    }
  }
  if (lane == 0) {
    R.meta[p] = m;
    R.rank[p] = rank;
  }
}


// Whether q belongs into p's row: the pair closer than MinDij + skin (+ slack)
template <bool PP>
__device__ __forceinline__ bool within_skin(const DevParams& P, const double4& p4, int cp,
                                            const double4& q4, int cq, double slack) {
  double Rij[3] = {__dsub_rn(q4.x, p4.x), __dsub_rn(q4.y, p4.y), __dsub_rn(q4.z, p4.z)};
#pragma unroll
  for (int k = 0; k < 3; k++) Rij[k] = min_image_rn(Rij[k], P.box, k);
  const double DijSq = sumsq3_rn(Rij);
  double md;
  if (PP) md = __dadd_rn(p4.w, q4.w);
  else md = __dsqrt_rn(min_dij_sq_rn<PP>(P, cp, p4.w, cq, q4.w));
  md = __dadd_rn(md, __dadd_rn(P.vl_skin, slack));
  return !(__dsub_rn(__dmul_rn(md, md), DijSq) <= 0.0);
}

// The row of particle p (cell c), built by one warp: the partners the sweep
// meets with p as "i" -- the own cell's list after p, then the half-shell
// cells (offset index kx + Nx*(ky + Ny*kz) > 0, AddAllNeighbours3D
// src/MCells.f90:456) in FirstNeighbour order, i.e. descending (kz, ky, kx),
// which is NeighbourParticles' list (src/MCells.f90:793-829) from p on.  Lane
// l < 14 holds the l-th of those lists; laid end to end they are tested 32
// elements at a time, two loads deep, and the hits appended in order, so a
// row costs the same few round trips whether its cells hold two particles or
// thirty.
template <bool PP>
__device__ __noinline__ void build_row(const DevParams& P, int n, int p, int c,
                                       const double4* __restrict__ X,
                                       const int* __restrict__ comp, const CellLists& L,
                                       const Rows& R, Counters* cnt, int tag) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const double4 p4 = ld32(X + p);
  const int cp = PP ? 0 : comp[p];
  int cx, cy, cz;
  cell_coords(P, c, cx, cy, cz);
  int cw = -1, len = 0;
  if (lane == 0) {
    cw = c;
  } else if (lane < 14) {
    const int o = 27 - lane;  // 26 .. 14: offsets in descending (kz, ky, kx)
    const int jx = cx + o % 3 - 1, jy = cy + (o / 3) % 3 - 1, jz = cz + o / 9 - 1;
    const bool ok = (P.pbc[0] || (jx >= 0 && jx < P.nx)) &&
                    (P.pbc[1] || (jy >= 0 && jy < P.ny)) && (P.pbc[2] || (jz >= 0 && jz < P.nz));
    if (ok)
      cw = P.coff + axis_wrap(jx, P.nx, P.pbc[0]) +
           P.nx * (axis_wrap(jy, P.ny, P.pbc[1]) + P.ny * axis_wrap(jz, P.nz, P.pbc[2]));
  }
  if (cw >= 0) len = L.slot_n[cw];
  const int* own = L.slot + (size_t)c * L.scap;
  // (p's place in its list; entries past the list's end are old ones)
  const int w0 = own[lane], w1 = lane + 32 < L.scap ? own[lane + 32] : -1;
  if (__any_sync(FULL, len < 0 || len > L.scap)) {
    build_row_links<PP>(P, n, p, c, X, comp, L, R, cnt, tag);
    return;
  }
  const int len0 = __shfl_sync(FULL, len, 0);
  const unsigned f0 = __ballot_sync(FULL, lane < len0 && w0 == p);
  const unsigned f1 = __ballot_sync(FULL, lane + 32 < len0 && w1 == p);
  if (!(f0 | f1)) {
    if (lane == 0) {
      atomicExch(&cnt->list_error, 1);
      set_abort(cnt, tag);
    }
    return;
  }
  const int rank = f0 ? __ffs(f0) - 1 : 31 + __ffs(f1);
  int skip = 0;  // entries of the lane's list that the row does not read
  if (lane == 0) {
    skip = rank + 1;
    len -= skip;
  }
  int incl = len;  // (0 on lanes >= 14)
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  const int T = __shfl_sync(FULL, incl, 13);
  const int excl = lane < 14 ? incl - len : INT_MAX;
  // the slot of element f of the lists laid end to end
  auto slot_of = [&](int f) -> size_t {
    int j = 0;
#pragma unroll
    for (int step = 8; step > 0; step >>= 1) {
      const int ex = __shfl_sync(FULL, excl, j + step);
      if (ex <= f) j += step;
    }
    const int cj = __shfl_sync(FULL, cw, j), sj = __shfl_sync(FULL, skip, j),
              ej = __shfl_sync(FULL, excl, j);
    return (size_t)cj * L.scap + (sj + f - ej);
  };
  int m = 0;
  for (int f = 0; f < T; f += 64) {
    const size_t i0 = slot_of(f + lane), i1 = slot_of(f + 32 + lane);
    const bool a0 = f + lane < T, a1 = f + 32 + lane < T;
    const int q0 = a0 ? L.slot[i0] : p, q1 = a1 ? L.slot[i1] : p;
    const double4 x0 = ld32(X + q0), x1 = ld32(X + q1);
    const bool h0 = a0 && within_skin<PP>(P, p4, cp, x0, PP ? 0 : comp[q0], 0.0);
    const bool h1 = a1 && within_skin<PP>(P, p4, cp, x1, PP ? 0 : comp[q1], 0.0);
    const unsigned b0 = __ballot_sync(FULL, h0), b1 = __ballot_sync(FULL, h1);
    const unsigned lt = (1u << lane) - 1u;
    const int k0 = m + __popc(b0 & lt), k1 = m + __popc(b0) + __popc(b1 & lt);
    if (h0 && k0 < R.kc) R.cand[(size_t)k0 * n + p] = q0;
    if (h1 && k1 < R.kc) R.cand[(size_t)k1 * n + p] = q1;
    m += __popc(b0) + __popc(b1);
  }
  if (lane != 0) return;
  if (m > R.kc) {
    atomicMax(&cnt->need_kc, m);
    atomicExch(&cnt->row_overflow, 1);
    set_abort(cnt, tag);
    R.meta[p] = 0;
    return;
  }
  R.meta[p] = m;
  R.rank[p] = rank;
}

// The same row by one thread, for a full rebuild: 32 neighbouring rows read
// the same cells through L1, so a warp builds them in about the round trips
// that it needs for one row on its own (1M rows: 1.5 ms a warp per row).
// false: a list does not fit the slots, nothing is written.
template <bool PP>
__device__ __forceinline__ bool build_row_thread(const DevParams& P, int n, int p, int c,
                                                 const double4* __restrict__ X,
                                                 const int* __restrict__ comp,
                                                 const CellLists& L, const Rows& R,
                                                 Counters* cnt, int tag) {
  const double4 p4 = ld32(X + p);
  const int cp = PP ? 0 : comp[p];
  int cx, cy, cz;
  cell_coords(P, c, cx, cy, cz);
  int m = 0, rank = -1;
#pragma unroll 1
  for (int l = 0; l < 14; l++) {
    int cw = c;
    if (l > 0) {
      const int o = 27 - l;
      const int jx = cx + o % 3 - 1, jy = cy + (o / 3) % 3 - 1, jz = cz + o / 9 - 1;
      const bool ok = (P.pbc[0] || (jx >= 0 && jx < P.nx)) &&
                      (P.pbc[1] || (jy >= 0 && jy < P.ny)) &&
                      (P.pbc[2] || (jz >= 0 && jz < P.nz));
      if (!ok) continue;
      cw = P.coff + axis_wrap(jx, P.nx, P.pbc[0]) +
           P.nx * (axis_wrap(jy, P.ny, P.pbc[1]) + P.ny * axis_wrap(jz, P.nz, P.pbc[2]));
    }
    const int4* sl = (const int4*)(L.slot + (size_t)cw * L.scap);
    int4 s = sl[0];  // (the first entries with the length)
    const int len = L.slot_n[cw];
    if (len < 0 || len > L.scap) return false;
    for (int k0 = 0; k0 < len; k0 += 4) {
      if (k0 > 0) s = sl[k0 >> 2];
      const int q[4] = {s.x, s.y, s.z, s.w};
      double4 x[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (k0 + u < len) x[u] = ld32(X + q[u]);
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (k0 + u >= len) continue;
        if (l == 0 && rank < 0) {  // the own list up to p: not read
          if (q[u] == p) rank = k0 + u;
          continue;
        }
        if (within_skin<PP>(P, p4, cp, x[u], PP ? 0 : comp[q[u]], 0.0)) {
          if (m < R.kc) R.cand[(size_t)m * n + p] = q[u];
          m++;
        }
      }
    }
    if (rank < 0) {  // p is not in its cell's list
      atomicExch(&cnt->list_error, 1);
      set_abort(cnt, tag);
      return true;
    }
  }
  if (m > R.kc) {
    atomicMax(&cnt->need_kc, m);
    atomicExch(&cnt->row_overflow, 1);
    set_abort(cnt, tag);
    R.meta[p] = 0;
    return true;
  }
  R.meta[p] = m;
  R.rank[p] = rank;
  return true;
}

// Arguments of the row and the test kernel (the same for both precisions).
struct TestArgs {
  const DevParams* P;
  const int* sysid;
  int n;
  const int* cell_cur;  // cell of every particle in this pass
  CellLists L;
  Rows R;
  const double4* X;
  const int* comp;
  const int* cand;
  const int* meta;
  int2* clist;
  unsigned char* cord;
  int* cstart;
  int* ccount;
  int cl_cap;
  Counters* cnt;
  int tag;
  // the cells whose particles are tested: [slab_c0, slab_c0 + slab_span)
  // (a slab of a decomposition, or every cell)
  int slab_c0;
  unsigned slab_span;
  // 1: of the rows that read a relinked cell, only those near a particle that
  // changed cell are rebuilt; 0: every row of a stamped cell
  int fine;
};

// The candidate rows this pass rebuilds (the body of k_rows; warp / nwarps:
// this warp's index among the warps that share the work):
//  - every row on a full rebuild, a thread per row;
//  - else the rows a relinked cell's movers change.  A relink keeps the
//    stayers of a list in their order and puts the arrivals first, so a row
//    that reads the cell changes only if a particle that left or entered it
//    is within MinDij + skin of the row's owner; one farther than that can
//    come no closer than MinDij + 0.2 skin before the next full rebuild
//    (every particle moves at most 0.4 skin in between), so a stale entry for
//    it in the row is tested and rejected, and its absence changes no
//    contact.  A warp takes one record (mover, cell) and one of the 14 cells
//    whose rows read that cell, its lanes check the owners there (a margin
//    errs towards rebuilding), and it builds the rows that are near and that
//    no other warp has claimed in this pass.  The rank (the place in the list)
//    of every particle of a relinked cell is rewritten.
//  - else, when more movers were recorded than the list holds, or in a slab
//    of a decomposition (the stamps of its ghost layer come by exchange),
//    every row of a stamped cell.
// The rows were rebuilt inside the test kernel before, each by the warp of
// its owner: one after another within a warp, whose block waited (box of
// 1M bidisperse spheres, 84 movers a pass: 300 us per test launch).
template <bool PP>
__device__ __forceinline__ void rows_body(const TestArgs& A, int warp, int nwarps) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  Counters* const cnt = A.cnt;
  const int abort1 = lane == 0 ? cnt->abort : 0;  // (one reading for the warp)
  const bool full = cnt->full_due != 0;
  const int stamp = cnt->pass_id + 1;
  const int nm = cnt->n_mlist[stamp & 1];
  if (__shfl_sync(FULL, abort1, 0)) return;
  const int n = A.n;
  const CellLists& L = A.L;
  auto build = [&](int p, int c) {
    build_row<PP>(sys_params(A.P, A.sysid, p), n, p, c, A.X, A.comp, L, A.R, cnt, A.tag);
  };
  if (full || !A.fine || nm > L.mcap) {
    for (int v = warp; v < (n + 31) / 32; v += nwarps) {
      const int p = v * 32 + lane;
      const int c = p < n ? A.cell_cur[p] : -1;
      bool need = p < n && (unsigned)(c - A.slab_c0) < A.slab_span;
      if (need)
        need = full ? !build_row_thread<PP>(sys_params(A.P, A.sysid, p), n, p, c, A.X, A.comp, L,
                                            A.R, cnt, A.tag)
                    : L.rflag[c] == stamp;
      unsigned todo = __ballot_sync(FULL, need);
      while (todo) {
        const int l = __ffs(todo) - 1;
        todo &= todo - 1u;
        build(__shfl_sync(FULL, p, l), __shfl_sync(FULL, c, l));
      }
    }
    return;
  }
  for (int item = warp; item < nm * 14; item += nwarps) {
    const int2 r = L.mlist[(size_t)(stamp & 1) * L.mcap + item / 14];
    const int o = item % 14;
    if ((unsigned)r.x >= (unsigned)n) continue;
    const DevParams& P = sys_params(A.P, A.sysid, r.x);
    const int b = reading_cell(P, r.y, o);
    if (b < 0) continue;
    const int len = L.slot_n[b];
    const double4 q4 = ld32(A.X + r.x);
    const int cq = PP ? 0 : A.comp[r.x];
    const int* sl = L.slot + (size_t)b * L.scap;
    const bool slots = len >= 0 && len <= L.scap;
    int at = L.head[b];  // (a list that does not fit the slots: its next 32)
    for (int k0 = 0; slots ? k0 < len : (at != -1 && k0 < n); k0 += 32) {
      int x = -1;
      if (slots) {
        if (k0 + lane < len) x = sl[k0 + lane];
      } else {
        for (int k = 0; k < 32 && at != -1; k++) {
          if (lane == k) x = at;
          at = L.next[at];
        }
      }
      bool need = false;
      if (x >= 0) {
        if (o == 13) A.R.rank[x] = k0 + lane;  // (the relinked cell itself)
        const double4 x4 = ld32(A.X + x);
        const double slack = 1.0e-9 * (1.0 + x4.w + q4.w);
        need = within_skin<PP>(P, x4, PP ? 0 : A.comp[x], q4, cq, slack) &&
               atomicExch(&L.rstamp[x], stamp) != stamp;
      }
      unsigned todo = __ballot_sync(FULL, need);
      while (todo) {
        const int l = __ffs(todo) - 1;
        todo &= todo - 1u;
        build(__shfl_sync(FULL, x, l), b);
      }
    }
  }
}

// Every particle tests its row; the contacts of a particle are written
// together and in row order, and the block takes room for its contacts in
// the list with one atomic (two block barriers, which every thread of the
// block meets).  (The pass's contact count and the list length it needs come
// from the pair kernel, or from here when the list overflows.)
//
// Rows are short and uneven (2.9 candidates on average, 8 in the longest of
// 32, at 1M spheres), so a warp lays its 32 rows end to end in shared memory
// and its lanes test one candidate each: 3 turns instead of two groups of
// four per thread.  (One turn at a time: two or four in flight cost the
// registers of one or two blocks more per SM and lose, 55 and 60 against 48 us
// per launch.)  The ballots of the turns give every contact's place.  A warp whose rows
// hold more than WIN candidates goes through them in windows, once to count
// and once more to write.
// (The body of k_test for block `vblock`, so that a persistent kernel can
// run it too.  NC: candidates read through the non-coherent path, which
// needs the rows unchanged for the whole launch; a kernel that runs several
// passes reads them coherently.)
template <bool NC>
__device__ __forceinline__ int ld_row(const int* a) {
  return NC ? __ldg(a) : *a;
}
constexpr int WIN = 256;
struct alignas(16) TestWarp {  // shared memory of one warp
  double4 x[32];               // the rows' owners
  int q[WIN];                  // candidates of the window
  unsigned short own[WIN];     // (component << 8) | lane of the owner
  unsigned mask[WIN / 32 + 1];  // contacts among them
  int pre[WIN / 32 + 1];       // contacts before each 32
};

template <bool PP, bool NC = true>
__device__ __forceinline__ void test_body(const TestArgs& A, int vblock, TestWarp* warps) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  TestWarp& W = warps[warp];
  const int p0 = vblock * blockDim.x + threadIdx.x;
  const int p = p0 < A.n ? p0 : 0;
  const int n = A.n;
  // the abort word, the particle's own data, row length and first candidates
  // are requested together (every row holds at least 4 entries' room);
  // nothing is written once the abort word is seen (the block still meets its
  // barriers)
  const bool live = A.cnt->abort == 0;
  const int meta = A.meta[p];
  int q0[4];
#pragma unroll
  for (int u = 0; u < 4; u++) q0[u] = ld_row<NC>(A.cand + (size_t)u * n + p);
  const double4 p4 = ld32(A.X + p);
  const int cp = PP ? 0 : A.comp[p];
  // (a slab of a decomposition tests only its own particles)
  bool valid = p0 < n;
  if (A.slab_span != 0xffffffffu && valid)
    valid = (unsigned)(A.cell_cur[p] - A.slab_c0) < A.slab_span;
  const int m = live && valid ? (meta & META_MASK) : 0;
  W.x[lane] = p4;
  int off = m;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL, off, o);
    if (lane >= o) off += y;
  }
  const int T = __shfl_sync(FULL, off, 31);
  off -= m;
  // one system: its box in registers (no image beyond an infinite bound)
  const DevParams& P0 = A.P[0];
  const bool one = A.sysid == nullptr;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  const double hx = P0.box.pbc[0] ? P0.box.half_lim[0] : inf;
  const double hy = P0.box.pbc[1] ? P0.box.half_lim[1] : inf;
  const double hz = P0.box.pbc[2] ? P0.box.half_lim[2] : inf;
  // candidates [w0, w0 + WIN) of the warp into W.q / W.own, their contact
  // ballots into W.mask, the running count into W.pre
  auto window = [&](int w0) {
    const int lo = w0 > off ? w0 - off : 0;
    const int hi = off + m < w0 + WIN ? m : w0 + WIN - off;
    const unsigned short own = (unsigned short)((cp << 8) | lane);
    int* const wq = W.q + (off - w0);
    unsigned short* const wo = W.own + (off - w0);
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k >= lo && k < hi) {
        wq[k] = q0[k];
        wo[k] = own;
      }
    for (int k0 = lo > 4 ? lo : 4; k0 < hi; k0 += 4) {
      int q[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (k0 + u < hi) q[u] = ld_row<NC>(A.cand + (size_t)(k0 + u) * n + p);
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (k0 + u < hi) {
          wq[k0 + u] = q[u];
          wo[k0 + u] = own;
        }
    }
    __syncwarp();
    const int Tw = T - w0 < WIN ? T - w0 : WIN;
    int run = 0;
    for (int f0 = 0; f0 < Tw; f0 += 32) {
      const int f = f0 + lane;
      bool hit = false;
      if (f < Tw) {
        const int q = W.q[f];
        const double4 xq = ld32(A.X + q);
        const int own_f = W.own[f];
        const double4 a = W.x[own_f & 31];
        double Rij[3] = {__dsub_rn(xq.x, a.x), __dsub_rn(xq.y, a.y), __dsub_rn(xq.z, a.z)};
        const DevParams* P = &P0;
        if (one) {
          if (!(fabs(Rij[0]) < hx)) Rij[0] = image_rn(Rij[0], P0.box, 0);
          if (!(fabs(Rij[1]) < hy)) Rij[1] = image_rn(Rij[1], P0.box, 1);
          if (!(fabs(Rij[2]) < hz)) Rij[2] = image_rn(Rij[2], P0.box, 2);
        } else {
          P = A.P + A.sysid[p0 - lane + (own_f & 31)];
#pragma unroll
          for (int k = 0; k < 3; k++) Rij[k] = min_image_rn(Rij[k], P->box, k);
        }
        const int cq = PP || P->nc == 1 ? 0 : A.comp[q];
        const double md = min_dij_sq_rn<PP>(*P, PP ? 0 : own_f >> 8, a.w, cq, xq.w);
        hit = __dsub_rn(md, sumsq3_rn(Rij)) > 0.0;
      }
      const unsigned b = __ballot_sync(FULL, hit);
      if (lane == 0) {
        W.mask[f0 >> 5] = b;
        W.pre[f0 >> 5] = run;
      }
      run += __popc(b);
    }
    if (lane == 0) {
      W.mask[(Tw + 31) >> 5] = 0u;
      W.pre[(Tw + 31) >> 5] = run;
    }
    __syncwarp();
  };
  // contacts among the window's first f candidates
  auto before = [&](int f) {
    return W.pre[f >> 5] + __popc(W.mask[f >> 5] & ((1u << (f & 31)) - 1u));
  };
  __shared__ int s_wsum[8];  // blocks of at most 256 threads
  __shared__ int s_base;
  int total = 0, start = 0, done = 0;  // done: contacts written from earlier windows
  // first the contacts are counted, then written
#pragma unroll 1
  for (int ph = 0; ph < 2; ph++) {
#pragma unroll 1
    for (int w0 = 0; w0 < T; w0 += WIN) {
      if (ph == 0 || T > WIN) window(w0);
      const int Tw = T - w0 < WIN ? T - w0 : WIN;
      // the lane's part of the window
      const int lo = off < w0 ? 0 : off - w0 < Tw ? off - w0 : Tw;
      const int hi = off + m < w0 ? 0 : off + m - w0 < Tw ? off + m - w0 : Tw;
      const int b_lo = before(lo), mine = before(hi) - b_lo;
      if (ph == 0) {
        total += mine;
        __syncwarp();
        continue;
      }
      const int base = start + done - b_lo;  // place of the row's contact k: base + before
      const int first = done - b_lo;         // its number among the owner's: first + before
      done += mine;
      for (int f = lane; f < ((Tw + 31) & ~31); f += 32) {
        const unsigned b = W.mask[f >> 5];
        const int o = f < Tw ? W.own[f] & 31 : 0;
        const int bo = __shfl_sync(FULL, base, o), fo = __shfl_sync(FULL, first, o);
        if ((b >> lane) & 1u) {
          const int k = W.pre[f >> 5] + __popc(b & ((1u << lane) - 1u));
          A.clist[bo + k] = make_int2(p0 - lane + o, W.q[f]);
          const int ord = fo + k;
          A.cord[bo + k] = (unsigned char)(ord < ORD_MAX ? ord : ORD_MAX);
        }
      }
      __syncwarp();
    }
    if (ph == 1) break;
    // one allocation per block (the warps' sums through shared memory, one
    // atomic on the pass's list length); a particle's contacts are contiguous
    int incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_wsum[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
      int acc = 0;
      for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
        const int t = s_wsum[w];
        s_wsum[w] = acc;
        acc += t;
      }
      s_base = acc > 0 ? atomicAdd(&A.cnt->n_contacts, acc) : 0;
    }
    __syncthreads();
    start = s_base + s_wsum[warp] + incl - total;
    if (live && valid) {
      A.cstart[p] = start;
      A.ccount[p] = total;
    }
    const bool over = live && start + total > A.cl_cap;
    if (over) {
      // the list is grown and the pass launched again
      atomicMax(&A.cnt->need_cl, start + total);
      atomicExch(&A.cnt->cl_overflow, 1);
      set_abort(A.cnt, A.tag);
    }
    if (__any_sync(FULL, over)) return;
  }
}

// ---------------------------------------------------------------------------
// Persistent launches: a 4-step chunk (8 force passes) as one cooperative
// launch whose blocks step through every pass's phases (relink, test, pair,
// fold), separated by grid-wide barriers.

// A grid-wide barrier over `expected` blocks (gridDim.x of a cooperative
// launch, so that every block is resident): an arrival counter and a
// generation word.  A block that waits longer than limit_ns nanoseconds
// (%globaltimer) sets cnt->barrier_timeout and cnt->abort and reports
// failure; its caller then returns, and the blocks still waiting give up in
// turn, so the launch always ends.
struct GridSync {
  unsigned* count;
  unsigned* gen;
  Counters* cnt;
  unsigned long long limit_ns;
  unsigned expected;
};

// A launch of one cluster (small systems): the hardware cluster barrier, the
// walls of each step of the launch (copied into the system's table after the
// step's predictor; NULL: walls at rest), whether escapes stop the launch, and
// the passes of its program, which it repeats (whole periods of the ring's
// rotation and of the history's double buffer).
struct ClusterRun {
  const dem_wall* walls;
  DevParams* table;
  int nw, stop;
  int period;
};
// release / acquire at cluster scope: what every thread of the cluster wrote
// before is visible to every thread after
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();  // (the aligned forms take whole warps; the phases end with lanes apart)
  asm volatile("barrier.cluster.arrive.release.aligned;\n"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* a) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
  return v;
}

// All threads of every block call; returns false after a timeout.  The
// block's thread 0 arrives with an acquire-release add (after the block
// barrier, so it releases the whole block's writes); the last to arrive
// resets the count and publishes the next generation with a release add;
// the others poll the generation with acquire loads.
__device__ __forceinline__ bool grid_sync(const GridSync& g) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned gen0 = ld_acquire_u32(g.gen);  // cannot advance before this block arrives
    unsigned prev;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;"
                 : "=r"(prev)
                 : "l"(g.count)
                 : "memory");
    if (prev == g.expected - 1u) {
      *(volatile unsigned*)g.count = 0u;
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(g.gen) : "memory");
    } else {
      const unsigned long long t0 = global_ns();
      while (ld_acquire_u32(g.gen) == gen0) {
        if (global_ns() - t0 > g.limit_ns) {
          atomicExch(&g.cnt->barrier_timeout, 1);
          atomicExch(&g.cnt->abort, 1);
          ok = 0;
          break;
        }
        __nanosleep(32);
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

struct NoView {};

// Blocks per SM of a cooperative chunk launch that has work for `want` blocks.
// Up to three on each of the 148 SMs the phases are chains of latencies, and
// 168 registers a thread are worth more than room for a fourth block (20,000
// spheres on a floor 82 us per step, 91 with four; 16 systems of 200 to 2,000
// spheres 80 and 84); past that a fourth block's warps hide more than its 0.2
// to 1.2 kB of spills a thread cost (216k jammed spheres 488, 524 with three;
// 1M dense 722 and 801; 64 systems of 200 to 20,000 352 and 363).
inline int chunk_blocks_per_sm(int want) { return want > 3 * 148 ? 4 : 3; }

// Host side: `k` (a chunk kernel) as one cluster of 16 blocks, or of 8 where
// the device does not take 16.
template <class K, class CP>
inline cudaError_t launch_cluster(K k, const CP* prog, int npass, ClusterRun cr,
                                  cudaStream_t st) {
  cudaError_t e =
      cudaFuncSetAttribute((const void*)k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  for (unsigned size = 16; size >= 8; size /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(size);
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = size;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int fit = 0;
    if (size > 8) {
      e = cudaOccupancyMaxActiveClusters(&fit, (const void*)k, &cfg);
      if (e != cudaSuccess || fit < 1) {
        (void)cudaGetLastError();
        continue;
      }
    }
    return cudaLaunchKernelEx(&cfg, k, prog, npass, GridSync{}, cr);
  }
  return cudaErrorLaunchOutOfResources;
}

// One force pass of a chunk: its relink, test and pass arguments, the
// integrator epilogue (EPI_PREDICT / EPI_CORRECT) and, for the mixed path,
// the FP32 record arrays it reads and writes.  16-byte aligned: blocks copy
// it into shared memory as int4.
template <class V4, class W2, class View>
struct alignas(16) ChunkPass {
  RelinkArgs rl;
  TestArgs t;
  PassArgs<V4, W2> a;
  View v;
  int epi;
};

// The list phases of a chunk as calls, so that each has its own register
// allocation within the kernel's budget (inlined together they spill 1-2 kB a
// thread).
template <class CP>
__device__ __noinline__ void chunk_relink(const CP& p, int warp, int nwarps, int* sh) {
  const RelinkArgs& R = p.rl;
  relink_body(R.PT, R.cellsys, R.L, R.par, R.n, R.update, R.stop_tag, R.cnt, warp, nwarps, sh);
}
template <bool PP, class CP>
__device__ __noinline__ void chunk_rows(const CP& p, int warp, int nwarps) {
  rows_body<PP>(p.t, warp, nwarps);
}
template <bool PP, class CP>
__device__ __noinline__ void chunk_test(const CP& p, TestWarp* warps) {
  const int nvb = (p.t.n + 127) / 128;
  for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
    test_body<PP, false>(p.t, vb, warps);
    __syncthreads();
  }
}

// The start of pass k of a cluster launch: its own tag (the pass number in the
// launch; the program repeats), the escape stop before a
// step's first pass, and the walls of the step before its second one (not
// past a stopped pass, which the host repeats with the walls as they stand;
// what stops the launch has done so before this pass, but for errors).
template <class CP>
__device__ __forceinline__ void cluster_pass(CP& p, const ClusterRun& c, int k) {
  if (threadIdx.x == 0) {
    p.t.tag = k;
    p.a.tag = k;
    p.rl.stop_tag = c.stop && (k & 1) == 0 ? k : -1;
  }
  if (c.walls && (k & 1) && blockIdx.x == 0 && *(volatile const int*)&p.rl.cnt->abort == 0) {
    const int words = c.nw * (int)(sizeof(dem_wall) / sizeof(double));
    const double* src = (const double*)(c.walls + (size_t)(k >> 1) * NWM);
    double* dst = (double*)c.table->walls;  // (one system)
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
}

// the pass `src` into the block's shared copy `dst`
template <class CP>
__device__ __forceinline__ void load_pass(CP& dst, const CP* __restrict__ src) {
  static_assert(sizeof(CP) % 16 == 0, "ChunkPass size");
  const int4* a = reinterpret_cast<const int4*>(src);
  int4* b = reinterpret_cast<int4*>(&dst);
  for (int i = threadIdx.x; i < (int)(sizeof(CP) / 16); i += blockDim.x) b[i] = a[i];
  __syncthreads();
}

}  // namespace dem
