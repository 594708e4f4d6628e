// The persistent device program of libxcal: one launch runs `iters` SIMPLE (or
// PISO) iterations, or one standalone Krylov solve; or, where the pressure CG is
// a kernel of its own (small meshes in one cluster, large ones on the whole
// GPU), what lies between two pressure solves.  Phases are separated by
// xcal::Sync barriers; every phase is "tile owned" (tile t of 256 rows is always
// processed by CTA t mod the CTA count), so a CTA may reduce over its tiles at
// the end of a phase sequence without another barrier.  Reference functions are
// cited at each phase; xcal_device.cuh states the arithmetic contract.
//
// A case runs on a group of CTAs numbered 0..vnb()-1 (vbid()): the whole grid
// of an ordinary launch, or the CTAs the serving kernel (bottom of this file)
// gives the case.
//
// XCAL_ONE: this unit is a build for numberings with sweeps by one CTA.
#ifndef XCAL_ONE
#define XCAL_ONE false
#endif
#include "xcal_device.cuh"
#include "xcal_kernel.h"

namespace xcal {

namespace {

// CTA index within the group running the case, and the group's size.
__shared__ int s_vbid, s_vnb;
__device__ __forceinline__ int vbid() { return s_vbid; }
__device__ __forceinline__ int vnb() { return s_vnb; }
// Scratch of the reductions and the phase timers.  File scope, so that the
// out-of-line solvers address them as shared memory and not through generic
// pointers.
constexpr int MAXTL = 8;                 // tiles per CTA whose warp sums are staged
__shared__ double s_sm[8 * MAXK];
__shared__ double s_out[MAXK];
__shared__ double s_ws[MAXTL * MAXK * 8];
__shared__ int s_ok;
__shared__ unsigned long long s_pacc[2 * NPH];   // per-phase cycles and counts


// Level-scheduled preconditioners (forward and backward sweeps): DILU, ILU(0).
template <typename T>
__device__ __forceinline__ bool leveled(const MatT<T> &A) {
  return A.precon == PRECON_DILU || A.precon == PRECON_ILU0;
}
template <typename T>
__device__ __forceinline__ void lev_setup_row(const MatT<T> &A, int i) {
  if (A.precon == PRECON_ILU0) ilu_setup_row(A, i);
  else dilu_setup_row(A, i);
}
template <int NS, typename T, class GetOut>
__device__ __forceinline__ void lev_fwd_row(const MatT<T> &A, const T (&in)[NS], GetOut geto, int i, int blev_i,
                                            T (&o)[NS]) {
  if (A.precon == PRECON_ILU0) ilu_fwd_row<NS>(A, in, geto, i, blev_i, o);
  else dilu_fwd_row<NS>(A, in, geto, i, blev_i, o);
}
template <int NS, typename T>
__device__ __forceinline__ void lev_bwd_row(const MatT<T> &A, const T *out, int i, T (&o)[NS]) {
  T oi[NS];
#pragma unroll
  for (int d = 0; d < NS; ++d) oi[d] = out[(size_t)i * NS + d];
  auto g = [&](int j, int d) { return out[(size_t)j * NS + d]; };
  if (A.precon == PRECON_ILU0) ilu_bwd_row_g<NS>(A, oi, g, i, o);
  else dilu_bwd_row_g<NS>(A, oi, g, i, o);
}

// State of the CTA's run.  The mesh scalars the solvers use are copied here
// from KParams: a solver called out of line takes a copy of the whole struct
// into registers instead of reaching through a pointer for each of them.
struct Ctx {
  const KParams *P;
  int n, np, ntiles, nfl, nbl;
  int n0, ring;   // rows of level 0 of a two-level numbering (0: other numberings); matrix tiles the dynamic shared memory holds
  const int *flev, *blev;
  // sweeps by one CTA: bytes of dynamic shared memory for the vector (-1: the
  // grid's CTAs sweep level by level), the rows listed level by level, items
  int sweep;
  const int *frow, *brow, *items, *lptr;
  Sync S;
  // Per-tile partial sums, two buffers of MAXK*ntiles used in turn by
  // successive reducing phases.  A CTA reads a reduction's partials after the
  // barrier that ends its phase while faster CTAs may already be writing the
  // next reduction's partials; with a single buffer that write could land
  // before the read.  The next write to the same buffer comes two reducing
  // phases later, behind a barrier every CTA reaches only after its read.
  double *part;
  int pw;   // buffer the next reducing phase writes
  __device__ __forceinline__ double *part_w() const { return part + (size_t)pw * MAXK * ntiles; }
  __device__ __forceinline__ const double *part_r() const { return part + (size_t)(pw ^ 1) * MAXK * ntiles; }
  // per-phase timers: thread 0 of CTA 0 charges the SM cycles between two
  // barrier exits to the phase class that was current at the second one
  bool timers;
  int tag;
  long long t_last;
  // Traversal direction of the tile loops, reversed at every barrier: a phase
  // then starts on the tiles the previous phase touched last, whose data are
  // the most likely still in L2 when the working set is larger than L2.  Every
  // row's values are independent of the order, so results are unchanged.
  int rev;
  __device__ __forceinline__ void phase(int t) { tag = t; }
  __device__ __forceinline__ void tick() {
    if (timers) {
      const long long t = clock64();
      s_pacc[tag] += (unsigned long long)(t - t_last);
      s_pacc[NPH + tag] += 1ull;
      t_last = t;
    }
  }
  // One value per tile summed over all tiles: put_part of every own tile
  // (over one or more phases), then end_sum, which is a barrier of the whole
  // group and gives every thread the canonical sum.
  __device__ __forceinline__ void put_part(int t, double v) { part_w()[t] = v; }
  __device__ __forceinline__ bool end_sum(double &out) {
    pw ^= 1;
    if (!sync()) return false;
    double r[1];
    final_sum<1>(part_r(), ntiles, s_sm, s_out, r);
    out = r[0];
    return true;
  }
  __device__ __forceinline__ bool sync() {
    rev ^= 1;
    const bool ok = S.sync(&s_ok);
    tick();
    return ok;
  }
};

__device__ __forceinline__ void ctx_mesh(Ctx &C, const KParams &P) {
  C.P = &P;
  C.n = P.n;
  C.np = P.np;
  C.ntiles = P.ntiles;
  C.nfl = P.nfl;
  C.nbl = P.nbl;
  C.n0 = P.n0;
  C.ring = P.ring;
  C.sweep = P.sweep;
  C.frow = P.frow;
  C.brow = P.brow;
  C.items = P.items;
  C.lptr = P.lptr;
  C.flev = P.flev;
  C.blev = P.blev;
}

// The mesh scalars and level arrays as the solvers read them: from the kernel's
// parameters, each read a constant-bank operand that need not stay in a
// register from one phase to the next; in the build whose solvers are called
// out of line, from their copy.
#if XCAL_ONE
__device__ __forceinline__ const Ctx &mesh_of(const Ctx &C) { return C; }
#else
__device__ __forceinline__ const KParams &mesh_of(const Ctx &C) { return *C.P; }
#endif

template <typename T>
__device__ __forceinline__ const MatT<T> &matU(const KParams &P) {
  if constexpr (sizeof(T) == 4) return P.AU32; else return P.AU;
}
template <typename T>
__device__ __forceinline__ const MatT<T> &matP(const KParams &P) {
  if constexpr (sizeof(T) == 4) return P.AP32; else return P.AP;
}
template <typename T>
__device__ __forceinline__ const KWorkT<T> &workU(const KParams &P) {
  if constexpr (sizeof(T) == 4) return P.wU32; else return P.wU;
}
template <typename T>
__device__ __forceinline__ const KWorkT<T> &workP(const KParams &P) {
  if constexpr (sizeof(T) == 4) return P.wP32; else return P.wP;
}

// ---------------------------------------------------------------- phases
// The CTA's tiles are vbid(), vbid() + vnb(), ...: own_tiles of them, the
// m-th in the phase's traversal direction being own_tile(m).
__device__ __forceinline__ int own_tiles(int nt) {
  const int B = vbid(), G = vnb();
  return B < nt ? (nt - 1 - B) / G + 1 : 0;
}
__device__ __forceinline__ int own_tile(int m, int cnt, int rev) {
  return vbid() + vnb() * (rev ? cnt - 1 - m : m);
}

template <class F>
__device__ __forceinline__ void tile_each(const Ctx &C, F f) {
  const auto &P = mesh_of(C);
  const int cnt = own_tiles(P.ntiles);
  for (int m = 0; m < cnt; ++m) {
    const int i = own_tile(m, cnt, C.rev) * TILE + threadIdx.x;
    if (i < P.n) f(i);
  }
}

// One row per thread per tile; with `reduce`, the K values returned by f are
// summed per tile with the canonical tree into part[k*ntiles + t] of the
// current partial-sum buffer (Ctx::part_w).  The warp
// stage of each tile's tree runs as the rows finish and is staged in shared
// memory; the 8-way stage of all the CTA's tiles runs once at the end, so the
// warps are not held at a block barrier per tile.
template <int K, class F>
__device__ __forceinline__ void tile_phase(Ctx &C, bool reduce, F f) {
  const auto &P = mesh_of(C);
  const int nt = P.ntiles, cnt = own_tiles(nt), rev = C.rev;
  if (!reduce) {
    for (int m = 0; m < cnt; ++m) {
      const int i = own_tile(m, cnt, rev) * TILE + threadIdx.x;
      double v[K];
      if (i < P.n) f(i, v);
    }
    return;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double *part = C.part_w();
  C.pw ^= 1;
  for (int m0 = 0; m0 < cnt; m0 += MAXTL) {   // chunks of at most MAXTL tiles
    const int tn = min(MAXTL, cnt - m0);
    for (int tl = 0; tl < tn; ++tl) {
      const int i = own_tile(m0 + tl, cnt, rev) * TILE + threadIdx.x;
      double v[K];
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] = 0.0;
      if (i < P.n) f(i, v);
#pragma unroll
      for (int k = 0; k < K; ++k) {
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) v[k] = v[k] + __shfl_down_sync(0xffffffffu, v[k], off);
        if (lane == 0) s_ws[(tl * K + k) * 8 + wid] = v[k];
      }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < tn * K; q += TPB) {
      const double *w = s_ws + q * 8;
      double a0 = w[0] + w[4], a1 = w[1] + w[5];
      const double a2 = w[2] + w[6], a3 = w[3] + w[7];
      a0 = a0 + a2;
      a1 = a1 + a3;
      a0 = a0 + a1;
      const int k = q % K, t = own_tile(m0 + q / K, cnt, rev);
      part[(size_t)k * nt + t] = a0;
    }
    __syncthreads();
  }
}

// Rows per thread in the phases of the general CG (any but that over a two-level
// numbering): the loads of two rows in flight, the arithmetic of the one-row
// routines.  ms per SIMPLE iteration, two rows / one: 128^3 Jacobi 14.2 / 14.6,
// mixed 11.8 / 11.3; 96^3 ILU(0) 8.02 / 8.10, DILU in the RCM order 209 / 193,
// mixed 167 / 136; 800^2 quads, Jacobi, 4.20 / 3.82.
template <typename T>
struct CgRows {
  static constexpr int R = 2;
};
// Row pairs pay when the CTAs hold two tiles or more each; with one tile per
// CTA or fewer (small meshes: one phase is a barrier and one row per thread)
// the one-row routines are faster.  Uniform across the CTAs of a run.
template <class PT>
__device__ __forceinline__ bool pairs_pay(const PT &P) { return P.ntiles >= 2 * vnb(); }

// tile_phase over R tiles at a time: the CTA takes its tiles (in the phase's
// direction) R by R, thread t row t of each (ii[r], ok[r] false past the
// mesh, where ii[r] is a valid row to read from); the per-tile reductions are
// those of tile_phase (each tile's canonical tree).
template <int K, int R, class F>
__device__ __forceinline__ void tile_phase_rows(Ctx &C, bool reduce, F f) {
  const auto &P = mesh_of(C);
  const int nt = P.ntiles, cnt = own_tiles(nt), rev = C.rev;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double *part = C.part_w();
  if (reduce) C.pw ^= 1;
  for (int m0 = 0; m0 < cnt; m0 += MAXTL) {
    const int tn = min(MAXTL, cnt - m0);
    for (int tl = 0; tl < tn; tl += R) {
      int ii[R];
      bool ok[R], tv[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        tv[r] = tl + r < tn;
        const int i = (tv[r] ? own_tile(m0 + tl + r, cnt, rev) : 0) * TILE + threadIdx.x;
        ok[r] = tv[r] && i < P.n;
        ii[r] = ok[r] ? i : 0;
      }
      double v[R][K];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int k = 0; k < K; ++k) v[r][k] = 0.0;
      f(ii, ok, v);
      if (reduce)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (!tv[r]) continue;
#pragma unroll
          for (int k = 0; k < K; ++k) {
            double x = v[r][k];
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) x = x + __shfl_down_sync(0xffffffffu, x, off);
            if (lane == 0) s_ws[((tl + r) * K + k) * 8 + wid] = x;
          }
        }
    }
    if (!reduce) continue;
    __syncthreads();
    for (int q = threadIdx.x; q < tn * K; q += TPB) {
      const double *w = s_ws + q * 8;
      double a0 = w[0] + w[4], a1 = w[1] + w[5];
      const double a2 = w[2] + w[6], a3 = w[3] + w[7];
      a0 = a0 + a2;
      a1 = a1 + a3;
      a0 = a0 + a1;
      const int k = q % K, t = own_tile(m0 + q / K, cnt, rev);
      part[(size_t)k * nt + t] = a0;
    }
    __syncthreads();
  }
}

template <class F>
__device__ __forceinline__ void grid_each(int count, F f) {
  for (int i = vbid() * TPB + threadIdx.x; i < count; i += vnb() * TPB) f(i);
}

template <int NS>
__device__ __forceinline__ void ld(const double *a, int i, double (&o)[NS]) {
#pragma unroll
  for (int d = 0; d < NS; ++d) o[d] = a[(size_t)i * NS + d];
}
template <int NS>
__device__ __forceinline__ void st(double *a, int i, const double (&o)[NS]) {
#pragma unroll
  for (int d = 0; d < NS; ++d) a[(size_t)i * NS + d] = o[d];
}

// ------------------------------------------------------- preconditioning
// Row-local part of M^{-1}: DILU forward level 0 (and the backward step of
// rows without upper neighbours) or a diagonal scaling.  Returns false when
// the row has no row-local part (DILU rows of level >= 1).
template <int NS, typename T, class PT>
__device__ __forceinline__ bool precon_local(const PT &P, const MatT<T> &A, int i, const T (&in)[NS],
                                             T (&o)[NS]) {
  if (A.precon == PRECON_DILU) {
    if (ldro(P.flev + i) != 0) return false;
#pragma unroll
    for (int d = 0; d < NS; ++d) o[d] = in[d];
    if (ldro(P.blev + i) == 0) {
      const T di = A.Dinv[i];
#pragma unroll
      for (int d = 0; d < NS; ++d) o[d] = o[d] * di;
    }
    return true;
  }
  if (A.precon == PRECON_ILU0) {
    if (ldro(P.flev + i) != 0) return false;
#pragma unroll
    for (int d = 0; d < NS; ++d) o[d] = in[d];
    if (ldro(P.blev + i) == 0) {
      const T u = A.fval[ldro(A.dpos + i)];
#pragma unroll
      for (int d = 0; d < NS; ++d) o[d] = o[d] / u;
    }
    return true;
  }
  const T di = A.Dinv[i];
#pragma unroll
  for (int d = 0; d < NS; ++d) o[d] = di * in[d];
  return true;
}

// The sweeps of a numbering with many narrow levels (the caller's own order,
// RCM: a level is a wavefront of a few dozen rows) by one CTA.  A barrier over
// the grid per level costs about 3.5 us whatever the level holds.  Here a level
// is cut into items of up to 32 rows, dealt to the CTA's warps in turn: a warp
// fetches the entries of its next item, a chain of dependent loads that the
// solution is no part of, while the other warps pass the levels between, and
// then works on the vector, which is in shared memory where it fits, when the
// block barrier of the level before is passed.  The other CTAs wait at a
// barrier, at most sweep_wait() levels long.  Row arithmetic is that of the row
// routines.
// (A count of the items done, polled by the warps, in place of the block
// barrier: its release waits for the fetches in flight, 1.4 us per level.)
extern __shared__ __align__(128) unsigned char s_dyn[];

struct SweepArgs {   // what the sweeps need of Ctx, by value: they are called out of line
  int n, nfl, nbl, sweep;
  const int *blev, *frow, *brow, *items, *lptr;
};

template <typename T>
struct SweepMat {   // what the level loop needs of the matrix
  const T *val, *Dinv;
  const int *col, *blev;
  int W, np;
};

// One row's entries on one side of the diagonal: for DILU forward the lower
// ones with their Dinv, backward the upper ones.
template <typename T, int WS>
struct SweepRow {
  int i;        // -1: none
  int last;     // forward: the row has no upper neighbours
  int c[WS];    // neighbour, -1: not on this side
  T a[WS], d[WS], di;
};
template <bool FWD, typename T, int WS>
__device__ __forceinline__ void sweep_load(const SweepMat<T> &A, int i, SweepRow<T, WS> &r) {
  r.i = i;
  const int ii = max(i, 0);
  r.di = A.Dinv[ii];
  r.last = FWD ? ldro(A.blev + ii) == 0 : 0;
#pragma unroll
  for (int k = 0; k < WS; ++k) {
    const int kk = k < A.W ? k : A.W - 1;
    const int c = (i >= 0 && k < A.W) ? ldro(A.col + (size_t)kk * A.np + ii) : -1;
    const bool use = FWD ? (c >= 0 && c < ii) : c > ii;
    r.c[k] = use ? c : -1;
    r.a[k] = A.val[(size_t)kk * A.np + ii];
    r.d[k] = FWD ? A.Dinv[use ? c : ii] : T(0);
  }
}

template <int NS, bool FWD, typename T, int WS>
__device__ __forceinline__ void sweep_row(const SweepRow<T, WS> &r, const T *in, T *x) {
  if (r.i < 0) return;
#pragma unroll
  for (int d = 0; d < NS; ++d) {
    T o = FWD ? in[(size_t)r.i * NS + d] : x[(size_t)r.i * NS + d] * r.di;
#pragma unroll
    for (int k = 0; k < WS; ++k) {
      const int j = r.c[k] >= 0 ? r.c[k] : r.i;
      const T t = o - r.a[k] * x[(size_t)j * NS + d] * (FWD ? r.d[k] : r.di);
      o = r.c[k] >= 0 ? t : o;
    }
    if (FWD && r.last) o = o * r.di;
    x[(size_t)r.i * NS + d] = o;
  }
}

// Levels [first, stop) of one direction.  Item q is rows[item[2q]..item[2q+1])
// of one level; ptr[l] is the first item of level l.  x is the vector solved
// for (out in global memory or its copy in shared memory), in the right-hand
// side of the forward sweep.
// Out of line, once per direction: the two rows held take most of the
// registers, and inlined the loop shared them with what its caller had live
// (user-built equation on a 6,500-cell BFS 70.6 -> 62.6 ms, SIMPLE in the caller's
// order on a 5k BFS 120 -> 105 ms per iteration).
template <int NS, bool FWD, typename T, int WS>
__device__ __noinline__ void sweep_levels(SweepMat<T> A, const int *rows, const int *item, const int *ptr, int first,
                                          int stop, const T *in, T *x) {
  constexpr int NW = TPB / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int q0 = ldro(ptr + first), nq = ldro(ptr + stop);
  auto row_of = [&](int q) {
    const int p = ldro(item + 2 * q) + lane;
    return p < ldro(item + 2 * q + 1) ? ldro(rows + p) : -1;
  };
  // own items q, q + NW, ...: the entries of the next one and the row of the
  // one after it are on their way.  Two buffers used in turn, not one copied
  // into the other: a copy would wait for the loads.
  SweepRow<T, WS> r0, r1;
  int q = q0 + wid, inext = -1;
  bool odd = false;
  if (q < nq) sweep_load<FWD>(A, row_of(q), r0);
  if (q + NW < nq) inext = row_of(q + NW);
  int end = ldro(ptr + first + 1);
  for (int l = first; l < stop; ++l) {
    const int end_next = ldro(ptr + min(l + 2, stop));
    for (; q < end; q += NW) {
      if (odd) {
        if (q + NW < nq) sweep_load<FWD>(A, inext, r0);
        sweep_row<NS, FWD>(r1, in, x);
      } else {
        if (q + NW < nq) sweep_load<FWD>(A, inext, r1);
        sweep_row<NS, FWD>(r0, in, x);
      }
      odd = !odd;
      if (q + 2 * NW < nq) inext = row_of(q + 2 * NW);
    }
    __syncthreads();
    end = end_next;
  }
}

template <int NS, typename T, int WS>
__device__ __forceinline__ void sweep_both(const SweepArgs &C, const MatT<T> &A, const int *fitem, const int *bitem,
                                           int f0, int f1, int b0, int b1, const T *in, T *x) {
  const int *fptr = C.lptr, *bptr = C.lptr + C.nfl + 1;
  const SweepMat<T> M{A.val, A.Dinv, A.col, C.blev, A.W, A.np};
  if (f0 < f1) sweep_levels<NS, true, T, WS>(M, C.frow, fitem, fptr, f0, f1, in, x);
  if (b0 < b1) sweep_levels<NS, false, T, WS>(M, C.brow, bitem, bptr, b0, b1, in, x);
}

// Levels of a sweep pair: forward from `first`, then backward from 1.
__device__ __forceinline__ int sweep_length(int nfl, int nbl, int first) { return max(0, nfl - first) + nbl - 1; }

template <int NS, typename T>
__device__ __noinline__ void sweep_by_one(SweepArgs C, MatT<T> A, const T *in, T *out, bool setup, int first, int lo,
                                          int hi) {
  // levels [lo, hi) of the pair: forward [f0, f1), backward [b0, b1)
  const int nf = max(0, C.nfl - first);
  const int f0 = first + min(lo, nf), f1 = first + min(hi, nf), b0 = 1 + max(lo - nf, 0), b1 = 1 + max(hi - nf, 0);
  const int tid = threadIdx.x, len = C.n * NS;
  const int *fptr = C.lptr, *bptr = C.lptr + C.nfl + 1;
  const int *fitem = C.items, *bitem = C.items + 2 * ldro(fptr + C.nfl);
  if (setup || A.precon != PRECON_DILU || A.W > WUNROLL) {
    // pivots on the way, or ILU(0) rows: level by level, nothing fetched
    // ahead, the vector in global memory
    for (int l = f0; l < f1; ++l) {
      const int end = ldro(fitem + 2 * (ldro(fptr + l + 1) - 1) + 1);
      for (int p = ldro(fitem + 2 * ldro(fptr + l)) + tid; p < end; p += TPB) {
        const int i = ldro(C.frow + p);
        if (setup) lev_setup_row(A, i);
        T iv[NS], o[NS];
#pragma unroll
        for (int d = 0; d < NS; ++d) iv[d] = in[(size_t)i * NS + d];
        lev_fwd_row<NS>(A, iv, [&](int j, int d) { return out[(size_t)j * NS + d]; }, i, ldro(C.blev + i), o);
#pragma unroll
        for (int d = 0; d < NS; ++d) out[(size_t)i * NS + d] = o[d];
      }
      __syncthreads();
    }
    for (int l = b0; l < b1; ++l) {
      const int end = ldro(bitem + 2 * (ldro(bptr + l + 1) - 1) + 1);
      for (int p = ldro(bitem + 2 * ldro(bptr + l)) + tid; p < end; p += TPB) {
        const int i = ldro(C.brow + p);
        T o[NS];
        lev_bwd_row<NS>(A, out, i, o);
#pragma unroll
        for (int d = 0; d < NS; ++d) out[(size_t)i * NS + d] = o[d];
      }
      __syncthreads();
    }
    return;
  }
  const bool local = (size_t)len * sizeof(T) <= (size_t)C.sweep;
  T *x = local ? (T *)s_dyn : out;
  if (local && lo == 0) {   // rows below `first` were done by the phase before
    for (int q = tid; q < len; q += TPB) x[q] = out[q];
    __syncthreads();
  }
  if (A.W <= 5) sweep_both<NS, T, 5>(C, A, fitem, bitem, f0, f1, b0, b1, in, x);
  else sweep_both<NS, T, WUNROLL>(C, A, fitem, bitem, f0, f1, b0, b1, in, x);
  if (local && hi == sweep_length(C.nfl, C.nbl, first))
    for (int q = tid; q < len; q += TPB) out[q] = x[q];
}

// Number of phases of M^{-1} after its producer phase.  The producer did the
// row-local part (and, with first_lvl == 2, forward level 1 as well).
template <class PT, typename T>
__device__ __forceinline__ int precon_tail_phases(const PT &P, const MatT<T> &A, bool setup, int first_lvl) {
  if (!leveled(A)) return setup ? 1 : 0;
  return max(0, P.nfl - first_lvl) + (P.nbl - 1);
}

// The remaining phases of M^{-1} (in -> out).  With `setup` the DILU pivots
// (update_preconditioner!) are computed level by level in the same phases.
// The last phase also computes the K partial sums red(i, v).
// ONE: with the sweeps by one CTA for the numberings that have them.
template <int NS, int K, bool ONE, typename T, class Red, int R = 1>
__device__ __forceinline__ bool precon_tail(Ctx &C, const MatT<T> &A, const T *in, T *out, bool setup, int first_lvl, Red red) {
  const auto &P = mesh_of(C);
  const int nph = precon_tail_phases(P, A, setup, first_lvl);
  C.phase(setup ? PH_PREC_SETUP : PH_KRY_PREC);
  bool applied = nph == 0 && setup;   // nothing left to apply: reduce in a phase of its own
  if constexpr (ONE) {
    if (C.sweep >= 0 && leveled(A)) {
      const int levels = sweep_length(C.nfl, C.nbl, first_lvl), step = sweep_wait(A.W);
      for (int lo = 0; lo < levels; lo += step) {
        if (vbid() == 0)
          sweep_by_one<NS, T>(SweepArgs{C.n, C.nfl, C.nbl, C.sweep, C.blev, C.frow, C.brow, C.items, C.lptr}, A, in,
                              out, setup, first_lvl, lo, min(levels, lo + step));
        if (!C.sync()) return false;
      }
      applied = true;
    }
  }
  if (applied) {
    tile_phase<K>(C, true, [&](int i, double (&v)[K]) { red(i, v); });
    return C.sync();
  }
  if constexpr (R > 1) {
    if (!setup && A.precon == PRECON_DILU && nph > 0 && pairs_pay(P)) {
      // the DILU levels R rows at a time; in a warp holding a row of the
      // level, rows outside it compute with what they read and store
      // nothing; a warp without one skips the rows (with a level-ordered
      // numbering whole tiles lie outside each level)
      int ph = 0;
      for (int l = first_lvl; l < P.nfl; ++l) {
        const bool last = (++ph == nph);
        tile_phase_rows<K, R>(C, last, [&](const int (&ii)[R], const bool (&ok)[R], double (&v)[R][K]) {
          bool at[R], any = false;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            at[r] = ok[r] && ldro(P.flev + ii[r]) == l;
            any = any || at[r];
          }
          if (__any_sync(0xffffffffu, any)) {
            T iv[R][NS], o[R][NS];
            int bl[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
              bl[r] = ldro(P.blev + ii[r]);
#pragma unroll
              for (int d = 0; d < NS; ++d) iv[r][d] = in[(size_t)ii[r] * NS + d];
            }
            dilu_fwd_rows<R, NS>(A, iv, [&](int j, int d) { return out[(size_t)j * NS + d]; }, ii, bl, o);
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (at[r])
#pragma unroll
                for (int d = 0; d < NS; ++d) out[(size_t)ii[r] * NS + d] = o[r][d];
          }
          if (last)
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (ok[r]) red(ii[r], v[r]);
        });
        if (!C.sync()) return false;
      }
      for (int l = 1; l < P.nbl; ++l) {
        const bool last = (++ph == nph);
        tile_phase_rows<K, R>(C, last, [&](const int (&ii)[R], const bool (&ok)[R], double (&v)[R][K]) {
          bool at[R], any = false;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            at[r] = ok[r] && ldro(P.blev + ii[r]) == l;
            any = any || at[r];
          }
          if (__any_sync(0xffffffffu, any)) {
            T o[R][NS];
            dilu_bwd_rows<R, NS>(A, out, ii, o);
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (at[r])
#pragma unroll
                for (int d = 0; d < NS; ++d) out[(size_t)ii[r] * NS + d] = o[r][d];
          }
          if (last)
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (ok[r]) red(ii[r], v[r]);
        });
        if (!C.sync()) return false;
      }
      return true;
    }
  }
  if (!leveled(A)) {
    if (!setup) return true;
    tile_phase<K>(C, true, [&](int i, double (&v)[K]) {
      diag_precon_setup_row(A, i);
      const T di = A.Dinv[i];
#pragma unroll
      for (int d = 0; d < NS; ++d) out[(size_t)i * NS + d] = di * in[(size_t)i * NS + d];
      red(i, v);
    });
    return C.sync();
  }
  int ph = 0;
  for (int l = first_lvl; l < P.nfl; ++l) {
    const bool last = (++ph == nph);
    tile_phase<K>(C, last, [&](int i, double (&v)[K]) {
      if (ldro(P.flev + i) == l) {
        if (setup) lev_setup_row(A, i);
        T iv[NS], o[NS];
#pragma unroll
        for (int d = 0; d < NS; ++d) iv[d] = in[(size_t)i * NS + d];
        lev_fwd_row<NS>(A, iv, [&](int j, int d) { return out[(size_t)j * NS + d]; }, i, ldro(P.blev + i), o);
#pragma unroll
        for (int d = 0; d < NS; ++d) out[(size_t)i * NS + d] = o[d];
      }
      if (last) red(i, v);
    });
    if (!C.sync()) return false;
  }
  for (int l = 1; l < P.nbl; ++l) {
    const bool last = (++ph == nph);
    tile_phase<K>(C, last, [&](int i, double (&v)[K]) {
      if (ldro(P.blev + i) == l) {
        T o[NS];
        lev_bwd_row<NS>(A, out, i, o);
#pragma unroll
        for (int d = 0; d < NS; ++d) out[(size_t)i * NS + d] = o[d];
      }
      if (last) red(i, v);
    });
    if (!C.sync()) return false;
  }
  return true;
}

// Krylov start for row i (Krylov.jl warm start): r0 = b - A*x0 in FP64 over
// the row just assembled, x = 0, the DILU pivot of level-0 rows and the
// row-local part of the first M^{-1}.  With T = float the row is also copied
// to the FP32 matrix the Krylov iterations use (iterative refinement: the
// FP64 residual r0 is the right-hand side of an FP32 correction solve).
// BiCGSTAB keeps r0 in q and preconditions into r[0]; CG keeps r[0] = r0 and
// preconditions into v[0].
template <int NS, typename T>
__device__ __forceinline__ void krylov_init_row(const KParams &P, const Mat &A64, const MatT<T> &A,
                                                const KWorkT<T> &w, const double (&b)[NS], const double *x0,
                                                int i, int solver) {
  if constexpr (sizeof(T) == 4) {
    // every entry, padding included (zero in the FP64 matrix)
    for (int k = 0; k < A.W; ++k) {
      const size_t e = (size_t)k * A.np + i;
      A.val[e] = (float)A64.val[e];
    }
  }
  double y[NS];
  T r0[NS];
  spmv_row<NS>(A64, i, [&](int j, int d) { return x0[(size_t)j * NS + d]; }, y);
#pragma unroll
  for (int d = 0; d < NS; ++d) {
    r0[d] = (T)(b[d] - y[d]);
    w.x[(size_t)i * NS + d] = T(0);
  }
  if (leveled(A) && ldro(P.flev + i) == 0) lev_setup_row(A, i);
  T o[NS];
  const bool dilu = leveled(A);
  if (solver != SOLVER_CG) {
#pragma unroll
    for (int d = 0; d < NS; ++d) w.q[(size_t)i * NS + d] = r0[d];
    if (dilu && precon_local<NS>(P, A, i, r0, o))
#pragma unroll
      for (int d = 0; d < NS; ++d) w.r[0][(size_t)i * NS + d] = o[d];
  } else {
#pragma unroll
    for (int d = 0; d < NS; ++d) w.r[0][(size_t)i * NS + d] = r0[d];
    if (dilu && precon_local<NS>(P, A, i, r0, o))
#pragma unroll
      for (int d = 0; d < NS; ++d) w.v[0][(size_t)i * NS + d] = o[d];
  }
}

// Set-up phases of M and its first application after the assembly phase,
// with the initial dot products (CG: <r,z>; BiCGSTAB: <b,r>, <r,r>), all
// accumulated in FP64.
template <int NS, bool ONE, typename T>
__device__ __forceinline__ bool krylov_start_inl(Ctx &C, const MatT<T> &A, const KWorkT<T> &w, const double *b, int solver) {
  if (solver != SOLVER_CG) {
    return precon_tail<NS, 2 * NS, ONE>(C, A, w.q, w.r[0], true, 1, [&](int i, double (&v)[2 * NS]) {
#pragma unroll
      for (int d = 0; d < NS; ++d) {
        const double rv = (double)w.r[0][(size_t)i * NS + d];
        v[2 * d] = b[(size_t)i * NS + d] * rv;
        v[2 * d + 1] = rv * rv;
      }
    });
  }
  return precon_tail<NS, NS, ONE>(C, A, w.r[0], w.v[0], true, 1, [&](int i, double (&v)[NS]) {
#pragma unroll
    for (int d = 0; d < NS; ++d)
      v[d] = (double)w.r[0][(size_t)i * NS + d] * (double)w.v[0][(size_t)i * NS + d];
  });
}

// A call inside the program costs all of it: a frame of 3 KB where 0.4 KB did,
// and up to 0.4 us a phase (quad 157^2, p by BiCGSTAB: 1.80 -> 2.16 ms per
// iteration).  So the numberings with sweeps by one CTA, whose time is in the
// sweeps, have a build of the program of their own (ONE), with start and
// solvers out of line; in the others everything is inlined.
template <int NS, typename T>
__device__ __noinline__ bool krylov_start_one(Ctx *state, MatT<T> A, KWorkT<T> w, const double *b, int solver) {
  Ctx C = *state;
  const bool ok = krylov_start_inl<NS, true, T>(C, A, w, b, solver);
  *state = C;
  return ok;
}
template <int NS, bool ONE, typename T>
__device__ __forceinline__ bool krylov_start(Ctx &C, const MatT<T> &A, const KWorkT<T> &w, const double *b,
                                             int solver) {
  if constexpr (!ONE) return krylov_start_inl<NS, false, T>(C, A, w, b, solver);
  const KParams *P = C.P;
  Ctx t = C;
  t.P = nullptr;
  const bool ok = krylov_start_one<NS, T>(&t, A, w, b, solver);
  C = t;
  C.P = P;
  return ok;
}

// ------------------------------------------------------------- BiCGSTAB
// Krylov.jl 0.9.5 bicgstab! with left preconditioner M, N = I, c = b.
// Entry: r[0] = M^{-1}(b - A x0), x = 0, partials <b,r>, <r,r> in part.
// Fused phases per iteration:
//   A  p = r + beta*(p - omega*v) (recomputed for neighbours), q = A p, M^-1 level 0
//   .. remaining M^-1 phases, last one reduces <b,v>
//   D  s = r - alpha*v (recomputed for neighbours), x += alpha*p, q = A s, M^-1 level 0
//   .. remaining M^-1 phases, last one reduces <t,s>, <t,t>
//   G  x += omega*s, r = s - omega*t, reduces <b,r>, <r,r>
// Vector updates are evaluated in FP64 and stored in T; dots accumulate in FP64.
template <int NS, bool ONE, typename T>
__device__ __forceinline__ bool bicgstab(Ctx &C, const MatT<T> &A, const KWorkT<T> &w, const double *bb, const KCfg &cfg,
                         int (&its)[NS], double (&rnorm_out)[NS]) {
  const auto &P = mesh_of(C);
  double red[2 * NS];
  final_sum<2 * NS>(C.part_r(), P.ntiles, s_sm, s_out, red);
  double rho[NS], alpha[NS], omega[NS], beta[NS], rnorm[NS], eps[NS], nrho[NS];
  unsigned active = 0;
#pragma unroll
  for (int d = 0; d < NS; ++d) {
    its[d] = 0;
    rnorm[d] = sqrt(red[2 * d + 1]);
    rho[d] = 1.0; alpha[d] = 1.0; omega[d] = 1.0; beta[d] = 0.0;
    eps[d] = 0.0; nrho[d] = 0.0;
    if (rnorm[d] == 0.0) continue;
    eps[d] = cfg.atol + cfg.rtol * rnorm[d];
    nrho[d] = red[2 * d];
    if (nrho[d] == 0.0) continue;
    const bool solved = rnorm[d] <= eps[d], tired = 0 >= cfg.itmax;
    if (!(solved || tired)) active |= 1u << d;
  }
  T *r = w.r[0];
  const int tail = precon_tail_phases(P, A, false, 1);
  int pc = 0;
  bool first = true;
  while (active) {
#pragma unroll
    for (int d = 0; d < NS; ++d)
      if (active & (1u << d)) { its[d] += 1; rho[d] = nrho[d]; }
    T *pn = w.p[pc], *po = w.p[pc ^ 1], *vn = w.v[pc], *vo = w.v[pc ^ 1];
    auto getp = [&](int j, int d) -> T {
      const size_t k = (size_t)j * NS + d;
      if (first) return r[k];
      const double pv = (double)po[k] + (-omega[d]) * (double)vo[k];
      return (T)((double)r[k] + beta[d] * pv);
    };
    // A: p update, q = A p, M^{-1} row-local part
    C.phase(PH_KRY_SPMV);
    tile_phase<NS>(C, tail == 0, [&](int i, double (&v)[NS]) {
      T y[NS], pi[NS], o[NS];
      spmv_row<NS>(A, i, getp, y);
#pragma unroll
      for (int d = 0; d < NS; ++d) pi[d] = getp(i, d);
#pragma unroll
      for (int d = 0; d < NS; ++d)
        if (active & (1u << d)) pn[(size_t)i * NS + d] = pi[d];
#pragma unroll
      for (int d = 0; d < NS; ++d) w.q[(size_t)i * NS + d] = y[d];
      if (precon_local<NS>(P, A, i, y, o))
#pragma unroll
        for (int d = 0; d < NS; ++d) vn[(size_t)i * NS + d] = o[d];
      if (tail == 0)
#pragma unroll
        for (int d = 0; d < NS; ++d) v[d] = bb[(size_t)i * NS + d] * (double)o[d];
    });
    if (!C.sync()) return false;
    if (!precon_tail<NS, NS, ONE>(C, A, (const T *)w.q, vn, false, 1, [&](int i, double (&v)[NS]) {
#pragma unroll
          for (int d = 0; d < NS; ++d) v[d] = bb[(size_t)i * NS + d] * (double)vn[(size_t)i * NS + d];
        }))
      return false;
    {
      double cv[NS];
      final_sum<NS>(C.part_r(), P.ntiles, s_sm, s_out, cv);
#pragma unroll
      for (int d = 0; d < NS; ++d)
        if (active & (1u << d)) alpha[d] = rho[d] / cv[d];
    }
    auto gets = [&](int j, int d) -> T {
      const size_t k = (size_t)j * NS + d;
      return vaxpy<T>(r[k], -alpha[d], vn[k]);
    };
    // D: s, x += alpha p, q = A s, M^{-1} row-local part
    C.phase(PH_KRY_SPMV);
    tile_phase<2 * NS>(C, tail == 0, [&](int i, double (&v)[2 * NS]) {
      T y[NS], o[NS], si[NS];
#pragma unroll
      for (int d = 0; d < NS; ++d) {
        const size_t k = (size_t)i * NS + d;
        si[d] = gets(i, d);
        if (active & (1u << d)) {
          w.s[k] = si[d];
          w.x[k] = vaxpy<T>(w.x[k], alpha[d], pn[k]);
        }
      }
      spmv_row<NS>(A, i, gets, y);
#pragma unroll
      for (int d = 0; d < NS; ++d) w.q[(size_t)i * NS + d] = y[d];
      if (precon_local<NS>(P, A, i, y, o))
#pragma unroll
        for (int d = 0; d < NS; ++d) w.t[(size_t)i * NS + d] = o[d];
      if (tail == 0)
#pragma unroll
        for (int d = 0; d < NS; ++d) {
          v[2 * d] = (double)o[d] * (double)si[d];
          v[2 * d + 1] = (double)o[d] * (double)o[d];
        }
    });
    if (!C.sync()) return false;
    if (!precon_tail<NS, 2 * NS, ONE>(C, A, (const T *)w.q, w.t, false, 1, [&](int i, double (&v)[2 * NS]) {
#pragma unroll
          for (int d = 0; d < NS; ++d) {
            const size_t k = (size_t)i * NS + d;
            const double tv = (double)w.t[k];
            v[2 * d] = tv * (double)w.s[k];
            v[2 * d + 1] = tv * tv;
          }
        }))
      return false;
    final_sum<2 * NS>(C.part_r(), P.ntiles, s_sm, s_out, red);
#pragma unroll
    for (int d = 0; d < NS; ++d)
      if (active & (1u << d)) omega[d] = red[2 * d] / red[2 * d + 1];
    // G: x += omega s, r = s - omega t, <b,r>, <r,r>
    C.phase(PH_KRY_VEC);
    tile_phase<2 * NS>(C, true, [&](int i, double (&v)[2 * NS]) {
#pragma unroll
      for (int d = 0; d < NS; ++d) {
        const size_t k = (size_t)i * NS + d;
        double rv = (double)r[k];
        if (active & (1u << d)) {
          w.x[k] = vaxpy<T>(w.x[k], omega[d], w.s[k]);
          const T rt = vaxpy<T>(w.s[k], -omega[d], w.t[k]);
          r[k] = rt;
          rv = (double)rt;
        }
        v[2 * d] = bb[k] * rv;
        v[2 * d + 1] = rv * rv;
      }
    });
    if (!C.sync()) return false;
    final_sum<2 * NS>(C.part_r(), P.ntiles, s_sm, s_out, red);
    unsigned cont = 0;
#pragma unroll
    for (int d = 0; d < NS; ++d) {
      if (!(active & (1u << d))) continue;
      nrho[d] = red[2 * d];
      beta[d] = (nrho[d] / rho[d]) * (alpha[d] / omega[d]);
      rnorm[d] = sqrt(red[2 * d + 1]);
      const bool mach = (rnorm[d] + 1.0 <= 1.0);
      const bool solved = (rnorm[d] <= eps[d]) || mach;
      const bool tired = its[d] >= cfg.itmax;
      const bool breakdown = (alpha[d] == 0.0 || isnan(alpha[d]));
      if (!(solved || tired || breakdown)) cont |= 1u << d;
    }
    active = cont;
    first = false;
    pc ^= 1;
  }
#pragma unroll
  for (int d = 0; d < NS; ++d) rnorm_out[d] = rnorm[d];
  return true;
}

// ------------------------------------------- CG over a two-level numbering
// The two-colour numbering (quad and hex meshes) puts the rows of DILU level
// 0 first: rows [0, n0) have only upper neighbours, rows [n0, n) only lower
// ones.  CG then needs no level arrays, and its phases touch only the rows
// they change (the arithmetic of each row is that of cg() below):
//   A  all rows: p = z + beta p, q = A p, <p, q>; x += alpha p of the
//      iteration before (its p is read here in any case)
//   B  level 1: r -= alpha q, z = M^-1 r (neighbours' r recomputed)
//   C  level 0: r -= alpha q, z = M^-1 r; <r, z>
// A tile's <r, z> is summed in the phase that completes it.
//
// RES: the CTA's matrix tiles (values and columns) are copied into shared
// memory at the start of the solve (the 256 entries of one row position are
// contiguous in the ELL layout) and stay there: after a barrier, which empties
// L1, the columns come from shared memory at once and the phase is one round
// of gathers long instead of two (BFS 47k, one tile per CTA: A 4.1 -> 3.6 us, B
// and C 4.0 -> 2.7; the grid barrier is 1.2 us of it, the sum of A and C 0.5).
// Otherwise the rows are read from global memory in every phase.
//
// The columns become addresses, so the rows are copied by each thread's own
// asynchronous 16-byte copies, all in flight together, whose completion is
// part of the instruction stream: there is no flag to wait for and no wait
// that could run out with the columns unset.
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
// 16 bytes into shared memory, through L2 (the matrix was written in this launch).
__device__ __forceinline__ void copy16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <typename T, int WT, bool RES>
__device__ __forceinline__ bool cg_two_level(Ctx &C, const MatT<T> &A, const KWorkT<T> &w, const KCfg &cfg, int &its_out,
                                             double &rn_out) {
  constexpr double EPS = 2.220446049250313e-16;
  constexpr int CAP = MAXTL * MAXK;   // tiles whose warp sums fit s_ws
  const int n = C.n, n0 = C.n0, np = A.np, nt = C.ntiles;
  const int W = WT < WUNROLL ? WT : A.W;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int B0 = vbid(), G = vnb();
  const int cnt = own_tiles(nt);
  const int t0 = (n0 - 1) / TILE, t1 = n0 / TILE;        // last tile with level-0 rows, first with level-1 rows
  const int c0 = own_tiles(t0 + 1);                      // own tiles with level-0 rows: m in [0, c0)
  const int m1 = t1 > B0 ? min(cnt, (t1 - B0 + G - 1) / G) : 0;   // with level-1 rows: m in [m1, cnt)
  T *sv = (T *)s_dyn;
  int *sc = (int *)(s_dyn + (size_t)C.ring * W * TILE * sizeof(T));
  if (RES) {
    // one row position at a time: the first threads take its values, the next its columns
    constexpr int V = 16 / sizeof(T), NV = TILE / V, NC = TILE / 4;
    static_assert(NV + NC <= TPB, "one copy per thread and row position");
    for (int m = 0; m < cnt; ++m)
      for (int k = 0; k < W; ++k) {
        const size_t g = (size_t)k * np + (size_t)(B0 + G * m) * TILE, l = (size_t)(m * W + k) * TILE;
        if (tid < NV) copy16(sv + l + V * tid, A.val + g + V * tid);
        else if (tid < NV + NC) copy16(sc + l + 4 * (tid - NV), A.col + g + 4 * (tid - NV));
      }
    copies_wait();
    __syncthreads();
  }
  // first entry of row i of own tile m; entry k is at [k * ks]
  const size_t ks = RES ? (size_t)TILE : (size_t)np;
  auto vals = [&](int m) -> const T * {
    return RES ? sv + (size_t)m * W * TILE + tid : A.val + (size_t)(B0 + G * m) * TILE + tid;
  };
  auto cols = [&](int m) -> const int * {
    return RES ? sc + (size_t)m * W * TILE + tid : A.col + (size_t)(B0 + G * m) * TILE + tid;
  };
  // warp sum of a tile's products into s_ws[q]; block sums of the staged own
  // tiles m0, m0+d, ... to the partials
  auto stage = [&](int q, double v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) s_ws[q * 8 + wid] = v;
  };
  auto tile_sums = [&](int m0, int d, int count) {
    __syncthreads();
    if (tid < count) {
      const double *ww = s_ws + tid * 8;
      double a0 = ww[0] + ww[4], a1 = ww[1] + ww[5];
      const double a2 = ww[2] + ww[6], a3 = ww[3] + ww[7];
      a0 = a0 + a2;
      a1 = a1 + a3;
      C.put_part(B0 + G * (m0 + d * tid), a0 + a1);
    }
  };

  double red[1];
  final_sum<1>(C.part_r(), nt, s_sm, s_out, red);
  const double sgn = (red[0] < 0.0) ? -1.0 : 1.0;
  double gamma = sgn * red[0], rnorm = sqrt(gamma), alpha = 0.0, beta = 0.0, pn2 = gamma;
  int its = 0;
  bool active = false;
  double eps = 0.0;
  if (gamma != 0.0) {
    eps = cfg.atol + cfg.rtol * rnorm;
    active = !(rnorm <= eps || 0 >= cfg.itmax);
  }
  T *z = w.v[0];
  T *ro = w.r[0], *rn = w.r[1], *pn = w.p[0], *pspare = w.p[1];
  // The first direction is z itself: z + beta z and x + alpha z with beta =
  // alpha = 0 (exact for finite z; a non-finite z makes gamma, and with it
  // alpha and the result, non-finite), so the row loop has no branch that
  // would keep its loads from being issued together.
  const T *po = z;
  bool pending = false;   // x still lacks alpha*po
  while (active) {
    // A
    C.phase(PH_KRY_SPMV);
    for (int m = 0, q = 0; m < cnt; ++m) {
      const int i = (B0 + G * m) * TILE + tid;
      const T *v = vals(m);
      const int *c = cols(m);
      double pq = 0.0;
      if (i < n) {
        const T xi = w.x[i];
        T y = T(0), pi = T(0), poi = T(0);
#pragma unroll
        for (int k = 0; k < WT; ++k) {
          const int kk = (WT < WUNROLL || k < W) ? k : W - 1;
          const int cj = (WT < WUNROLL || k < W) ? c[kk * ks] : -1;
          const int j = cj >= 0 ? cj : i;
          const T oj = po[j], pj = vaxpy<T>(z[j], beta, oj);
          const T t = y + v[kk * ks] * pj;
          y = cj >= 0 ? t : y;
          if (cj == i) {
            pi = pj;
            poi = oj;
          }
        }
        w.x[i] = vaxpy<T>(xi, alpha, poi);
        pn[i] = pi;
        w.q[i] = y;
        pq = (double)pi * (double)y;
      }
      stage(q, pq);
      if (++q == CAP || m + 1 == cnt) {
        tile_sums(m + 1 - q, 1, q);
        q = 0;
        if (m + 1 < cnt) __syncthreads();
      }
    }
    pending = false;
    double s;
    if (!C.end_sum(s)) return false;
    const double pAp = sgn * s;
    if (pAp <= EPS * pn2 && fabs(pAp) <= EPS * pn2) break;   // zero curvature: stop
    alpha = gamma / pAp;
    // B
    C.phase(PH_KRY_PREC);
    for (int m = cnt - 1, q = 0; m >= m1; --m) {
      const int i = (B0 + G * m) * TILE + tid;
      const T *v = vals(m);
      const int *c = cols(m);
      double rz = 0.0;
      if (i < n && i >= n0) {
        const T ri = vaxpy<T>(ro[i], -alpha, w.q[i]), di = A.Dinv[i];
        T o = ri;
#pragma unroll
        for (int k = 0; k < WT - 1; ++k) {   // the diagonal is the last entry
          const int kk = (WT < WUNROLL || k < W - 1) ? k : 0;
          const int cj = (WT < WUNROLL || k < W - 1) ? c[kk * ks] : -1;
          const bool use = cj >= 0 && cj < i;
          const int j = use ? cj : i;
          const T t = o - v[kk * ks] * vaxpy<T>(ro[j], -alpha, w.q[j]) * A.Dinv[j];
          o = use ? t : o;
        }
        o = o * di;
        rn[i] = ri;
        z[i] = o;
        rz = (double)ri * (double)o;
      }
      if (m >= c0) {   // no level-0 rows: the tile is complete
        stage(q, rz);
        if (++q == CAP || m == max(m1, c0)) {
          tile_sums(m + q - 1, -1, q);
          q = 0;
          __syncthreads();
        }
      }
    }
    if (!C.sync()) return false;
    // C
    C.phase(PH_KRY_PREC);
    for (int m = c0 - 1, q = 0; m >= 0; --m) {
      const int i = (B0 + G * m) * TILE + tid;
      const T *v = vals(m);
      const int *c = cols(m);
      double rz = 0.0;
      if (i < n0) {
        const T ri = vaxpy<T>(ro[i], -alpha, w.q[i]);
        const T di = A.Dinv[i];
        T o = ri * di;
#pragma unroll
        for (int k = 1; k < WT; ++k) {   // the diagonal is the first entry
          const int kk = (WT < WUNROLL || k < W) ? k : W - 1;
          const int cj = (WT < WUNROLL || k < W) ? c[kk * ks] : -1;
          const bool use = cj > i;
          const int j = use ? cj : i;
          const T t = o - v[kk * ks] * z[j] * di;
          o = use ? t : o;
        }
        rn[i] = ri;
        z[i] = o;
        rz = (double)ri * (double)o;
      } else if (i < n) {   // level-1 rows of the tile that holds both levels
        rz = (double)rn[i] * (double)z[i];
      }
      stage(q, rz);
      if (++q == CAP || m == 0) {
        tile_sums(m + q - 1, -1, q);
        q = 0;
        if (m > 0) __syncthreads();
      }
    }
    if (!C.end_sum(s)) return false;
    const double gn = sgn * s;
    rnorm = sqrt(gn);
    const bool solved = (rnorm <= eps) || (rnorm + 1.0 <= 1.0);
    if (!solved) {
      beta = gn / gamma;
      pn2 = gn + (beta * beta) * pn2;
      gamma = gn;
    }
    its += 1;
    active = !(solved || its >= cfg.itmax);
    pending = true;
    T *tp = ro;
    ro = rn;
    rn = tp;
    tp = pn;
    pn = pspare;
    pspare = tp;
    po = tp;
  }
  if (pending)   // x += alpha p of the last iteration: own rows, read by this thread only before the next barrier
    for (int m = 0; m < cnt; ++m) {
      const int i = (B0 + G * m) * TILE + tid;
      if (i < n) w.x[i] = vaxpy<T>(w.x[i], alpha, po[i]);
    }
  its_out = its;
  rn_out = rnorm;
  return true;
}

// ------------------------------------------------------------------- CG
// Krylov.jl 0.9.5 cg! with preconditioner M.  The sign of <r,z> at the start
// selects the formulation: for a negative definite system CG runs on (-A)x=-b,
// i.e. <r,z> and <p,Ap> enter with their sign flipped (negation is exact).
// Entry: r[0] = b - A x0, v[0] = M^{-1} r, x = 0, partial <r,z> in part.
// Fused phases per iteration:
//   A  p = z + beta*p (recomputed for neighbours), q = A p, reduces <p,q>
//   B  x += alpha p, r -= alpha q, M^-1 levels 0 and 1 (level-0 values of
//      neighbours recomputed), backward step of rows without upper neighbours
//   .. remaining M^-1 phases, the last reduces <r,z>
template <int NS, bool ONE, typename T>
__device__ __forceinline__ bool cg(Ctx &C, const MatT<T> &A, const KWorkT<T> &w, const KCfg &cfg, int (&its)[NS],
                   double (&rnorm_out)[NS]) {
  const auto &P = mesh_of(C);
  const double EPS = 2.220446049250313e-16;
  double red[NS];
  final_sum<NS>(C.part_r(), P.ntiles, s_sm, s_out, red);
  double gamma[NS], sgn[NS], rnorm[NS], pn2[NS], eps[NS], alpha[NS], beta[NS];
  unsigned active = 0;
#pragma unroll
  for (int d = 0; d < NS; ++d) {
    its[d] = 0;
    sgn[d] = (red[d] < 0.0) ? -1.0 : 1.0;
    gamma[d] = sgn[d] * red[d];
    rnorm[d] = sqrt(gamma[d]);
    alpha[d] = 0.0; beta[d] = 0.0; pn2[d] = gamma[d]; eps[d] = 0.0;
    if (gamma[d] == 0.0) continue;
    eps[d] = cfg.atol + cfg.rtol * rnorm[d];
    const bool solved = rnorm[d] <= eps[d], tired = 0 >= cfg.itmax;
    if (!(solved || tired)) active |= 1u << d;
  }
  const T *z = w.v[0];
  T *zw = w.v[0];
  const bool dilu = leveled(A);
  const bool lvl1 = dilu && P.nfl >= 2;
  const int tail = dilu ? precon_tail_phases(P, A, false, 2) : 0;
  int rc = 0, pc = 0;
  bool first = true;
  while (active) {
    T *pn = w.p[pc], *po = w.p[pc ^ 1];
    auto getp = [&](int j, int d) -> T {
      const size_t k = (size_t)j * NS + d;
      if (first) return z[k];
      return vaxpy<T>(z[k], beta[d], po[k]);
    };
    // A: p update, q = A p, <p,q>
    C.phase(PH_KRY_SPMV);
    if (CgRows<T>::R > 1 && pairs_pay(P)) {
      constexpr int R = CgRows<T>::R;
      tile_phase_rows<NS, R>(C, true, [&](const int (&ii)[R], const bool (&ok)[R], double (&v)[R][NS]) {
        T y[R][NS];
        spmv_rows<R, NS>(A, ii, getp, y);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (!ok[r]) continue;
          const int i = ii[r];
#pragma unroll
          for (int d = 0; d < NS; ++d) {
            const T pi = getp(i, d);
            if (active & (1u << d)) pn[(size_t)i * NS + d] = pi;
            v[r][d] = (double)pi * (double)y[r][d];
            w.q[(size_t)i * NS + d] = y[r][d];
          }
        }
      });
    } else {
      tile_phase<NS>(C, true, [&](int i, double (&v)[NS]) {
        T y[NS];
        spmv_row<NS>(A, i, getp, y);
#pragma unroll
        for (int d = 0; d < NS; ++d) {
          const T pi = getp(i, d);
          if (active & (1u << d)) pn[(size_t)i * NS + d] = pi;
          v[d] = (double)pi * (double)y[d];
          w.q[(size_t)i * NS + d] = y[d];
        }
      });
    }
    if (!C.sync()) return false;
    final_sum<NS>(C.part_r(), P.ntiles, s_sm, s_out, red);
    unsigned upd = 0;
#pragma unroll
    for (int d = 0; d < NS; ++d) {
      if (!(active & (1u << d))) continue;
      const double pAp = sgn[d] * red[d];
      if (pAp <= EPS * pn2[d] && fabs(pAp) <= EPS * pn2[d]) continue;   // zero curvature: stop
      alpha[d] = gamma[d] / pAp;
      upd |= 1u << d;
    }
    active = upd;
    if (!active) break;
    T *ro = w.r[rc], *rn = w.r[rc ^ 1];
    auto getr = [&](int j, int d) -> T {
      const size_t k = (size_t)j * NS + d;
      return vaxpy<T>(ro[k], -alpha[d], w.q[k]);
    };
    // B: x, r updates and M^{-1} levels 0/1
    C.phase(PH_KRY_PREC);
    if (CgRows<T>::R > 1 && pairs_pay(P)) {
      if (A.precon == PRECON_DILU) {
        // R rows at a time; a DILU row of level 0 or 1 is one forward row
        // (level 0: no lower neighbours, then its diagonal step when it has
        // no upper ones), the row-local part of precon_local for level 0
        constexpr int R = CgRows<T>::R;
        tile_phase_rows<NS, R>(C, tail == 0, [&](const int (&ii)[R], const bool (&ok)[R], double (&v)[R][NS]) {
          T rr[R][NS], o[R][NS];
          int fl[R], bl[R];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int i = ii[r];
            fl[r] = ldro(P.flev + i);
            bl[r] = ldro(P.blev + i);
#pragma unroll
            for (int d = 0; d < NS; ++d) {
              const size_t k = (size_t)i * NS + d;
              rr[r][d] = getr(i, d);
              if (ok[r] && (active & (1u << d))) {
                w.x[k] = vaxpy<T>(w.x[k], alpha[d], pn[k]);
                rn[k] = rr[r][d];
              }
            }
          }
          // only level-1 rows have lower neighbours to sum over; a warp
          // without one takes the row-local step (level 0: o = r, scaled by
          // the pivot's inverse when the row has no upper neighbours)
          bool any = false;
#pragma unroll
          for (int r = 0; r < R; ++r) any = any || (ok[r] && lvl1 && fl[r] == 1);
          if (__any_sync(0xffffffffu, any)) {
            dilu_fwd_rows<R, NS>(A, rr, getr, ii, bl, o);
          } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
              for (int d = 0; d < NS; ++d) o[r][d] = rr[r][d];
              if (bl[r] == 0) {
                const T di = A.Dinv[ii[r]];
#pragma unroll
                for (int d = 0; d < NS; ++d) o[r][d] = o[r][d] * di;
              }
            }
          }
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (!ok[r]) continue;
            const bool have = fl[r] == 0 || (lvl1 && fl[r] == 1);
            if (have)
#pragma unroll
              for (int d = 0; d < NS; ++d) zw[(size_t)ii[r] * NS + d] = o[r][d];
            if (tail == 0)
#pragma unroll
              for (int d = 0; d < NS; ++d) v[r][d] = (double)rr[r][d] * (double)o[r][d];
          }
        });
        goto phase_b_done;
      }
    }
    tile_phase<NS>(C, tail == 0, [&](int i, double (&v)[NS]) {
      T rr[NS], o[NS];
#pragma unroll
      for (int d = 0; d < NS; ++d) {
        const size_t k = (size_t)i * NS + d;
        rr[d] = getr(i, d);
        if (active & (1u << d)) {
          w.x[k] = vaxpy<T>(w.x[k], alpha[d], pn[k]);
          rn[k] = rr[d];
        }
      }
      bool have;
      have = precon_local<NS>(P, A, i, rr, o);
      if (!have && lvl1 && ldro(P.flev + i) == 1) {
        lev_fwd_row<NS>(A, rr, getr, i, ldro(P.blev + i), o);
        have = true;
      }
      if (have)
#pragma unroll
        for (int d = 0; d < NS; ++d) zw[(size_t)i * NS + d] = o[d];
      if (tail == 0)
#pragma unroll
        for (int d = 0; d < NS; ++d) v[d] = (double)rr[d] * (double)o[d];
    });
  phase_b_done:
    if (!C.sync()) return false;
    if (dilu) {
      auto rz = [&](int i, double (&v)[NS]) {
#pragma unroll
        for (int d = 0; d < NS; ++d) v[d] = (double)rn[(size_t)i * NS + d] * (double)z[(size_t)i * NS + d];
      };
      if (!precon_tail<NS, NS, ONE, T, decltype(rz), CgRows<T>::R>(C, A, (const T *)rn, zw, false, 2, rz)) return false;
    }
    final_sum<NS>(C.part_r(), P.ntiles, s_sm, s_out, red);
    unsigned cont = 0;
#pragma unroll
    for (int d = 0; d < NS; ++d) {
      if (!(active & (1u << d))) continue;
      const double gn = sgn[d] * red[d];
      rnorm[d] = sqrt(gn);
      const bool mach = (rnorm[d] + 1.0 <= 1.0);
      const bool solved = (rnorm[d] <= eps[d]) || mach;
      if (!solved) {
        beta[d] = gn / gamma[d];
        pn2[d] = gn + (beta[d] * beta[d]) * pn2[d];
        gamma[d] = gn;
      }
      its[d] += 1;
      const bool tired = its[d] >= cfg.itmax;
      if (!(solved || tired)) cont |= 1u << d;
    }
    active = cont;
    first = false;
    rc ^= 1;
    pc ^= 1;
  }
#pragma unroll
  for (int d = 0; d < NS; ++d) rnorm_out[d] = rnorm[d];
  return true;
}

// ---------------------------------------------------------------- GMRES
// Krylov.jl 0.9.5 gmres! with left preconditioner M, N = I, restart = false
// (the basis grows up to itmax vectors), no reorthogonalisation: modified
// Gram-Schmidt Arnoldi, QR of the Hessenberg matrix by Givens rotations
// (SymOrtho, sym_givens), back substitution for y at the end, x = V y.
// Entry (krylov_start, as for BiCGSTAB): r[0] = M^{-1}(b - A x0), x = 0,
// partials <b,r>, <r,r>.  Phases of inner iteration k:
//   P1  V_k = src/div (stored; recomputed for neighbours), t = A V_k,
//       M^{-1} row-local part
//   ..  remaining M^{-1} phases, the last reduces h_1 = <V_1, q>
//   Mi  q -= h_{i-1} V_{i-1}, reduces h_i = <V_i, q>        (i = 2..k)
//   N   q -= h_k V_k, reduces <q, q>
// Every CTA's thread 0 then updates its copy of the rotations (c, s, z) and
// the new column; CTA 0 also stores the column of R for the back substitution.
__device__ __forceinline__ double sgn1(double a) { return a > 0.0 ? 1.0 : (a < 0.0 ? -1.0 : a); }

__device__ __forceinline__ void sym_givens(double a, double b, double &c, double &s, double &rho) {
  if (b == 0.0) {
    c = (a == 0.0) ? 1.0 : sgn1(a);
    s = 0.0;
    rho = fabs(a);
  } else if (a == 0.0) {
    c = 0.0;
    s = sgn1(b);
    rho = fabs(b);
  } else if (fabs(b) > fabs(a)) {
    const double t = a / b;
    s = sgn1(b) / sqrt(1.0 + t * t);
    c = s * t;
    rho = b / s;
  } else {
    const double t = b / a;
    c = sgn1(a) / sqrt(1.0 + t * t);
    s = c * t;
    rho = a / c;
  }
}

template <int NS, bool ONE, typename T>
__device__ __forceinline__ bool gmres(Ctx &C, const MatT<T> &A, const KWorkT<T> &w, const KCfg &cfg, int (&its)[NS],
                      double (&rnorm_out)[NS]) {
  const auto &P = mesh_of(C);
  const double BTOL = 1.8189894035458565e-12;   // eps(Float64)^(3/4) = 2^-39
  double red[2 * NS];
  final_sum<2 * NS>(C.part_r(), P.ntiles, s_sm, s_out, red);
  const int G1 = w.gmax + 1;
  const int kmax = min(cfg.itmax, w.gmax);
  double *gws = w.gws + (size_t)vbid() * NS * 4 * G1;
  const size_t rs = (size_t)w.gmax * (w.gmax + 1) / 2;
  double beta0[NS], rnorm[NS], eps[NS], hbis[NS];
  unsigned active = 0;
#pragma unroll
  for (int d = 0; d < NS; ++d) {
    its[d] = 0;
    beta0[d] = sqrt(red[2 * d + 1]);
    rnorm[d] = beta0[d];
    hbis[d] = beta0[d];
    eps[d] = 0.0;
    if (beta0[d] == 0.0) continue;        // x = 0 is a zero-residual solution
    eps[d] = cfg.atol + cfg.rtol * rnorm[d];
    const bool solved = rnorm[d] <= eps[d], tired = 0 >= cfg.itmax;
    if (!(solved || tired)) active |= 1u << d;
  }
  if (threadIdx.x == 0)
#pragma unroll
    for (int d = 0; d < NS; ++d) gws[(size_t)d * 4 * G1 + 2 * G1] = beta0[d];   // z_1 = beta
  const unsigned ran = active;
  const T *r0 = w.r[0];
  T *qb[2] = {w.v[0], w.v[1]};
  const size_t nv = (size_t)P.n * NS;
  const int tail = precon_tail_phases(P, A, false, 1);
  int k = 0;
  while (active) {
    ++k;
    const T *src = (k == 1) ? r0 : qb[(k - 1) & 1];
    T *qn = qb[k & 1];
    T *Vk = w.V + (size_t)(k - 1) * nv;
    double div[NS];
#pragma unroll
    for (int d = 0; d < NS; ++d) div[d] = (k == 1) ? beta0[d] : hbis[d];
    auto getv = [&](int j, int d) -> T { return (T)((double)src[(size_t)j * NS + d] / div[d]); };
    // P1: V_k, t = A V_k, M^{-1} row-local part
    C.phase(PH_KRY_SPMV);
    tile_phase<NS>(C, tail == 0, [&](int i, double (&v)[NS]) {
      T y[NS], o[NS], vk[NS];
      spmv_row<NS>(A, i, getv, y);
#pragma unroll
      for (int d = 0; d < NS; ++d) {
        vk[d] = getv(i, d);
        Vk[(size_t)i * NS + d] = vk[d];
        w.t[(size_t)i * NS + d] = y[d];
      }
      if (precon_local<NS>(P, A, i, y, o))
#pragma unroll
        for (int d = 0; d < NS; ++d) qn[(size_t)i * NS + d] = o[d];
      if (tail == 0)
#pragma unroll
        for (int d = 0; d < NS; ++d) {
          const double v1 = (k == 1) ? (double)vk[d] : (double)w.V[(size_t)i * NS + d];
          v[d] = v1 * (double)o[d];
        }
    });
    if (!C.sync()) return false;
    if (!precon_tail<NS, NS, ONE>(C, A, (const T *)w.t, qn, false, 1, [&](int i, double (&v)[NS]) {
#pragma unroll
          for (int d = 0; d < NS; ++d)
            v[d] = (double)w.V[(size_t)i * NS + d] * (double)qn[(size_t)i * NS + d];
        }))
      return false;
    double h[NS];
    final_sum<NS>(C.part_r(), P.ntiles, s_sm, s_out, h);
    if (threadIdx.x == 0)
#pragma unroll
      for (int d = 0; d < NS; ++d) gws[(size_t)d * 4 * G1 + 3 * G1] = h[d];
    // modified Gram-Schmidt against V_2..V_k, each dot after the previous update
    for (int m = 2; m <= k + 1; ++m) {
      const T *Vp = w.V + (size_t)(m - 2) * nv;
      const T *Vm = w.V + (size_t)(m - 1) * nv;
      const bool norm = (m == k + 1);
      C.phase(PH_KRY_VEC);
      tile_phase<NS>(C, true, [&](int i, double (&v)[NS]) {
#pragma unroll
        for (int d = 0; d < NS; ++d) {
          const size_t q = (size_t)i * NS + d;
          const T qv = vaxpy<T>(qn[q], -h[d], Vp[q]);
          qn[q] = qv;
          v[d] = norm ? (double)qv * (double)qv : (double)Vm[q] * (double)qv;
        }
      });
      if (!C.sync()) return false;
      final_sum<NS>(C.part_r(), P.ntiles, s_sm, s_out, h);
      if (!norm && threadIdx.x == 0)
#pragma unroll
        for (int d = 0; d < NS; ++d) gws[(size_t)d * 4 * G1 + 3 * G1 + (m - 1)] = h[d];
    }
#pragma unroll
    for (int d = 0; d < NS; ++d) hbis[d] = sqrt(h[d]);
    // Givens: previous rotations on the new column, then the new rotation
    if (threadIdx.x == 0) {
#pragma unroll
      for (int d = 0; d < NS; ++d) {
        if (!(active & (1u << d))) continue;
        double *cs = gws + (size_t)d * 4 * G1, *sn = cs + G1, *zz = sn + G1, *col = zz + G1;
        for (int i = 0; i < k - 1; ++i) {
          const double tmp = cs[i] * col[i] + sn[i] * col[i + 1];
          col[i + 1] = sn[i] * col[i] - cs[i] * col[i + 1];
          col[i] = tmp;
        }
        double c_, s_, rho;
        sym_givens(col[k - 1], hbis[d], c_, s_, rho);
        cs[k - 1] = c_;
        sn[k - 1] = s_;
        col[k - 1] = rho;
        const double zeta = s_ * zz[k - 1];
        zz[k - 1] = c_ * zz[k - 1];
        zz[k] = zeta;
        s_out[d] = fabs(zeta);
        if (vbid() == 0) {
          double *Rc = w.gR + (size_t)d * rs + (size_t)(k - 1) * k / 2;
          for (int i = 0; i < k; ++i) Rc[i] = col[i];
        }
      }
    }
    __syncthreads();
    unsigned cont = 0;
#pragma unroll
    for (int d = 0; d < NS; ++d) {
      if (!(active & (1u << d))) continue;
      rnorm[d] = s_out[d];
      its[d] = k;
      const bool mach = (rnorm[d] + 1.0 <= 1.0);
      const bool solved = (rnorm[d] <= eps[d]) || mach;
      const bool breakdown = hbis[d] <= BTOL;
      const bool tired = k >= kmax;
      if (!(solved || tired || breakdown)) cont |= 1u << d;
    }
    __syncthreads();
    active = cont;
  }
  if (ran) {
    // R complete (CTA 0's stores) after this barrier; y by back substitution
    C.phase(PH_KRY_VEC);
    if (!C.sync()) return false;
    if (threadIdx.x == 0) {
#pragma unroll
      for (int d = 0; d < NS; ++d) {
        if (!(ran & (1u << d))) continue;
        const int kd = its[d];
        double *zz = gws + (size_t)d * 4 * G1 + 2 * G1, *y = zz + G1;
        const double *R = w.gR + (size_t)d * rs;
        for (int i = 0; i < kd; ++i) y[i] = zz[i];
        for (int i = kd - 1; i >= 0; --i) {
          double yi = y[i];
          for (int j = kd - 1; j >= i + 1; --j) yi = yi - R[(size_t)j * (j + 1) / 2 + i] * y[j];
          const double rii = R[(size_t)i * (i + 1) / 2 + i];
          y[i] = (fabs(rii) <= BTOL) ? 0.0 : yi / rii;
        }
      }
    }
    __syncthreads();
    tile_each(C, [&](int i) {
#pragma unroll
      for (int d = 0; d < NS; ++d) {
        if (!(ran & (1u << d))) continue;
        const double *y = gws + (size_t)d * 4 * G1 + 3 * G1;
        const size_t q = (size_t)i * NS + d;
        double acc = (double)w.x[q];
        for (int m = 0; m < its[d]; ++m) acc = acc + y[m] * (double)w.V[(size_t)m * nv + q];
        w.x[q] = (T)acc;
      }
    });
    if (!C.sync()) return false;
  }
#pragma unroll
  for (int d = 0; d < NS; ++d) rnorm_out[d] = rnorm[d];
  return true;
}

// The solvers of the ONE build, once per component count.  The state is
// copied in and back, so that the caller's own stays in registers; matrix and
// vectors are read from shared memory (kept in registers they spilled).
__shared__ __align__(16) unsigned char s_matrix[sizeof(Mat)], s_work[sizeof(KWork)];
template <int NS, typename T>
__device__ __noinline__ bool krylov_general(Ctx *state, const double *b, KCfg cfg, int *its, double *rn) {
  Ctx C = *state;
  const MatT<T> &A = *(const MatT<T> *)s_matrix;
  const KWorkT<T> &w = *(const KWorkT<T> *)s_work;
  int it[NS];
  double r[NS];
  bool ok;
  if (cfg.solver == SOLVER_BICGSTAB) ok = bicgstab<NS, true>(C, A, w, b, cfg, it, r);
  else if (cfg.solver == SOLVER_GMRES) ok = gmres<NS, true>(C, A, w, cfg, it, r);
  else ok = cg<NS, true>(C, A, w, cfg, it, r);
#pragma unroll
  for (int d = 0; d < NS; ++d) {
    its[d] = it[d];
    rn[d] = r[d];
  }
  *state = C;
  return ok;
}
template <int NS, typename T>
__device__ __forceinline__ bool krylov(Ctx &C, const MatT<T> &A, const KWorkT<T> &w, const double *b, const KCfg &cfg,
                                       int (&its)[NS], double (&rn)[NS]) {
  __syncthreads();
  if (threadIdx.x == 0) {
    *(MatT<T> *)s_matrix = A;
    *(KWorkT<T> *)s_work = w;
  }
  __syncthreads();
  const KParams *P = C.P;
  Ctx t = C;
  t.P = nullptr;   // were the parameters' address to leave the kernel, every read of them would go through memory
  int it[NS];
  double r[NS];
  const bool ok = krylov_general<NS, T>(&t, b, cfg, it, r);
#pragma unroll
  for (int d = 0; d < NS; ++d) {
    its[d] = it[d];
    rn[d] = r[d];
  }
  C = t;
  C.P = P;
  return ok;
}

template <int NS, bool ONE, typename T>
__device__ __forceinline__ bool solve_vector(Ctx &C, const MatT<T> &A, const KWorkT<T> &w, const double *b,
                                             const KCfg &cfg, int (&its)[NS], double (&rn)[NS]) {
  if constexpr (ONE) {
    return krylov<NS, T>(C, A, w, b, cfg, its, rn);
  } else {
    if (cfg.solver == SOLVER_BICGSTAB) return bicgstab<NS, false>(C, A, w, b, cfg, its, rn);
    if (cfg.solver == SOLVER_GMRES) return gmres<NS, false>(C, A, w, cfg, its, rn);
    return cg<NS, false>(C, A, w, cfg, its, rn);
  }
}

// Pressure solve of a mesh of DIM dimensions.
template <int DIM, bool ONE, typename T>
__device__ __forceinline__ bool solve_pressure(Ctx &C, const MatT<T> &A, const KWorkT<T> &w, const double *b,
                                               const KCfg &cfg, int (&its)[1], double (&rn)[1]) {
  if constexpr (!ONE) {   // a two-level numbering has no sweeps by one CTA
    constexpr int WT = DIM == 2 ? 5 : DIM == 3 ? 7 : WUNROLL;   // rows of a quad or hex mesh
    if (cfg.solver == SOLVER_CG && A.precon == PRECON_DILU && C.n0 > 0 && A.W <= WUNROLL) {
      // (large meshes run the CG as a kernel of its own; here the rows of tiles
      // that do not fit are those of a standalone solve, of a serving case or of
      // a launch form that was asked for)
      if (C.ring * vnb() < C.ntiles) {
        if (WT < WUNROLL && A.W == WT) return cg_two_level<T, WT, false>(C, A, w, cfg, its[0], rn[0]);
        return cg_two_level<T, WUNROLL, false>(C, A, w, cfg, its[0], rn[0]);
      }
      if (WT < WUNROLL && A.W == WT) return cg_two_level<T, WT, true>(C, A, w, cfg, its[0], rn[0]);
      return cg_two_level<T, WUNROLL, true>(C, A, w, cfg, its[0], rn[0]);
    }
  }
  return solve_vector<1, ONE>(C, A, w, b, cfg, its, rn);
}

// -------------------------------------------------------------- assembly
// Momentum row (ux/uy[/uz] share A): _discretise! with Time, Divergence(mdotf),
// -Laplacian(nueff) and -Source(grad p) (Solvers_1_SIMPLE.jl:21-35,
// Discretise_2_generated_distretisation.jl:5-81, Discretise_1_schemes.jl:11-113),
// then apply_boundary_conditions! (Discretise_4_apply_bcs.jl:7-44 with the functors
// of Discretise_3_boundary_conditions.jl:4-209), implicit_relaxation!
// (Solve_1_api.jl:54-60) and inverse_diagonal! (Solvers_0_functions.jl:77-88).
template <int NS>
__device__ __forceinline__ void momentum_row(const KParams &P, int i, bool relax, double (&b)[NS]) {
  const Mat &A = P.AU;
  const double vol = ldro(P.vol + i);
  double acc = 0.0;
  for (int k = 0; k < P.Wf; ++k) {
    const size_t e = (size_t)k * P.np + i;
    const int f = ldro(P.f_face + e);
    if (f < 0) break;
    const double ns = (double)ldro(P.f_sign + e);
    const int pos = ldro(P.f_pos + e);
    double t2;
    const double mf = P.mdot[f];
    if (P.div == DIV_UPWIND) {
      const double ap = 1.0 * (mf * ns);
      acc += jmax(ap, 0.0);
      t2 = -jmax(-ap, 0.0);
    } else {
      const int nb = ldro(P.f_nbr + e);
      const double ax = ldro(P.fcx + f) - ldro(P.ccx + i), ay = ldro(P.fcy + f) - ldro(P.ccy + i),
                   az = ldro(P.fcz + f) - ldro(P.ccz + i);
      const double bx = ldro(P.ccx + nb) - ldro(P.ccx + i), by = ldro(P.ccy + nb) - ldro(P.ccy + i),
                   bz = ldro(P.ccz + nb) - ldro(P.ccz + i);
      const double weight = sqrt((ax * ax + ay * ay) + az * az) / sqrt((bx * bx + by * by) + bz * bz);
      const double omw = 1.0 - weight;
      const double ap = 1.0 * (mf * ns);
      acc += ap * omw;
      t2 = ap * weight;
    }
    const double ap3 = -1.0 * ((-P.nueff[f]) * ldro(P.area + f)) / ldro(P.delta + f);
    acc += ap3;
    const double t3 = -ap3;
    const double base = ldro(P.f_first + e) ? 0.0 : A.val[pos];
    A.val[pos] = (base + t2) + t3;
  }
  double prev[NS];
#pragma unroll
  for (int d = 0; d < NS; ++d) { prev[d] = P.U[(size_t)i * NS + d]; b[d] = 0.0; }
  if (P.time == TIME_EULER) {
    const double rdt = 1 / P.dt;
    acc += vol * rdt;
#pragma unroll
    for (int d = 0; d < NS; ++d) b[d] += prev[d] * vol * rdt;
  }
#pragma unroll
  for (int d = 0; d < NS; ++d) b[d] += -1.0 * P.gp[(size_t)i * NS + d] * vol;
  const FieldBC &bc = P.bcU;
  for (int q = ldro(bc.a_ptr + i); q < ldro(bc.a_ptr + i + 1); ++q) {
    const int f = ldro(bc.a_face + q);
    const BcEntry &e = bc.tab[ldro(bc.a_bc + q)];
    const double ap = 1.0 * P.mdot[f];
    if (P.div == DIV_UPWIND) {
      if (e.type == BC_DIRICHLET) {
#pragma unroll
        for (int d = 0; d < NS; ++d) b[d] -= ap * e.v[d];
      } else if (e.type == BC_NEUMANN || e.type == BC_KWALL || e.type == BC_OMEGAWALL) {
        acc += jmax(ap, 0.0);
      }
    } else {
      if (e.type == BC_DIRICHLET) {
#pragma unroll
        for (int d = 0; d < NS; ++d) b[d] += 1.0 * ((-P.mdot[f]) * e.v[d]);
      } else if (e.type == BC_NEUMANN || e.type == BC_KWALL || e.type == BC_OMEGAWALL) {
        acc += ap;
      }
    }
    if (e.type == BC_DIRICHLET) {
      const double flux = P.nueff[f] * ldro(P.area + f) / ldro(P.delta + f);
      const double apl = -1.0 * (-flux);
      acc += apl;
#pragma unroll
      for (int d = 0; d < NS; ++d) b[d] += apl * e.v[d];
    }
  }
  if (relax) {
    acc /= P.aU;
#pragma unroll
    for (int d = 0; d < NS; ++d) b[d] += (1.0 - P.aU) * acc * prev[d];
  }
  A.val[ldro(A.dpos + i)] = acc;
  P.rD[i] = vol / acc;
  st<NS>(P.bU, i, b);
}

// u . S_f of a face vector field (flux!/div!: psif[fID] . (area*normal))
template <int NS>
__device__ __forceinline__ double face_dot_S(const KParams &P, const double *uf, int f) {
  const double a = ldro(P.area + f);
  double s = uf[(size_t)f * NS] * (a * ldro(P.fnx + f)) + uf[(size_t)f * NS + 1] * (a * ldro(P.fny + f));
  if (NS == 3) s = s + uf[(size_t)f * NS + 2] * (a * ldro(P.fnz + f));
  return s;
}

// Pressure row: div!(divHv, Uf) (Calculate_0_divergence.jl:75-107) then
// Laplacian(rDf, p) == Source(divHv) with BCs and setReference!
// (Solvers_1_SIMPLE.jl:37-39,154-157, Solve_1_api.jl:62-69).
template <int NS>
__device__ __forceinline__ double pressure_row(const KParams &P, int i) {
  const Mat &A = P.AP;
  const double vol = ldro(P.vol + i);
  double dv = 0.0;
  for (int k = 0; k < P.Wf; ++k) {
    const size_t e = (size_t)k * P.np + i;
    const int f = ldro(P.f_face + e);
    if (f < 0) break;
    dv += face_dot_S<NS>(P, P.UfH, f) * (double)ldro(P.f_sign + e) / vol;
  }
  for (int q = ldro(P.cb_ptr + i); q < ldro(P.cb_ptr + i + 1); ++q)
    dv += face_dot_S<NS>(P, P.UfH, ldro(P.cb_face + q)) / vol;
  P.divH[i] = dv;
  double acc = 0.0;
  for (int k = 0; k < P.Wf; ++k) {
    const size_t e = (size_t)k * P.np + i;
    const int f = ldro(P.f_face + e);
    if (f < 0) break;
    const int pos = ldro(P.f_pos + e);
    const double ap = 1.0 * ((-P.rDf[f]) * ldro(P.area + f)) / ldro(P.delta + f);
    acc += ap;
    const double base = ldro(P.f_first + e) ? 0.0 : A.val[pos];
    A.val[pos] = base + (-ap);
  }
  double b = 0.0;
  b += 1.0 * dv * vol;
  const FieldBC &bc = P.bcP;
  for (int q = ldro(bc.a_ptr + i); q < ldro(bc.a_ptr + i + 1); ++q) {
    const int f = ldro(bc.a_face + q);
    const BcEntry &e = bc.tab[ldro(bc.a_bc + q)];
    if (e.type == BC_DIRICHLET) {
      const double flux = P.rDf[f] * ldro(P.area + f) / ldro(P.delta + f);
      const double ap = 1.0 * (-flux);
      acc += ap;
      b += ap * e.v[0];
    }
  }
  if (P.has_pref && i == P.ref_cell) {
    b += acc * P.pref;
    acc += acc;
  }
  A.val[ldro(A.dpos + i)] = acc;
  P.bP[i] = b;
  return b;
}

// H! sums (Solvers_0_functions.jl:110-140): H = (b - sum_n A_cn U_n) * (1/A_cc),
// ux's matrix for every component, neighbours in face order.
template <int NS>
__device__ __forceinline__ void H_row(const KParams &P, int i, const double (&bb)[NS]) {
  const Mat &A = P.AU;
  double sum[NS];
#pragma unroll
  for (int d = 0; d < NS; ++d) sum[d] = 0.0;
  for (int k = 0; k < P.Wf; ++k) {
    const size_t e = (size_t)k * P.np + i;
    const int f = ldro(P.f_face + e);
    if (f < 0) break;
    const int nb = ldro(P.f_nbr + e);
    const double a = A.val[ldro(P.f_pos + e)];
#pragma unroll
    for (int d = 0; d < NS; ++d) sum[d] += a * P.U[(size_t)nb * NS + d];
  }
  const double rDc = 1 / A.val[ldro(A.dpos + i)];
#pragma unroll
  for (int d = 0; d < NS; ++d) P.H[(size_t)i * NS + d] = (bb[d] - sum[d]) * rDc;
}

// ------------------------------------------------------------ face fields
// interpolate! (Calculate_2_interpolation.jl:241-277) plus correct_boundaries!
// (:135-237) for a vector cell field.
template <int NS>
__device__ __forceinline__ void face_vector(const KParams &P, const double *cellv, int f, double (&u)[NS]) {
  const double w = ldro(P.wgt + f);
  const double omw = 1.0 - w;
  const int a = ldro(P.o1 + f), b = ldro(P.o2 + f);
#pragma unroll
  for (int d = 0; d < NS; ++d) u[d] = w * cellv[(size_t)a * NS + d] + omw * cellv[(size_t)b * NS + d];
  if (f < P.nbf) {
    const int bi = ldro(P.bcU.fbc + f);
    if (bi >= 0) {
      const BcEntry &e = P.bcU.tab[bi];
#pragma unroll
      for (int d = 0; d < NS; ++d) u[d] = (e.type == BC_DIRICHLET) ? e.v[d] : cellv[(size_t)a * NS + d];
    }
  }
}

// flux!(mdotf, Uf) (Solvers_0_functions.jl:65-73) from the face-interpolated U.
template <int NS>
__device__ __forceinline__ void face_mdot(const KParams &P, int f) {
  double u[NS];
  face_vector<NS>(P, P.U, f, u);
  if (P.model == 1)
#pragma unroll
    for (int d = 0; d < NS; ++d) P.UfH[(size_t)f * NS + d] = u[d];
  const double a = ldro(P.area + f);
  double m = u[0] * (a * ldro(P.fnx + f)) + u[1] * (a * ldro(P.fny + f));
  if (NS == 3) m = m + u[2] * (a * ldro(P.fnz + f));
  P.mdot[f] = m;
}

// correct_interpolation! (Calculate_0_gradient.jl:146-173), internal face f.
template <int NS>
__device__ __forceinline__ double midpoint_corrected(const KParams &P, int f) {
  const double w = 0.5;
  const int a = ldro(P.o1 + f), b = ldro(P.o2 + f);
  const double phifp = w * (P.p[a] + P.p[b]);
  const double g0 = w * (P.gp[(size_t)a * NS] + P.gp[(size_t)b * NS]);
  const double g1 = w * (P.gp[(size_t)a * NS + 1] + P.gp[(size_t)b * NS + 1]);
  const double r0 = ldro(P.fcx + f) - w * (ldro(P.ccx + a) + ldro(P.ccx + b));
  const double r1 = ldro(P.fcy + f) - w * (ldro(P.ccy + a) + ldro(P.ccy + b));
  double dt = g0 * r0 + g1 * r1;
  if (NS == 3) {
    const double g2 = w * (P.gp[(size_t)a * NS + 2] + P.gp[(size_t)b * NS + 2]);
    const double r2 = ldro(P.fcz + f) - w * (ldro(P.ccz + a) + ldro(P.ccz + b));
    dt = dt + g2 * r2;
  }
  return phifp + dt;
}

// grad!(grad p) for the scheme in use, starting from a synchronised pf of the
// first interpolation.  With correct_u the last Green-Gauss pass also applies
// correct_velocity! (Solvers_0_functions.jl:90-99): U = H - grad(p)*rD.
template <int NS>
__device__ __forceinline__ bool gradient_p(Ctx &C, bool correct_u) {
  const KParams &P = *C.P;
  const int npass = (P.grad == GRAD_MIDPOINT) ? 3 : 1;
  for (int pass = 0; pass < npass; ++pass) {
    const bool last = (pass == npass - 1);
    C.phase(PH_GRAD);
    tile_each(C, [&](int i) {
      double g[NS];
      green_gauss_row<NS>(P, P.pf, i, g);
      st<NS>(P.gp, i, g);
      if (last && correct_u) {
        const double rdi = P.rD[i];
#pragma unroll
        for (int d = 0; d < NS; ++d) P.U[(size_t)i * NS + d] = P.H[(size_t)i * NS + d] - g[d] * rdi;
      }
    });
    if (!C.sync()) return false;
    if (!last) {
      C.phase(PH_FACE);
      grid_each(P.nf - P.nbf, [&](int q) {
        const int f = P.nbf + q;
        P.pf[f] = midpoint_corrected<NS>(P, f);
      });
      if (!C.sync()) return false;
    }
  }
  return true;
}

// ------------------------------------------------------------- k-omega
// Wilcox k-omega of RANSModels_kOmega.jl:114-415 and RANSModels_functions.jl:5-88.
constexpr double KW_BPLUS = 0.09, KW_ALPHA1 = 0.52, KW_BETA1 = 0.072, KW_SIGK = 0.5, KW_SIGW = 0.5;   // get_coeffs

__device__ __forceinline__ double nut_wall_fn(double nu, double yplus, double kappa, double E) {
  return jmax(nu * (yplus * kappa / log(jmax(E * yplus, 1.0 + 1e-4)) - 1), 0.0);
}

// omega of a wall cell (constraint!/set_cell_value!, :364-448)
__device__ __forceinline__ double omega_wall(const KParams &P, const BcEntry &e, double kc, double y) {
  const double wvis = 6.0 * P.nu / (e.beta1 * (y * y));
  const double wlog = sqrt(kc) / (e.c25 * e.kappa * y);
  const double yplus = e.c25 * y * sqrt(kc) / P.nu;
  return (yplus > e.ylam) ? wlog : wvis;
}

// Transport row of k or omega: Time + Divergence(mdotf) - Laplacian(nueff) +
// Si(D) == Source(P) (:191-207) with BCs (Discretise_3_boundary_conditions.jl),
// implicit_relaxation! and, for omega, constrain_equation! (:346-399).
__device__ __forceinline__ double scalar_row(const KParams &P, const Mat &A, int i, const double *phi,
                                             const double *gam, const double *Si, const double *src,
                                             const FieldBC &bc, double alpha, int div, int time, bool omega) {
  const double vol = ldro(P.vol + i);
  double acc = 0.0;
  for (int k = 0; k < P.Wf; ++k) {
    const size_t e = (size_t)k * P.np + i;
    const int f = ldro(P.f_face + e);
    if (f < 0) break;
    const double ns = (double)ldro(P.f_sign + e);
    const int pos = ldro(P.f_pos + e);
    double t2;
    const double mf = P.mdot[f];
    if (div == DIV_UPWIND) {
      const double ap = 1.0 * (mf * ns);
      acc += jmax(ap, 0.0);
      t2 = -jmax(-ap, 0.0);
    } else {
      const int nb = ldro(P.f_nbr + e);
      const double ax = ldro(P.fcx + f) - ldro(P.ccx + i), ay = ldro(P.fcy + f) - ldro(P.ccy + i),
                   az = ldro(P.fcz + f) - ldro(P.ccz + i);
      const double bx = ldro(P.ccx + nb) - ldro(P.ccx + i), by = ldro(P.ccy + nb) - ldro(P.ccy + i),
                   bz = ldro(P.ccz + nb) - ldro(P.ccz + i);
      const double weight = sqrt((ax * ax + ay * ay) + az * az) / sqrt((bx * bx + by * by) + bz * bz);
      const double omw = 1.0 - weight;
      const double ap = 1.0 * (mf * ns);
      acc += ap * omw;
      t2 = ap * weight;
    }
    const double ap3 = -1.0 * ((-gam[f]) * ldro(P.area + f)) / ldro(P.delta + f);
    acc += ap3;
    const double t3 = -ap3;
    const double base = ldro(P.f_first + e) ? 0.0 : A.val[pos];
    A.val[pos] = (base + t2) + t3;
  }
  const double prev = phi[i];
  double b = 0.0;
  if (time == TIME_EULER) {
    const double rdt = 1 / P.dt;
    acc += vol * rdt;
    b += prev * vol * rdt;
  }
  acc += 1.0 * Si[i] * vol;
  b += 1.0 * src[i] * vol;
  for (int q = ldro(bc.a_ptr + i); q < ldro(bc.a_ptr + i + 1); ++q) {
    const int f = ldro(bc.a_face + q);
    const BcEntry &e = bc.tab[ldro(bc.a_bc + q)];
    const double ap = 1.0 * P.mdot[f];
    const bool neu = (e.type == BC_NEUMANN || e.type == BC_KWALL || e.type == BC_OMEGAWALL);
    if (div == DIV_UPWIND) {
      if (e.type == BC_DIRICHLET) b -= ap * e.v[0];
      else if (neu) acc += jmax(ap, 0.0);
    } else {
      if (e.type == BC_DIRICHLET) b += 1.0 * ((-P.mdot[f]) * e.v[0]);
      else if (neu) acc += ap;
    }
    if (e.type == BC_DIRICHLET) {
      const double flux = gam[f] * ldro(P.area + f) / ldro(P.delta + f);
      const double apl = -1.0 * (-flux);
      acc += apl;
      b += apl * e.v[0];
    }
    if (e.type == BC_OMEGAWALL) {
      const double flux = 1.0 * Si[i];
      b += flux * phi[i] * vol;
    }
  }
  acc /= alpha;
  b += (1.0 - alpha) * acc * prev;
  if (omega)
    for (int q = ldro(bc.a_ptr + i); q < ldro(bc.a_ptr + i + 1); ++q) {
      const BcEntry &e = bc.tab[ldro(bc.a_bc + q)];
      if (e.type != BC_OMEGAWALL) continue;
      const double wc = omega_wall(P, e, P.k[i], ldro(P.delta + ldro(bc.a_face + q)));
      b += acc * wc;
      acc += acc;
    }
  A.val[ldro(A.dpos + i)] = acc;
  return b;
}

// grad!(gradU, Uf, U) Orthogonal (Calculate_0_gradient.jl:106-112) for cell i:
// g[d][j] = dU_d/dx_j by Green-Gauss of the face values in UfH.
template <int NS>
__device__ __forceinline__ void grad_u_row(const KParams &P, int i, double (&g)[3][3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int j = 0; j < 3; ++j) g[d][j] = 0.0;
  for (int k = 0; k < P.Wf; ++k) {
    const size_t e = (size_t)k * P.np + i;
    const int f = ldro(P.f_face + e);
    if (f < 0) break;
    const double ns = (double)ldro(P.f_sign + e);
    const double a = ldro(P.area + f);
    const double sx = (a * ldro(P.fnx + f)) * ns, sy = (a * ldro(P.fny + f)) * ns, sz = (a * ldro(P.fnz + f)) * ns;
#pragma unroll
    for (int d = 0; d < NS; ++d) {
      const double v = P.UfH[(size_t)f * NS + d];
      g[d][0] += v * sx;
      g[d][1] += v * sy;
      if (NS == 3) g[d][2] += v * sz;
    }
  }
  const double vol = ldro(P.vol + i);
#pragma unroll
  for (int d = 0; d < NS; ++d)
#pragma unroll
    for (int j = 0; j < NS; ++j) g[d][j] /= vol;
  for (int q = ldro(P.cb_ptr + i); q < ldro(P.cb_ptr + i + 1); ++q) {
    const int f = ldro(P.cb_face + q);
    const double a = ldro(P.area + f);
    const double sx = a * ldro(P.fnx + f), sy = a * ldro(P.fny + f), sz = a * ldro(P.fnz + f);
#pragma unroll
    for (int d = 0; d < NS; ++d) {
      const double v = P.UfH[(size_t)f * NS + d];
      double bx = v * sx, by = v * sy;
      bx /= vol;
      by /= vol;
      g[d][0] += bx;
      g[d][1] += by;
      if (NS == 3) {
        double bz = v * sz;
        bz /= vol;
        g[d][2] += bz;
      }
    }
  }
}

// bound!(field, eps()) for the rows of forward level l: the reference's
// sequential loop (later cells see updated values) in level order.
__device__ __forceinline__ void bound_row(const KParams &P, double *fld, int i) {
  const double EPS = 2.220446049250313e-16;
  double sum_flux = 0.0;
  int cnt = 0;
  for (int k = 0; k < P.Wf; ++k) {
    const size_t e = (size_t)k * P.np + i;
    if (ldro(P.f_face + e) < 0) break;
    sum_flux += jmax(fld[ldro(P.f_nbr + e)], EPS);
    cnt += 1;
  }
  const double average = sum_flux / (double)cnt;
  const double fi = fld[i];
  fld[i] = jmax(jmax(fi, average * (signbit(fi) ? 1.0 : 0.0)), EPS);
}

template <int NS, typename T, bool ONE>
__device__ __forceinline__ bool turbulence(Ctx &C) {
  const KParams &P = *C.P;
  const double nu = P.nu;
  // production, destruction, effective diffusivities (turbulence!, :256-272)
  C.phase(PH_TURB);
  tile_each(C, [&](int i) {
    double g[3][3];
    grad_u_row<NS>(P, i, g);
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int j = 0; j < 3; ++j) P.G[(size_t)i * 9 + 3 * d + j] = g[d][j];
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < NS; ++j)
#pragma unroll
      for (int k = 0; k < NS; ++k) {
        const double Sjk = 0.5 * (g[k][j] + g[j][k]);
        s += Sjk * Sjk;
      }
    const double pk = s * 2.0;
    P.Pw[i] = KW_ALPHA1 * pk;
    const double wi = P.w[i];
    P.Dw[i] = KW_BETA1 * wi;
    P.Dk[i] = KW_BPLUS * wi;
    double pki = P.nut[i] * pk;
    const FieldBC &bc = P.bcK;
    for (int q = ldro(bc.a_ptr + i); q < ldro(bc.a_ptr + i + 1); ++q) {   // correct_production!
      const BcEntry &e = bc.tab[ldro(bc.a_bc + q)];
      if (e.type != BC_KWALL) continue;
      const int f = ldro(bc.a_face + q);
      const double delta = ldro(P.delta + f);
      const double nx = ldro(P.fnx + f), ny = ldro(P.fny + f), nz = ldro(P.fnz + f);
      const double kc = P.k[i];
      const double uStar = e.c25 * sqrt(kc);
      const double dUdy = uStar / (e.kappa * delta);
      const double yplus = e.c25 * delta * sqrt(kc) / nu;
      const double nutw = nut_wall_fn(nu, yplus, e.kappa, e.E);
      const double ux = P.U[(size_t)i * NS] - 0.0, uy = P.U[(size_t)i * NS + 1] - 0.0;
      const double uz = (NS == 3 ? P.U[(size_t)i * NS + 2] : P.Uz2[i]) - 0.0;
      const double dn = (ux * nx + uy * ny) + uz * nz;
      const double gx = (ux - nx * dn) / delta, gy = (uy - ny * dn) / delta, gz = (uz - nz * dn) / delta;
      const double mag = sqrt((gx * gx + gy * gy) + gz * gz);
      if (yplus > e.ylam) pki = (nu + nutw) * mag * dUdy;
    }
    P.Pk[i] = pki;
  });
  grid_each(P.nf, [&](int f) {
    P.nueffw[f] = nu + KW_SIGW * P.nutf[f];
    P.nueffk[f] = nu + KW_SIGK * P.nutf[f];
  });
  if (!C.sync()) return false;
  const KWorkT<T> &wk = workP<T>(P);
  for (int eq = 0; eq < 2; ++eq) {   // omega first, then k
    const bool om = (eq == 0);
    MatT<T> A = matP<T>(P);
    A.precon = om ? P.precW : P.precK;
    double *phi = om ? P.w : P.k;
    const KCfg &cfg = om ? P.kW : P.kK;
    C.phase(PH_TURB);
    tile_each(C, [&](int i) {
      double b[1];
      b[0] = om ? scalar_row(P, P.AP, i, phi, P.nueffw, P.Dw, P.Pw, P.bcW, P.aW, P.divW, P.timeW, true)
                : scalar_row(P, P.AP, i, phi, P.nueffk, P.Dk, P.Pk, P.bcK, P.aK, P.divK, P.timeK, false);
      P.bP[i] = b[0];
      krylov_init_row<1, T>(P, P.AP, A, wk, b, phi, i, cfg.solver);
    });
    if (!C.sync()) return false;
    if (!krylov_start<1, ONE>(C, A, wk, P.bP, cfg.solver)) return false;
    int its[1];
    double rn[1];
    if (!solve_vector<1, ONE>(C, A, wk, P.bP, cfg, its, rn)) return false;
    // run! copy-back, then constrain_boundary! for omega (:401-448)
    C.phase(PH_TURB);
    tile_each(C, [&](int i) {
      double v = (double)wk.x[i] + phi[i];
      if (om) {
        const FieldBC &bc = P.bcW;
        for (int q = ldro(bc.a_ptr + i); q < ldro(bc.a_ptr + i + 1); ++q) {
          const BcEntry &e = bc.tab[ldro(bc.a_bc + q)];
          if (e.type != BC_OMEGAWALL) continue;
          v = omega_wall(P, e, P.k[i], ldro(P.delta + ldro(bc.a_face + q)));
        }
      }
      phi[i] = v;
    });
    if (!C.sync()) return false;
    for (int l = 0; l < P.nfl; ++l) {   // bound!(phi, eps()); after k also nut = k/omega
      tile_each(C, [&](int i) {
        if (ldro(P.flev + i) != l) return;
        bound_row(P, phi, i);
        if (!om) P.nut[i] = P.k[i] / P.w[i];
      });
      if (!C.sync()) return false;
    }
  }
  // interpolate!(nutf, nut) + correct_boundaries! + correct_eddy_viscosity! (:496-536)
  // and update_nueff! (Solvers_0_functions.jl:1-11)
  C.phase(PH_TURB);
  grid_each(P.nf, [&](int f) {
    double v = face_scalar(P, P.nut, f, P.bcN, false);
    if (f < P.nbf) {
      const int bi = ldro(P.bcN.fbc + f);
      if (bi >= 0 && P.bcN.tab[bi].type == BC_NUTWALL) {
        const BcEntry &e = P.bcN.tab[bi];
        const int c = ldro(P.o1 + f);
        const double yplus = e.c25 * ldro(P.delta + f) * sqrt(P.k[c]) / nu;
        const double nutw = nut_wall_fn(nu, yplus, e.kappa, e.E);
        if (yplus > e.ylam) v = nutw;
      }
    }
    P.nutf[f] = v;
    P.nueff[f] = nu + v;
  });
  return C.sync();
}

// ------------------------------------------------------------- programs
// A run is a chain of steps, one pressure solve each: step k = it*ncorr +
// corr.  before_solve does everything between two solves up to the start of
// solve k, after_solve everything that follows solve k-1 up to the end of its
// corrector and, with the last corrector, of its iteration.
template <int NS, typename T, bool ONE>
struct Simple {
  Ctx &C;
  const bool piso;
  const int ncorr;
  bool finite;   // Krylov residual norms of this iteration all finite

  // set-up before the loop (Solvers_1_SIMPLE.jl:114-119)
  __device__ __forceinline__ bool setup() {
    const KParams &P = *C.P;
    const bool mid = (P.grad == GRAD_MIDPOINT);
    const double nu = P.nu;
    C.phase(PH_SETUP);
    grid_each(P.nf, [&](int f) {
      face_mdot<NS>(P, f);
      P.pf[f] = face_scalar(P, P.p, f, P.bcP, mid);
      if (P.model == 1) P.nutf[f] = 0.0;   // initialise_RANS: a fresh face field
      P.nueff[f] = (P.model == 1) ? nu + 0.0 : nu;
    });
    if (!C.sync()) return false;
    if (!gradient_p<NS>(C, false)) return false;
    C.phase(PH_SETUP);
    return true;
  }

  __device__ __forceinline__ bool before_solve(int k) {
    const KParams &P = *C.P;
    const int it = k / ncorr, corr = k - it * ncorr;
    if (corr == 0) {
      finite = true;
      // ---- momentum: assemble, start Krylov, set up M, solve
      const MatT<T> &AUT = matU<T>(P);
      const KWorkT<T> &wU = workU<T>(P);
      C.phase(PH_MOM_ASM);
      tile_each(C, [&](int i) {
        double b[NS];
        momentum_row<NS>(P, i, !piso, b);
        krylov_init_row<NS, T>(P, P.AU, AUT, wU, b, P.U, i, P.kU.solver);
      });
      if (!C.sync()) return false;
      if (!krylov_start<NS, ONE>(C, AUT, wU, P.bU, P.kU.solver)) return false;
      int itsU[NS];
      double rnU[NS];
      if (!solve_vector<NS, ONE>(C, AUT, wU, P.bU, P.kU, itsU, rnU)) return false;
#pragma unroll
      for (int d = 0; d < NS; ++d) finite = finite && isfinite(rnU[d]);
      // run! copy-back: U = x + x0
      C.phase(PH_UPDATE);
      tile_each(C, [&](int i) {
#pragma unroll
        for (int d = 0; d < NS; ++d) {
          const size_t q = (size_t)i * NS + d;
          P.U[q] = (double)wU.x[q] + P.U[q];
        }
      });
      if (!C.sync()) return false;
      // ---- residual!(R_ux..), remove_pressure_source!, H!
      C.phase(PH_RESID);
      tile_phase<2 * NS>(C, true, [&](int i, double (&v)[2 * NS]) {
        double y[NS], bb[NS];
        spmv_row<NS>(P.AU, i, [&](int j, int d) { return P.U[(size_t)j * NS + d]; }, y);
        const double vol = ldro(P.vol + i);
        ld<NS>(P.bU, i, bb);
#pragma unroll
        for (int d = 0; d < NS; ++d) {
          const double df = y[d] - bb[d];
          v[2 * d] = df * df;
          v[2 * d + 1] = bb[d] * bb[d];
          bb[d] -= -1.0 * P.gp[(size_t)i * NS + d] * vol;
        }
        st<NS>(P.bU, i, bb);
        H_row<NS>(P, i, bb);
      });
      if (!C.sync()) return false;
      double red[2 * NS];
      final_sum<2 * NS>(C.part_r(), P.ntiles, s_sm, s_out, red);
      if (vbid() == 0 && threadIdx.x == 0) {
#pragma unroll
        for (int d = 0; d < NS; ++d) {
          P.R[(size_t)it * 4 + d] = sqrt(red[2 * d] / (double)P.n) / sqrt(red[2 * d + 1]);
          P.kry[(size_t)it * 5 + d] = itsU[d];
        }
        P.step->finite = finite ? 1 : 0;
      }
    } else {   // H! again with the corrected U (PISO corrector loop)
      C.phase(PH_RESID);
      tile_each(C, [&](int i) {
        double bb[NS];
        ld<NS>(P.bU, i, bb);
        H_row<NS>(P, i, bb);
      });
      if (!C.sync()) return false;
    }
    // interpolate!(rDf, rD); interpolate!(Uf, Hv) + correct_boundaries!
    C.phase(PH_FACE);
    grid_each(P.nf, [&](int f) {
      const double w = ldro(P.wgt + f);
      const double omw = 1.0 - w;
      P.rDf[f] = w * P.rD[ldro(P.o1 + f)] + omw * P.rD[ldro(P.o2 + f)];
      double u[NS];
      face_vector<NS>(P, P.H, f, u);
#pragma unroll
      for (int d = 0; d < NS; ++d) P.UfH[(size_t)f * NS + d] = u[d];
    });
    if (!C.sync()) return false;
    // div! + pressure assembly + Krylov start
    const MatT<T> &APT = matP<T>(P);
    const KWorkT<T> &wP = workP<T>(P);
    C.phase(PH_P_ASM);
    tile_each(C, [&](int i) {
      double b[1];
      b[0] = pressure_row<NS>(P, i);
      krylov_init_row<1, T>(P, P.AP, APT, wP, b, P.p, i, P.kP.solver);
    });
    if (!C.sync()) return false;
    return krylov_start<1, ONE>(C, APT, wP, P.bP, P.kP.solver);
  }

  // After solve k with `its` iterations and residual norm rn; stop: the run
  // ends with this iteration.
  __device__ __forceinline__ bool after_solve(int k, int its, double rn, bool &stop) {
    const KParams &P = *C.P;
    const bool mid = (P.grad == GRAD_MIDPOINT);
    const int it = k / ncorr, corr = k - it * ncorr;
    const KWorkT<T> &wP = workP<T>(P);
    finite = finite && isfinite(rn);
    // run! copy-back then explicit_relaxation!(p, prev, alpha_p)
    C.phase(PH_UPDATE);
    tile_each(C, [&](int i) {
      const double pn = (double)wP.x[i] + P.p[i];
      const double p0 = P.p[i];
      P.p[i] = p0 + P.aP * (pn - p0);
    });
    if (!C.sync()) return false;
    // residual!(R_p) and the face interpolation of grad!(grad p)
    C.phase(PH_RESID);
    tile_phase<2>(C, true, [&](int i, double (&v)[2]) {
      double y[1];
      spmv_row<1>(P.AP, i, [&](int j, int d) { return P.p[j]; }, y);
      const double bb = P.bP[i];
      const double df = y[0] - bb;
      v[0] = df * df;
      v[1] = bb * bb;
    });
    grid_each(P.nf, [&](int f) { P.pf[f] = face_scalar(P, P.p, f, P.bcP, mid); });
    if (!C.sync()) return false;
    double red[2];
    final_sum<2>(C.part_r(), P.ntiles, s_sm, s_out, red);
    const double Rp = sqrt(red[0] / (double)P.n) / sqrt(red[1]);
    if (vbid() == 0 && threadIdx.x == 0) {
      P.R[(size_t)it * 4 + 3] = Rp;
      P.kry[(size_t)it * 5 + 3] = its;
      P.step->finite = finite ? 1 : 0;
    }
    if (!gradient_p<NS>(C, true)) return false;
    // interpolate!(Uf, U) + correct_boundaries! + flux!(mdotf, Uf)
    C.phase(PH_FACE);
    grid_each(P.nf, [&](int f) { face_mdot<NS>(P, f); });
    if (!C.sync()) return false;
    if constexpr (NS == 2) {   // k-omega is a 2D model (xcal_case_setup refuses it in 3D)
      if (P.model == 1 && !turbulence<NS, T, ONE>(C)) return false;
    }
    if (corr + 1 < ncorr) return true;
    const bool lead = vbid() == 0 && threadIdx.x == 0;
    // XCAL_FLAG_ABORT_ON_NAN (no reference counterpart): stop a diverged run.
    // The residuals R_* themselves may be 0/0 = NaN on a healthy run (a zero
    // right-hand side, e.g. uy at the first iteration), so the test uses the
    // Krylov residual norms, which are finite whenever A, b and x0 are.
    if (P.abort_nan && !finite) {
      if (lead) P.bar->nonfinite = 1;
      stop = true;
    } else if (!piso) {
      // convergence test (Solvers_1_SIMPLE.jl:200-215); every CTA reads the
      // same residuals (CTA 0 stored the momentum ones several barriers ago),
      // so all take the same branch
      bool c = Rp <= P.conv;
#pragma unroll
      for (int d = 0; d < NS; ++d) c = c && (P.R[(size_t)it * 4 + d] <= P.conv);
      stop = c;
    }
    if (lead) *P.done = it + 1;
    return true;
  }
};

// The chain of a run.  step < 0: all of it.  Otherwise one link, for
// meshes whose pressure solve is a kernel of its own (xcal_cg_kernel,
// xcal_cg_cluster_kernel): launch
// `step` does what follows solve step-1 and what leads to solve `step`, and
// P.step carries the solve's results and the state of the run between them.
template <int NS, typename T, bool ONE>
__device__ __forceinline__ void simple_program(Ctx &C, int iters, bool piso, int step) {
  const KParams &P = *C.P;
  Simple<NS, T, ONE> S{C, piso, piso ? 2 : 1, true};
  const int total = iters * S.ncorr;
  int its[1] = {0};
  double rn[1] = {0.0};
  if (step > 0) {
    S.finite = P.step->finite != 0;
    its[0] = P.step->its;
    rn[0] = P.step->rnorm;
  } else if (!S.setup()) {
    return;
  }
  for (int k = max(step, 0);; ++k) {
    if (k > 0) {
      bool stop = false;
      if (!S.after_solve(k - 1, its[0], rn[0], stop)) return;
      if (stop) {
        if (vbid() == 0 && threadIdx.x == 0) P.step->stop = 1;
        return;
      }
    }
    if (k == total) return;
    if (!S.before_solve(k)) return;
    if (step >= 0) {
      if (vbid() == 0 && threadIdx.x == 0) P.step->pw = C.pw;
      return;
    }
    if (!solve_pressure<NS, ONE>(C, matP<T>(P), workP<T>(P), P.bP, P.kP, its, rn)) return;
  }
}

template <bool ONE>
__device__ __forceinline__ void solve_program(Ctx &C) {
  const KParams &P = *C.P;
  C.phase(PH_P_ASM);
  tile_each(C, [&](int i) {
    double b[1] = {P.sb[i]};
    krylov_init_row<1, double>(P, P.AU, P.AU, P.wU, b, P.U, i, P.solve_solver);
  });
  if (!C.sync()) return;
  if (!krylov_start<1, ONE>(C, P.AU, P.wU, P.sb, P.solve_solver)) return;
  KCfg cfg;
  cfg.solver = P.solve_solver;
  cfg.itmax = P.solve_itmax;
  cfg.atol = P.solve_atol;
  cfg.rtol = P.solve_rtol;
  int its[1];
  double rn[1];
  if (!solve_pressure<1, ONE>(C, P.AU, P.wU, P.sb, cfg, its, rn)) return;
  tile_each(C, [&](int i) { P.U[i] = P.wU.x[i] + P.U[i]; });
  if (vbid() == 0 && threadIdx.x == 0) {
    P.solve_out[0] = (double)its[0];
    P.solve_out[1] = rn[0];
    *P.done = 1;
  }
}

}  // namespace

// State of a launch whose CTAs are all of one group.
__device__ __forceinline__ void launch_begin(Ctx &C, const KParams &prm) {
  ctx_mesh(C, prm);
  C.S.bar = prm.bar;
  C.S.mode = prm.mode;
  C.S.nb = gridDim.x;
  if (threadIdx.x == 0) {
    s_vbid = blockIdx.x;
    s_vnb = gridDim.x;
  }
  __syncthreads();
  C.S.extra = (unsigned)prm.bar_extra;
  C.S.timeout_ns = prm.bar_timeout_ns ? prm.bar_timeout_ns : BARRIER_TIMEOUT_NS;
  C.S.epoch = 0;
  C.part = prm.part;
  C.pw = 0;
  C.rev = 0;
  C.timers = prm.phase != nullptr && blockIdx.x == 0 && threadIdx.x == 0;
  C.tag = PH_SETUP;
  if (C.timers) {
    for (int k = 0; k < 2 * NPH; ++k) s_pacc[k] = 0ull;
    C.t_last = clock64();
  }
}
// The timers are added up over the launches of a run.  `again`: another launch
// with the same barrier word follows, so the last CTA out clears its count.
__device__ __forceinline__ void launch_end(Ctx &C, const KParams &prm, bool again) {
  if (C.timers)
    for (int k = 0; k < 2 * NPH; ++k) prm.phase[k] += s_pacc[k];
  if (!again) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned out = atomicAdd(&prm.bar->exits, 1u);
    if (out + 1u == gridDim.x) {
      prm.bar->count = 0ull;
      prm.bar->exits = 0u;
    }
  }
}

#if defined(XCAL_CG)
// The pressure solve of a large mesh (rows of which the CTAs cannot keep in
// shared memory) as a kernel of its own.  Its phases stream the matrix with a
// few dependent gathers per row, and what hides their latency is warps: this
// kernel needs few registers, so MB = 8 CTAs fit an SM where the program's
// register budget allows 4.  128^3 FP64, 278 MB in A and 134 in B or C: 63 and
// 28 us (4.4 and 4.8 TB/s), against 69 and 56 of the general CG in the program.
// In the program's 64 registers the same phases took 88 and 40 us, with the
// rows streamed through shared memory by bulk copies 80 and 33.
template <typename T, int WT, int MB>
__global__ void __launch_bounds__(TPB, MB) xcal_cg_kernel(const __grid_constant__ KParams prm) {
  if (ld_volatile_i32(&prm.bar->err) || ld_volatile_i32(&prm.step->stop)) return;
  Ctx C;
  launch_begin(C, prm);
  C.pw = prm.step->pw;
  int its;
  double rn;
  if (cg_two_level<T, WT, false>(C, matP<T>(prm), workP<T>(prm), prm.kP, its, rn) && vbid() == 0 && threadIdx.x == 0) {
    prm.step->its = its;
    prm.step->rnorm = rn;
  }
  launch_end(C, prm, true);
}

// The pressure solve of a small mesh as one cluster of CTAs holding all of it
// in shared memory: matrix rows, preconditioner and Krylov vectors.  A row's
// neighbours are read through distributed shared memory (their addresses are
// worked out once, in place of the column indices), tile sums are stored
// straight into every CTA's copy of the partials, and the barrier is the
// cluster's own, so no phase goes through L2.  Row arithmetic and sums are
// those of cg_two_level.
//
// A CTA holds a chunk of the tiles with level-0 rows and the same chunk of
// the others: its rows are close together in the mesh, so most neighbours
// are its own, and a CTA that has tiles has work in each phase.  (Both splits
// round alike, so shares differ by up to two tiles: of 16 tiles on 16 CTAs,
// eight CTAs hold two and eight none.)  Up to four tiles at a time, one per 256
// threads (threads for tiles that are not there slow the barriers down: cavity
// 40^2 A 2.57 -> 2.28 us, B and C 1.64 -> 1.54).
enum { CV_Z = 0, CV_P = 1, CV_R = 3, CV_Q = 5, CV_D = 6, CV_X = 7 };   // vectors (p and r twice)
static_assert(CV_X + 1 == CGC_VECTORS, "vectors of a row");

__device__ __forceinline__ unsigned cluster_addr(unsigned a, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ double ld_cluster(unsigned a, double) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float ld_cluster(unsigned a, float) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void st_cluster(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <typename T, int WT>
__global__ void __launch_bounds__(CGC_TPB, 1) xcal_cg_cluster_kernel(const __grid_constant__ KParams prm, int slots) {
  __shared__ double part[2][CGC_TILES];
  __shared__ double ws[CGC_SLOTS * 8];
  __shared__ double sm[8];
  if (ld_volatile_i32(&prm.bar->err) || ld_volatile_i32(&prm.step->stop)) return;
  constexpr double EPS = 2.220446049250313e-16;
  const MatT<T> &A = matP<T>(prm);
  const KWorkT<T> &w = workP<T>(prm);
  const int n = prm.n, n0 = prm.n0, np = prm.np, nt = prm.ntiles;
  const int W = WT < WUNROLL ? WT : A.W;
  const int tid = threadIdx.x, lane = tid & 31, tl = tid >> 8, r = tid & 255, wt = (tid >> 5) & 7;
  const int G = gridDim.x, b = blockIdx.x, groups = blockDim.x / TILE;
  // tiles [0, N0) hold level-0 rows, the rest only level-1 rows; tile N0-1 may hold both
  const int N0 = (n0 - 1) / TILE + 1, N1 = nt - N0;
  const int a0 = chunk(b, N0, G), k0 = chunk(b + 1, N0, G) - a0;                // own level-0 tiles: slots [0, k0)
  const int a1 = N0 + chunk(b, N1, G), cnt = k0 + chunk(b + 1, N1, G) - chunk(b, N1, G);   // the others: [k0, cnt)
  const int L = slots * TILE;
  T *vec = (T *)s_dyn, *val = vec + (size_t)CGC_VECTORS * L;
  unsigned *adr = (unsigned *)(val + (size_t)W * L);
  const unsigned vec0 = smem_u32(vec);
  auto tile_of = [&](int s) { return s < k0 ? a0 + s : a1 + (s - k0); };
  const bool timer = prm.phase != nullptr && b == 0 && tid == 0;
  long long t_last = timer ? clock64() : 0, acc[2] = {0, 0}, num[2] = {0, 0};
  auto tick = [&](int what) {
    if (timer) {
      const long long t = clock64();
      acc[what] += t - t_last;
      num[what] += 1;
      t_last = t;
    }
  };
  // rows into shared memory; entry k's neighbour as the address of its z in
  // the cluster, with bit 0 for the diagonal and bit 1 for padding
  for (int s = tl; s < cnt; s += groups) {
    const int l = s * TILE + r, i = tile_of(s) * TILE + r;
    const bool on = i < n;
    vec[CV_Z * L + l] = on ? w.v[0][i] : T(0);
    vec[CV_R * L + l] = on ? w.r[0][i] : T(0);
    vec[CV_D * L + l] = on ? A.Dinv[i] : T(0);
    vec[CV_X * L + l] = T(0);
    const unsigned own = vec0 + (unsigned)(l * sizeof(T));
    for (int k = 0; k < W; ++k) {
      const int c = A.col[(size_t)k * np + i];
      val[(size_t)k * L + l] = A.val[(size_t)k * np + i];
      unsigned a = cluster_addr(own, b) | 2u;
      if (c >= 0) {
        const int t = c / TILE, g = t < N0 ? t : t - N0, N = t < N0 ? N0 : N1;
        const int o = (int)(((long long)(g + 1) * G - 1) / N);   // its CTA
        const int slot = g - chunk(o, N, G) + (t < N0 ? 0 : chunk(o + 1, N0, G) - chunk(o, N0, G));
        a = cluster_addr(vec0 + (unsigned)((slot * TILE + c % TILE) * sizeof(T)), o) | (c == i ? 1u : 0u);
      }
      adr[(size_t)k * L + l] = a;
    }
  }
  int par = 0;
  {
    const double *p0 = prm.part + (size_t)(prm.step->pw ^ 1) * MAXK * nt;
    for (int q = tid; q < nt; q += (int)blockDim.x) part[par][q] = p0[q];
  }
  cluster_sync();
  // canonical sum of the tiles' partials (final_sum's tree; one tile per lane)
  auto total = [&]() -> double {
    if (tid < TPB) {
      double a = tid < nt ? part[par][tid] : 0.0;
#pragma unroll
      for (int off = 16; off >= 1; off >>= 1) a = a + __shfl_down_sync(0xffffffffu, a, off);
      if (lane == 0) sm[tid >> 5] = a;
    }
    __syncthreads();
    par ^= 1;
    double x0 = sm[0] + sm[4], x1 = sm[1] + sm[5];
    const double x2 = sm[2] + sm[6], x3 = sm[3] + sm[7];
    x0 = x0 + x2;
    x1 = x1 + x3;
    return x0 + x1;
  };
  auto stage = [&](int s, double v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) ws[s * 8 + wt] = v;
  };
  // every own tile's sum to every CTA, then the barrier
  auto exchange = [&]() {
    __syncthreads();
    for (int q = tid; q < cnt * G; q += (int)blockDim.x) {
      const int s = q / G;
      const double *ww = ws + s * 8;
      double x0 = ww[0] + ww[4], x1 = ww[1] + ww[5];
      const double x2 = ww[2] + ww[6], x3 = ww[3] + ww[7];
      x0 = x0 + x2;
      x1 = x1 + x3;
      st_cluster(cluster_addr(smem_u32(&part[par][tile_of(s)]), q - s * G), x0 + x1);
    }
    cluster_sync();
  };

  double s0 = total();
  const double sgn = (s0 < 0.0) ? -1.0 : 1.0;
  double gamma = sgn * s0, rnorm = sqrt(gamma), alpha = 0.0, beta = 0.0, pn2 = gamma, eps = 0.0;
  int its = 0;
  bool active = false;
  const KCfg &cfg = prm.kP;
  if (gamma != 0.0) {
    eps = cfg.atol + cfg.rtol * rnorm;
    active = !(rnorm <= eps || 0 >= cfg.itmax);
  }
  int ro = CV_R, rn = CV_R + 1, po = CV_Z, pn = CV_P, pspare = CV_P + 1;   // first direction: as in cg_two_level
  bool pending = false;
  const int sB = (k0 > 0 && tile_of(k0 - 1) == N0 - 1 && n0 < N0 * TILE) ? k0 - 1 : k0;   // first slot with level-1 rows
  while (active) {
    // A
    {
      const unsigned opo = (unsigned)(po * L * sizeof(T));
      for (int s = tl; s < cnt; s += groups) {
        const int l = s * TILE + r;
        T y = T(0), pi = T(0), poi = T(0);
#pragma unroll
        for (int k = 0; k < WT; ++k) {
          const int kk = (WT < WUNROLL || k < W) ? k : W - 1;
          const unsigned a = (WT < WUNROLL || k < W) ? adr[kk * L + l] : 2u | (unsigned)vec0;
          const unsigned ad = (a & 2u) ? adr[l] & ~3u : a & ~3u;
          const T oj = ld_cluster(ad + opo, T()), pj = vaxpy<T>(ld_cluster(ad, T()), beta, oj);
          const T t = y + val[kk * L + l] * pj;
          y = (a & 2u) ? y : t;
          if (a & 1u) {
            pi = pj;
            poi = oj;
          }
        }
        vec[CV_X * L + l] = vaxpy<T>(vec[CV_X * L + l], alpha, poi);
        vec[pn * L + l] = pi;
        vec[CV_Q * L + l] = y;
        stage(s, (double)pi * (double)y);
      }
      pending = false;
      exchange();
      s0 = total();
      tick(0);
    }
    const double pAp = sgn * s0;
    if (pAp <= EPS * pn2 && fabs(pAp) <= EPS * pn2) break;   // zero curvature: stop
    alpha = gamma / pAp;
    const unsigned oro = (unsigned)(ro * L * sizeof(T)), oq = (unsigned)(CV_Q * L * sizeof(T)),
                   od = (unsigned)(CV_D * L * sizeof(T));
    // B
    for (int s = sB + tl; s < cnt; s += groups) {
      const int l = s * TILE + r, i = tile_of(s) * TILE + r;
      double rz = 0.0;
      if (i < n && i >= n0) {
        const T ri = vaxpy<T>(vec[ro * L + l], -alpha, vec[CV_Q * L + l]);
        T o = ri;
#pragma unroll
        for (int k = 0; k < WT - 1; ++k) {
          const int kk = (WT < WUNROLL || k < W - 1) ? k : 0;
          const unsigned a = (WT < WUNROLL || k < W - 1) ? adr[kk * L + l] : 2u;
          const bool use = (a & 3u) == 0u;
          const unsigned ad = use ? a : adr[l] & ~3u;
          const T t = o - val[kk * L + l] * vaxpy<T>(ld_cluster(ad + oro, T()), -alpha, ld_cluster(ad + oq, T())) *
                              ld_cluster(ad + od, T());
          o = use ? t : o;
        }
        o = o * vec[CV_D * L + l];
        vec[rn * L + l] = ri;
        vec[CV_Z * L + l] = o;
        rz = (double)ri * (double)o;
      }
      if (s >= k0) stage(s, rz);
    }
    cluster_sync();
    tick(1);
    // C
    for (int s = tl; s < k0; s += groups) {
      const int l = s * TILE + r, i = tile_of(s) * TILE + r;
      double rz = 0.0;
      if (i < n0) {
        const T ri = vaxpy<T>(vec[ro * L + l], -alpha, vec[CV_Q * L + l]);
        const T di = vec[CV_D * L + l];
        T o = ri * di;
#pragma unroll
        for (int k = 1; k < WT; ++k) {
          const int kk = (WT < WUNROLL || k < W) ? k : W - 1;
          const unsigned a = (WT < WUNROLL || k < W) ? adr[kk * L + l] : 2u;
          const bool use = (a & 3u) == 0u;
          const unsigned ad = use ? a : adr[l] & ~3u;
          const T t = o - val[kk * L + l] * ld_cluster(ad, T()) * di;
          o = use ? t : o;
        }
        vec[rn * L + l] = ri;
        vec[CV_Z * L + l] = o;
        rz = (double)ri * (double)o;
      } else if (i < n) {   // level-1 rows of the tile that holds both levels
        rz = (double)vec[rn * L + l] * (double)vec[CV_Z * L + l];
      }
      stage(s, rz);
    }
    exchange();
    s0 = total();
    tick(1);
    const double gn = sgn * s0;
    rnorm = sqrt(gn);
    const bool solved = (rnorm <= eps) || (rnorm + 1.0 <= 1.0);
    if (!solved) {
      beta = gn / gamma;
      pn2 = gn + (beta * beta) * pn2;
      gamma = gn;
    }
    its += 1;
    active = !(solved || its >= cfg.itmax);
    pending = true;
    int tp = ro;
    ro = rn;
    rn = tp;
    tp = pn;
    pn = pspare;
    pspare = tp;
    po = tp;
  }
  for (int s = tl; s < cnt; s += groups) {
    const int l = s * TILE + r, i = tile_of(s) * TILE + r;
    const T x = vec[CV_X * L + l];
    if (i < n) w.x[i] = pending ? vaxpy<T>(x, alpha, vec[po * L + l]) : x;
  }
  if (b == 0 && tid == 0) {
    prm.step->its = its;
    prm.step->rnorm = rnorm;
  }
  if (timer) {
    prm.phase[PH_KRY_SPMV] += acc[0];
    prm.phase[PH_KRY_PREC] += acc[1];
    prm.phase[NPH + PH_KRY_SPMV] += num[0];
    prm.phase[NPH + PH_KRY_PREC] += num[1];
  }
  cluster_sync();   // no CTA leaves while another may still reach its memory
}
#endif

// KParams is passed by value: the fields live in the kernel's constant
// parameter bank instead of occupying registers.  T is the scalar type of
// the Krylov iterations (double: FP64 path; float: mixed path).  MB is the
// number of resident CTAs per SM the register budget is sized for: 2 (128
// registers, few spills) suits meshes with about one tile per CTA, where a
// phase is barrier-latency bound; 4 (64 registers, more spills, twice the
// warps in flight) suits large meshes, where a phase is memory-latency bound.
// ONE: the build for numberings with sweeps by one CTA (KParams::sweep >= 0).
template <int NS, typename T, int MB, bool ONE>
__global__ void __launch_bounds__(TPB, MB) xcal_program_kernel(const __grid_constant__ KParams prm, int prog, int iters,
                                                               int step) {
  if (step > 0 && (ld_volatile_i32(&prm.bar->err) || ld_volatile_i32(&prm.step->stop))) return;
  Ctx C;
  launch_begin(C, prm);
  if (prog == PROG_SOLVE) {
    if constexpr (NS == 1 && sizeof(T) == 8) solve_program<ONE>(C);
  } else {
    if constexpr (NS >= 2) simple_program<NS, T, ONE>(C, iters, prog == PROG_PISO, step);
  }
  launch_end(C, prm, step >= 0);
}

// ------------------------------------------------------------- serving
// The packed serving form: one persistent launch (all of it co-resident)
// whose CTAs take cases from the host.  Each CTA polls its mail word in
// mapped host memory; the host gives a case to a group of CTAs (any CTAs,
// numbered 0..nblk-1 inside the group), which copy the case's image from
// pinned host memory into its device region, run SIMPLE to the case's
// tolerance or iteration cap with a barrier of their own, write the results
// to pinned host memory and go back to polling.  Every wait is bounded: the
// group barrier by its 2 s limit, an idle CTA by the host's heartbeat (it
// leaves when the heartbeat stops for idle_limit_ns, or on shutdown).
__device__ __forceinline__ unsigned long long ld_acquire_sys_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys_i32(int *p, int v) {
  asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned atom_add_acqrel_u32(unsigned *p, unsigned v) {
  unsigned old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

template <int NS, typename T, int MB, bool ONE>
__global__ void __launch_bounds__(TPB, MB) xcal_serve_kernel(ServeMail *mail, const ServeCtl *ctl) {
  __shared__ ServeJob sJ;   // the job record, read once per job
  __shared__ const ServeJob *s_job;
  __shared__ int s_cmd;
  static_assert(sizeof(ServeJob) % 8 == 0, "job record copied in 8-byte words");
  ServeMail *m = mail + blockIdx.x;
  unsigned long long seen = 0;
  if (threadIdx.x == 0) seen = *(volatile unsigned long long *)&m->ack;
  for (;;) {
    if (threadIdx.x == 0) {
      int cmd = 0;
      unsigned long long hb = *(volatile const unsigned long long *)&ctl->heartbeat;
      unsigned long long t_hb = globaltimer();
      const unsigned long long limit = ctl->idle_limit_ns;
      unsigned nap = 256, polls = 0;
      for (;;) {
        const unsigned long long q = ld_acquire_sys_u64(&m->seq);
        if (q != seen) {
          seen = q;
          cmd = 1;
          break;
        }
        if ((++polls & 15u) == 0u) {
          if (*(volatile const unsigned *)&ctl->shutdown) break;
          const unsigned long long h2 = *(volatile const unsigned long long *)&ctl->heartbeat, now = globaltimer();
          if (h2 != hb) {
            hb = h2;
            t_hb = now;
          } else if (now - t_hb > limit) {
            break;
          }
        }
        __nanosleep(nap);
        if (nap < 32768u) nap <<= 1;
      }
      if (cmd) {
        // mail fields through volatile loads: the same words held earlier
        // jobs' values, which this SM may still have cached
        s_job = *(ServeJob *const volatile *)&m->job;
        s_vbid = *(volatile const int *)&m->vbid;
        s_vnb = *(volatile const int *)&m->nblk;
        *(volatile unsigned long long *)&m->ack = seen;
      }
      s_cmd = cmd;
    }
    __syncthreads();
    if (!s_cmd) return;
    // The job record and the case image live in pinned host memory whose
    // regions are reused by later jobs: read them with ld.global.cv (fetch
    // again, never from a cached line).
    {
      const unsigned long long *src = (const unsigned long long *)s_job;
      unsigned long long *dst = (unsigned long long *)&sJ;
      for (int k = threadIdx.x; k < (int)(sizeof(ServeJob) / 8); k += TPB) dst[k] = __ldcv(src + k);
    }
    __syncthreads();
    const ServeJob &J = sJ;
    const KParams &sP = sJ.prm;
    const int B = vbid(), G = vnb();
    // this CTA's share of the region: image copy, then zero part
    {
      const uint4 *src = J.src;
      uint4 *dst = J.dst;
      const unsigned long long c16 = J.copy16, z16 = J.zero16;
      for (unsigned long long q = (unsigned long long)B * TPB + threadIdx.x; q < c16; q += (unsigned long long)G * TPB)
        dst[q] = __ldcv(src + q);
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
      for (unsigned long long q = (unsigned long long)B * TPB + threadIdx.x; q < z16; q += (unsigned long long)G * TPB)
        dst[c16 + q] = zero;
    }
    Ctx C;
    ctx_mesh(C, sP);
    C.S.bar = sP.bar;
    C.S.mode = SYNC_GRID;
    C.S.nb = G;
    C.S.extra = 0;
    C.S.timeout_ns = BARRIER_TIMEOUT_NS;
    C.S.epoch = 0;
    C.part = sP.part;
    C.pw = 0;
    C.rev = 0;
    C.timers = false;
    C.tag = PH_SETUP;
    C.t_last = 0;
    if (C.sync()) simple_program<NS, T, ONE>(C, J.iters, J.prog == PROG_PISO, -1);
    C.sync();   // the run's results (fields, histories, done) complete
    // results to pinned host memory, this CTA's share
    {
      const int n = sP.n;
      const int dn = *(volatile const int *)sP.done;
      for (int q = B * TPB + threadIdx.x; q < n * NS; q += G * TPB) J.out_U[q] = sP.U[q];
      for (int q = B * TPB + threadIdx.x; q < n; q += G * TPB) J.out_p[q] = sP.p[q];
      for (int q = B * TPB + threadIdx.x; q < dn * 4; q += G * TPB) J.out_R[q] = sP.R[q];
      for (int q = B * TPB + threadIdx.x; q < dn * 5; q += G * TPB) J.out_kry[q] = sP.kry[q];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence_system();
      const unsigned prev = atom_add_acqrel_u32(J.exits, 1u);
      if (prev + 1u == (unsigned)G) {
        // last CTA of the group out: state for the host, then the group's
        // barrier word and exit count reset for the next case that uses them
        volatile Bar *b = sP.bar;
        J.out_state[0] = *(volatile const int *)sP.done;
        J.out_state[1] = b->err;
        J.out_state[2] = b->nonfinite;
        b->count = 0ull;
        b->err = 0;
        b->nonfinite = 0;
        *(volatile unsigned *)J.exits = 0u;
        __threadfence_system();
        st_release_sys_i32(J.out_state + 3, 1);
      }
    }
    __syncthreads();
  }
}

// One translation unit per instantiation (build.py compiles this file once per
// XCAL_INST value, in parallel); the launcher table lives in xcal_launch.cu.
#if defined(XCAL_INST)
#define XCAL_CAT2(a, b) a##b
#define XCAL_CAT(a, b) XCAL_CAT2(a, b)
#ifndef XCAL_MB
#define XCAL_MB 2
#endif
#if defined(XCAL_CG)
const void *XCAL_CAT(cg_kernel_, XCAL_INST)(int W) {
  if (W == 5) return (const void *)xcal_cg_kernel<XCAL_T, 5, XCAL_MB>;
  if (W == 7) return (const void *)xcal_cg_kernel<XCAL_T, 7, XCAL_MB>;
  return (const void *)xcal_cg_kernel<XCAL_T, WUNROLL, XCAL_MB>;
}
const void *XCAL_CAT(cgc_kernel_, XCAL_INST)(int W) {
  if (W == 5) return (const void *)xcal_cg_cluster_kernel<XCAL_T, 5>;
  if (W == 7) return (const void *)xcal_cg_cluster_kernel<XCAL_T, 7>;
  return (const void *)xcal_cg_cluster_kernel<XCAL_T, WUNROLL>;
}
#elif defined(XCAL_SERVE_ONLY)
template __global__ void xcal_serve_kernel<XCAL_NS, XCAL_T, XCAL_MB, XCAL_ONE>(ServeMail *, const ServeCtl *);
const void *XCAL_CAT(serve_kernel_, XCAL_INST)() {
  return (const void *)xcal_serve_kernel<XCAL_NS, XCAL_T, XCAL_MB, XCAL_ONE>;
}
#else
template __global__ void xcal_program_kernel<XCAL_NS, XCAL_T, XCAL_MB, XCAL_ONE>(const __grid_constant__ KParams, int,
                                                                                 int, int);
const void *XCAL_CAT(program_kernel_, XCAL_INST)() {
  return (const void *)xcal_program_kernel<XCAL_NS, XCAL_T, XCAL_MB, XCAL_ONE>;
}
#endif
#endif

}  // namespace xcal
