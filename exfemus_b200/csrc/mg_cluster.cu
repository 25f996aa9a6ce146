// mg_cluster.cu -- the lower part of a scalar system's V-cycle (MGStep, src/MGSolverBase.C:
// 212-289, with Gauss-Seidel sweeps) in ONE launch of one thread-block cluster.
//
// What bounds these levels is not data but dependent phases: a sweep is one phase per
// colour (9 in 2D, 27 in 3D), a cycle smooths every lower level 4 to 12 times, and a phase
// that is a kernel of its own costs 2.5-2.8 us (launch boundary 1.3 us, then descriptor,
// row and iterate loads one after the other).  Here the phases of a level and all levels
// below it run in one kernel: every CTA holds the whole iterate in its shared memory, in
// colour order, an updated value is sent to all CTAs by asynchronous stores that complete
// on the receivers' mbarriers, and the next rows are loaded while the values travel.
//
// A phase is then latency: about 270 cycles of row product (FP64 adds and shuffles), 170 to
// send, 600 until the slowest CTA's values arrive.  Measured on the way (FP64, 65 x 65
// lattice): plain remote stores and a cluster barrier with release / acquire 2,500 cycles a
// phase (1,200 of them the release), 8-byte stores to 16 CTAs 2,000 (the packets bound it:
// hence colour order and vectors), descriptors read from global memory in the phase +500.
// V-cycle of the 32 x 32 conduction workload (4 levels, 180 phases): 0.45 -> 0.17 ms; of a
// 128 x 64 scalar system (6 levels, the four below the top here) 0.63 -> 0.37 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <vector>

#include "cluster.cuh"
#include "exf_internal.h"
#include "mg_cluster_plan.h"

namespace exf {

// 512 threads: 256 cost 7% more on the 129 x 129 lattice (rounds of rows), 1024 spill
static constexpr int kCluNT = 512;
// Rows of the coarsest level up to which its product runs in the cluster.  It reads n^2
// doubles through at most 16 SMs; above, the descent and the ascent are two launches around
// the product on all SMs.  Two-level V-cycle with one pre- and post-sweep, in one launch and
// in three (FP64, us): n = 289 37 and 39, 625 42 and 41, 729 (3D) 92 and 92, 1225 56 and 52,
// 2401 113 and 80, 4761 629 and 168.
static constexpr int kCluCoarse = 700;
// lanes per row; a warp's rows are consecutive in colour order, so their new values leave
// as vectors
static constexpr int clu_lpr(int dim) { return dim == 2 ? 8 : 16; }

template <class T>
struct CluLevel {
  int N, Np, steps, act, mat;  // nodes, padded positions, steps of a sweep, active CTAs, entries
                               // of a CTA's rows in shared memory (0: not there)
  const int4 *tab;             // CluTable
  const int *first;
  const int2 *ent;
  const int2 *step;
  const int *node;             // -1: padding
  const int *col;              // positions of the columns
  const T *vv;
  T *x, *b, *r;
  const int *r_ptr, *r_col;    // restriction of this level's residual: rows of the level below
  const T *r_val;
  const double *r_mask;
  const int *p_ptr, *p_col;    // prolongation from the level below: rows of this level
  const T *p_val;
};
template <class T>
struct CluArgs {
  CluLevel<T> lev[kCluMaxLev];  // lev[0] the coarsest level
  int hi;                       // levels hi .. 1 are smoothed
  int nu_pre, nu_post;          // sweeps of a level below the top
  int nu_pre_hi, nu_post_hi;    // sweeps of level hi
  int reverse;
  int part;                     // 1: descent, 2: coarsest product, 4: ascent
  int steps, xlen, mlen;        // most steps of a level, longest iterate, most entries of a CTA
  int *wait_flag;
  T damp;
  int overwrite;                // correction factor 0: x = P x_c, as prolong_add
  const double *inv;            // coarsest inverse, gauge mask
  const double *gmask;
};

// the phases' barrier: the CTA alone, or the cluster
__device__ __forceinline__ void phase_sync(int act) {
  if (act == 1) {
    __syncthreads();
  } else {
    cluster_arrive();
    cluster_wait();
  }
}

// A level as a CTA holds it in shared memory: the iterate by position (colour order), and
// step after step the row of each of the CTA's groups: {position or -1, first entry,
// entries (0: padding), diagonal entry - first entry}, the reciprocal of the diagonal entry
// and the rhs; where they fit (mat), the rows' entries too.
template <class T>
struct CluSmem {
  T *x;
  int4 *d;         // [steps][groups of the CTA]
  T *inv, *b;
  int2 *step;      // CluStep
  T *v;            // entries (mat)
  int *c;
  uint64_t *bar;   // two mbarriers: the values of a colour, alternating
  unsigned phase;  // colours exchanged so far
  int *wait_flag;
  bool ok;         // no bounded wait has run out
};

template <class T, int E>
struct RowSlot {  // a lane's entries of one row (column -1: none)
  int c[E];
  T v[E];
};

// entries E * u + lane of row q; the diagonal entry is left out (DIAG: kept)
template <class T, int LPR, int E, bool DIAG>
__device__ __forceinline__ void load_row(const int *col, const T *vv, const int4 q, int lane, RowSlot<T, E> &s) {
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int i = e * LPR + lane;
    s.c[e] = -1;
    if (i < q.z && (DIAG || i != q.w)) {
      s.c[e] = col[q.y + i];
      s.v[e] = vv[q.y + i];
    }
  }
}

// sum of the products of row q with the iterate over the group's lanes (in every lane)
template <class T, int LPR, int E, bool DIAG>
__device__ __forceinline__ T row_dot(const int *col, const T *vv, const RowSlot<T, E> &s, const int4 q, int lane,
                                     const T *x) {
  T acc = T(0);
#pragma unroll
  for (int e = 0; e < E; e++)
    if (s.c[e] >= 0) acc += s.v[e] * x[s.c[e]];
  for (int i = E * LPR + lane; i < q.z; i += LPR)  // rows of more than E * LPR entries
    if (DIAG || i != q.w) acc += vv[q.y + i] * x[col[q.y + i]];
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// the level's rows of this CTA into shared memory
template <class T, int LPR>
__device__ __forceinline__ void load_level(const CluLevel<T> &L, int rank, CluSmem<T> &S) {
  const int n = L.steps * (kCluNT / LPR);
  const int4 *tab = L.tab + (long)rank * n;
  for (int i = threadIdx.x; i < L.steps; i += kCluNT) S.step[i] = L.step[i];
  for (int q = threadIdx.x; q < n; q += kCluNT) {
    const int4 d = tab[q];
    T inv = T(0), b = T(0);
    if (d.z > 0) {
      inv = T(1) / L.vv[d.y + d.w];
      b = L.b[L.node[d.x]];
    }
    S.inv[q] = inv;
    S.b[q] = b;
    S.d[q] = L.mat ? make_int4(d.x, L.first[(long)rank * n + q], d.z, d.w) : d;
  }
  const int2 *ent = L.ent + (long)rank * L.mat;
#pragma unroll 4
  for (int i = threadIdx.x; i < L.mat; i += kCluNT) {
    const int2 e = ent[i];
    S.c[i] = e.y;
    S.v[i] = L.vv[e.x];
  }
}

template <class T>
__device__ __forceinline__ void fill_x(const CluLevel<T> &L, bool zero, CluSmem<T> &S) {
  for (int i = threadIdx.x; i < L.Np; i += kCluNT) {
    const int n = L.node[i];
    S.x[i] = zero || n < 0 ? T(0) : L.x[n];
  }
}
template <class T>
__device__ __forceinline__ void store_x(const CluLevel<T> &L, int gt, int nth, const CluSmem<T> &S) {
  for (int i = gt; i < L.Np; i += nth) {
    const int n = L.node[i];
    if (n >= 0) L.x[n] = S.x[i];
  }
}

// nsw sweeps of one level: the steps of all sweeps form one sequence.  With several CTAs a
// warp's new values are sent to every CTA, and a warp starts a colour when the CTA's mbarrier
// of the colour before has completed.  Colours alternate between two mbarriers; a phase p
// completes when all of colour p's bytes have arrived AND each of the CTA's warps has
// arrived, which a warp does after it has seen phase p - 2.  Two rules keep the order:
//  * no warp is left behind: phase p + 2 waits for the arrival of every warp of the CTA, so
//    its parity cannot turn back under a warp that still tests phase p (a warp without rows
//    in two colours running would otherwise wait for a phase that is over);
//  * no value arrives early: a CTA sends colour p + 2 after its phase p + 1, hence after the
//    sends of colour p + 1 of EVERY CTA (plan_cluster deals each CTA a unit in each colour,
//    padding if need be), hence after phase p of every CTA: its bytes cannot count as colour
//    p's, nor can it overwrite a value that a warp still reads for colour p + 1 (that warp
//    has not sent yet).
// A warp whose wait runs out leaves the sweep; so do, each after its own limit, the warps that
// wait for it (a flag looked at before every send and arrival instead: 4% of a V-cycle).
// Entries that are not in shared memory (!MAT) are loaded two or three steps ahead.
template <class T, int LPR, int E, bool MAT>
__device__ __forceinline__ void sweep_level(const CluLevel<T> &L, int nsw, int reverse, CluSmem<T> &S) {
  constexpr int GC = kCluNT / LPR, RW = 32 / LPR;
  constexpr int PK = RW * sizeof(T) > 16 ? RW * sizeof(T) / 16 : 1;  // vectors per warp and CTA
  constexpr int VL = RW / PK;                                        // values per vector
  constexpr int PF = MAT ? 1 : (E > 4 ? 2 : 3);
  const int g = threadIdx.x / LPR, lane = threadIdx.x % LPR, wl = threadIdx.x & 31;
  const int *col = MAT ? S.c : L.col;
  const T *vv = MAT ? S.v : L.vv;
  const int steps = L.steps, total = nsw * steps, bit = reverse ? 2 : 1;
  const int4 *sd = S.d + g;
  const T *sinv = S.inv + g, *sb = S.b + g;
  // step i of a sweep is step s0 + i * dir of the tables
  const int s0 = reverse ? steps - 1 : 0, dir = reverse ? -1 : 1;
  // the warps arrive for a colour once they have sent the colour before (while its values
  // travel), thread 0 with the colour's bytes, which the step before it in the order holds
  auto arrive = [&](unsigned phase, int next) {
    if (wl > 0) return;
    const unsigned count = reverse ? (unsigned)next >> 16 : (unsigned)next & 0xffffu;
    if (threadIdx.x > 0) mbar_arrive(&S.bar[phase & 1]);
    else mbar_arrive_tx(&S.bar[phase & 1], count * (unsigned)sizeof(T));
  };
  const unsigned dst = (unsigned)wl / PK;  // the CTA this lane sends to, its vector
  const int hv = wl % PK;
  unsigned ax = 0, ab = 0;
  const bool sender = L.act > 1 && dst < (unsigned)L.act;
  if (sender) {
    ax = cluster_addr(S.x + hv * VL, dst);
    ab = cluster_addr(S.bar, dst);
  }
  if (L.act > 1 && total > 0) arrive(S.phase, S.step[steps - 1 - s0].x);
  RowSlot<T, E> s[PF];
  int ld = s0, nld = 0;  // table step of the next load
  auto load = [&](RowSlot<T, E> &r) {
    load_row<T, LPR, E, false>(col, vv, sd[ld * GC], lane, r);
    ld += dir;
    if (++nld == steps) {
      nld = 0;
      ld = s0;
    }
  };
#pragma unroll
  for (int u = 0; u < PF; u++)
    if (u < total) load(s[u]);
  int cs = s0, ncs = 0;  // table step being computed
  for (int it = 0; it < total; it += PF) {
#pragma unroll
    for (int u = 0; u < PF; u++) {
      if (it + u < total) {
        const int4 q = sd[cs * GC];
        const int2 st = S.step[cs];
        const T xn = (sb[cs * GC] - row_dot<T, LPR, E, false>(col, vv, s[u], q, lane, S.x)) * sinv[cs * GC];
        if (L.act == 1) {
          if (q.x >= 0 && lane == 0) S.x[q.x] = xn;
        } else {
          const int p0 = __shfl_sync(0xffffffffu, q.x, 0);  // the warp's first position
          if (p0 >= 0) {
            const unsigned bar = ab + (S.phase & 1) * 8, at = ax + (unsigned)(p0 * sizeof(T));
            const T v0 = __shfl_sync(0xffffffffu, xn, (hv * VL) * LPR);
            const T v1 = __shfl_sync(0xffffffffu, xn, (hv * VL + 1) * LPR);
            if constexpr (VL == 2) {
              if (sender) cluster_send2(at, v0, v1, bar);
            } else {
              const T v2 = __shfl_sync(0xffffffffu, xn, 2 * LPR), v3 = __shfl_sync(0xffffffffu, xn, 3 * LPR);
              if (sender) cluster_send4(at, v0, v1, v2, v3, bar);
            }
          }
        }
        cs += dir;
        if (++ncs == steps) {
          ncs = 0;
          cs = s0;
        }
        if (it + u + PF < total) load(s[u]);
        if (st.y & bit) {
          if (L.act == 1) {
            __syncthreads();
          } else {
            if (it + u + 1 < total) arrive(S.phase + 1, st.x);
            if (!__all_sync(0xffffffffu, mbar_wait(&S.bar[S.phase & 1], (S.phase >> 1) & 1))) {
              S.ok = false;  // the warp sends and arrives no more, here and on the other shared levels
              atomicOr(S.wait_flag, kWaitCluster);
              return;
            }
            S.phase++;
          }
        }
      }
    }
  }
}

template <class T, int LPR, int E>
__device__ __forceinline__ void sweeps(const CluLevel<T> &L, int nsw, int reverse, CluSmem<T> &S) {
  if (L.act > 1 && !S.ok) return;  // (a level of one CTA has no waits but the CTA's barriers)
  if (L.mat) sweep_level<T, LPR, E, true>(L, nsw, reverse, S);
  else sweep_level<T, LPR, E, false>(L, nsw, reverse, S);
}

template <class T, int LPR, int E>
__global__ void __launch_bounds__(kCluNT, 1) k_mg_cluster(const __grid_constant__ CluArgs<T> A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint64_t s_bar[2];
  constexpr int GC = kCluNT / LPR;
  const int rank = (int)cluster_rank();
  const int csize = (int)cluster_size();
  const int tid = threadIdx.x;
  const int lane = tid % LPR;
  CluSmem<T> S;
  S.d = reinterpret_cast<int4 *>(smem_raw);
  S.inv = reinterpret_cast<T *>(S.d + (size_t)A.steps * GC);
  S.b = S.inv + (size_t)A.steps * GC;
  S.step = reinterpret_cast<int2 *>(S.b + (size_t)A.steps * GC);
  S.x = reinterpret_cast<T *>(S.step + A.steps);
  S.v = S.x + A.xlen;
  S.c = reinterpret_cast<int *>(S.v + A.mlen);
  S.bar = s_bar;
  S.phase = 0;
  S.wait_flag = A.wait_flag;
  S.ok = true;
  if (tid == 0) {
    mbar_init(&s_bar[0], kCluNT / 32);
    mbar_init(&s_bar[1], kCluNT / 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (csize > 1) {  // every CTA's mbarriers exist before the first value is sent
    cluster_arrive();
    cluster_wait();
  }
  EXF_PDL_WAIT();
  // A level's work is done by its first `act` CTAs; with act == 1 the others are not even at
  // its barriers.  down: x = 0 (or given), pre-smoothing, residual, restriction
  int l = A.hi;
  if (!(A.part & 1)) {  // the ascent alone: where the descent ends
    l = 0;
    if (rank > 0)
      while (l < A.hi && A.lev[l + 1].act == 1) l++;
  }
  for (; (A.part & 1) && l >= 1; l--) {
    const CluLevel<T> &L = A.lev[l];
    if (L.act == 1 && rank > 0) break;  // the levels from here down belong to CTA 0
    const bool in = rank < L.act;
    const int nth = L.act * kCluNT, gt = rank * kCluNT + tid;
    if (in) {
      load_level<T, LPR>(L, rank, S);
      fill_x(L, l < A.hi, S);
    }
    phase_sync(L.act);
    if (in) {
      sweeps<T, LPR, E>(L, l == A.hi ? A.nu_pre_hi : A.nu_pre, A.reverse, S);
      // r = b - A x of every row; x back to global memory
      const int *col = L.mat ? S.c : L.col;
      const T *vv = L.mat ? S.v : L.vv;
#pragma unroll 2
      for (int st = 0; st < L.steps; st++) {
        const int at = st * GC + tid / LPR;
        const int4 q = S.d[at];
        RowSlot<T, E> s;
        load_row<T, LPR, E, true>(col, vv, q, lane, s);
        const T acc = row_dot<T, LPR, E, true>(col, vv, s, q, lane, S.x);
        if (q.z > 0 && lane == 0) L.r[L.node[q.x]] = S.b[at] - acc;
      }
      store_x(L, gt, nth, S);
    }
    phase_sync(L.act);
    if (in) {  // b of the level below, LPR lanes per row
      const CluLevel<T> &Cl = A.lev[l - 1];
      const int G = nth / LPR, gid = gt / LPR;
      for (int r0 = 0; r0 < Cl.N; r0 += G) {
        const int c = r0 + gid;
        T acc = T(0);
        if (c < Cl.N)
          for (int k = L.r_ptr[c] + lane; k < L.r_ptr[c + 1]; k += LPR) acc += L.r_val[k] * L.r[L.r_col[k]];
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (c < Cl.N && lane == 0) Cl.b[c] = (T)L.r_mask[c] * acc;
      }
    }
    phase_sync(L.act);
  }
  // coarsest level: x = A0^{-1} (b * gmask), a warp per row
  const int act1 = A.lev[1].act;
  if (l == 0 && (A.part & 2)) {
    const CluLevel<T> &L = A.lev[0];
    const int n = L.N, w = (rank * kCluNT + tid) >> 5, wl = tid & 31;
    const int nw = (act1 == 1 ? 1 : csize) * (kCluNT / 32);
    for (int row = w; row < n; row += nw) {
      double acc = 0.;
      for (int j = wl; j < n; j += 32) acc += A.inv[(long)row * n + j] * (A.gmask[j] * (double)L.b[j]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (wl == 0) L.x[row] = (T)acc;
    }
    phase_sync(act1);
  }
  if (!(A.part & 4)) return;
  l++;  // CTAs that left the descent rejoin at the lowest level they share
  // up: x += damp * P x_c (or x = P x_c), post-smoothing
  bool apart = act1 == 1;  // CTA 0 is on its own
  for (; l <= A.hi; l++) {
    const CluLevel<T> &L = A.lev[l];
    if (apart && L.act > 1) {  // the whole cluster meets again above CTA 0's levels
      cluster_arrive();
      cluster_wait();
      apart = false;
    }
    const bool in = rank < L.act;
    const int nth = L.act * kCluNT, gt = rank * kCluNT + tid;
    if (in) {
      const T *xc = A.lev[l - 1].x;
      for (int f = gt; f < L.N; f += nth) {
        T acc = T(0);
        for (int k = L.p_ptr[f]; k < L.p_ptr[f + 1]; k++) acc += L.p_val[k] * xc[L.p_col[k]];
        L.x[f] = A.overwrite ? acc : L.x[f] + A.damp * acc;
      }
      load_level<T, LPR>(L, rank, S);
    }
    phase_sync(L.act);
    if (in) fill_x(L, false, S);
    phase_sync(L.act);  // every iterate is filled before the first value is sent
    if (in) {
      sweeps<T, LPR, E>(L, l == A.hi ? A.nu_post_hi : A.nu_post, A.reverse, S);
      store_x(L, gt, nth, S);
    }
    phase_sync(L.act);
  }
}

// ------------------------------------------------------------------ host side
template <class T>
struct CV;
template <>
struct CV<double> {
  static const double *vv(const SysLevel &L) { return L.A.vv.p; }
  static const double *val(const Transfer &t) { return t.val.p; }
  static double *x(SysLevel &L) { return L.x.p; }
  static double *b(SysLevel &L) { return L.b.p; }
  static double *r(SysLevel &L) { return L.r.p; }
};
template <>
struct CV<float> {
  static const float *vv(const SysLevel &L) { return L.A32.vv.p; }
  static const float *val(const Transfer &t) { return t.val32.p; }
  static float *x(SysLevel &L) { return L.x32.p; }
  static float *b(SysLevel &L) { return L.b32.p; }
  static float *r(SysLevel &L) { return L.r32.p; }
};

template <class T>
static auto cluster_kernel(int dim) {
  return dim == 2 ? k_mg_cluster<T, clu_lpr(2), 4> : k_mg_cluster<T, clu_lpr(3), 8>;
}

// largest usable cluster of both kernels on the current device (at most 16), 0: none
static int cluster_fit(int dim) {
  int best = 16;
  auto probe = [&](auto kern) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCluSmem) != cudaSuccess) {
      cudaGetLastError();
      best = 0;
      return;
    }
    for (; best >= 1; best >>= 1) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(best);
      cfg.blockDim = dim3(kCluNT);
      cfg.dynamicSmemBytes = kCluSmem;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = best;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n >= 1) return;
      cudaGetLastError();
    }
  };
  probe(cluster_kernel<double>(dim));
  probe(cluster_kernel<float>(dim));
  return best;
}

__global__ void k_clu_columns(const int *qq_col, const int *pos, long nqq, int *col) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nqq) col[k] = pos[qq_col[k]];
}
// the copy of each CTA's entries, 8 threads per row
__global__ void k_clu_entries(const int4 *tab, const int *first, int ntab, int per_cta, int entries, const int *col,
                              int2 *ent) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) / 8;
  if (t >= ntab) return;
  const int4 d = tab[t];
  int2 *o = ent + (long)(t / per_cta) * entries + first[t];
  for (int i = threadIdx.x % 8; i < d.z; i += 8) o[i] = make_int2(d.y + i, col[d.y + i]);
}

// Tables of a scalar system's levels for the cluster kernel (plan_cluster), at its first
// Gauss-Seidel solve, so that systems solved otherwise do not pay for them: the patterns of
// all candidate levels in one download, all tables in one block of device memory.  Levels
// without tables (no cluster on the device, no memory) keep a launch per colour.
int cluster_ready(exf_sys *s) {
  if (s->clu_ready) return EXF_OK;
  s->clu_ready = true;
  const int dev = s->mesh->device;
  int hi = 0;
  while (hi + 1 < s->nlev && hi + 1 < kCluMaxLev && s->L[hi + 1].N <= cluster_rows(s->dim, 1 << 20)) hi++;
  if (s->nv1 != 0 || hi < 1 || dev < 0 || dev >= 64) return EXF_OK;
  static std::atomic<int> fit[2][64];  // per dimension and device: cluster size + 1
  int most = fit[s->dim == 2][dev].load(std::memory_order_acquire) - 1;
  if (most < 0) {
    most = cluster_fit(s->dim);
    fit[s->dim == 2][dev].store(most + 1, std::memory_order_release);
  }
  if (most < 1) return EXF_OK;
  std::vector<std::vector<int>> qp(hi + 1), diag(hi + 1), items(hi + 1);
  for (int l = 1; l <= hi; l++) {
    SysLevel &L = s->L[l];
    qp[l].resize(L.N + 1);
    diag[l].resize(L.N);
    items[l].resize(L.N);
    EXF_CUDA(cudaMemcpyAsync(qp[l].data(), L.qq_ptr.p, (L.N + 1) * sizeof(int), cudaMemcpyDeviceToHost, s->stream));
    EXF_CUDA(cudaMemcpyAsync(diag[l].data(), L.diag_pos.p, L.N * sizeof(int), cudaMemcpyDeviceToHost, s->stream));
    EXF_CUDA(cudaMemcpyAsync(items[l].data(), L.col_items.p, L.N * sizeof(int), cudaMemcpyDeviceToHost, s->stream));
  }
  EXF_CUDA(cudaStreamSynchronize(s->stream));
  const int lpr = clu_lpr(s->dim), gc = kCluNT / lpr;
  // each table 16-byte aligned: tab, first, step, node and the nodes' positions of every
  // level, then the columns' positions and the CTAs' entries (filled on the device)
  std::vector<int4> mem;
  auto put = [&](const auto &h) {
    const size_t at = mem.size(), bytes = h.size() * sizeof(h[0]);
    mem.resize(at + (bytes + 15) / 16);
    if (bytes) memcpy(&mem[at], h.data(), bytes);
    return at;
  };
  static_assert(sizeof(CluRow) == sizeof(int4) && sizeof(CluStep) == sizeof(int2), "tables are copied as they are");
  struct At {
    size_t tab, first, step, node, pos, col, ent;
  };
  std::vector<At> at(hi + 1);
  for (int l = 1; l <= hi; l++) {
    SysLevel &L = s->L[l];
    CluTable &C = L.clu;
    const CluPlan P = plan_cluster(L.N, qp[l].data(), diag[l].data(), L.ncolour, L.col_off.data(), items[l].data(), lpr,
                                   kCluNT, most);
    C.act = P.act;
    C.Np = (int)P.node.size();
    C.steps = (int)P.step.size();
    // entries that fit no CTA's shared memory are read from the level's arrays
    C.entries = (size_t)P.entries * (4 + sizeof(float)) > kCluSmem ? 0 : P.entries;
    at[l] = {put(P.tab), put(P.first), put(P.step), put(P.node), put(P.pos), 0, 0};
  }
  size_t len = mem.size();
  for (int l = 1; l <= hi; l++) {
    at[l].col = len;
    at[l].ent = at[l].col + ((size_t)s->L[l].nqq + 3) / 4;
    len = at[l].ent + (size_t)s->L[l].clu.act * s->L[l].clu.entries / 2;
  }
  if (s->clu_mem.alloc(len) != EXF_OK) return EXF_OK;
  int4 *d = s->clu_mem.p;
  EXF_CUDA(cudaMemcpyAsync(d, mem.data(), mem.size() * sizeof(int4), cudaMemcpyHostToDevice, s->stream));
  // every CTA copies C.entries entries: those beyond its rows are entry 0
  EXF_CUDA(cudaMemsetAsync(d + mem.size(), 0, (len - mem.size()) * sizeof(int4), s->stream));
  for (int l = 1; l <= hi; l++) {
    SysLevel &L = s->L[l];
    CluTable &C = L.clu;
    int *col = reinterpret_cast<int *>(d + at[l].col);
    int2 *ent = reinterpret_cast<int2 *>(d + at[l].ent);
    C.tab = d + at[l].tab;
    C.first = reinterpret_cast<const int *>(d + at[l].first);
    C.step = reinterpret_cast<const int2 *>(d + at[l].step);
    C.node = reinterpret_cast<const int *>(d + at[l].node);
    C.col = col;
    C.ent = ent;
    k_clu_columns<<<(unsigned)((L.nqq + 255) / 256), 256, 0, s->stream>>>(
        L.qq_col.p, reinterpret_cast<const int *>(d + at[l].pos), L.nqq, col);
    EXF_COUNT(1);
    if (C.entries) {
      const int n = C.steps * gc;
      k_clu_entries<<<(unsigned)(((long)C.act * n * 8 + 255) / 256), 256, 0, s->stream>>>(C.tab, C.first, C.act * n, n,
                                                                                         C.entries, col, ent);
      EXF_COUNT(1);
    }
  }
  EXF_LAUNCH_CHECK();
  EXF_CUDA(cudaStreamSynchronize(s->stream));
  for (int l = 1; l <= hi; l++) s->L[l].clu.ok = true;
  return EXF_OK;
}

static bool shape_of(const exf_sys *s, int hi, size_t elem, CluShape &S) {
  return cluster_shape(hi, elem, kCluNT / clu_lpr(s->dim), [&](int l) -> const CluTable & { return s->L[l].clu; }, S);
}

// whether levels `lev` .. 0 run in the cluster kernel with values of `elem` bytes, level lev
// with `sweeps` sweeps per cycle
bool mg_cluster_level(const exf_sys *s, int lev, size_t elem, int sweeps) {
  CluShape S;
  return s->nv1 == 0 && s->L[lev].N <= cluster_rows(s->dim, sweeps) && shape_of(s, lev, elem, S);
}

// levels hi .. 0 of one V-cycle (gamma 1): x of level hi, from b of level hi; one launch, or
// three with a large coarsest level
template <class T>
int mg_cluster(exf_sys *s, int hi, const exf_mg_params *p, int mul_hi) {
  CluArgs<T> A = {};
  CluShape S;
  if (!shape_of(s, hi, sizeof(T), S)) {
    set_error("level %d does not fit the cluster cycle", hi);
    return EXF_ERR_UNSUPPORTED;
  }
  for (int l = hi; l >= 0; l--) {
    SysLevel &L = s->L[l];
    CluLevel<T> &d = A.lev[l];
    d.N = L.N;
    d.x = CV<T>::x(L);
    d.b = CV<T>::b(L);
    d.r = CV<T>::r(L);
    if (l == 0) break;
    d.Np = L.clu.Np;
    d.steps = L.clu.steps;
    d.act = L.clu.act;
    d.mat = S.mat[l];
    d.tab = L.clu.tab;
    d.first = L.clu.first;
    d.ent = L.clu.ent;
    d.step = L.clu.step;
    d.node = L.clu.node;
    d.col = L.clu.col;
    d.vv = CV<T>::vv(L);
    SysLevel &C = s->L[l - 1];
    d.r_ptr = C.Rq.ptr.p;
    d.r_col = C.Rq.col.p;
    d.r_val = CV<T>::val(C.Rq);
    d.r_mask = C.rmask.p;
    d.p_ptr = L.Pq.ptr.p;
    d.p_col = L.Pq.col.p;
    d.p_val = CV<T>::val(L.Pq);
  }
  A.steps = S.steps;
  A.xlen = S.xlen;
  A.mlen = S.mlen;
  A.hi = hi;
  const int mul = p->double_below_top ? 2 : 1;
  A.nu_pre = p->nu_pre * mul;
  A.nu_post = p->nu_post * mul;
  A.nu_pre_hi = p->nu_pre * mul_hi;
  A.nu_post_hi = p->nu_post * mul_hi;
  A.reverse = p->reverse_colours ? 1 : 0;
  A.damp = (T)p->corr_damp;
  A.overwrite = p->corr_damp == 0. ? 1 : 0;
  A.inv = s->coarse_inv.p;
  A.gmask = s->gmask0.p;
  A.wait_flag = s->wait_flag.p;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S.act);
  cfg.blockDim = dim3(kCluNT);
  cfg.dynamicSmemBytes = S.smem;
  cfg.stream = s->stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = S.act;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  if (s->L[0].N <= kCluCoarse) {
    A.part = 7;
    EXF_CUDA(cudaLaunchKernelEx(&cfg, cluster_kernel<T>(s->dim), A));
    EXF_COUNT(1);
    return EXF_OK;
  }
  A.part = 1;
  EXF_CUDA(cudaLaunchKernelEx(&cfg, cluster_kernel<T>(s->dim), A));
  EXF_TRY(coarse_apply<T>(s, A.lev[0].b, A.lev[0].x));
  A.part = 4;
  EXF_CUDA(cudaLaunchKernelEx(&cfg, cluster_kernel<T>(s->dim), A));
  EXF_COUNT(2);
  return EXF_OK;
}
template int mg_cluster<double>(exf_sys *, int, const exf_mg_params *, int);
template int mg_cluster<float>(exf_sys *, int, const exf_mg_params *, int);

}  // namespace exf
