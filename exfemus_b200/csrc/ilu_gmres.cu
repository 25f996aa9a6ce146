// ilu_gmres.cu -- the reference's default level solver for scalar equations: LASPACK's
// GMRESIter (restart 30) left-preconditioned by ILUPrecond, selected by SOLVERT GMRESM
// with the default ILU_PRECONDM (template_appl/nse/DATA/MGSclass_conf.h:101,
// contrib/matrix/linear_solverM.h:200-205, contrib/matrix/laspack_linear_solverM.C:91-96).
//
// ILU (contrib/laspack/factor.c:25-320, the non-symmetric row-wise branch): row i takes
// the set S of its columns <= i, gathers the current entries (S_a, S_b) of the rows in S
// into a dense |S| x |S| matrix, eliminates, and writes back row i's lower entries, its
// diagonal and the entries (S_a, i) of the earlier rows: the factor is stored on the
// matrix's own pattern and the preconditioner is
//   y = (D + U)^-1 D (D + L)^-1 c     (ILUPrecond, contrib/laspack/precond.c:75-110)
// with the triangular solves of MulInv_QV (contrib/laspack/operats.c:1049-1290).  Every
// elimination step, product, sum and division is done in the reference's order with
// explicitly rounded operations (no fused multiply-add), so the factor and the
// preconditioner give the reference's bits.
//
// The row recurrences run sync-free: a warp takes the next row from a ticket counter
// (rows by dependency level, see level_order), waits until the rows it depends on are
// published (bounded acquire loads: of a generation flag per row in the factorisation, of
// the value itself in the triangular solves), computes, and publishes its row (release
// store).  A warp only waits on rows with earlier tickets, which running
// warps hold, so the recurrences always progress; a wait that runs out sets the system's
// wait flag, which the host reports as EXF_ERR_CUDA.  Time is set by the dependency depth
// of the numbering (the level-nested numbering: about 770 levels for the 257 x 257 nodes
// of a 128 x 128 quad9 level), not by bandwidth.
//
// GMRES (contrib/laspack/itersolv.c:1341-1510): MaxIter = the smoothing count, modified
// Gram-Schmidt, Givens rotations, the reference's relative-residual test (rtc.c:48-70)
// before every restart cycle; the scalars live on the device and a converged call skips
// the rest of its kernels, so a smoothing call is a fixed kernel sequence that a CUDA
// graph can hold.  Vector updates use the reference's rounding (a product, then a sum);
// inner products and norms are parallel reductions, so GMRES iterates agree with the
// reference's to rounding, not bitwise.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

#include "cluster.cuh"
#include "exf_internal.h"
#include "ilu_stream.h"

namespace exf {

__device__ __forceinline__ int ld_acq(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_rel(int *p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// the triangular solves publish each row's value itself: the output vector is filled with
// this NaN pattern (which arithmetic does not produce) first, and a row's value replaces it
// with a release store
constexpr unsigned long long kNotReady = 0x7FF4C0FFEE000001ull;
__device__ __forceinline__ double ld_acq_f64(const double *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return __longlong_as_double((long long)v);
}
__device__ __forceinline__ void st_rel_f64(double *p, double v) {
  asm volatile("st.release.gpu.global.b64 [%0], %1;" ::"l"(p), "l"((unsigned long long)__double_as_longlong(v))
               : "memory");
}
// bounded wait for the published value of row j (0 if the wait ran out; the flag is set)
__device__ __forceinline__ double wait_val(const double *v, int j, int *err) {
  for (int t = 0; t < (1 << 20); t++) {
    const double x = ld_acq_f64(v + j);
    if ((unsigned long long)__double_as_longlong(x) != kNotReady) return x;
    if ((t & 255) == 255 && *(volatile int *)err) return 0.;
    __nanosleep(32);
  }
  atomicOr(err, kWaitIlu);
  return 0.;
}

// bounded wait until row j is published in generation gen; false if it ran out (or an
// earlier wait of the launch did)
__device__ __forceinline__ bool wait_row(const int *flag, int j, int gen, int *err) {
  for (int t = 0; t < (1 << 20); t++) {
    if (ld_acq(flag + j) >= gen) return true;
    if ((t & 255) == 255 && *(volatile int *)err) return false;
    __nanosleep(64);
  }
  atomicOr(err, kWaitIlu);
  return false;
}

// position of c in the sorted list a[0..n), -1 if absent
__device__ __forceinline__ int bsearch_i(const int *a, int n, int c) {
  int lo = 0, hi = n - 1;
  while (lo <= hi) {
    const int m = (lo + hi) >> 1, v = a[m];
    if (v == c) return m;
    if (v < c) lo = m + 1;
    else hi = m - 1;
  }
  return -1;
}

// a[j >> 5] of a per-lane register array without a dynamic register index
template <int KU>
__device__ __forceinline__ double pick(const double (&a)[KU], int u) {
  double v = a[0];
#pragma unroll
  for (int q = 1; q < KU; q++)
    if (q == u) v = a[q];
  return v;
}

// ctl[0]: ticket, ctl[1]: generation (factorisation), ctl[2]: zero-pivot row + 1
__global__ void k_ilu_arm(int *ctl, const int *skip) {
  if (skip && *skip) return;
  ctl[0] = 0;
  ctl[1] += 1;
}
// before a triangular solve: the output marked unpublished, the ticket reset
__global__ void k_ilu_prep(double *v, long n, int *ctl, const int *skip) {
  if (skip && *skip) return;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) ctl[0] = 0;
  if (i < n) v[i] = __longlong_as_double((long long)kNotReady);
}

// one warp per row; MAXL >= the longest lower row + 1; f holds a copy of the matrix on
// entry and the factor on exit; invd[i] = 1 / the factor's diagonal
template <int MAXL, int NW>
__global__ void __launch_bounds__(32 * NW) k_ilu_factor(int N, const int *__restrict__ ord, const int *__restrict__ ptr,
                                                        const int *__restrict__ col, const int *__restrict__ dpos,
                                                        double *f, double *invd, int *flag, int *ctl, int *err) {
  constexpr int KU = (MAXL + 31) / 32;
  extern __shared__ double ilu_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *Lm = ilu_smem + (size_t)warp * MAXL * (MAXL + 1);
  // per warp: S, each S row's first entry and entry count, the offsets of the rows'
  // entries in the flattened gather, and the position of column i in each S row
  int *Sc = reinterpret_cast<int *>(ilu_smem + (size_t)NW * MAXL * (MAXL + 1)) + warp * 5 * MAXL;
  int *Rb = Sc + MAXL, *Off = Rb + MAXL, *Pi = Off + MAXL + 1;  // Off holds MAXL + 1 entries
  const int gen = ctl[1];
  auto Lat = [&](int a, int b) -> double & { return Lm[a * (MAXL + 1) + b]; };
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(ctl, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= N) return;
    const int i = ord[t];
    const int k0 = ptr[i], kd = dpos[i], LD = kd - k0 + 1;
    if (LD > MAXL) {  // the host sizes MAXL from the pattern: not reached
      if (lane == 0) atomicOr(err, kWaitIlu);
      if (lane == 0) st_rel(flag + i, gen);
      continue;
    }
    for (int a = lane; a < LD; a += 32) {
      const int r = col[k0 + a];
      Sc[a] = r;
      Rb[a] = ptr[r];
      Off[a + 1] = ptr[r + 1] - Rb[a];  // the row's entry count, summed below
      Pi[a] = -1;
    }
    for (int a = lane; a < LD - 1; a += 32) wait_row(flag, Sc[a], gen, err);
    for (int t = lane; t < LD * (MAXL + 1); t += 32) Lm[t] = 0.;
    __syncwarp();
    if (lane == 0) {
      Off[0] = 0;
      for (int a = 0; a < LD; a++) Off[a + 1] += Off[a];
    }
    __syncwarp();
    // the entries (S_a, S_b) of the rows in S, columns <= i, gathered by all lanes over the
    // rows' concatenated entries, four entries per lane in flight
    const int T = Off[LD];
    for (int e0 = 0; e0 < T; e0 += 128) {
      int kk[4], cc[4], aa[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int e = e0 + 32 * q + lane;
        kk[q] = -1;
        if (e < T) {
          int lo = 0, hi = LD - 1;  // the row a with Off[a] <= e < Off[a + 1]
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (Off[mid] <= e) lo = mid;
            else hi = mid - 1;
          }
          aa[q] = lo;
          kk[q] = Rb[lo] + (e - Off[lo]);
          cc[q] = col[kk[q]];
        }
      }
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (kk[q] >= 0 && cc[q] <= i) {
          const int b = bsearch_i(Sc, LD, cc[q]);
          if (b >= 0) Lat(aa[q], b) = f[kk[q]];
          if (cc[q] == i) Pi[aa[q]] = kk[q];
        }
    }
    __syncwarp();
    const int last = LD - 1;
    double lk[KU], uk[KU];  // row i's lower entries and the column-i entries of rows S_k
#pragma unroll
    for (int u = 0; u < KU; u++) {
      const int k = lane + 32 * u;
      lk[u] = k < last ? Lat(last, k) : 0.;
      uk[u] = k < last ? Lat(k, last) : 0.;
    }
    // L[last][k] -= L[last][j] * L[j][k] / L[j][j] and, independent of it,
    // L[k][last] -= L[j][last] * L[k][j] / L[j][j]: the two chains of divisions side by side
    for (int j = 0; j < last; j++) {
      const double lj = __shfl_sync(0xffffffffu, pick(lk, j >> 5), j & 31);
      const double uj = __shfl_sync(0xffffffffu, pick(uk, j >> 5), j & 31), djj = Lat(j, j);
#pragma unroll
      for (int u = 0; u < KU; u++) {
        const int k = lane + 32 * u;
        if (k > j && k < last) {
          lk[u] = __dsub_rn(lk[u], __ddiv_rn(__dmul_rn(lj, Lat(j, k)), djj));
          uk[u] = __dsub_rn(uk[u], __ddiv_rn(__dmul_rn(uj, Lat(k, j)), djj));
        }
      }
    }
    // L[last][last] -= L[j][last] * L[last][j] / L[j][j]: the terms at once, then in order
    double qd[KU];
#pragma unroll
    for (int u = 0; u < KU; u++) {
      const int k = lane + 32 * u;
      qd[u] = k < last ? __ddiv_rn(__dmul_rn(uk[u], lk[u]), Lat(k, k)) : 0.;
    }
    double d = Lat(last, last);
    for (int j = 0; j < last; j++) d = __dsub_rn(d, __shfl_sync(0xffffffffu, pick(qd, j >> 5), j & 31));
    if (fabs(d) < 10. * DBL_MIN && lane == 0) atomicCAS(ctl + 2, 0, i + 1);  // LASZeroPivotErr
#pragma unroll
    for (int u = 0; u < KU; u++) {
      const int k = lane + 32 * u;
      if (k < last) {
        f[k0 + k] = lk[u];
        if (Pi[k] >= 0) f[Pi[k]] = uk[u];  // entry (S_k, i) of the earlier row S_k
        else atomicOr(err, kWaitIlu);           // LASILUStructErr: the pattern is symmetric here
      }
    }
    if (lane == 0) {
      f[kd] = d;
      invd[i] = __ddiv_rn(1., d);
    }
    __threadfence();
    __syncwarp();
    if (lane == 0) st_rel(flag + i, gen);
  }
}

// The factorisation where every row has at most kFacMax entries up to its diagonal (2D
// meshes) and levels are narrow (fac_one_cta), by one CTA, a dependency level at a time, a warp per row.  The general kernel
// above pays, per level, the flag round trip through L2 and a gather whose places are
// searched for: 25 us.  Here the places are found once per system (k_ilu_struct), the
// entries of a warp's next row are on their way while it eliminates the current one, and
// a level ends with the CTA's barrier.  Same operations, same order, same bits.
constexpr int kFacMax = 11, kFacLd = kFacMax + 1;
constexpr int kFacCap = 128;  // places of a row: at most kFacMax^2
static_assert(kFacMax * kFacMax <= kFacCap && kFacMax * kFacLd < 255, "a place is a byte, 255 none");

// row t of the level order: {row, first entry, first of its places, diagonal entry}; its
// places, a word each: entry << 8 | place in the dense block; and the entries (S_a, i) of the
// rows in S.  COUNT: the number of its places alone.
template <bool COUNT>
__global__ void k_ilu_struct(int N, const int *__restrict__ ord, const int *__restrict__ ptr,
                             const int *__restrict__ col, const int *__restrict__ dpos, int *cnt,
                             const int *__restrict__ off, int4 *row, unsigned *ent, int *pos) {
  const int t = (int)(((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (t >= N) return;
  const int i = ord[t], k0 = ptr[i], kd = dpos[i], LD = kd - k0 + 1;
  const int S = lane < LD ? col[k0 + lane] : -1;
  int n = 0;
  for (int a = 0; a < LD; a++) {
    const int r = __shfl_sync(0xffffffffu, S, a), rb = ptr[r], re = ptr[r + 1];
    for (int e0 = rb; e0 < re; e0 += 32) {
      const int k = e0 + lane, c = k < re ? col[k] : -2;
      int b = -1;
      for (int q = 0; q < LD; q++)
        if (__shfl_sync(0xffffffffu, S, q) == c) b = q;
      const unsigned m = __ballot_sync(0xffffffffu, b >= 0);
      if constexpr (!COUNT) {
        if (b >= 0) ent[off[t] + n + __popc(m & ((1u << lane) - 1u))] = (unsigned)k << 8 | (unsigned)(a * kFacLd + b);
        if (c == i) pos[t * 16 + a] = k;
      }
      n += __popc(m);
    }
  }
  if (lane > 0) return;
  if constexpr (COUNT) {
    cnt[t] = n;
  } else {
    row[t] = make_int4(i, k0, off[t], kd);
    if (t == N - 1) row[N] = make_int4(0, 0, off[N], 0);
  }
}

__global__ void __launch_bounds__(1024) k_ilu_factor_cta(int nlev, const int *__restrict__ loff,
                                                         const int4 *__restrict__ row, const unsigned *__restrict__ ent,
                                                         const int *__restrict__ pos, double *f, double *invd, int *ctl) {
  __shared__ double s_blk[32][kFacMax * kFacLd + 4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *B = s_blk[warp];
  int4 rw = make_int4(0, 0, 0, 0);
  constexpr unsigned kNone = 0xffffffffu;
  unsigned e[kFacCap / 32];
  int pi = 0;
  auto fetch = [&](int t) {
    rw = row[t];
    const int n = row[t + 1].z - rw.z;
    pi = lane < 16 ? pos[t * 16 + lane] : 0;
#pragma unroll
    for (int q = 0; q < kFacCap / 32; q++) e[q] = 32 * q + lane < n ? ent[rw.z + 32 * q + lane] : kNone;
  };
  int lo = loff[0], hi = loff[1], hi2 = nlev > 1 ? loff[2] : hi;
  if (lo + warp < hi) fetch(lo + warp);
  for (int l = 0; l < nlev; l++) {
    const int hi3 = l + 3 <= nlev ? loff[l + 3] : hi2;
    bool have = lo + warp < hi;
    for (int t = lo + warp; t < hi; t += 32) {
      double g[kFacCap / 32];
#pragma unroll
      for (int q = 0; q < kFacCap / 32; q++) g[q] = e[q] != kNone ? f[e[q] >> 8] : 0.;
      for (int q = lane; q < kFacMax * kFacLd; q += 32) B[q] = 0.;
      __syncwarp();
#pragma unroll
      for (int q = 0; q < kFacCap / 32; q++)
        if (e[q] != kNone) B[e[q] & 255u] = g[q];
      __syncwarp();
      const int i = rw.x, k0 = rw.y, kd = rw.w, last = kd - k0, pk = pi;
      // the warp's next row, of this level or the next
      const int tn = t + 32 < hi ? t + 32 : hi + warp;
      if (tn < (t + 32 < hi ? hi : hi2)) fetch(tn);
      double lk = lane < last ? B[last * kFacLd + lane] : 0., uk = lane < last ? B[lane * kFacLd + last] : 0.;
      for (int j = 0; j < last; j++) {
        const double lj = __shfl_sync(0xffffffffu, lk, j), uj = __shfl_sync(0xffffffffu, uk, j);
        const double djj = B[j * kFacLd + j];
        if (lane > j && lane < last) {
          lk = __dsub_rn(lk, __ddiv_rn(__dmul_rn(lj, B[j * kFacLd + lane]), djj));
          uk = __dsub_rn(uk, __ddiv_rn(__dmul_rn(uj, B[lane * kFacLd + j]), djj));
        }
      }
      const double qd = lane < last ? __ddiv_rn(__dmul_rn(uk, lk), B[lane * kFacLd + lane]) : 0.;
      double d = B[last * kFacLd + last];
      for (int j = 0; j < last; j++) d = __dsub_rn(d, __shfl_sync(0xffffffffu, qd, j));
      if (fabs(d) < 10. * DBL_MIN && lane == 0) atomicCAS(ctl + 2, 0, i + 1);  // LASZeroPivotErr
      if (lane < last) {
        f[k0 + lane] = lk;
        f[pk] = uk;
      }
      if (lane == 0) {
        f[kd] = d;
        invd[i] = __ddiv_rn(1., d);
      }
      __syncwarp();
    }
    if (!have && hi + warp < hi2) fetch(hi + warp);
    lo = hi;
    hi = hi2;
    hi2 = hi3;
    __syncthreads();
  }
}

// w = (D + L)^-1 c: Sum = 0, Sum -= l_ik w_k over the row's lower entries in column
// order, Sum += c_i, w_i = Sum / d_i (as the product with the stored inverse)
__global__ void __launch_bounds__(128) k_ilu_lower(int N, const int *__restrict__ ord, const int *__restrict__ ptr,
                                                   const int *__restrict__ col,
                                                   const int *__restrict__ dpos, const double *__restrict__ f,
                                                   const double *__restrict__ invd, const double *c, double *w,
                                                   int *ctl, int *err, const int *skip) {
  if (skip && *skip) return;
  const int lane = threadIdx.x & 31;
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(ctl, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= N) return;
    const int i = ord[t];
    const int k0 = ptr[i], nl = dpos[i] - k0;
    const double ci = c[i], di = invd[i];  // loaded before the waits, off the critical path
    double s = 0.;
    for (int base = 0; base < nl; base += 32) {
      double p = 0.;
      if (base + lane < nl) {
        const int k = k0 + base + lane;
        const double fk = f[k];
        p = __dmul_rn(fk, wait_val(w, col[k], err));
      }
      const int n = min(32, nl - base);
      for (int t = 0; t < n; t++) s = __dsub_rn(s, __shfl_sync(0xffffffffu, p, t));
    }
    s = __dadd_rn(s, ci);
    if (lane == 0) st_rel_f64(w + i, __dmul_rn(s, di));
  }
}

// y = (D + U)^-1 (D w): Sum -= u_ik y_k over the upper entries from the row's end,
// Sum += d_i w_i, y_i = Sum / d_i (rows by level of the upper entries)
__global__ void __launch_bounds__(128) k_ilu_upper(int N, const int *__restrict__ ord, const int *__restrict__ ptr,
                                                   const int *__restrict__ col,
                                                   const int *__restrict__ dpos, const double *__restrict__ f,
                                                   const double *__restrict__ invd, const double *w, double *y,
                                                   int *ctl, int *err, const int *skip) {
  if (skip && *skip) return;
  const int lane = threadIdx.x & 31;
  for (;;) {
    int t0 = 0;
    if (lane == 0) t0 = atomicAdd(ctl, 1);
    t0 = __shfl_sync(0xffffffffu, t0, 0);
    if (t0 >= N) return;
    const int i = ord[t0];
    const int kd = dpos[i], k1 = ptr[i + 1], nu = k1 - 1 - kd;
    const double zi = __dadd_rn(0., __dmul_rn(f[kd], w[i])), di = invd[i];  // Mul_QV of the diagonal: 0 + d_i w_i
    double s = 0.;
    for (int base = 0; base < nu; base += 32) {
      double p = 0.;
      if (base + lane < nu) {
        const int k = k1 - 1 - base - lane;  // from the row's end
        const double fk = f[k];
        p = __dmul_rn(fk, wait_val(y, col[k], err));
      }
      const int n = min(32, nu - base);
      for (int t = 0; t < n; t++) s = __dsub_rn(s, __shfl_sync(0xffffffffu, p, t));
    }
    s = __dadd_rn(s, zi);
    if (lane == 0) st_rel_f64(y + i, __dmul_rn(s, di));
  }
}


// ILUPrecond of a level whose vector fits one CTA's shared memory and whose dependency levels
// are narrow (tri_one_cta): both triangular solves in one launch of one CTA, dependency level after dependency level.  What bounds a solve is
// the round trip from a row's value to the rows that read it, once per level: 3 us through
// L2 between warps (the kernels above).  Here a few warps solve in turn, a thread per row,
// doing the reference's operations in the reference's order, and the values stay in shared
// memory.  Their instructions are then the bound, so the factor comes as a stream in the order of its
// use (another warp copies it into shared-memory stages), in records of up to 32 rows of one
// level (build_tri_stream).  Absent entries and rows point to a zero behind the vector
// (s - 0 * 0 leaves the bits of s).  v holds c, then w = (D + L)^-1 c, then y, in place: a
// row reads its own c (w) before it replaces it.
//
// The owner of a chunk's last record frees the chunk's stage.  By then every record of the
// chunk has been solved, hence loaded, and no warp has anything else to read there: a record
// holds the place of its warp's next one.  A warp's test of a stage's phase is safe too: the
// chunk it waits for holds its own unsolved record, so the stage cannot have moved on, and
// the chunk before it in the stage is not later than that of the record it has just solved
// (kTriStages = kTriWarps), so that one was there.
constexpr int kTriThreads = 256;
static_assert(kTriStages >= kTriWarps, "a warp's next record is at most kTriWarps chunks on");
static_assert(sizeof(TriWord) == sizeof(uint4) && sizeof(TriPair) == sizeof(int2), "streams are copied as they are");
constexpr size_t kTriSmem = 224 * 1024;

struct TriSmem {
  uint4 st[kTriStages][kTriWords];
  uint64_t full[kTriStages], empty[kTriStages], turn[kTriWarps];
  double part[32];  // sums of rows that continue in the next record
};
struct TriRow {  // a lane's row of a record, loaded a record ahead
  int g, flags, i;
  double inv, dia;
  int c[kTriE];
  double a[kTriE];
};
__device__ __forceinline__ void tri_load(TriRow &t, const uint4 *rec, const uint4 h, int lane) {
  t.g = (int)h.x;
  t.flags = (int)h.y;
  const int *q = reinterpret_cast<const int *>(rec + 1) + lane;
  const double *d = reinterpret_cast<const double *>(rec + 9) + lane;
  const int *col = reinterpret_cast<const int *>(rec + 41) + lane;
  const double *val = reinterpret_cast<const double *>(rec + 41 + 32 * t.g) + lane;
  t.i = q[0];
  t.inv = d[0];
  t.dia = d[32];
#pragma unroll
  for (int g = 0; g < kTriE / 4; g++)
    if (g < t.g) {
#pragma unroll
      for (int u = 4 * g; u < 4 * g + 4; u++) {
        t.c[u] = col[u * 32];
        t.a[u] = val[u * 32];
      }
    }
}
__device__ __forceinline__ void tri_solve(const TriRow &t, double *v, double *part, int lane, bool upper) {
  double s = t.flags & 1 ? 0. : part[lane];
  const double w = v[t.i];
  double x[kTriE];
#pragma unroll
  for (int g = 0; g < kTriE / 4; g++)  // every gather before the first product
    if (g < t.g) {
#pragma unroll
      for (int u = 4 * g; u < 4 * g + 4; u++) x[u] = v[t.c[u]];
    }
#pragma unroll
  for (int g = 0; g < kTriE / 4; g++)
    if (g < t.g) {
      double p[4];
#pragma unroll
      for (int u = 0; u < 4; u++) p[u] = __dmul_rn(t.a[4 * g + u], x[4 * g + u]);
#pragma unroll
      for (int u = 0; u < 4; u++) s = __dsub_rn(s, p[u]);
    }
  if (t.flags & 2)  // lower: (Sum + c_i) / d; upper: (Sum + (0 + d_i w_i)) / d
    v[t.i] = __dmul_rn(__dadd_rn(s, upper ? __dadd_rn(0., __dmul_rn(t.dia, w)) : w), t.inv);
  else part[lane] = s;
}

__global__ void __launch_bounds__(kTriThreads) k_ilu_tri(int N, const uint4 *__restrict__ str,
                                                         const int2 *__restrict__ chunk, int nch, int nlo, int nrec,
                                                         const uint4 first, const double *c, double *y, int *err,
                                                         const int *skip) {
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char tri_raw[];
  TriSmem &S = *reinterpret_cast<TriSmem *>(tri_raw);
  double *v = reinterpret_cast<double *>(tri_raw + sizeof(TriSmem));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    for (int k = 0; k < kTriStages; k++) {
      mbar_init(&S.full[k], 1);
      mbar_init(&S.empty[k], 1);
    }
    for (int k = 0; k < kTriWarps; k++) mbar_init(&S.turn[k], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    v[N] = 0.;
  }
#pragma unroll 4
  for (int i = tid; i < N; i += kTriThreads) v[i] = c[i];
  __syncthreads();
  if (tid == 32 * kTriWarps) {  // producer: chunk after chunk
    int it = 0;
    bool ok = true;
    int2 ch = chunk[0];
    for (; it < nch; it++) {
      const int k = it % kTriStages;
      if (it >= kTriStages && !mbar_wait(&S.empty[k], ((it / kTriStages) - 1) & 1)) {
        ok = false;
        break;
      }
      mbar_arrive_tx(&S.full[k], (unsigned)ch.y * 16u);
      bulk_g2s(&S.st[k][0], str + ch.x, (unsigned)ch.y * 16u, &S.full[k]);
      if (it + 1 < nch) ch = chunk[it + 1];
    }
    if (!ok) {  // the copies already issued land before the CTA leaves
      atomicOr(err, kWaitIlu);
      for (int j = max(0, it - kTriStages); j < it; j++) mbar_wait(&S.full[j % kTriStages], (j / kTriStages) & 1);
    }
  } else if (warp < kTriWarps) {
    // the warps solve the records in turn; while one solves, the others load their next
    TriRow t;
    int ci = 0;  // chunk of the record in hand
    bool good = true, have = false;
    static_assert(kTriWarps == 4, "a first place for each warp");
    unsigned next = warp == 0 ? first.x : warp == 1 ? first.y : warp == 2 ? first.z : first.w;
    auto fetch = [&]() {
      ci += next >> 24;
      const int k = ci % kTriStages;
      if (good && !mbar_wait(&S.full[k], (ci / kTriStages) & 1)) {
        atomicOr(err, kWaitIlu);
        good = false;
      }
      have = good;
      if (!have) return;
      const uint4 *r = &S.st[k][next & 0xffffffu];
      const uint4 h = r[0];
      next = h.w;
      tri_load(t, r, h, lane);
    };
    if (warp < nrec) fetch();
    for (int k = warp, turn = warp == 0 ? -1 : 0; k < nrec; k += kTriWarps, turn++) {
      if (turn >= 0 && !mbar_wait(&S.turn[warp], turn & 1)) {  // record k - 1 is solved
        atomicOr(err, kWaitIlu);
        good = have = false;  // the turns go on without further work
      }
      if (have) tri_solve(t, v, S.part, lane, k >= nlo);
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&S.turn[(warp + 1) % kTriWarps]);
        // the last record of a chunk (all its others are solved) frees the chunk's stage
        if (have && (t.flags & 4)) mbar_arrive(&S.empty[ci % kTriStages]);
      }
      have = false;
      if (k + kTriWarps < nrec) fetch();
    }
  }
  __syncthreads();
#pragma unroll 4
  for (int i = tid; i < N; i += kTriThreads) y[i] = v[i];
}

// the factor's values into the streams: {double of the stream, entry of f or ~row of 1 / d}
__global__ void k_ilu_stream(const int2 *__restrict__ src, int n, const double *__restrict__ f,
                             const double *__restrict__ invd, double *__restrict__ str) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int2 e = src[i];
  str[e.x] = e.y >= 0 ? f[e.y] : invd[~e.y];
}

// ------------------------------------------------------------------- GMRES scalars
// gm_sc: [0] ||b||^2, [1] ||v1||^2 (the residual), [2] the last inner product, [4] the
// norm a vector is scaled by, H(i, k) = h[i][k], S(k) = s[k], C1/C2 the rotations, Y(k)
// = y[k] (1-based as in GMRESIter); gm_ctl[0] != 0: the call has converged, skip
constexpr int kGmSteps = 30;  // SetGMRESRestart(30), laspack_linear_solverM.C:91
__host__ __device__ constexpr int gmH(int i, int k) { return 16 + i * 32 + k; }
__host__ __device__ constexpr int gmS(int k) { return 1008 + k; }
__host__ __device__ constexpr int gmC1(int k) { return 1040 + k; }
__host__ __device__ constexpr int gmC2(int k) { return 1072 + k; }
__host__ __device__ constexpr int gmY(int k) { return 1104 + k; }
constexpr int kGmScalars = 1136;

template <int NT>
__global__ void __launch_bounds__(NT) k_gm_dot_part(const double *__restrict__ a, const double *__restrict__ b,
                                                    long n, double *part) {
  __shared__ double sh[NT / 32];
  double v = 0.;
  for (long i = (long)blockIdx.x * NT + threadIdx.x; i < n; i += (long)gridDim.x * NT) v += a[i] * b[i];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.;
    for (int k = 0; k < NT / 32; k++) t += sh[k];
    part[blockIdx.x] = t;
  }
}
__global__ void k_gm_dot_fin(const double *__restrict__ part, int np, double *out) {
  __shared__ double sh[8];
  double v = 0.;
  for (int i = threadIdx.x; i < np; i += 256) v += part[i];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.;
    for (int k = 0; k < 8; k++) t += sh[k];
    *out = t;
  }
}

// RTCResult (rtc.c:48-70): converged when ||r|| < eps ||b|| (or b = 0 and 1 + ||r|| = 1)
__global__ void k_gm_rtc(const double *sc, int *ctl, double eps) {
  const double rn = sqrt(sc[1]), bn = sqrt(sc[0]);
  const bool conv = rn < eps * bn || (fabs(bn) < 10. * DBL_MIN && fabs((1. + rn) - 1.) < 10. * DBL_EPSILON);
  ctl[0] = conv ? 1 : 0;
}
__global__ void k_gm_reset(int *ctl) { ctl[0] = 0; }

// s[1] = ||v1|| after preconditioning; the vector is then scaled by 1 / s[1]
__global__ void k_gm_first(double *sc) {
  sc[gmS(1)] = __dsqrt_rn(sc[2]);
  sc[4] = sc[gmS(1)];
}

// v *= 1 / *den (MulAsgn_VS with the reciprocal formed once)
__global__ void k_gm_scale(double *v, long n, const double *den, const int *skip) {
  if (*skip) return;
  const double f = __ddiv_rn(1., *den);
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = __dmul_rn(v[i], f);
}
// v -= h vk (SubAsgn_VV(v, Mul_SV(h, vk)))
__global__ void k_gm_axpy(double *v, const double *__restrict__ vk, long n, const double *h, const int *skip) {
  if (*skip) return;
  const double hh = *h;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = __dsub_rn(v[i], __dmul_rn(hh, vk[i]));
}

// h[i][i+1] = ||v_{i+1}|| (the last inner product), then the Q-R update of column i and
// of s (itersolv.c, the "Q-R algorithm" block)
__device__ __forceinline__ void gm_qr_column(double *sc, int i, double nrm) {
  sc[gmH(i, i + 1)] = nrm;
  sc[4] = nrm;
  for (int k = 1; k < i; k++) {
    const double hk = sc[gmH(i, k)], hk1 = sc[gmH(i, k + 1)];
    const double h1 = __dadd_rn(__dmul_rn(sc[gmC1(k)], hk), __dmul_rn(sc[gmC2(k)], hk1));
    const double h2 = __dadd_rn(__dmul_rn(-sc[gmC2(k)], hk), __dmul_rn(sc[gmC1(k)], hk1));
    sc[gmH(i, k)] = h1;
    sc[gmH(i, k + 1)] = h2;
  }
  const double hii = sc[gmH(i, i)], hi1 = sc[gmH(i, i + 1)];
  const double r = __dsqrt_rn(__dadd_rn(__dmul_rn(hii, hii), __dmul_rn(hi1, hi1)));
  sc[gmC1(i)] = __ddiv_rn(hii, r);
  sc[gmC2(i)] = __ddiv_rn(hi1, r);
  sc[gmH(i, i)] = r;
  sc[gmH(i, i + 1)] = 0.;
  sc[gmS(i + 1)] = __dmul_rn(-sc[gmC2(i)], sc[gmS(i)]);
  sc[gmS(i)] = __dmul_rn(sc[gmC1(i)], sc[gmS(i)]);
}
__global__ void k_gm_qr(double *sc, int i) { gm_qr_column(sc, i, __dsqrt_rn(sc[2])); }

// H y = s by back substitution (s is overwritten, as in the reference)
__global__ void k_gm_solve(double *sc, int ni) {
  for (int j = ni; j > 0; j--) {
    sc[gmY(j)] = __ddiv_rn(sc[gmS(j)], sc[gmH(j, j)]);
    for (int k = j - 1; k > 0; k--) sc[gmS(k)] = __dsub_rn(sc[gmS(k)], __dmul_rn(sc[gmH(j, k)], sc[gmY(j)]));
  }
}

// x += y_j v_j for j = ni .. 1 (AddAsgn_VV(x, Mul_SV(y[j], v[j])))
__global__ void k_gm_update(double *x, const double *__restrict__ V, long n, int ni, const double *sc,
                            const int *skip) {
  if (*skip) return;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double xi = x[i];
  for (int j = ni; j > 0; j--) xi = __dadd_rn(xi, __dmul_rn(sc[gmY(j)], V[(long)(j - 1) * n + i]));
  x[i] = xi;
}
__global__ void k_gm_copy(const double *src, double *dst) { *dst = *src; }

// The same steps for a vector that fits one CTA's shared memory: an Arnoldi step is 3 i + 5
// launches of 2-3 us above, whatever the size, and one launch here.
constexpr int kGmCta = 1024;
constexpr size_t kGmSmem = 200 * 1024;

// block sum, the same value in every thread
__device__ __forceinline__ double gm_sum(double v, double *sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();  // sh is free again
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  v = sh[threadIdx.x & 31];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// ||b||^2 and the relative-residual test of a call's start
__global__ void __launch_bounds__(kGmCta) k_gm_begin(const double *__restrict__ b, int n, double *sc, int *ctl,
                                                     double eps) {
  __shared__ double sh[kGmCta / 32];
  double v = 0.;
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += kGmCta) v += b[i] * b[i];
  v = gm_sum(v, sh);
  if (threadIdx.x > 0) return;
  sc[0] = v;
  const double rn = sqrt(sc[1]), bn = sqrt(v);
  const bool conv = rn < eps * bn || (fabs(bn) < 10. * DBL_MIN && fabs((1. + rn) - 1.) < 10. * DBL_EPSILON);
  ctl[0] = conv ? 1 : 0;
}
// v[1] to unit length, s[1] its norm (i = 0); or v[i + 1] orthogonalised against v[1 .. i]
// (modified Gram-Schmidt), the Q-R update of column i, and to unit length
__global__ void __launch_bounds__(kGmCta) k_gm_step(double *V, int n, int i, double *sc, const int *skip) {
  if (*skip) return;
  extern __shared__ double gm_v[];
  __shared__ double sh[kGmCta / 32];
  double *w = V + (long)i * n;
#pragma unroll 4
  for (int q = threadIdx.x; q < n; q += kGmCta) gm_v[q] = w[q];
  for (int k = 1; k <= i; k++) {
    const double *vk = V + (long)(k - 1) * n;
    double d = 0.;
#pragma unroll 4
    for (int q = threadIdx.x; q < n; q += kGmCta) d += gm_v[q] * vk[q];
    const double h = gm_sum(d, sh);
    if (threadIdx.x == 0) sc[gmH(i, k)] = h;
#pragma unroll 4
    for (int q = threadIdx.x; q < n; q += kGmCta) gm_v[q] = __dsub_rn(gm_v[q], __dmul_rn(h, vk[q]));
  }
  double d = 0.;
#pragma unroll 4
  for (int q = threadIdx.x; q < n; q += kGmCta) d += gm_v[q] * gm_v[q];
  const double nrm = __dsqrt_rn(gm_sum(d, sh)), f = __ddiv_rn(1., nrm);
#pragma unroll 4
  for (int q = threadIdx.x; q < n; q += kGmCta) w[q] = __dmul_rn(gm_v[q], f);
  if (threadIdx.x > 0) return;
  if (i == 0) {
    sc[gmS(1)] = nrm;
  } else {
    gm_qr_column(sc, i, nrm);
  }
}

// ------------------------------------------------------------------- host side
static int ilu_grid(exf_sys *s) { return s->nsm * 2; }

static int dot_dev(exf_sys *s, SysLevel &L, const double *a, const double *b, long n, double *out) {
  constexpr int G = 296;
  if (L.gm_part.n < (size_t)G) EXF_TRY(L.gm_part.alloc(G));
  k_gm_dot_part<256><<<G, 256, 0, s->stream>>>(a, b, n, L.gm_part.p);
  k_gm_dot_fin<<<1, 256, 0, s->stream>>>(L.gm_part.p, G, out);
  EXF_COUNT(2);
  return EXF_OK;
}

// y = ILUPrecond(c) on level lev (y may be c); kernels skipped while *skip != 0
static int ilu_apply_dev(exf_sys *s, int lev, const double *c, double *y, const int *skip) {
  SysLevel &L = s->L[lev];
  const int N = L.N, G = ilu_grid(s);
  if (L.ilu_nsrc) {  // the streams exist: one CTA
    k_ilu_tri<<<1, kTriThreads, sizeof(TriSmem) + (size_t)(N + 1) * sizeof(double), s->stream>>>(
        N, L.ilu_str.p, L.ilu_chunk.p, L.ilu_nchunk, L.ilu_nrec[0], L.ilu_nrec[0] + L.ilu_nrec[1], L.ilu_first, c, y,
        s->wait_flag.p, skip);
    EXF_COUNT(1);
    EXF_LAUNCH_CHECK();
    return EXF_OK;
  }
  const unsigned g = (unsigned)((N + 255) / 256);
  k_ilu_prep<<<g, 256, 0, s->stream>>>(L.gm_w.p, N, L.ilu_ctl.p, skip);
  k_ilu_lower<<<G, 128, 0, s->stream>>>(N, L.ilu_ord_lo.p, L.qq_ptr.p, L.qq_col.p, L.diag_pos.p, L.ilu_f.p,
                                        L.ilu_inv.p, c, L.gm_w.p, L.ilu_ctl.p, s->wait_flag.p, skip);
  k_ilu_prep<<<g, 256, 0, s->stream>>>(y, N, L.ilu_ctl.p, skip);
  k_ilu_upper<<<G, 128, 0, s->stream>>>(N, L.ilu_ord_up.p, L.qq_ptr.p, L.qq_col.p, L.diag_pos.p, L.ilu_f.p,
                                        L.ilu_inv.p, L.gm_w.p, y, L.ilu_ctl.p, s->wait_flag.p, skip);
  EXF_COUNT(4);
  EXF_LAUNCH_CHECK();
  return EXF_OK;
}

template <int MAXL, int NW>
static int launch_factor(exf_sys *s, SysLevel &L) {
  const size_t smem = (size_t)NW * (MAXL * (MAXL + 1) * sizeof(double) + 5 * MAXL * sizeof(int));
  auto kern = k_ilu_factor<MAXL, NW>;
  EXF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_ilu_arm<<<1, 1, 0, s->stream>>>(L.ilu_ctl.p, nullptr);
  kern<<<s->nsm * 4, 32 * NW, smem, s->stream>>>(L.N, L.ilu_ord_lo.p, L.qq_ptr.p, L.qq_col.p, L.diag_pos.p, L.ilu_f.p, L.ilu_inv.p,
                                                   L.ilu_flag.p, L.ilu_ctl.p, s->wait_flag.p);
  EXF_COUNT(2);
  EXF_LAUNCH_CHECK();
  return EXF_OK;
}

// The streams of k_ilu_tri for one level, from the pattern (fixed per system); without memory
// for them the level is solved on all SMs
static int build_streams(exf_sys *s, SysLevel &L, const std::vector<int> &ptr, const std::vector<int> &col,
                         const std::vector<int> &dp) {
  if (sizeof(TriSmem) + (size_t)(L.N + 1) * sizeof(double) > kTriSmem) return EXF_OK;
  EXF_CUDA(cudaFuncSetAttribute(k_ilu_tri, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTriSmem));
  const TriStream T = build_tri_stream(ptr, col, dp);
  if (!tri_one_cta(T.nrec, T.depth)) return EXF_OK;
  if (L.ilu_str.alloc(T.str.size()) != EXF_OK || L.ilu_src.alloc(T.src.size()) != EXF_OK ||
      L.ilu_chunk.alloc(T.chunk.size()) != EXF_OK) {
    L.ilu_str.release();
    L.ilu_src.release();
    return EXF_OK;
  }
  EXF_CUDA(cudaMemcpyAsync(L.ilu_str.p, T.str.data(), T.str.size() * sizeof(uint4), cudaMemcpyHostToDevice, s->stream));
  EXF_CUDA(cudaMemcpyAsync(L.ilu_src.p, T.src.data(), T.src.size() * sizeof(int2), cudaMemcpyHostToDevice, s->stream));
  EXF_CUDA(cudaMemcpyAsync(L.ilu_chunk.p, T.chunk.data(), T.chunk.size() * sizeof(int2), cudaMemcpyHostToDevice,
                           s->stream));
  EXF_CUDA(cudaStreamSynchronize(s->stream));
  L.ilu_nchunk = (int)T.chunk.size();
  for (int u = 0; u < 2; u++) L.ilu_nrec[u] = T.nrec[u];
  L.ilu_first = make_uint4(T.first[0], T.first[1], T.first[2], T.first[3]);
  L.ilu_nsrc = (int)T.src.size();
  return EXF_OK;
}

// The places of k_ilu_factor_cta for one level, from the pattern and the rows' dependency
// levels (fixed per system); without memory for them the level is factored on all SMs
static int build_places(exf_sys *s, SysLevel &L, const std::vector<int> &lv) {
  const int N = L.N;
  std::vector<int> loff(L.ilu_depth[0] + 1, 0), off(N + 1, 0);
  for (int i = 0; i < N; i++) loff[lv[i] + 1]++;
  for (int l = 0; l < L.ilu_depth[0]; l++) loff[l + 1] += loff[l];
  DBuf<int> d_off;
  if (d_off.alloc(N + 1) != EXF_OK) return EXF_OK;
  const unsigned g = (unsigned)(((long)N * 32 + 255) / 256);
  k_ilu_struct<true><<<g, 256, 0, s->stream>>>(N, L.ilu_ord_lo.p, L.qq_ptr.p, L.qq_col.p, L.diag_pos.p, d_off.p, nullptr,
                                               nullptr, nullptr, nullptr);
  EXF_LAUNCH_CHECK();
  EXF_CUDA(cudaMemcpyAsync(off.data() + 1, d_off.p, N * sizeof(int), cudaMemcpyDeviceToHost, s->stream));
  EXF_CUDA(cudaStreamSynchronize(s->stream));
  for (int t = 0; t < N; t++) off[t + 1] += off[t];
  if (L.ilu_loff.alloc(loff.size()) != EXF_OK || L.ilu_ent.alloc(off[N]) != EXF_OK ||
      L.ilu_pos.alloc((size_t)N * 16) != EXF_OK || L.ilu_row.alloc(N + 1) != EXF_OK) {
    L.ilu_ent.release();
    L.ilu_pos.release();
    L.ilu_row.release();
    return EXF_OK;
  }
  EXF_TRY(L.ilu_pos.zero(s->stream));
  EXF_CUDA(cudaMemcpyAsync(L.ilu_loff.p, loff.data(), loff.size() * sizeof(int), cudaMemcpyHostToDevice, s->stream));
  EXF_CUDA(cudaMemcpyAsync(d_off.p, off.data(), off.size() * sizeof(int), cudaMemcpyHostToDevice, s->stream));
  k_ilu_struct<false><<<g, 256, 0, s->stream>>>(N, L.ilu_ord_lo.p, L.qq_ptr.p, L.qq_col.p, L.diag_pos.p, nullptr,
                                                d_off.p, L.ilu_row.p, L.ilu_ent.p, L.ilu_pos.p);
  EXF_LAUNCH_CHECK();
  EXF_COUNT(2);
  EXF_CUDA(cudaStreamSynchronize(s->stream));
  return EXF_OK;
}

// ILUFactor of level lev's matrix, once per assembly (outside graph capture)
int ilu_ready(exf_sys *s, int lev) {
  SysLevel &L = s->L[lev];
  if (L.ilu_ok) return EXF_OK;
  if (s->nv1 != 0) {
    set_error("GMRES + ILU smoothing needs a scalar system: the Navier-Stokes pressure block has zero "
              "diagonal entries, on which LASPACK's ILU stops (LASZeroInDiagErr)");
    return EXF_ERR_UNSUPPORTED;
  }
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  EXF_CUDA(cudaStreamIsCapturing(s->stream, &cs));
  if (cs != cudaStreamCaptureStatusNone) {
    set_error("the ILU factor of level %d is stale inside a graph capture", lev);
    return EXF_ERR_STATE;
  }
  const int N = L.N;
  if (L.ilu_maxl == 0) {  // from the pattern, fixed per system
    std::vector<int> ptr(N + 1), dp(N), col(L.nqq);
    EXF_CUDA(cudaMemcpyAsync(ptr.data(), L.qq_ptr.p, (N + 1) * sizeof(int), cudaMemcpyDeviceToHost, s->stream));
    EXF_CUDA(cudaMemcpyAsync(dp.data(), L.diag_pos.p, N * sizeof(int), cudaMemcpyDeviceToHost, s->stream));
    EXF_CUDA(cudaMemcpyAsync(col.data(), L.qq_col.p, L.nqq * sizeof(int), cudaMemcpyDeviceToHost, s->stream));
    EXF_CUDA(cudaStreamSynchronize(s->stream));
    int m = 1;
    for (int i = 0; i < N; i++) m = std::max(m, dp[i] - ptr[i] + 1);
    std::vector<int> lo, up, lv;
    L.ilu_depth[0] = level_order(ptr, col, dp, false, lo, &lv);
    L.ilu_depth[1] = level_order(ptr, col, dp, true, up);
    EXF_TRY(L.ilu_ord_lo.alloc(N));
    EXF_TRY(L.ilu_ord_up.alloc(N));
    EXF_CUDA(cudaMemcpyAsync(L.ilu_ord_lo.p, lo.data(), N * sizeof(int), cudaMemcpyHostToDevice, s->stream));
    EXF_CUDA(cudaMemcpyAsync(L.ilu_ord_up.p, up.data(), N * sizeof(int), cudaMemcpyHostToDevice, s->stream));
    EXF_CUDA(cudaStreamSynchronize(s->stream));
    EXF_TRY(build_streams(s, L, ptr, col, dp));
    // (entries in 24 bits, places in 8)
    if (m <= kFacMax && N <= (1 << 18) && L.nqq < (1 << 24) - 1 && fac_one_cta(N, L.ilu_depth[0]))
      EXF_TRY(build_places(s, L, lv));
    L.ilu_maxl = m;
    s->buf_epoch++;
  }
  if (L.ilu_maxl > 128) {
    set_error("ILU: a row of level %d has %d entries left of the diagonal (at most 127 supported)", lev,
              L.ilu_maxl - 1);
    return EXF_ERR_UNSUPPORTED;
  }
  if (L.ilu_f.n != (size_t)L.nqq) {
    EXF_TRY(L.ilu_f.alloc(L.nqq));
    EXF_TRY(L.ilu_inv.alloc(N));
    EXF_TRY(L.ilu_flag.alloc(N));
    EXF_TRY(L.ilu_flag.zero(s->stream));
    EXF_TRY(L.ilu_ctl.alloc(4));
    EXF_TRY(L.ilu_ctl.zero(s->stream));
    s->buf_epoch++;
  }
  EXF_CUDA(cudaMemcpyAsync(L.ilu_f.p, L.A.vv.p, L.nqq * sizeof(double), cudaMemcpyDeviceToDevice, s->stream));
  EXF_CUDA(cudaMemsetAsync(L.ilu_ctl.p + 2, 0, sizeof(int), s->stream));
  if (L.ilu_row.p) {
    k_ilu_factor_cta<<<1, 1024, 0, s->stream>>>(L.ilu_depth[0], L.ilu_loff.p, L.ilu_row.p, L.ilu_ent.p, L.ilu_pos.p,
                                                L.ilu_f.p, L.ilu_inv.p, L.ilu_ctl.p);
    EXF_COUNT(1);
    EXF_LAUNCH_CHECK();
  } else if (L.ilu_maxl <= 16) EXF_TRY((launch_factor<16, 2>(s, L)));
  else if (L.ilu_maxl <= 32) EXF_TRY((launch_factor<32, 2>(s, L)));
  else if (L.ilu_maxl <= 64) EXF_TRY((launch_factor<64, 2>(s, L)));
  else EXF_TRY((launch_factor<128, 1>(s, L)));
  if (L.ilu_nsrc) {
    k_ilu_stream<<<(L.ilu_nsrc + 255) / 256, 256, 0, s->stream>>>(L.ilu_src.p, L.ilu_nsrc, L.ilu_f.p, L.ilu_inv.p,
                                                                  reinterpret_cast<double *>(L.ilu_str.p));
    EXF_COUNT(1);
    EXF_LAUNCH_CHECK();
  }
  int zp = 0;
  EXF_CUDA(cudaMemcpyAsync(&zp, L.ilu_ctl.p + 2, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
  EXF_CUDA(cudaStreamSynchronize(s->stream));
  EXF_TRY(device_wait_status(s));
  if (zp) {
    set_error("ILU: zero pivot in row %d of level %d (LASZeroPivotErr)", zp - 1, lev);
    return EXF_ERR_SINGULAR;
  }
  L.ilu_ok = true;
  return EXF_OK;
}

int ilu_apply(exf_sys *s, int lev, const double *c, double *y) {
  EXF_TRY(ilu_ready(s, lev));
  SysLevel &L = s->L[lev];
  if (L.gm_w.n < (size_t)L.ndof) EXF_TRY(L.gm_w.alloc(L.ndof));
  return ilu_apply_dev(s, lev, c, y, nullptr);
}

// one call of the level solver: GMRESIter(A, x, b, m, ILUPrecond) with RTC accuracy eps;
// with acc, *acc = the squared residual of its last test (LastAcc times ||b||)
int gmres_smooth(exf_sys *s, int lev, double eps, int m, double *x, const double *b, double *acc) {
  EXF_TRY(ilu_ready(s, lev));
  SysLevel &L = s->L[lev];
  const long n = L.ndof;
  const int kmax = std::min(m, kGmSteps);
  if (L.gm_V.n < (size_t)(kmax + 1) * n || L.gm_w.n < (size_t)n || L.gm_t.n < (size_t)n || !L.gm_sc.p) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    EXF_CUDA(cudaStreamIsCapturing(s->stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) {
      set_error("GMRES work space of level %d sized inside a graph capture", lev);
      return EXF_ERR_STATE;
    }
    if (L.gm_V.n < (size_t)(kmax + 1) * n) EXF_TRY(L.gm_V.alloc((size_t)(kmax + 1) * n));
    if (L.gm_w.n < (size_t)n) EXF_TRY(L.gm_w.alloc(n));
    if (L.gm_t.n < (size_t)n) EXF_TRY(L.gm_t.alloc(n));
    if (!L.gm_sc.p) {
      EXF_TRY(L.gm_sc.alloc(kGmScalars));
      EXF_TRY(L.gm_sc.zero(s->stream));
      EXF_TRY(L.gm_ctl.alloc(4));
    }
    s->buf_epoch++;
  }
  double *sc = L.gm_sc.p, *V = L.gm_V.p;
  int *ctl = L.gm_ctl.p;
  auto vk = [&](int k) { return V + (long)(k - 1) * n; };  // v[k], 1-based
  const unsigned g = (unsigned)((n + 255) / 256);
  const bool small = (size_t)n * sizeof(double) <= kGmSmem;  // one CTA per step
  if (small)
    EXF_CUDA(cudaFuncSetAttribute(k_gm_step, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGmSmem));
  auto step = [&](int i) {
    k_gm_step<<<1, kGmCta, (size_t)n * sizeof(double), s->stream>>>(V, (int)n, i, sc, ctl);
    EXF_COUNT(1);
  };
  if (small) {
    EXF_TRY(spmv_resid<double>(s, lev, x, b, vk(1), sc + 1));  // v[1] = b - A x
    k_gm_begin<<<1, kGmCta, 0, s->stream>>>(b, (int)n, sc, ctl, eps);
    EXF_COUNT(1);
  } else {
    k_gm_reset<<<1, 1, 0, s->stream>>>(ctl);
    EXF_TRY(dot_dev(s, L, b, b, n, sc));                       // bNorm
    EXF_TRY(spmv_resid<double>(s, lev, x, b, vk(1), sc + 1));  // v[1] = b - A x
  }
  for (int iter = 0; iter < m;) {
    if (!small || iter > 0) {
      k_gm_rtc<<<1, 1, 0, s->stream>>>(sc, ctl, eps);
      EXF_COUNT(1);
    }
    EXF_TRY(ilu_apply_dev(s, lev, vk(1), vk(1), ctl));
    if (small) {
      step(0);
    } else {
      EXF_TRY(dot_dev(s, L, vk(1), vk(1), n, sc + 2));
      k_gm_first<<<1, 1, 0, s->stream>>>(sc);
      k_gm_scale<<<g, 256, 0, s->stream>>>(vk(1), n, sc + 4, ctl);
      EXF_COUNT(2);
    }
    const int ni = std::min(kGmSteps, m - iter);
    for (int i = 1; i <= ni; i++) {
      EXF_TRY(spmv_resid<double>(s, lev, vk(i), nullptr, L.gm_t.p, nullptr));  // A v[i]
      EXF_TRY(ilu_apply_dev(s, lev, L.gm_t.p, vk(i + 1), ctl));
      if (small) {
        step(i);
        continue;
      }
      for (int k = 1; k <= i; k++) {  // modified Gram-Schmidt
        EXF_TRY(dot_dev(s, L, vk(i + 1), vk(k), n, sc + gmH(i, k)));
        k_gm_axpy<<<g, 256, 0, s->stream>>>(vk(i + 1), vk(k), n, sc + gmH(i, k), ctl);
        EXF_COUNT(1);
      }
      EXF_TRY(dot_dev(s, L, vk(i + 1), vk(i + 1), n, sc + 2));
      k_gm_qr<<<1, 1, 0, s->stream>>>(sc, i);
      k_gm_scale<<<g, 256, 0, s->stream>>>(vk(i + 1), n, sc + 4, ctl);
      EXF_COUNT(2);
    }
    iter += ni;
    k_gm_solve<<<1, 1, 0, s->stream>>>(sc, ni);
    k_gm_update<<<g, 256, 0, s->stream>>>(x, V, n, ni, sc, ctl);
    EXF_COUNT(2);
    EXF_TRY(spmv_resid<double>(s, lev, x, b, vk(1), sc + 1));  // the new residual
  }
  if (acc) {
    k_gm_copy<<<1, 1, 0, s->stream>>>(sc + 1, acc);
    EXF_COUNT(1);
  }
  EXF_LAUNCH_CHECK();
  return EXF_OK;
}

}  // namespace exf
