// mg_cluster_plan.h -- which CTA, warp and step of the cluster kernel (mg_cluster.cu) updates
// which row of a scalar level, and which levels fit one launch.  Host code on plain arrays,
// no CUDA types, so that the rules the kernel's exchange rests on can be checked without a
// device.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace exf {

constexpr int kCluMaxLev = 10;
constexpr size_t kCluSmem = 224 * 1024;  // dynamic shared memory of a CTA
constexpr size_t kCluRep = 152 * 1024;   // of these, the iterate at most

struct CluRow {  // a row group's row in one step
  int pos, k0, len, diag;  // position or -1 (none), first entry, entries (0: padding), diagonal - first
};
struct CluStep {
  int next, flags;  // positions of the colour after its own, of the one before << 16 (both
                    // cyclic); 1: last step of its colour, 2: first step of it
};
struct CluPlan {
  int act = 1;      // CTAs that share the level
  int entries = 0;  // most matrix entries of a CTA, a multiple of 4
  std::vector<int> node, pos;  // node at each position (-1 padding), position of each node
  std::vector<CluStep> step;   // steps of a sweep
  std::vector<CluRow> tab;     // [act][steps][groups]
  std::vector<int> first;      // [act][steps][groups] first of the row's entries in the CTA's copy
};

// qp: row pointers, diag: absolute diagonal entries, items: the nodes by colour; lpr lanes
// per row, CTAs of nt threads, `most` CTAs in the cluster; less than 2^15 positions.
//
// Positions are the nodes in colour order (a colour's rows longest first, so that a warp's
// rows are alike, each colour padded to whole warps); a colour's units of one warp are dealt
// round-robin to the CTAs.  A CTA's send in a colour tells the others that it has seen the
// colour before complete, and its two mbarriers serve alternate colours: so EVERY CTA has a
// unit in EVERY colour.  A colour with fewer units than CTAs gets units of padding.
inline CluPlan plan_cluster(int N, const int *qp, const int *diag, int ncolour, const int *col_off, const int *items,
                            int lpr, int nt, int most) {
  CluPlan P;
  const int gc = nt / lpr, rw = 32 / lpr, nw = nt / 32;
  int rows = 0;
  for (int c = 0; c < ncolour; c++) rows = std::max(rows, col_off[c + 1] - col_off[c]);
  // CTA 0 alone where a colour's rows fit its groups (its barrier costs a fifth of an
  // exchange), otherwise the whole cluster (just enough CTAs for the rows: 2-6% slower)
  P.act = rows <= gc ? 1 : most;
  P.pos.assign(N, -1);
  int longest = 0;
  for (int i = 0; i < N; i++) longest = std::max(longest, qp[i + 1] - qp[i]);
  std::vector<int> cbase(ncolour), rounds(ncolour), units(ncolour), at(longest + 1), used;
  for (int c = 0; c < ncolour; c++) {
    const int n = col_off[c + 1] - col_off[c];
    units[c] = (n + rw - 1) / rw;
    if (n > 0 && P.act > 1) units[c] = std::max(units[c], P.act);
    cbase[c] = (int)P.node.size();
    P.node.resize(cbase[c] + units[c] * rw, -1);
    // longest rows first, rows of one length in the items' order
    std::fill(at.begin(), at.end(), 0);
    for (const int *v = items + col_off[c]; v != items + col_off[c + 1]; v++) at[qp[*v + 1] - qp[*v]]++;
    for (int len = longest, p = cbase[c]; len >= 0; len--) {
      const int k = at[len];
      at[len] = p;
      p += k;
    }
    for (const int *v = items + col_off[c]; v != items + col_off[c + 1]; v++) {
      const int p = at[qp[*v + 1] - qp[*v]]++;
      P.node[p] = *v;
      P.pos[*v] = p;
    }
    rounds[c] = (units[c] + P.act * nw - 1) / (P.act * nw);
    if (rounds[c] > 0) used.push_back(c);
  }
  for (size_t k = 0; k < used.size(); k++) {
    const int c = used[k], after = used[(k + 1) % used.size()], before = used[(k + used.size() - 1) % used.size()];
    for (int r = 0; r < rounds[c]; r++)
      P.step.push_back({units[after] * rw | units[before] * rw << 16, (r == rounds[c] - 1 ? 1 : 0) | (r == 0 ? 2 : 0)});
  }
  const int steps = (int)P.step.size();
  P.tab.assign((size_t)P.act * steps * gc, CluRow{-1, 0, 0, -1});
  int st0 = 0;
  for (int c = 0; c < ncolour; c++) {
    int cta = 0, slot = st0 * gc;  // of the unit: slot = step, warp and group
    for (int u = 0, p = cbase[c]; u < units[c]; u++) {
      CluRow *t = &P.tab[(size_t)cta * steps * gc + slot];
      for (int g = 0; g < rw; g++, p++) {
        const int v = P.node[p];
        if (v >= 0) t[g] = {p, qp[v], qp[v + 1] - qp[v], diag[v] - qp[v]};
        else if (g == 0) t[g] = {p, 0, 0, -1};  // a unit of padding: it sends, nothing reads it
      }
      if (++cta == P.act) {
        cta = 0;
        slot += rw;
      }
    }
    st0 += rounds[c];
  }
  P.first.assign(P.tab.size(), 0);
  for (int r = 0; r < P.act; r++) {
    int at = 0;
    for (size_t q = (size_t)r * steps * gc; q < (size_t)(r + 1) * steps * gc; q++) {
      P.first[q] = at;
      at += P.tab[q].len;
    }
    P.entries = std::max(P.entries, (at + 3) & ~3);
  }
  return P;
}

// Most rows of a level that is faster in the cluster than with a launch per colour, with
// `sweeps` sweeps per cycle.  A sweep in the cluster grows with the rows (16 SMs) while
// launches cost the same up to here, and the restriction, prolongation and residual that go
// with the level lose from the start.  V-cycle down from such a level, cluster and launches
// (us): 2D FP64 9,409 rows 2 sweeps 122 and 120, 12,769 rows 2 sweeps 135 and 124, 4 sweeps
// 188 and 187, 16,641 rows 8 sweeps 329 and 320, 12 sweeps 446 and 447; FP32 12,769 rows 4
// sweeps 163 and 166, 16,641 rows 4 sweeps 177 and 170, 8 sweeps 261 and 277, 25,921 rows 12
// sweeps 446 and 396; 6,561 rows 1 sweep 91 and 93, 0 sweeps 73 and 64.  3D FP32 18,785 rows 2
// sweeps 230 and 231, 25,625 rows 2 sweeps 247 and 239, 4 sweeps 373 and 394, 30,625 rows 8
// sweeps 733 and 707; FP64 18,785 rows 1 sweep 195 and 201, 2 sweeps 264 and 298.
constexpr int cluster_rows(int dim, int sweeps) {
  return sweeps < 1    ? 0
         : dim == 3    ? 26000 - 14000 / sweeps
         : sweeps == 1 ? 6600
                       : 18300 - 18000 / sweeps;
}

// Dynamic shared memory of a CTA: the step tables (rows, reciprocals, rhs), the steps, the
// iterate and the copied entries, sized for the largest of a launch's levels each
constexpr size_t cluster_smem(size_t elem, int gc, int steps, int xlen, int mlen) {
  return (size_t)steps * gc * (16 + 2 * elem) + (size_t)steps * 8 + (size_t)xlen * elem + (size_t)mlen * (4 + elem);
}

struct CluShape {
  int act = 1, steps = 0, xlen = 0, mlen = 0;  // CTAs, most steps, longest iterate, most entries of a CTA
  int mat[kCluMaxLev] = {0};                   // entries of a CTA in shared memory per level (0: not there)
  size_t smem = 0;
};
// Whether levels hi .. 1 fit one launch with values of `elem` bytes, and its sizes; lev(l)
// gives a level's ok, act, steps, Np and entries.  Both the choice of the cluster path and
// the launch use this.  CTAs above 0 leave the descent at the first level of one CTA, so a
// coarser level must not need more CTAs than a finer one.
template <class Lev>
inline bool cluster_shape(int hi, size_t elem, int gc, Lev lev, CluShape &S) {
  S = CluShape();
  if (hi < 1 || hi >= kCluMaxLev) return false;
  for (int l = 1; l <= hi; l++) {
    const auto &C = lev(l);
    if (!C.ok || (size_t)C.Np * elem > kCluRep || C.act < S.act) return false;
    S.act = C.act;
    S.steps = std::max(S.steps, (C.steps + 1) & ~1);  // 16-byte alignment of what follows the steps
    S.xlen = std::max(S.xlen, (C.Np + 3) & ~3);
  }
  if (cluster_smem(elem, gc, S.steps, S.xlen, 0) > kCluSmem) return false;
  for (int l = 1; l <= hi; l++) {  // the rows' entries of the levels where they fit beside the tables
    const int n = lev(l).entries;
    S.mat[l] = n > 0 && cluster_smem(elem, gc, S.steps, S.xlen, n) <= kCluSmem ? n : 0;
    S.mlen = std::max(S.mlen, S.mat[l]);
  }
  S.smem = cluster_smem(elem, gc, S.steps, S.xlen, S.mlen);
  return true;
}

}  // namespace exf
