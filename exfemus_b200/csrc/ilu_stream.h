// ilu_stream.h -- the order and the records in which one CTA solves a level's triangular
// systems (k_ilu_tri, ilu_gmres.cu).  Host code on plain arrays, no CUDA types, so that the
// rules the kernel rests on can be checked without a device.
#pragma once
#include <algorithm>
#include <cstdint>
#include <utility>
#include <vector>

namespace exf {

constexpr int kTriE = 24, kTriStages = 4, kTriWarps = 4;
constexpr int tri_words(int M) { return 41 + 24 * M; }  // M: a multiple of 4
constexpr int kTriWords = 2 * tri_words(kTriE);         // a stage: two records at least

struct TriWord {
  uint32_t x, y, z, w;
};
struct TriPair {
  int x, y;
};
struct TriStream {
  std::vector<TriWord> str;
  std::vector<TriPair> src;    // {double of the stream, entry of the factor or ~row of 1 / d}
  std::vector<TriPair> chunk;  // {first word, words}
  int nrec[2] = {0, 0};        // records of the lower, the upper solve
  int depth[2] = {0, 0};       // their dependency levels
  uint32_t first[kTriWarps] = {0};  // places of the first records, from chunk 0
};

// The rows in the order their tickets hand them out: by dependency level (the longest
// chain of lower, or upper, entries leading to the row), index order within a level.
// Every row depends only on rows of earlier levels, so a warp still waits only on earlier
// tickets, and the rows of a level run together instead of one index after the other
// (consecutive rows of the level-nested numbering mostly depend on each other).
// Returns the number of levels.
inline int level_order(const std::vector<int> &ptr, const std::vector<int> &col, const std::vector<int> &dp, bool upper,
                       std::vector<int> &ord, std::vector<int> *level = nullptr) {
  const int N = (int)dp.size();
  std::vector<int> lv(N, 0);
  int nl = 0;
  for (int q = 0; q < N; q++) {
    const int i = upper ? N - 1 - q : q;
    int l = 0;
    const int a = upper ? dp[i] + 1 : ptr[i], e = upper ? ptr[i + 1] : dp[i];
    for (int k = a; k < e; k++) l = std::max(l, lv[col[k]] + 1);
    lv[i] = l;
    nl = std::max(nl, l + 1);
  }
  std::vector<int> cnt(nl + 1, 0);
  for (int i = 0; i < N; i++) cnt[lv[i] + 1]++;
  for (int l = 0; l < nl; l++) cnt[l + 1] += cnt[l];
  ord.assign(N, 0);
  for (int i = 0; i < N; i++) ord[cnt[lv[i]]++] = i;
  if (level) *level = std::move(lv);
  return nl;
}

// The streams of one level from its pattern (ptr, col, diagonal entries dp): the rows by
// dependency level, a level's rows longest first, consecutive records packed into chunks.
// Records of up to 32 rows of one level and up to kTriE entries of each, in planes of 32:
//   {groups of 4 entries, 1: first of its rows | 2: last | 4: last of its chunk, 16-byte
//   words, place of the record kTriWarps on: chunks ahead << 24 | word in the chunk},
//   row[32], 1 / d [32], d[32], index[entries][32], value[entries][32]
// A row of more entries continues in the next record.  Absent entries and rows point to
// index N.  The place is what a warp needs to go from its record to its next: it never reads
// the header of a record it does not solve, since that record's chunk may be over (its
// stage handed to the next chunk) by the time it would.
inline TriStream build_tri_stream(const std::vector<int> &ptr, const std::vector<int> &col, const std::vector<int> &dp) {
  TriStream T;
  const int N = (int)dp.size();
  std::vector<TriPair> rec;  // {chunk, first word}
  for (int up = 0; up < 2; up++) {
    std::vector<int> ord, lv;
    T.depth[up] = level_order(ptr, col, dp, up == 1, ord, &lv);
    auto len = [&](int i) { return up ? ptr[i + 1] - 1 - dp[i] : dp[i] - ptr[i]; };
    for (int a = 0; a < N;) {
      int e = a;
      while (e < N && lv[ord[e]] == lv[ord[a]]) e++;
      std::stable_sort(ord.begin() + a, ord.begin() + e, [&](int x, int y) { return len(x) > len(y); });
      for (; a < e; a += 32) {
        const int R = std::min(32, e - a), most = len(ord[a]);
        for (int j0 = 0; j0 == 0 || j0 < most; j0 += kTriE) {
          const int M = (std::min(kTriE, most - j0) + 3) & ~3, w = tri_words(M);
          const size_t o = T.str.size();
          if (T.chunk.empty() || T.chunk.back().y + w > kTriWords) T.chunk.push_back({(int)o, 0});
          T.chunk.back().y += w;
          rec.push_back({(int)T.chunk.size() - 1, (int)o});
          T.nrec[up]++;
          T.str.resize(o + w, TriWord{0u, 0u, 0u, 0u});
          T.str[o] = {(uint32_t)M / 4, (j0 == 0 ? 1u : 0u) | (j0 + kTriE >= most ? 2u : 0u), (uint32_t)w, 0u};
          int *row = reinterpret_cast<int *>(&T.str[o + 1]), *ix = reinterpret_cast<int *>(&T.str[o + 41]);
          for (int k = 0; k < 32; k++) row[k] = N;
          for (int k = 0; k < 32 * M; k++) ix[k] = N;
          for (int r = 0; r < R; r++) {
            const int i = ord[a + r];
            row[r] = i;
            T.src.push_back({(int)(2 * (o + 9)) + r, ~i});
            T.src.push_back({(int)(2 * (o + 25)) + r, dp[i]});
            for (int j = j0; j < std::min(len(i), j0 + M); j++) {
              const int k = up ? ptr[i + 1] - 1 - j : ptr[i] + j;  // upper: from the row's end
              ix[(j - j0) * 32 + r] = col[k];
              T.src.push_back({(int)(2 * (o + 41 + 8 * M)) + (j - j0) * 32 + r, k});
            }
          }
        }
      }
      a = e;
    }
  }
  auto place = [&](const TriPair &r, int from) {
    return (uint32_t)(r.x - from) << 24 | (uint32_t)(r.y - T.chunk[r.x].x);
  };
  for (size_t k = 0; k < rec.size(); k++) {
    if (k < kTriWarps) T.first[k] = place(rec[k], 0);
    if (k + kTriWarps < rec.size()) T.str[rec[k].y].w = place(rec[k + kTriWarps], rec[k].x);
    if (k + 1 == rec.size() || rec[k + 1].x != rec[k].x) T.str[rec[k].y].y |= 4u;
  }
  return T;
}

// One CTA solves record after record, 0.31 us each; the kernels on all SMs pay a round trip
// through L2 per dependency level, 3.0 us in 2D and 5 to 6.4 us in 3D.  ILUPrecond, one CTA
// and all SMs (us): level-nested numbering 65 x 65 nodes (442 records, 390 levels) 138 and
// 1172, 129 x 129 (1379, 774) 415 and 2339, 25^3 (2858, 582) 860 and 3735; numbered at random
// within each nesting class, where levels are few and wide, 65 x 65 (296, 54) 97 and 190,
// 129 x 129 (1064, 50) 336 and 185, 25^3 (2045, 240) 641 and 1221.
inline bool tri_one_cta(const int nrec[2], const int depth[2]) {
  return nrec[0] + nrec[1] <= 9 * (depth[0] + depth[1]);
}
// The factorisation (rows of at most kFacMax entries up to the diagonal): one CTA takes 3 us
// and 0.2 us per row of a level's 32-row rounds, all SMs 25 us per level.  Factorisation, one
// CTA and all SMs (ms), level-nested numbering: 33 x 33 nodes (11 rows per level) 0.62 and
// 2.4, 65 x 65 (22) 1.5 and 4.9, 129 x 129 (43) 4.5 and 9.9, 257 x 257 (86) 15.9 and 19.9.
inline bool fac_one_cta(int N, int depth) { return N <= 100 * depth; }

}  // namespace exf
