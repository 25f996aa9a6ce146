"""The record stream of the one-CTA triangular solves (csrc/ilu_stream.h, host code compiled
here with g++): the places lead each warp through its own records without a look at another
one's, and the records in order, replayed as the kernel solves them, give the triangular
solves bit for bit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "exfemus_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "ilu_stream.h"
template <class T> static void all(const T &v) { for (auto &p : v) printf("%d %d ", p.x, p.y); }
int main() {
  int N;
  if (scanf("%d", &N) != 1) return 1;
  std::vector<int> ptr(N + 1, 0), dp(N), col;
  for (int i = 0; i < N; i++) {
    int n;
    if (scanf("%d", &n) != 1) return 1;
    ptr[i + 1] = ptr[i] + n;
    for (int k = 0, c; k < n; k++) {
      if (scanf("%d", &c) != 1) return 1;
      if (c == i) dp[i] = ptr[i] + k;
      col.push_back(c);
    }
  }
  const exf::TriStream T = exf::build_tri_stream(ptr, col, dp);
  printf("%d %d %d %d ", exf::tri_one_cta(T.nrec, T.depth), exf::fac_one_cta(N, T.depth[0]), T.depth[0], T.depth[1]);
  printf("%d %d %d %d %d %d %d %d ", exf::kTriStages, exf::kTriWarps, exf::kTriWords, (int)T.str.size(),
         (int)T.src.size(), (int)T.chunk.size(), T.nrec[0], T.nrec[1]);
  for (int w = 0; w < exf::kTriWarps; w++) printf("%u ", T.first[w]);
  all(T.chunk);
  all(T.src);
  for (auto &w : T.str) printf("%u %u %u %u ", w.x, w.y, w.z, w.w);
}
"""


@pytest.fixture(scope="module")
def builder(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("stream")
    (d / "s.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / "s.cpp"), "-o", str(d / "s")], check=True)

    def run(rows):
        text = "%d\n" % len(rows) + "\n".join("%d %s" % (len(r), " ".join(map(str, r))) for r in rows)
        out = subprocess.run([str(d / "s")], input=text, capture_output=True, text=True, check=True).stdout.split()
        v = np.array([int(x) for x in out], np.int64)
        cta, v = v[:4], v[4:]
        stages, warps, words, nstr, nsrc, nch, lo, up = v[:8]
        o = 8 + warps
        first = v[8:o]
        chunk, o = v[o:o + 2 * nch].reshape(nch, 2), o + 2 * nch
        src, o = v[o:o + 2 * nsrc].reshape(nsrc, 2), o + 2 * nsrc
        return dict(stages=stages, warps=warps, words=words, first=first, chunk=chunk, src=src,
                    str=v[o:].reshape(nstr, 4).astype(np.uint32), nlo=lo, nrec=lo + up, tri_cta=bool(cta[0]),
                    fac_cta=bool(cta[1]), depth=cta[2:])

    return run


def lattice(nx, ny, seed=None):
    """Quad9 rows of an (nx x ny)-node lattice; nodes renumbered at random for a seed."""
    at = np.arange(nx * ny) if seed is None else np.random.default_rng(seed).permutation(nx * ny)
    rows = [set() for _ in range(nx * ny)]
    for ey in range(0, ny - 1, 2):
        for ex in range(0, nx - 1, 2):
            el = [int(at[(ey + j) * nx + ex + i]) for j in range(3) for i in range(3)]
            for a in el:
                rows[a].update(el)
    return [sorted(r) for r in rows]


def arrow(n):
    """One long last row (several records), and wide levels before it."""
    rows = [[i, n - 1] for i in range(n - 1)]
    return rows + [list(range(n))]


CASES = {"one": [[0]], "two": [[0, 1], [0, 1]], "lattice": lattice(17, 9), "random": lattice(33, 17, 1),
         "arrow": arrow(83)}


@pytest.mark.parametrize("name", list(CASES))
def test_places_lead_through_the_own_records(builder, name):
    t = builder(CASES[name])
    chunk, words = t["chunk"], t["str"]
    assert np.all(chunk[:, 1] <= t["words"]) and chunk[:, 1].sum() == len(words)
    order = []  # records in stream order: (chunk, word in the chunk)
    for c, (start, n) in enumerate(chunk):
        at = 0
        while at < n:
            order.append((c, at))
            at += int(words[start + at][2])
        assert at == n
    assert len(order) == t["nrec"]
    last = [k + 1 == len(order) or order[k + 1][0] != order[k][0] for k in range(len(order))]
    for w in range(min(t["warps"], t["nrec"])):
        c, place = 0, int(t["first"][w])
        for k in range(w, t["nrec"], t["warps"]):
            ahead = place >> 24
            # the stage of the next chunk held an earlier chunk that this warp, or the owner
            # of a record solved before its own, has been in
            assert ahead <= t["stages"]
            c += ahead
            assert (c, place & 0xffffff) == order[k]
            head = words[chunk[c][0] + (place & 0xffffff)]
            assert bool(head[1] & 4) == last[k]
            place = int(head[3])


@pytest.mark.parametrize("name", list(CASES))
def test_replayed_records_are_the_triangular_solves(builder, name):
    rows = CASES[name]
    N = len(rows)
    t = builder(rows)
    rng = np.random.default_rng(7)
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    f = rng.standard_normal(ptr[-1])
    dp = np.array([ptr[i] + rows[i].index(i) for i in range(N)])
    inv = 1.0 / f[dp]
    c = rng.standard_normal(N)
    val = np.ascontiguousarray(t["str"]).reshape(-1).view(np.float64).copy()
    for at, e in t["src"]:
        val[at] = f[e] if e >= 0 else inv[~e]
    ints = t["str"].reshape(-1).view(np.int32)
    v, part = np.append(c, 0.0), np.zeros(32)
    k = o = 0
    while o < len(t["str"]):
        g, flags, n, _ = (int(x) for x in t["str"][o])
        for lane in range(32):
            i = ints[4 * (o + 1) + lane]
            s = 0.0 if flags & 1 else part[lane]
            for u in range(4 * g):
                s = s - val[2 * (o + 41 + 8 * 4 * g) + 32 * u + lane] * v[ints[4 * (o + 41) + 32 * u + lane]]
            own = v[i] if k < t["nlo"] else 0.0 + val[2 * (o + 25) + lane] * v[i]
            if flags & 2:
                v[i] = (s + own) * val[2 * (o + 9) + lane]
            else:
                part[lane] = s
        o, k = o + n, k + 1
    w, y = np.zeros(N), np.zeros(N)
    for i in range(N):
        s = 0.0
        for q in range(ptr[i], dp[i]):
            s = s - f[q] * w[rows[i][q - ptr[i]]]
        w[i] = (s + c[i]) * inv[i]
    for i in range(N - 1, -1, -1):
        s = 0.0
        for q in range(ptr[i + 1] - 1, dp[i], -1):
            s = s - f[q] * y[rows[i][q - ptr[i]]]
        y[i] = (s + (0.0 + f[dp[i]] * w[i])) * inv[i]
    assert k == t["nrec"] and v[N] == 0.0
    assert np.array_equal(v[:N], y)


def test_wide_levels_stay_on_all_sms(builder):
    """Narrow levels (a row depends on the one before) go to one CTA, few wide levels do not."""
    t = builder(lattice(33, 17))
    assert t["tri_cta"] and t["fac_cta"]
    t = builder(lattice(129, 129, 3))
    assert sum(t["depth"]) < 100 and t["nrec"] > 1000
    assert not t["tri_cta"] and not t["fac_cta"]
    t = builder(lattice(65, 65, 3))  # a third of the records a level: still the one CTA's
    assert t["tri_cta"]
