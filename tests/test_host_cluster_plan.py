"""How the cluster kernel's rows are dealt to CTAs and warps (csrc/mg_cluster_plan.h, host
code compiled here with g++), and a model of the kernel's exchange on such plans: warps and
messages proceed in any order that the two mbarriers of a CTA admit."""
import os
import random
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "exfemus_b200", "csrc")
NT, MOST = 512, 16

PROGRAM = r"""
#include <cstdio>
#include "mg_cluster_plan.h"
int main() {
  int N, nc, lpr, nt, most;
  if (scanf("%d %d %d %d %d", &N, &nc, &lpr, &nt, &most) != 5) return 1;
  std::vector<int> qp(N + 1, 0), diag(N), off(nc + 1, 0), col(N), items(N);
  for (int i = 0; i < N; i++) {
    int len;
    if (scanf("%d %d", &col[i], &len) != 2) return 1;
    qp[i + 1] = qp[i] + len;
    diag[i] = qp[i] + len / 2;
    off[col[i] + 1]++;
  }
  for (int c = 0; c < nc; c++) off[c + 1] += off[c];
  std::vector<int> at(off.begin(), off.end() - 1);
  for (int i = 0; i < N; i++) items[at[col[i]]++] = i;
  const exf::CluPlan P = exf::plan_cluster(N, qp.data(), diag.data(), nc, off.data(), items.data(), lpr, nt, most);
  printf("%d %d %d %d\n", P.act, P.entries, (int)P.node.size(), (int)P.step.size());
  for (int v : P.node) printf("%d ", v);
  for (int v : P.pos) printf("%d ", v);
  for (auto &s : P.step) printf("%d %d ", s.next, s.flags);
  for (size_t q = 0; q < P.tab.size(); q++)
    printf("%d %d %d %d %d ", P.tab[q].pos, P.tab[q].k0, P.tab[q].len, P.tab[q].diag, P.first[q]);
}
"""


def compile_cpp(d, name):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / (name + ".cpp")), "-o", str(d / name)], check=True)


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(PROGRAM)
    compile_cpp(d, "plan")

    def run(colour, length, lpr):
        nc = int(colour.max()) + 1
        text = "%d %d %d %d %d\n" % (colour.size, nc, lpr, NT, MOST)
        text += "\n".join("%d %d" % cl for cl in zip(colour, length))
        out = subprocess.run([str(d / "plan")], input=text, capture_output=True, text=True, check=True).stdout.split()
        v = np.array([int(x) for x in out])
        act, entries, npos, steps = v[:4]
        o = 4
        node, o = v[o:o + npos], o + npos
        pos, o = v[o:o + colour.size], o + colour.size
        step, o = v[o:o + 2 * steps].reshape(steps, 2), o + 2 * steps
        tab = v[o:].reshape(act, steps, NT // lpr, 5)
        return dict(act=act, entries=entries, node=node, pos=pos, step=step, tab=tab, rw=32 // lpr,
                    nw=NT // 32)

    return run


def lattice(*n):
    """Colours i % 3 + 3 (j % 3) + 9 (k % 3) and row lengths of a Q2 lattice."""
    idx = np.indices(n[::-1])[::-1]
    colour = sum((3 ** d) * (i % 3) for d, i in enumerate(idx))
    length = np.prod([np.where(i % 2 == 0, np.where((i == 0) | (i == m - 1), 3, 5), 3) for i, m in zip(idx, n)], axis=0)
    return colour.ravel(), length.ravel()


def uneven(*sizes):
    """A first-fit colouring's shape: large first colours, a few nodes in the last."""
    rng = np.random.default_rng(len(sizes))
    colour = rng.permutation(np.repeat(np.arange(len(sizes)), sizes))
    return colour, rng.integers(9, 26, colour.size)


LEVELS = {
    "33x17": (lattice(33, 17), 8),     # 55 rows a colour in the last line class: 14 warps of rows for 16 CTAs
    "17x9": (lattice(17, 9), 8),       # one CTA
    "129x129": (lattice(129, 129), 8),  # several rounds a colour
    "17x5x9": (lattice(17, 5, 9), 16),
    "65x17x17": (lattice(65, 17, 17), 16),
    "uneven": (uneven(300, 260, 90, 65, 40, 7, 1, 1), 8),
    "empty colour": (lattice(200, 2), 8),
    "uneven3d": (uneven(200, 33, 32, 31, 5, 2, 1, 1, 1), 16),
}


def units(p):
    """units[colour][cta][warp]: bytes / 4 of the values that the warp sends in the colour."""
    ends = np.cumsum((p["step"][:, 1] & 2) > 0) - 1
    out = np.zeros((ends[-1] + 1, p["act"], p["nw"]), int)
    lead = p["tab"][:, :, ::p["rw"], 0]  # position of a warp's first group: -1 sends nothing
    for s in range(len(ends)):
        out[ends[s]] += (lead[:, s, :] >= 0) * p["rw"]
    return out


@pytest.mark.parametrize("name", list(LEVELS))
def test_plan(planner, name):
    (colour, length), lpr = LEVELS[name]
    p = planner(colour, length, lpr)
    pos, node, tab, rw = p["pos"], p["node"], p["tab"], p["rw"]
    assert np.array_equal(node[pos], np.arange(colour.size)) and (node >= 0).sum() == colour.size
    rows = tab[tab[..., 2] > 0]
    assert np.array_equal(np.sort(rows[:, 0]), np.sort(pos))  # every row once
    qp = np.concatenate([[0], np.cumsum(length)])
    v = node[rows[:, 0]]
    assert np.array_equal(rows[:, 1], qp[v]) and np.array_equal(rows[:, 2], length[v])
    assert np.all((rows[:, 3] >= 0) & (rows[:, 3] < rows[:, 2]))
    assert (tab[..., 2].sum(axis=(1, 2)) <= p["entries"]).all()
    # a warp's groups hold consecutive positions from a multiple of the vector's length
    lead = tab[:, :, ::rw, 0]
    assert np.all((lead < 0) | (lead % rw == 0))
    # a step names the values that all CTAs together send in the colours around its own
    col_of_step = np.cumsum((p["step"][:, 1] & 2) > 0) - 1
    u = units(p)
    assert len(u) == len(np.unique(colour)) == ((p["step"][:, 1] & 1) > 0).sum()
    for c in range(len(u)):
        assert np.all(p["step"][col_of_step == c, 0] & 0xffff == u[(c + 1) % len(u)].sum())
        assert np.all(p["step"][col_of_step == c, 0] >> 16 == u[c - 1].sum())
    if p["act"] > 1:
        assert np.all(u.sum(axis=2) > 0), "a CTA sends nothing in a colour"


def exchange(u, sweeps, rng, all_warps_arrive=True):
    """Runs the exchange of sweep_level in a random order; returns what went wrong, or None."""
    ncol, act, nw = u.shape
    P = ncol * sweeps
    done = np.zeros((act, 2), int)          # completed phases of each mbarrier
    need = nw if all_warps_arrive else 1
    pend, tx = np.full((act, 2), need), np.zeros((act, 2), int)
    got = np.zeros((act, P), int)
    total = u.sum(axis=(1, 2))
    slow = rng.choice(["none", "cta", "warp"])
    who = rng.randrange(act), rng.randrange(nw)
    msgs, late = [], []

    def complete(r, b):
        if pend[r, b] == 0 and tx[r, b] == 0:
            done[r, b] += 1
            pend[r, b] = need

    def arrive(r, w, p):
        if p < P and (all_warps_arrive or w == 0):
            pend[r, p & 1] -= 1
            tx[r, p & 1] += total[p % ncol] if w == 0 else 0
            complete(r, p & 1)

    at = np.zeros((act, nw), int)
    sent = np.zeros((act, nw), bool)
    for r in range(act):
        for w in range(nw):
            arrive(r, w, 0)

    def step(r, w):
        p = at[r, w]
        if p >= P:
            return None, False
        if not sent[r, w]:
            sent[r, w] = True
            arrive(r, w, p + 1)  # it has seen colour p - 1
            if u[p % ncol, r, w]:
                for q in range(act):
                    (late if slow == "cta" and q == who[0] else msgs).append((q, p, u[p % ncol, r, w]))
            return None, True
        if (done[r, p & 1] & 1) == ((p >> 1) & 1):
            return None, False
        if got[r, p] != total[p % ncol]:
            return "cta %d warp %d passes colour %d before its values" % (r, w, p), True
        at[r, w], sent[r, w] = p + 1, False
        return None, True

    everyone = [(r, w) for r in range(act) for w in range(nw)]
    while True:
        moved = False
        for box in (msgs, late) if not msgs else (msgs,):
            for _ in range(rng.randint(0, len(box))):
                k = rng.randrange(len(box))
                box[k], box[-1] = box[-1], box[k]
                q, p, n = box.pop()
                got[q, p] += n
                tx[q, p & 1] -= n
                complete(q, p & 1)
                moved = True
        rng.shuffle(everyone)
        for r, w in everyone:
            if slow == "warp" and (r, w) == who and rng.random() < 0.9 and moved:
                continue
            bad, m = step(r, w)
            if bad:
                return bad
            moved = moved or m
        if np.all(at == P):
            return None
        if not moved and not msgs and not late and not any(step(r, w)[1] for r, w in everyone):
            return "a warp waits for a phase that is over"


@pytest.mark.parametrize("name", ["33x17", "17x5x9", "uneven", "uneven3d"])
def test_exchange_in_any_order(planner, name):
    (colour, length), lpr = LEVELS[name]
    u = units(planner(colour, length, lpr))
    if u.shape[1] == 1:
        pytest.skip("one CTA: no exchange")
    for seed in range(6):
        assert exchange(u, 2, random.Random(seed)) is None, seed


def test_the_model_sees_a_missing_unit_and_a_missing_arrival(planner):
    """Without the padding units, and with only one warp bound to the phases."""
    (colour, length), lpr = LEVELS["33x17"]
    u = units(planner(colour, length, lpr))
    bare = u.copy()
    bare[6:, 14:] = 0  # the last line class has 14 warps of rows
    assert any(exchange(bare, 2, random.Random(s)) for s in range(20))
    assert any(exchange(u, 2, random.Random(s), all_warps_arrive=False) for s in range(20))


SHAPE = r"""
#include <cstdio>
#include "mg_cluster_plan.h"
struct Lev { int ok, act, steps, Np, entries; };
int main() {
  int hi, elem, gc;
  if (scanf("%d %d %d", &hi, &elem, &gc) != 3) return 1;
  std::vector<Lev> L(hi + 1);
  for (int l = 1; l <= hi; l++)
    if (scanf("%d %d %d %d %d", &L[l].ok, &L[l].act, &L[l].steps, &L[l].Np, &L[l].entries) != 5) return 1;
  exf::CluShape S;
  const bool ok = exf::cluster_shape(hi, elem, gc, [&](int l) -> const Lev & { return L[l]; }, S);
  printf("%d %d %d %d %d %zu", ok, S.act, S.steps, S.xlen, S.mlen, S.smem);
  for (int l = 1; l <= hi && l < exf::kCluMaxLev; l++) printf(" %d", S.mat[l]);
}
"""


def test_levels_of_a_launch(tmp_path):
    """Levels that fit alone but not together, and a coarse level of more CTAs than the next."""
    (tmp_path / "shape.cpp").write_text(SHAPE)
    compile_cpp(tmp_path, "shape")

    def shape(levels, elem=8, gc=64):
        text = "%d %d %d\n" % (len(levels), elem, gc) + "\n".join("%d %d %d %d %d" % lev for lev in levels)
        out = subprocess.run([str(tmp_path / "shape")], input=text, capture_output=True, text=True, check=True)
        v = [int(x) for x in out.stdout.split()]
        return bool(v[0]), dict(act=v[1], steps=v[2], xlen=v[3], mlen=v[4], smem=v[5], mat=v[6:])

    smem = lambda steps, xlen, mlen: steps * 64 * 32 + steps * 8 + xlen * 8 + mlen * 12  # noqa: E731
    ok, s = shape([(1, 1, 9, 81, 1000), (1, 16, 9, 2000, 900), (1, 16, 27, 17001, 0)])
    assert ok and s["act"] == 16 and s["steps"] == 28 and s["xlen"] == 17004
    assert s["mat"] == [1000, 900, 0] and s["mlen"] == 1000 and s["smem"] == smem(28, 17004, 1000) <= 224 * 1024
    many_steps, long = (1, 16, 60, 2000, 0), (1, 16, 9, 19000, 0)
    assert shape([many_steps])[0] and shape([(1, 16, 9, 2000, 0), long])[0]
    assert smem(60, 19000, 0) > 224 * 1024 and not shape([many_steps, long])[0]
    # an odd step count at the limit is rounded up before it is compared
    assert smem(41, 18132, 0) <= 224 * 1024 < smem(42, 18132, 0) and not shape([(1, 16, 41, 18132, 0)])[0]
    assert not shape([(1, 16, 9, 500, 0), (1, 1, 9, 600, 0)])[0]
    assert not shape([(0, 1, 9, 81, 0)])[0] and not shape([(1, 1, 9, 81, 0)] * 10)[0]
