"""The one-CTA kernels of the GMRES + ILU level solver (needs a B200): ILUPrecond bit for bit
against a restatement of LASPACK's ILUFactor / MulInv_QV in plain Python (every operation
in its order, contrib/laspack/factor.c:25-320, operats.c:1049-1290), on levels with more
than 32 rows per dependency level and (3D) rows longer than a record; a smoother call of
one, several and more than 30 iterations against GMRESIter restated on host arrays."""
import numpy as np
import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib, workloads

pytestmark = pytest.mark.gpu


def system(dim, nlev, n0):
    m = ex.Mesh(dim, nlev, n0, (0, 2, 0, 1, 0, 1)[:2 * dim])
    t = ex.MGSolT(m)
    t.GenBc(_lib.BC_HEAT_DIRICHLET)
    t.phys = ex.phys(inv_dt=2.0)
    t.set_source(workloads.heat_source(m.nel(nlev - 1)))
    t.assemble_all()
    return t


def ilu_apply(rp, col, val, c):
    n = len(rp) - 1
    f = val.copy()
    at = [{int(col[k]): k for k in range(rp[i], rp[i + 1])} for i in range(n)]
    for i in range(n):
        S = [j for j in sorted(at[i]) if j <= i]
        L = {(a, b): f[at[a][b]] for a in S for b in S if b in at[a]}
        g = lambda a, b: L.get((a, b), 0.0)  # noqa: E731
        low, upp = {k: g(i, k) for k in S[:-1]}, {k: g(k, i) for k in S[:-1]}
        for q, j in enumerate(S[:-1]):
            for k in S[q + 1:-1]:
                low[k] = low[k] - (low[j] * g(j, k)) / g(j, j)
                upp[k] = upp[k] - (upp[j] * g(k, j)) / g(j, j)
        d = g(i, i)
        for j in S[:-1]:
            d = d - (upp[j] * low[j]) / g(j, j)
            f[at[i][j]], f[at[j][i]] = low[j], upp[j]
        f[at[i][i]] = d
    inv = [1.0 / f[at[i][i]] for i in range(n)]
    w = np.zeros(n)
    for i in range(n):
        s = 0.0
        for j in sorted(at[i]):
            if j < i:
                s = s - f[at[i][j]] * w[j]
        w[i] = (s + c[i]) * inv[i]
    y = np.zeros(n)
    for i in range(n - 1, -1, -1):
        s = 0.0
        for j in sorted(at[i], reverse=True):
            if j > i:
                s = s - f[at[i][j]] * y[j]
        y[i] = (s + (0.0 + f[at[i][i]] * w[i])) * inv[i]
    return y


@pytest.mark.parametrize("dim,nlev,n0", [(2, 1, (1, 1)), (2, 3, (5, 3)), (2, 4, (3, 2)), (3, 1, (2, 1, 3)),
                                         (3, 2, (2, 1, 2))])
def test_ilu_apply_bitwise(gpu_lib, dim, nlev, n0):
    t = system(dim, nlev, n0)
    for lev in range(nlev):
        rp, col, val = t.csr(lev)
        c = np.random.default_rng(lev).standard_normal(t.ndof(lev))
        assert np.array_equal(t.ilu_apply(lev, c), ilu_apply(rp, col, val, c)), lev


def gmres(A, M, x, b, m, restart=30):
    it = 0
    while it < m:
        k = min(restart, m - it)
        v = M(b - A(x))
        beta = np.linalg.norm(v)
        V, H = [v / beta], np.zeros((k + 1, k))
        for i in range(k):
            w = M(A(V[i]))
            for j in range(i + 1):
                H[j, i] = w @ V[j]
                w = w - H[j, i] * V[j]
            H[i + 1, i] = np.linalg.norm(w)
            V.append(w / H[i + 1, i])
        e = np.zeros(k + 1)
        e[0] = beta
        x = x + np.column_stack(V[:k]) @ np.linalg.lstsq(H, e, rcond=None)[0]
        it += k
    return x


@pytest.mark.parametrize("dim,nlev,n0", [(2, 3, (4, 3)), (3, 2, (2, 1, 2))])
@pytest.mark.parametrize("m", [1, 4, 33])
def test_smoother_call(gpu_lib, dim, nlev, n0, m):
    t = system(dim, nlev, n0)
    p = ex.mg_params(smoother=_lib.SMOOTH_GMRES_ILU, eps=1e-30)
    rng = np.random.default_rng(m)
    for lev in range(nlev):
        x, b = rng.standard_normal(t.ndof(lev)), rng.standard_normal(t.ndof(lev))
        got = t.smooth(lev, p, m, x, b)
        want = gmres(lambda u: t.spmv(lev, u), lambda u: t.ilu_apply(lev, u), x, b, m)
        # least squares here, rotations there: rounding of m <= 33 steps of a system whose
        # preconditioned condition number is below 1e3
        assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want), lev


def test_converged_call_leaves_x(gpu_lib):
    t = system(2, 3, (4, 3))
    x = np.random.default_rng(3).standard_normal(t.ndof(2))
    p = ex.mg_params(smoother=_lib.SMOOTH_GMRES_ILU, eps=1e-6)
    assert np.array_equal(t.smooth(2, p, 4, x, t.spmv(2, x)), x)
