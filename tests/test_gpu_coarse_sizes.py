"""Coarsest-level factorisation at the sizes where its panel kernel changes (one row per
thread on 256 or 512 threads, three rows on 512, the shared-memory panel above 1536 rows),
against a dense solve.  The explicit inverse's forward error is bounded by a modest multiple
of cond(A) n 2^-53; the bound used is that product."""
import numpy as np
import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib

pytestmark = pytest.mark.gpu

# (elements x, y): (2 x + 1)(2 y + 1) rows
SIZES = [(1, 1, 9), (7, 8, 255), (6, 10, 273), (3, 36, 511), (9, 13, 513), (2, 153, 1535), (14, 26, 1537)]


@pytest.mark.parametrize("nx,ny,n", SIZES, ids=lambda v: str(v))
def test_coarse_inverse_against_dense_solve(nx, ny, n, gpu_lib):
    m = ex.Mesh(2, 2, (nx, ny), (0, 1, 0, 1))
    t = ex.MGSolT(m)
    t.GenBc(_lib.BC_HEAT_DIRICHLET)
    t.phys = ex.phys()
    t.set_xold(np.zeros(t.ntop_dof))
    t.assemble_all()
    assert t.ndof(0) == n
    rp, col = t.pattern(0)
    A = np.zeros((n, n))
    A[np.repeat(np.arange(n), np.diff(rp)), col] = t.matrix(0)
    b = np.random.default_rng(n).standard_normal(n)
    ref = np.linalg.solve(A, b)
    x = t.coarse_solve(b)
    assert np.linalg.norm(x - ref) <= np.linalg.cond(A) * n * 2.0 ** -53 * np.linalg.norm(ref)
