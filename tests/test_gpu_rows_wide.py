"""FP64 Vanka row sweeps of 2D levels above one wave of rows (8 lanes hold a row's 16 sums),
against the CPU oracle; and residual calls that alternate levels on one system (they share
the system's vectors), against b - A x."""
import numpy as np
import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib

from conftest import or_mg, or_phys, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reverse", [0, 1])
def test_large_level_sweep_matches_oracle(reverse, oracle_mod, gpu_lib):
    """144 x 128 elements: about 29,000 star rows per colour, above the 18,944 of one wave at
    16 lanes; an interior row has 25 blocks (two rounds of the 8 lanes' two loads), a corner
    row 9.  One sweep; the bound is the other sweep comparisons' 1e-12."""
    n0, nlev = (9, 8), 5
    gm, om = ex.Mesh(2, nlev, n0, (0, 1, 0, 1)), oracle_mod.OrMesh(2, nlev, n0, (0, 1, 0, 1))
    ns, osys = ex.MGSolNS(gm), oracle_mod.OrSys(om, 1)
    ns.GenBc(_lib.BC_CAVITY)
    osys.bc_preset(_lib.BC_CAVITY)
    ns.phys = ex.phys(inv_re=0.02)
    rng = np.random.default_rng(5)
    top = nlev - 1
    xold = 0.3 * rng.standard_normal(ns.ndof(top))
    ns.set_xold(xold)
    ns.assemble_all()
    osys.assemble_all(or_phys(oracle_mod, inv_re=0.02), xold=xold)
    x, b = rng.standard_normal(ns.ndof(top)), rng.standard_normal(ns.ndof(top))
    kw = dict(smoother=_lib.SMOOTH_VANKA, omega=0.4, reverse_colours=reverse)
    g = ns.smooth(top, ex.mg_params(vanka_kernel=_lib.VANKA_ROWS, **kw), 1, x, b)
    o = osys.smooth(top, or_mg(oracle_mod, **kw), 1, x, b)
    assert rel(g, o) < 1e-12


def test_residuals_of_alternating_levels(gpu_lib):
    gm = ex.Mesh(3, 3, (2, 1, 1), (0, 2, 0, 1, 0, 1))
    ns = ex.MGSolNS(gm)
    ns.GenBc(_lib.BC_CHANNEL)
    ns.phys = ex.phys(inv_re=0.1)
    rng = np.random.default_rng(6)
    ns.set_xold(rng.standard_normal(ns.ntop_dof))
    ns.assemble_all()
    for lev in (0, 2, 1, 2, 0):
        x, b = rng.standard_normal(ns.ndof(lev)), rng.standard_normal(ns.ndof(lev))
        ax = ns.spmv(lev, x)
        assert np.abs(ns.resid(lev, x, b) - (b - ax)).max() <= 1e-13 * (np.abs(ax).max() + np.abs(b).max())
