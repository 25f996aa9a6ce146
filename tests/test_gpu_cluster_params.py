"""Cycle parameters at the edges of their meaning, on levels in the cluster kernel and on
levels above it (needs a B200), against the cycle composed from the library's unit operations."""
import numpy as np
import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib, workloads

from conftest import rel

pytestmark = pytest.mark.gpu


def compose(s, p, lev, x, b):
    """MGStep on host arrays; a correction factor of zero replaces x by P x_c, as exf_prolong
    does and as a cycle of one launch per colour always did."""
    if lev == 0:
        return s.coarse_solve(b)
    mul = 2 if lev < s.nlev - 1 else 1
    x = s.smooth(lev, p, p.nu_pre * mul, x, b)
    bc = s.restrict(lev - 1, s.resid(lev, x, b))
    y = s.prolong(lev, compose(s, p, lev - 1, np.zeros(bc.size), bc))
    x = x + p.corr_damp * y if p.corr_damp else y
    return s.smooth(lev, p, p.nu_post * mul, x, b)


@pytest.mark.parametrize("damp", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("dim,nlev,n0", [(2, 3, (3, 2)), (2, 6, (4, 2)), (3, 2, (2, 2, 2))])
def test_correction_factor(gpu_lib, dim, nlev, n0, damp):
    m = ex.Mesh(dim, nlev, n0, (0, 2, 0, 1, 0, 1)[:2 * dim])
    t = ex.MGSolT(m)
    t.GenBc(_lib.BC_HEAT_DIRICHLET)
    t.phys = ex.phys(inv_dt=3.0)
    rng = np.random.default_rng(nlev)
    t.set_source(workloads.heat_source(m.nel(nlev - 1)))
    t.set_xold(rng.standard_normal(t.ntop_dof))
    t.assemble_all()
    x0 = rng.standard_normal(t.ntop_dof)
    p = ex.mg_params(max_cycles=1, eps=1e-30, corr_damp=damp)
    t.set_x(x0)
    t.solve(p)
    # a cycle is a few thousand roundings of 1.1e-16 in operators whose sweeps contract
    assert rel(t.x(), compose(t, p, nlev - 1, x0, t.rhs())) <= 1e-12


@pytest.mark.parametrize("dim,n0", [(2, (12, 13)), (2, (13, 13)), (2, (24, 5)), (3, (4, 4, 4)), (3, (5, 3, 4))])
def test_coarsest_product_inside_and_outside_the_launch(gpu_lib, dim, n0):
    """Coarsest levels on either side of the line at 700 rows: 675, 729, 539, 729 and 693."""
    m = ex.Mesh(dim, 2, n0, (0, 2, 0, 1, 0, 1)[:2 * dim])
    t = ex.MGSolT(m)
    t.GenBc(_lib.BC_HEAT_DIRICHLET)
    t.phys = ex.phys(inv_dt=3.0)
    rng = np.random.default_rng(n0[0])
    t.set_source(workloads.heat_source(m.nel(1)))
    t.set_xold(rng.standard_normal(t.ntop_dof))
    t.assemble_all()
    x0 = rng.standard_normal(t.ntop_dof)
    p = ex.mg_params(max_cycles=1, eps=1e-30)
    t.set_x(x0)
    t.solve(p)
    one = t.x()
    # a cycle is a few thousand roundings of 1.1e-16 in operators whose sweeps contract
    assert rel(one, compose(t, p, 1, x0, t.rhs())) <= 1e-12
    outs = []
    for graph in (0, 1):
        t.set_x(x0)
        t.solve(ex.mg_params(max_cycles=3, eps=1e-30, use_graph=graph))
        outs.append(t.x())
    assert np.array_equal(outs[0], outs[1])
