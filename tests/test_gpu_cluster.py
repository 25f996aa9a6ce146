"""One V-cycle of scalar systems whose lower levels run in the cluster kernel (needs a
B200), against the same cycle composed from the library's unit operations (level by level:
smoothing, residual, restriction, coarse solve, prolongation): sizes at the edges of the
row groups, of a single CTA, of the shared memory, with a top level above the cluster's
and odd element counts, both colour orders, and without pre- or post-smoothing."""
import numpy as np
import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib, workloads

from conftest import rel

pytestmark = pytest.mark.gpu

CASES = [
    # dim, levels, level-0 elements, pre / post sweeps, reversed colours
    (2, 2, (1, 1), (1, 1), 0),
    (2, 3, (3, 1), (2, 0), 1),
    (2, 4, (3, 5), (0, 2), 0),
    (2, 4, (7, 2), (2, 3), 1),
    (2, 5, (4, 4), (1, 2), 0),    # 129 x 129 lattice: several rounds per colour
    (2, 6, (4, 2), (2, 2), 1),    # 257 x 129: the FP64 top level has its own launches
    (3, 2, (2, 1, 3), (2, 2), 0),
    (3, 3, (3, 2, 2), (1, 1), 1),
    (3, 3, (8, 2, 2), (1, 2), 0),  # 65 x 17 x 17: the matrix stays in global memory
    (3, 4, (3, 1, 2), (2, 1), 0),
]


def compose(s, p, lev, x, b):
    """MGStep on host arrays: sweeps doubled below the top, correction 0.95 P x_c."""
    if lev == 0:
        return s.coarse_solve(b)
    mul = 2 if lev < s.nlev - 1 else 1
    x = s.smooth(lev, p, p.nu_pre * mul, x, b)
    bc = s.restrict(lev - 1, s.resid(lev, x, b))
    x = x + p.corr_damp * s.prolong(lev, compose(s, p, lev - 1, np.zeros(bc.size), bc))
    return s.smooth(lev, p, p.nu_post * mul, x, b)


@pytest.mark.parametrize("dim,nlev,n0,nu,reverse", CASES)
def test_cycle_equals_the_composed_cycle(gpu_lib, dim, nlev, n0, nu, reverse):
    m = ex.Mesh(dim, nlev, n0, (0, 2, 0, 1, 0, 1)[:2 * dim])
    t = ex.MGSolT(m)
    t.GenBc(_lib.BC_HEAT_DIRICHLET)
    t.phys = ex.phys(inv_dt=3.0)
    rng = np.random.default_rng(dim * 100 + nlev)
    t.set_source(workloads.heat_source(m.nel(nlev - 1)))
    t.set_xold(rng.standard_normal(t.ntop_dof))
    t.assemble_all()
    x0 = rng.standard_normal(t.ntop_dof)
    p = ex.mg_params(nu_pre=nu[0], nu_post=nu[1], max_cycles=1, eps=1e-30, reverse_colours=reverse)
    t.set_x(x0)
    t.solve(p)
    one = t.x()
    # a cycle is a few thousand roundings of 1.1e-16 in operators whose sweeps contract
    assert rel(one, compose(t, p, nlev - 1, x0, t.rhs())) <= 1e-12
    # the same bits again, and from the device loop (three cycles)
    t.set_x(x0)
    t.solve(p)
    assert np.array_equal(t.x(), one)
    outs = []
    for graph in (0, 1):
        t.set_x(x0)
        t.solve(ex.mg_params(nu_pre=nu[0], nu_post=nu[1], max_cycles=3, eps=1e-30, reverse_colours=reverse,
                             use_graph=graph))
        outs.append(t.x())
    assert np.array_equal(outs[0], outs[1])
    # FP32 cycles: three defect corrections end within the FP32 cycle's own relative
    # error (1e-5) of what the FP64 cycles leave of the error
    t.set_x(x0)
    t.solve(ex.mg_params(nu_pre=nu[0], nu_post=nu[1], max_cycles=3, eps=1e-30, reverse_colours=reverse,
                         precision=_lib.PREC_MIXED))
    assert np.linalg.norm(t.x() - outs[0]) <= 1e-5 * np.linalg.norm(x0 - outs[0])
