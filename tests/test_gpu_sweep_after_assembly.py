"""Sweeps that are the first launches after an assembly use the new matrix (needs a B200): the
smoothers read it before they wait for the launch before them."""
import ctypes as C

import numpy as np
import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,dim,nlev,n0", [("T", 2, 5, (4, 4)), ("T", 3, 3, (3, 2, 2)), ("NS", 2, 4, (4, 4)),
                                              ("NS", 3, 2, (4, 2, 2))])
def test_first_sweeps_after_assembly(gpu_lib, kind, dim, nlev, n0):
    m = ex.Mesh(dim, nlev, n0, (0, 1, 0, 1, 0, 1)[:2 * dim])
    s = (ex.MGSolNS if kind == "NS" else ex.MGSolT)(m)
    s.GenBc((_lib.BC_CAVITY if dim == 2 else _lib.BC_CHANNEL) if kind == "NS" else _lib.BC_HEAT_DIRICHLET)
    rng = np.random.default_rng(nlev)
    s.set_xold(0.1 * rng.standard_normal(s.ntop_dof))
    if kind == "T":
        s.set_source(workloads.heat_source(m.nel(nlev - 1)))
    top = nlev - 1
    p = ex.mg_params(smoother=_lib.SMOOTH_VANKA if kind == "NS" else _lib.SMOOTH_GS)
    x0, ms = rng.standard_normal(s.ntop_dof), C.c_double()
    for inv_dt in (1.0, 1000.0, 30.0):
        s.phys = ex.phys(inv_re=0.01, inv_dt=inv_dt)
        s.set_x(x0)
        s.assemble_all()
        # a warm-up sweep and a timed one on the top level's x and b
        _lib.check(s.L.exf_time_op(s.h, 1, top, C.byref(p), C.byref(s.phys), 1, C.byref(ms)))
        assert np.array_equal(s.x(), s.smooth(top, p, 2, x0, s.rhs())), inv_dt
