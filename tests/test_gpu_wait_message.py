"""The error of a bounded wait that ran out names the kernel it ran out in (needs a B200)."""
import ctypes as C

import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib

pytestmark = pytest.mark.gpu


def test_the_error_names_the_kernel(gpu_lib):
    t = ex.MGSolT(ex.Mesh(2, 2, (2, 2), (0, 1, 0, 1)))
    t.GenBc(_lib.BC_HEAT_DIRICHLET)
    t.assemble_all()
    p, ms = ex.mg_params(), C.c_double()
    # the probe waits, bounded, on a barrier phase that nothing completes
    assert t.L.exf_time_op(t.h, 6, 0, C.byref(p), C.byref(t.phys), 1, C.byref(ms)) == _lib.EXF_ERR_CUDA
    msg = t.L.exf_last_error().decode()
    assert "wait probe" in msg and "Vanka" not in msg and "cluster" not in msg and "ILU" not in msg
    assert t.solve(ex.mg_params(eps=1e-8)).converged  # the flag is clear again
