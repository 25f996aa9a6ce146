"""The one-launch-per-colour Vanka kernel of small 2D levels (needs a B200): AUTO against the
ROWS pair, bit for bit (same sums in the same order), on odd element counts, one to three
sweeps (an odd number of colours in all leaves the iterate in the second buffer), both
colour orders, FP64, FP16 blocks and FP32 blocks, and on an uploaded mesh whose colouring
is not the lattice's."""
import ctypes as C

import numpy as np
import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib

pytestmark = pytest.mark.gpu


def cavity(mesh):
    ns = ex.MGSolNS(mesh)
    ns.GenBc(_lib.BC_CAVITY)
    ns.phys = ex.phys(inv_re=0.02)
    xyz, N = mesh.xyz(), mesh.ntop
    x = np.zeros(ns.ntop_dof)
    x[:N] = np.sin(3.0 * xyz[0]) * xyz[1]
    x[N:2 * N] = 0.3 * np.cos(2.0 * xyz[1])
    ns.set_xold(x)
    ns.assemble_all()
    return ns


def meshes():
    yield ex.Mesh(2, 2, (1, 1), (0, 1, 0, 1))
    yield ex.Mesh(2, 3, (3, 5), (0, 1, 0, 1))
    yield ex.Mesh(2, 4, (7, 2), (0, 1, 0, 1))
    a = ex.Mesh.refine_arrays(2, 3, *_coarse())
    yield ex.Mesh.upload(2, a["nnodes"], _coarse()[0], a["xyz"], a["conn"], a["neigh"], a["parent"])


def _coarse():
    """A skewed 2 x 3 quad9 box, nodes numbered vertices first."""
    nx, ny = 2, 3
    pts = {}

    def node(i, j):
        return pts.setdefault((i, j), len(pts))

    for j in range(0, 2 * ny + 1, 2):
        for i in range(0, 2 * nx + 1, 2):
            node(i, j)
    nvert = len(pts)
    conn = []
    for ey in range(ny):
        for ex_ in range(nx):
            i, j = 2 * ex_, 2 * ey
            conn.append([node(i + a, j + b) for a, b in
                         ((0, 0), (2, 0), (2, 2), (0, 2), (1, 0), (2, 1), (1, 2), (0, 1), (1, 1))])
    xyz = np.zeros((2, len(pts)))
    for (i, j), n in pts.items():
        xyz[:, n] = i / (2.0 * nx) + 0.05 * j / (2.0 * ny), j / (2.0 * ny)
    return nvert, xyz, np.array(conn, np.int32)


@pytest.mark.parametrize("nsweeps,reverse", [(1, 0), (2, 1), (3, 0)])
def test_sweeps_have_the_row_kernels_bits(gpu_lib, nsweeps, reverse):
    for mesh in meshes():
        ns = cavity(mesh)
        rng = np.random.default_rng(nsweeps)
        for lev in range(1, ns.nlev):
            x, b = rng.standard_normal(ns.ndof(lev)), rng.standard_normal(ns.ndof(lev))
            outs = [ns.smooth(lev, ex.mg_params(smoother=_lib.SMOOTH_VANKA, omega=0.4, reverse_colours=reverse,
                                                vanka_kernel=k), nsweeps, x, b)
                    for k in (_lib.VANKA_AUTO, _lib.VANKA_ROWS)]
            assert np.array_equal(outs[0], outs[1]), lev


@pytest.mark.parametrize("fp32_blocks", [0, 1])
def test_mixed_cycles_have_the_row_kernels_bits(gpu_lib, fp32_blocks):
    """Cycle by cycle; whether the multigrid converges on such a mesh is not the question
    (the skewed one diverges with either kernel), so status and history are compared too."""
    for mesh in meshes():
        ns = cavity(mesh)
        outs = []
        for k in (_lib.VANKA_AUTO, _lib.VANKA_ROWS):
            ns.set_x(ns.xold())
            p = ex.mg_params(smoother=_lib.SMOOTH_VANKA, omega=0.4, nu_pre=3, nu_post=2, max_cycles=3, eps=1e-30,
                             precision=_lib.PREC_MIXED, fp32_blocks=fp32_blocks, vanka_kernel=k)
            st = _lib.ExfSolveStats()
            rc = ns.L.exf_mg_solve(ns.h, C.byref(p), C.byref(st))
            outs.append((rc, np.array(st.hist[:st.cycles]), ns.x()))
        assert outs[0][0] == outs[1][0] and outs[0][1].size >= 1
        assert np.array_equal(outs[0][1], outs[1][1], equal_nan=True)
        assert np.array_equal(outs[0][2], outs[1][2], equal_nan=True)
