"""One V-cycle of a scalar system on uploaded meshes whose levels run in the cluster kernel
(needs a B200): interior nodes shifted by 1e-10 put the first-fit colouring's order at
random inside each lattice line, which leaves a few nodes in the last colours, so CTAs have
colours without a row of their own; against the cycle composed from the library's unit
operations."""
import numpy as np
import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib, workloads

from conftest import rel
from test_gpu_cluster import compose
from test_gpu_upload import structured_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reverse", [0, 1])
@pytest.mark.parametrize("dim,nlev,n0", [(2, 4, (4, 2)), (2, 5, (3, 4)), (3, 3, (4, 2, 2))])
def test_cycle_on_an_uploaded_mesh(gpu_lib, dim, nlev, n0, reverse):
    gm = ex.Mesh(dim, nlev, n0, (0, 2, 0, 1, 0, 1)[:2 * dim])
    arrays = structured_arrays(gm, n0)
    rng = np.random.default_rng(dim * 10 + nlev)
    xyz = np.array(arrays["xyz"])
    inside = np.all([(xyz[d] > 0) & (xyz[d] < xyz[d].max()) for d in range(dim)], axis=0)
    for d in range(dim):
        xyz[d, inside] += 1e-10 * rng.uniform(-1, 1, inside.sum())
    m = ex.Mesh.upload(**dict(arrays, xyz=xyz))
    t = ex.MGSolT(m)
    t.GenBc(_lib.BC_HEAT_DIRICHLET)
    t.phys = ex.phys(inv_dt=3.0)
    t.set_source(workloads.heat_source(m.nel(nlev - 1)))
    t.set_xold(rng.standard_normal(t.ntop_dof))
    t.assemble_all()
    # fewer than 16 warps of rows in a colour (4 rows a warp in 2D, 2 in 3D)
    assert np.bincount(t.colours(nlev - 1)[1]).min() < (64 if dim == 2 else 32)
    x0 = rng.standard_normal(t.ntop_dof)
    p = ex.mg_params(max_cycles=1, eps=1e-30, reverse_colours=reverse)
    outs = []
    for _ in range(5):
        t.set_x(x0)
        t.solve(p)
        outs.append(t.x())
    # a cycle is a few thousand roundings of 1.1e-16 in operators whose sweeps contract
    assert rel(outs[0], compose(t, p, nlev - 1, x0, t.rhs())) <= 1e-12
    assert all(np.array_equal(o, outs[0]) for o in outs[1:])
