"""Assembly with every coefficient in play (advecting velocity, upwinding, mass term, Robin
sides, buoyancy) on stretched boxes, against the CPU oracle.

The node-pair integrals deal a 3D element's 27 x 27 pairs to threads in groups of rows
(temperature: a warp per row; Navier-Stokes: three rows a thread); one element, and element
counts that are no multiple of anything, reach every row and both directions of a colour.
An entry is a sum of 27 products of at most ten factors per element and at most eight
elements, in the oracle's order: (27 + 8 + 10) * 2^-53 = 5e-15 of the largest magnitude;
1e-12 as for the other assembly comparisons."""
import numpy as np
import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib

from conftest import or_phys

pytestmark = pytest.mark.gpu

BOXES = [
    (3, 2, (1, 1, 1), (0, 2, 0, 0.5, 0, 1.3)),
    (3, 2, (3, 1, 2), (-1, 2, 0, 0.7, 0.2, 1.9)),
    (2, 2, (1, 1), (0, 2, 0, 0.5)),
    (2, 2, (3, 5), (-1, 2, 0, 0.7)),
]


@pytest.mark.parametrize("kind", ["T", "NS"])
@pytest.mark.parametrize("box", BOXES, ids=lambda b: "x".join(map(str, b[2])))
def test_coupled_assembly_matches_oracle(box, kind, oracle_mod, gpu_lib):
    dim, nlev, n0, ext = box
    rng = np.random.default_rng(11)
    gm, om = ex.Mesh(dim, nlev, n0, ext), oracle_mod.OrMesh(dim, nlev, n0, ext)
    ns, t = ex.MGSolNS(gm), ex.MGSolT(gm)
    ns.couple(t)
    t.couple(ns)
    pk = dict(inv_re=0.07, inv_prdl=1.4, inv_dt=3.0, upwind_ns=0.8, upwind_t=0.6, buoy=0.9, dirg=(0.3, 1.0, -0.2))
    gs = t if kind == "T" else ns
    osys = oracle_mod.OrSys(om, 0 if kind == "T" else 1)
    preset = _lib.BC_HEAT_DIRICHLET if kind == "T" else (_lib.BC_CAVITY if dim == 2 else _lib.BC_CHANNEL)
    osys.bc_preset(preset)
    gs.GenBc(preset)
    if kind == "T":  # Robin on the x = max side, Dirichlet elsewhere
        b0, b1 = osys.bc()
        side = om.xyz()[0] == ext[1]
        b0[:om.ntop][side] = 1
        b1[:om.ntop][side] = 2
        osys.set_bc(b0, b1)
        gs.set_bc(b0, b1)
    gs.phys = ex.phys(**pk)
    xns, xt = rng.standard_normal(ns.ntop_dof), rng.standard_normal(t.ntop_dof)
    ns.set_xold(xns)
    t.set_xold(xt)
    qe = rng.random(om.nel(nlev - 1)) if kind == "T" else None
    if qe is not None:
        t.set_source(qe)
    gs.assemble_all()
    if kind == "T":
        osys.assemble_all(or_phys(oracle_mod, **pk), xold=xt, vel=xns, qe=qe)
    else:
        osys.assemble_all(or_phys(oracle_mod, **pk), xold=xns, temp=xt)
    for lev in range(nlev):
        g, o = gs.matrix(lev), osys.matrix(lev)
        assert np.abs(g - o).max() <= 1e-12 * np.abs(o).max(), (lev, np.abs(g - o).max() / np.abs(o).max())
    g, o = gs.rhs(), osys.rhs()
    assert np.abs(g - o).max() <= 1e-12 * np.abs(o).max()
