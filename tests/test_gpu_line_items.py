"""The Gauss-point stages whose contractions run a thread per line of points
and variable (vspace.cuh), at the orders and shapes that take them: lines that
do not fill a group's last round of threads, one to three elements, pairs,
single elements, curved geometry."""
import numpy as np
import pytest

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu

PER, ISO = C.P_, dg.ISOTHERMAL_WALL


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("shape,n", [("box", (2, 1, 1)), ("box", (3, 1, 1)), ("shear", (3, 2, 2)), ("sine", (2, 3, 3))],
                         ids=["pair", "single", "pairs", "curved"])
@pytest.mark.parametrize("p", [1, 2, 4, 5, 6])
def test_stages_match_the_nodal_form(p, n, shape):
    """FP64: two RK4 steps against the nodal form, whose contractions are per
    point, 1e-13 (the bar of the two forms elsewhere).  Mixed: the update of
    one RK4 step of the mixed form against the FP64 one, 2e-5, the bar of a
    single FP32 residual, to which the update of a short step is
    proportional."""
    nx, ny, nz = n
    walls = shape == "sine"
    if walls:
        nodes, q, bounds = C.sine_nodes(nx, ny, nz, 2, 2.0, 1.0, 1.0, 0.03, walls=True), 2, [PER, PER, C.NS_, ISO, PER, PER]
    else:
        nodes, q = C.box_nodes(nx, ny, nz, 1, 2.0, 1.0, 1.0, shear=0.3 if shape == "shear" else 0.0), 1
        bounds = [PER] * 6 if shape == "shear" else [C.F_, C.F_, C.NS_, ISO, PER, PER]
    mesh = dg.Mesh(nx, ny, nz, p, q, nodes, bounds)
    prm = C.params(mu=1e-2, u=0.3, source=(0.0, 0.1, -0.2, 0.05, 0.0))
    U = C.random_state(prm, mesh.nelem, mesh.nb, np.random.default_rng(p), 0.005)
    dt = 2e-4 / (p + 1)
    out = {}
    for form in (dg.STEP_GAUSS, dg.STEP_NODAL):
        with dg.Solver(mesh, prm) as s:
            s.set_prandtl(0.71)
            s.set_step_form(form)
            s.set_state(U)
            norms = s.step(dg.RK4, dt, 2)
            out[form] = s.get_state(), np.array(norms)
    assert rel(out[dg.STEP_GAUSS][0], out[dg.STEP_NODAL][0]) < 1e-13
    assert rel(out[dg.STEP_GAUSS][1], out[dg.STEP_NODAL][1]) < 1e-10
    new = {}
    for precision in (dg.FP64, dg.MIXED_FP32):
        with dg.Solver(mesh, prm, precision=precision) as s:
            s.set_prandtl(0.71)
            s.set_state(U)
            s.step(dg.RK4, dt, 1)
            new[precision] = s.get_state()
    assert rel(new[dg.MIXED_FP32] - U, new[dg.FP64] - U) < 2e-5
