"""The element counts and shapes at which the FP64 and the mixed stage change
their kernels (line_kernels, mixed_line)."""
import numpy as np
import pytest

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu

# p, elements on either side of a line, shape
FP64 = [(1, (12, 14, 7), "box"), (1, (12, 11, 9), "box"), (1, (16, 37, 4), "shear"), (1, (13, 14, 14), "shear"), (1, (16, 37, 4), "sine"),
        (1, (13, 14, 14), "sine"), (2, (16, 37, 2), "box"), (2, (12, 11, 9), "box"), (2, (16, 37, 4), "shear"), (2, (3, 23, 37), "sine"),
        (2, (12, 37, 12), "sine"), (2, (73, 73, 1), "sine"), (2, (11, 37, 16), "sine"), (2, (16, 17, 24), "shear"), (3, (16, 37, 4), "sine"),
        (3, (3, 23, 37), "sine"), (3, (20, 37, 4), "sine"), (3, (3, 7, 141), "sine"), (4, (7, 7, 12), "box"), (4, (6, 10, 10), "box"),
        (4, (7, 10, 9), "shear"), (4, (7, 10, 9), "sine")]
MIXED = [(2, (3, 13, 77), "box"), (2, (3, 13, 79), "box"), (2, (48, 37, 4), "sine"), (2, (22, 17, 19), "sine"), (2, (16, 37, 16), "sine"),
         (3, (38, 37, 4), "box"), (3, (19, 37, 8), "box"), (3, (13, 19, 23), "box")]


def mesh_of(p, n, shape):
    if shape == "sine":
        return dg.Mesh(*n, p, 2, C.sine_nodes(*n, 2, 2.0, 1.0, 1.0, 0.02, walls=True), [C.P_, C.P_, C.NS_, dg.ISOTHERMAL_WALL, C.P_, C.P_])
    nodes = C.box_nodes(*n, 1, 2.0, 1.0, 1.0, shear=0.3 if shape == "shear" else 0.0)
    return dg.Mesh(*n, p, 1, nodes, [C.P_] * 6 if shape == "shear" else [C.P_, C.P_, C.NS_, dg.ISOTHERMAL_WALL, C.P_, C.P_])


def step(mesh, prm, U, dt, precision=dg.FP64, form=dg.STEP_GAUSS):
    with dg.Solver(mesh, prm, precision=precision) as s:
        s.set_prandtl(0.71)
        s.set_step_form(form)
        s.set_state(U)
        norms = s.step(dg.RK4, dt, 1)
        return s.get_state(), norms


@pytest.mark.parametrize("p,n,shape", FP64, ids=lambda v: str(v).replace(" ", ""))
def test_fp64_stages_match_the_nodal_form(p, n, shape):
    """An RK4 step against the nodal form: 1e-13 for the state and 1e-10 for the
    printed norm, the bars of the two forms elsewhere."""
    mesh, prm = mesh_of(p, n, shape), C.params(mu=1e-2, u=0.3, source=(0.0, 0.1, -0.2, 0.05, 0.0))
    U = C.random_state(prm, mesh.nelem, mesh.nb, np.random.default_rng(p), 0.005)
    (a, na), (b, nb) = (step(mesh, prm, U, 1e-5, form=f) for f in (dg.STEP_GAUSS, dg.STEP_NODAL))
    assert np.linalg.norm(a - b) < 1e-13 * np.linalg.norm(b)
    assert abs(na[0] - nb[0]) < 1e-10 * nb[0]


@pytest.mark.parametrize("p,n,shape", MIXED, ids=lambda v: str(v).replace(" ", ""))
def test_mixed_updates_follow_fp64(p, n, shape):
    """The update of an RK4 step against the FP64 one, 2e-5, the bar of a
    single FP32 residual."""
    mesh, prm = mesh_of(p, n, shape), C.params(mu=1e-2, u=0.3, source=(0.0, 0.1, -0.2, 0.05, 0.0))
    U = C.random_state(prm, mesh.nelem, mesh.nb, np.random.default_rng(p), 0.005)
    a, b = (step(mesh, prm, U, 1e-5, precision=q)[0] - U for q in (dg.MIXED_FP32, dg.FP64))
    assert np.linalg.norm(a - b) < 2e-5 * np.linalg.norm(b)
