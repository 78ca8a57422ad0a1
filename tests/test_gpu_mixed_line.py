"""The mixed Gauss-point kernels whose lanes own lines of points (mstage.cuh),
chosen by the element count of a mesh."""
import numpy as np
import pytest

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu

PER, ISO = C.P_, dg.ISOTHERMAL_WALL

# pairs (even element counts) and single elements: the copies along z put the
# mesh on either side of the counts at which the kernels change
SIZES = [(1, (6, 5, 4), (40,)), (1, (7, 5, 3), (23,)), (2, (7, 5, 3), (23,)), (3, (6, 5, 4), (42,)), (3, (7, 5, 3), (23, 49))]


def step(nodes, n, p, q, bounds, U, pr, precision=dg.MIXED_FP32):
    prm = C.params(mu=1e-2, u=0.3, source=(0.0, 0.1, -0.2, 0.05, 0.0))
    with dg.Solver(dg.Mesh(*n, p, q, nodes, bounds), prm, precision=precision) as s:
        s.set_prandtl(pr)
        s.set_state(U)
        s.step(dg.RK4, 2e-4 / (p + 1), 1)
        s.step(dg.TVDRK3, 2e-4 / (p + 1), 1)
        return s.get_state()


@pytest.mark.parametrize("shape,pr", [("box", 0.71), ("shear", 0.0)], ids=["box_heat", "shear"])
@pytest.mark.parametrize("p,n,copies", SIZES)
def test_copies_of_a_periodic_mesh_step_alike(p, n, copies, shape, pr):
    """A mesh periodic in z and a state on it, put one after the other along z,
    step as the single one does.  Kernels that round an FP32 value differently
    move the update by some 2e-7 of itself (pairs against single elements, 2.3
    to 3.4e-7 over p = 1..4); the same FP32 values and FP64 roundings, 1e-16 of
    the state and 1e-11 of the update, stay below 1e-9.  (Affine meshes: on
    curved ones a shift along z alone moves the update by 2 to 4e-8, by the
    rounding of the geometry.)"""
    nx, ny, nz = n
    X = C.box_nodes(nx, ny, nz, 1, 2.0, 1.0, 1.0, shear=0.25 if shape == "shear" else 0.0)
    bounds = [PER] * 6 if shape == "shear" else [C.F_, C.F_, C.NS_, ISO, PER, PER]
    prm = C.params(mu=1e-2, u=0.3)
    U = C.random_state(prm, nx * ny * nz, (p + 1) ** 3, np.random.default_rng(p), 0.005)
    one = step(X, n, p, 1, bounds, U, pr) - U
    for m in copies:
        Xm = np.tile(X.reshape(-1, 3), (m, 1, 1))
        Xm[:, :, 2] += np.arange(m)[:, None]
        many = step(Xm.ravel(), (nx, ny, nz * m), p, 1, bounds, np.tile(U, m), pr).reshape(m, -1) - U
        assert np.linalg.norm(many - one) < 1e-9 * np.linalg.norm(many)


@pytest.mark.parametrize("pr", [0.0, 0.71], ids=["plain", "heat"])
@pytest.mark.parametrize("p,n", [(1, (14, 13, 13)), (1, (14, 13, 14)), (2, (14, 13, 13)), (3, (1, 1, 1)), (3, (7, 5, 3)), (3, (14, 13, 13))])
def test_curved_updates_follow_fp64(p, n, pr):
    """On curved elements, on either side of the counts: the update against
    the FP64 one, 2e-5, the bar of a single FP32 residual."""
    X = C.sine_nodes(*n, 2, 2.0, 1.0, 1.0, 0.03, walls=True)
    bounds = [PER, PER, C.NS_, ISO, PER, PER]
    U = C.random_state(C.params(mu=1e-2, u=0.3), n[0] * n[1] * n[2], (p + 1) ** 3, np.random.default_rng(p), 0.005)
    a, b = (step(X, n, p, 2, bounds, U, pr, precision) - U for precision in (dg.MIXED_FP32, dg.FP64))
    assert np.linalg.norm(a - b) < 2e-5 * np.linalg.norm(b)
