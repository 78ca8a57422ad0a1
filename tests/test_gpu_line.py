"""The FP64 Gauss-point kernels whose lanes own lines of Gauss points
(lstage.cuh), at the element counts and shapes that choose between their
forms and leave a warp's lanes or the last warp's elements unused."""
import numpy as np
import pytest

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu

PER, ISO = C.P_, dg.ISOTHERMAL_WALL
CHANNEL = [C.IN_, C.OUT_, C.NS_, C.W_, PER, PER]


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def mesh_of(shape, n, p, bounds):
    nx, ny, nz = n
    if shape == "sine":
        nodes, q = C.sine_nodes(nx, ny, nz, 2, 2.0, 1.0, 1.0, 0.03, walls=bounds[2] != PER), 2
    elif shape == "mirror":  # box elements whose first and second edges point down their axes
        X = C.box_nodes(nx, ny, nz, 1, 2.0, 1.0, 1.0).reshape(-1, 3)
        X[:, :2] *= -1.0
        nodes, q = X.ravel(), 1
    else:
        nodes, q = C.box_nodes(nx, ny, nz, 1, 2.0, 1.0, 1.0, shear=0.3 if shape == "shear" else 0.0), 1
    return dg.Mesh(nx, ny, nz, p, q, nodes, bounds)


# p = 1: 4 elements a warp from 216 elements; p = 2: an element a warp up to
# 1184 elements, then 3; p = 3: one; p = 4: one from 350 elements
SIZES = [(1, (6, 6, 5)), (1, (6, 6, 6)), (1, (7, 7, 5)), (2, (1, 1, 2)), (2, (37, 8, 4)), (2, (12, 11, 9)), (2, (13, 10, 10)),
         (2, (11, 11, 11)), (3, (1, 2, 1)), (3, (5, 3, 3)), (4, (6, 6, 6)), (4, (7, 10, 5)), (4, (13, 9, 3))]


@pytest.mark.parametrize("shape,bounds,pr", [("box", CHANNEL, 0.0), ("box", [C.F_, C.F_, ISO, C.F_, C.F_, ISO], 0.71),
                                             ("shear", [PER] * 6, 0.0), ("mirror", [C.F_, C.F_, C.NS_, C.W_, PER, PER], 0.71),
                                             ("sine", [PER, PER, C.NS_, ISO, PER, PER], 0.71)],
                         ids=["box", "box_heat", "shear", "mirror", "sine_heat"])
@pytest.mark.parametrize("p,n", SIZES)
def test_line_kernels_match_the_nodal_form(p, n, shape, bounds, pr):
    """Two RK4 steps and a TVD-RK3 step against the nodal form, whose kernels
    share none of the line kernels' contractions or exchanges and are pinned
    to the oracle: the bar of the two forms elsewhere, 1e-13 for the state; the
    printed norm, a sum over a residual with cancellation, 1e-10.  Box
    elements along the axes take the axis-frame kernels, sheared and mirrored
    ones the general affine ones, curved ones the per-point geometry."""
    mesh = mesh_of(shape, n, p, bounds)
    prm = C.params(mu=1e-2, u=0.3, source=(0.0, 0.1, -0.2, 0.05, 0.0))
    U = C.random_state(prm, mesh.nelem, mesh.nb, np.random.default_rng(p), 0.005)
    out = {}
    for form in (dg.STEP_GAUSS, dg.STEP_NODAL):
        with dg.Solver(mesh, prm) as s:
            s.set_prandtl(pr)
            s.set_step_form(form)
            s.set_state(U)
            norms = [*s.step(dg.RK4, 2e-4 / (p + 1), 2), *s.step(dg.TVDRK3, 2e-4 / (p + 1), 1)]
            out[form] = s.get_state(), np.array(norms)
    assert rel(out[dg.STEP_GAUSS][0], out[dg.STEP_NODAL][0]) < 1e-13
    assert rel(out[dg.STEP_GAUSS][1], out[dg.STEP_NODAL][1]) < 1e-10


@pytest.mark.parametrize("shape,bounds,pr", [("box", [C.F_, C.F_, ISO, C.F_, C.F_, ISO], 0.71), ("shear", [PER] * 6, 0.0),
                                             ("sine", [PER, PER, C.NS_, ISO, PER, PER], 0.71)],
                         ids=["box_heat", "shear", "sine_heat"])
@pytest.mark.parametrize("p,n", [(1, (6, 6, 6)), (1, (7, 7, 5)), (2, (12, 11, 9)), (2, (11, 11, 11)), (3, (5, 3, 3)),
                                 (4, (7, 10, 5))])
def test_line_adjoint_matches_the_nodal_form(p, n, shape, bounds, pr):
    """The gradient of one recorded RK4 step in the state and the parameters
    against the nodal form's: the bar of the two forms' gradients elsewhere,
    1e-12; each parameter's, whose viscosity term the nodal form takes as a
    difference of two residuals, 1e-8."""
    mesh = mesh_of(shape, n, p, bounds)
    prm = C.params(mu=1e-2, u=0.3, source=(0.0, 0.1, -0.2, 0.05, 0.0))
    rng = np.random.default_rng(p)
    U = C.random_state(prm, mesh.nelem, mesh.nb, rng, 0.005)
    lam = rng.standard_normal(U.shape)
    out = {}
    for form in (dg.STEP_GAUSS, dg.STEP_NODAL):
        with dg.Solver(mesh, prm) as s:
            s.set_prandtl(pr)
            s.set_step_form(form)
            s.set_state(U)
            s.forward_record(dg.RK4, 2e-4 / (p + 1), 1, 1)
            out[form] = s.backward_params(lam)
    (ga, pa), (gb, pb) = out[dg.STEP_GAUSS], out[dg.STEP_NODAL]
    assert rel(ga, gb) < 1e-12
    assert np.all(np.abs(pa - pb) <= 1e-8 * np.abs(pb)), (pa, pb)


@pytest.mark.parametrize("shape,bounds", [("box", CHANNEL), ("shear", [PER] * 6), ("sine", [PER, PER, C.NS_, C.NS_, PER, PER])],
                         ids=["box", "shear", "sine"])
@pytest.mark.parametrize("p,n", [(1, (6, 6, 6)), (1, (7, 7, 5)), (2, (12, 11, 9)), (2, (12, 12, 12)), (3, (5, 3, 3)),
                                 (4, (7, 10, 5))])
def test_line_residual_and_product(p, n, shape, bounds):
    """R and f of a nodal state against the nodal kernels, which a mixed
    handle with the heat flux off does not take but a Prandtl number large
    enough to vanish from every sum does: kq = mu gamma / Pr = 1e-300.  The bar
    of residuals against the oracle, 1e-11.  The product with a vector against
    the difference of two such residuals, whose truncation (h^2) and rounding
    (1e-12 / h) meet at h = 1e-4: 1e-6."""
    mesh = mesh_of(shape, n, p, bounds)
    prm = C.params(mu=1e-2, u=0.3, source=(0.0, 0.1, -0.2, 0.05, 0.0))
    rng = np.random.default_rng(p)
    U = C.random_state(prm, mesh.nelem, mesh.nb, rng, 0.005)
    lam, v = rng.standard_normal(U.shape), rng.standard_normal(U.shape)
    with dg.Solver(mesh, prm) as s:
        R, f = s.residual(U)
        g = s.residual_vjp(U, lam)
        s.set_prandtl(1e298)
        R0, f0 = s.residual(U)
        assert rel(R, R0) < 1e-11 and rel(f, f0) < 1e-11
        h = 1e-4
        fd = lam @ (s.residual(U + h * v)[1] - s.residual(U - h * v)[1]) / (2 * h)
    assert abs(g @ v - fd) < 1e-6 * np.linalg.norm(g) * np.linalg.norm(v)
