"""The residual of a nodal state and its VJP through the line kernels against
the same through the kernels with a thread per node: a mesh periodic in z small
enough to take the latter, and copies of it along z that take the former."""
import numpy as np
import pytest

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu

PER, ISO = C.P_, dg.ISOTHERMAL_WALL


@pytest.mark.parametrize("shape,bounds", [("box", [C.F_, C.F_, C.NS_, ISO, PER, PER]), ("box", [C.W_, C.F_, C.W_, C.NS_, PER, PER]),
                                          ("shear", [PER] * 6), ("sine", [PER, PER, C.NS_, ISO, PER, PER])],
                         ids=["box_iso", "box_slip", "shear", "sine_iso"])
@pytest.mark.parametrize("pr", [0.0, 0.71], ids=["plain", "heat"])
@pytest.mark.parametrize("p,copies", [(1, 2), (2, 12), (4, 3)])
def test_copies_of_a_periodic_mesh(p, copies, pr, shape, bounds):
    """140 elements, below the 216 (p = 1), 1185 (p = 2; residual 1600) and
    350 (p = 4) from which the line kernels are taken, and 2, 12 and 3 copies
    (with the heat flux the residual keeps the nodal kernels).  The extent
    along z is dyadic, so a copy has the same geometry bit for bit and what is
    left is the rounding of two orders of summation: each product lies within
    1e-14 of the exact one, bar 1e-12; R and f have the bar of residuals,
    1e-11."""
    n = nx, ny, nz = 7, 5, 4
    if shape == "sine":
        nodes, q = C.sine_nodes(*n, 2, 2.0, 1.0, 1.0, 0.03, walls=True), 2
    else:
        nodes, q = C.box_nodes(*n, 1, 2.0, 1.0, 1.0, shear=0.25 if shape == "shear" else 0.0), 1
    X = nodes.reshape(-1, 3)
    many = np.tile(X, (copies, 1, 1))
    many[:, :, 2] += np.arange(copies)[:, None]
    prm = C.params(mu=1e-2, u=0.3, source=(0.0, 0.1, -0.2, 0.05, 0.0))
    rng = np.random.default_rng(p)
    U = C.random_state(prm, nx * ny * nz, (p + 1) ** 3, rng, 0.005)
    lam = rng.standard_normal(U.size)
    out = []
    for m, Xm in ((1, X), (copies, many)):
        with dg.Solver(dg.Mesh(nx, ny, nz * m, p, q, Xm.ravel(), bounds), prm) as s:
            s.set_prandtl(pr)
            g = s.residual_vjp(np.tile(U, m), np.tile(lam, m))
            out.append([v.reshape(m, -1) for v in (*s.residual(np.tile(U, m)), g)])
    for one, copy, bar in zip(*out, (1e-11, 1e-11, 1e-12)):
        assert np.linalg.norm(copy - one) < bar * np.linalg.norm(copy)
