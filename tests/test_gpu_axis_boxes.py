"""Which meshes the kernels in axis frames may take: boxes whose nodes lie
exactly on the axes' lines, not ones whose metric nearly does."""
import numpy as np
import pytest

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 3, 4])
def test_flat_elements_with_a_slight_tilt(p):
    """Elements 1e-5 high and 1/8 long, tilted by y += 9e-14 x (1e-8 of the
    height over the length): a shear layer u(eta), with density and pressure
    constant and no other velocity, has no flux across its layers and
    f = tilt dFx/dy, of the momentum along x and the energy.  f is projected
    on that profile: 1 with the metric as it is (0.90 at p = 1 by the
    discretisation, the CPU oracle's value), 0 with the metric of boxes.  The
    rounding of the pressure, from energies 100 times as large, leaves noise
    of up to the size of f in a value, independent over the 8 (p + 1)^3 values
    and more of a column of elements: 0.13 in the projection at p = 1.
    Bar 0.5."""
    n = (8, 8, 8)  # (x and z dyadic: their Jacobian is exact, so the tilt is all there is beside the diagonal)
    ly, tilt = 8e-5, 9e-14
    nodes = C.box_nodes(*n, 1, 1.0, ly, 1.0).reshape(-1, 3).copy()
    nodes[:, 1] += tilt * nodes[:, 0]
    mesh = dg.Mesh(*n, p, 1, nodes.ravel(), [C.P_] * 6)
    y = C.node_coords(*n, p, 1, C.box_nodes(*n, 1, 1.0, ly, 1.0))[..., 1]  # of the untilted mesh: a function of eta
    one, k = np.ones_like(y), 2 * np.pi / ly
    u, du = 10.0 + 2.0 * np.sin(k * y), 2.0 * k * np.cos(k * y)
    U = C.state_from_primitives(one, u, 0 * one, 0 * one, one / 1.4, 1.4)
    with dg.Solver(mesh, C.params(mu=0.0)) as s:
        f = s.residual(U.ravel())[1].reshape(U.shape)
    for r, dF in ((1, 2.0 * u * du), (4, (2.5 + 1.5 * u * u) * du)):
        assert abs(np.sum(f[:, r] * tilt * dF) / np.sum((tilt * dF) ** 2) - 1.0) < 0.5
