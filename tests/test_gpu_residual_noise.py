"""The rounding of a nodal residual does not depend on the kernels that form it."""
import numpy as np
import pytest

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["box", "shear"])
@pytest.mark.parametrize("p,n", [(3, (12, 12, 12)), (4, (9, 9, 9))])
def test_uniform_stream(p, n, shape):
    """f of a uniform stream is rounding alone, most of it from the jumps of
    the face traces.  Formed by the line kernels, and by the nodal ones (a heat
    flux that vanishes from every sum): both from the nodal traces, so alike
    but for the order of the volume term's sums: within 30% (traces
    extrapolated from Gauss points give twice the nodal kernels')."""
    mesh = dg.Mesh(*n, p, 1, C.box_nodes(*n, 1, 2.0, 1.0, 1.0, shear=0.3 if shape == "shear" else 0.0), [C.P_] * 6)
    one = np.ones((mesh.nelem, mesh.nb))
    U = C.state_from_primitives(one, 0.3 * one, 0.2 * one, 0.1 * one, one / 1.4, 1.4).ravel()
    with dg.Solver(mesh, C.params(mu=1e-2)) as s:
        f = s.residual(U)[1]
        s.set_prandtl(1e298)
        nodal = s.residual(U)[1]
    assert np.linalg.norm(f) < 1.3 * np.linalg.norm(nodal)
