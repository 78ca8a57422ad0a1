"""A captured step is captured again, its norm on a branch of its own, when
enough steps have run."""
import numpy as np
import pytest

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [dg.STEP_GAUSS, dg.STEP_NODAL])
@pytest.mark.parametrize("scheme", [dg.RK4, dg.TVDRK3])
def test_short_calls_equal_one_long_call(scheme, form):
    """70 steps in one call (branched from its start) and in calls of 1, 62, 1,
    1 and 5 (captured again before the fifth): the same states and norms, bit
    for bit."""
    mesh = dg.Mesh(3, 2, 2, 2, 1, C.box_nodes(3, 2, 2, 1, 2.0, 1.0, 1.0), [C.F_, C.F_, C.NS_, C.W_, C.P_, C.P_])
    prm = C.params(mu=1e-2, u=0.3)
    U = C.random_state(prm, mesh.nelem, mesh.nb, np.random.default_rng(1), 0.005)
    out = []
    for calls in ((70,), (1, 62, 1, 1, 5)):
        with dg.Solver(mesh, prm) as s:
            s.set_step_form(form)
            s.set_state(U)
            norms = [x for n in calls for x in s.step(scheme, 1e-5, n)]
            out.append((s.get_state(), np.array(norms)))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
