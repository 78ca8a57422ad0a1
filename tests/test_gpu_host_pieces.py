"""Host calls step a state in pieces whose number goes by its size."""
import numpy as np
import pytest

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu


# 1080 and 5000 bytes an element: on either side of 1.5, 12 and 22 MB
@pytest.mark.parametrize("precision", [dg.FP64, dg.MIXED_FP32])
@pytest.mark.parametrize("p,n", [(2, (1, 1, 1)), (2, (11, 9, 14)), (2, (11, 9, 15)), (4, (17, 13, 10)), (4, (17, 13, 11)),
                                 (4, (18, 18, 13)), (4, (18, 18, 14))])
def test_step_host_equals_set_step_get(p, n, precision):
    """Two calls of two steps on the host state, the second in place and
    queued behind the first, against set_state, step and get_state: pieces
    change no result."""
    nodes = C.box_nodes(*n, 1, 2.0, 1.0, 1.0)
    prm = C.params(mu=1e-2, u=0.3)
    mesh = dg.Mesh(*n, p, 1, nodes, [C.F_, C.F_, C.NS_, C.W_, C.P_, C.P_])
    U = C.random_state(prm, mesh.nelem, mesh.nb, np.random.default_rng(p), 0.005)
    with dg.Solver(mesh, prm, precision=precision) as s:
        s.set_state(U)
        s.step(dg.RK4, 1e-4, 2)
        V = s.get_state()
        s.set_state(V)
        s.step(dg.RK4, 1e-4, 2)
        want = s.get_state()
        out = np.empty_like(U)
        s.step_host(dg.RK4, 1e-4, 2, U, out, wait=False)
        s.step_host(dg.RK4, 1e-4, 2, out, out, wait=False)
        s.synchronize()
    assert np.array_equal(out, want)
