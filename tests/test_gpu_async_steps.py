"""Queued host calls return before the calls ahead of them have run."""
import numpy as np
import pytest
import torch

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu


def test_a_long_call_queues_behind_a_short_one():
    """60 steps, then 64 of the same size, both queued: when the second call
    returns the first one's output is still the NaN that it held (its 60 steps
    of some 0.5 ms each are not over), and the state that comes out is that of
    the blocking calls, bit for bit.  A blocking call of another step size
    beforehand has made room for 128 norms, so nothing has to be allocated;
    no norms are asked for, whose copy to pageable memory would wait."""
    n, dt = (24, 24, 24), 1e-5
    mesh = dg.Mesh(*n, 3, 1, C.box_nodes(*n, 1, 2.0, 1.0, 1.0), [C.P_] * 6)
    prm = C.params(mu=1e-2, u=0.3)
    U = C.random_state(prm, mesh.nelem, mesh.nb, np.random.default_rng(1), 0.005)
    pinned = [torch.empty(U.size, dtype=torch.float64).pin_memory().numpy() for _ in range(3)]
    a, b, c = pinned
    with dg.Solver(mesh, prm) as s:
        a[:] = U
        s.step_host(dg.RK4, dt, 60, a, b)
        s.step_host(dg.RK4, dt, 64, b, c)
        want = c.copy()
    with dg.Solver(mesh, prm) as s:
        s.set_state(U)
        s.step(dg.RK4, 0.5 * dt, 128)
        s.step_host(dg.RK4, dt, 3, a, b)  # the graph of dt, and the call's events and streams
        s.synchronize()
        b[:] = np.nan
        s.step_host(dg.RK4, dt, 60, a, b, norms=False, wait=False)
        s.step_host(dg.RK4, dt, 64, b, c, norms=False, wait=False)
        queued = np.isnan(b[0])
        s.synchronize()
        assert queued
        assert np.array_equal(c, want)
