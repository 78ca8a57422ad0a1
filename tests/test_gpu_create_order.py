"""What dgb_create leaves queued comes before the handle's later work."""
import threading
import time

import numpy as np
import pytest
import torch

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [dg.FP64, dg.MIXED_FP32])
def test_a_busy_default_stream_does_not_reach_the_state(precision):
    """While another thread keeps some 10 ms of work on the default stream, a
    handle is made, given a state and stepped on its own stream, which does
    not wait for the default one: the state and the step are those of an idle
    device.  (A state cleared on the default stream would be cleared after
    it was set.)"""
    mesh = dg.Mesh(6, 5, 4, 3, 1, C.box_nodes(6, 5, 4, 1, 2.0, 1.0, 1.0), [C.F_, C.F_, C.NS_, dg.ISOTHERMAL_WALL, C.P_, C.P_])
    prm = C.params(mu=1e-2, u=0.3)
    U = C.random_state(prm, mesh.nelem, mesh.nb, np.random.default_rng(1), 0.005)

    def run():
        with dg.Solver(mesh, prm, precision=precision) as s:
            s.set_state(U)
            torch.cuda.synchronize()
            got = s.get_state()
            s.step(dg.RK4, 1e-5, 2)
            return got, s.get_state()

    want = run()
    stop = threading.Event()

    def load():
        while not stop.is_set():
            torch.cuda._sleep(20_000_000)
            time.sleep(0.008)

    other = threading.Thread(target=load)
    other.start()
    try:
        outs = [run() for _ in range(3)]
    finally:
        stop.set()
        other.join()
    for got, stepped in outs:
        assert np.array_equal(got, U)
        assert np.array_equal(stepped, want[1])
