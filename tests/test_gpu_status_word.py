"""The status of steps whose norm kernel runs beside the stages: both set bits
of one word."""
import numpy as np
import pytest

import dgpr_b200 as dg
from tests import cases as C

pytestmark = pytest.mark.gpu


# 1 step: the norm between two stages; 64 and more: on a branch of its own
@pytest.mark.parametrize("nsteps", [1, 63, 64, 200])
@pytest.mark.parametrize("form", [dg.STEP_GAUSS, dg.STEP_NODAL])
@pytest.mark.parametrize("precision", [dg.FP64, dg.MIXED_FP32])
def test_status_does_not_depend_on_the_branch(precision, form, nsteps):
    """An inflow without a Mach root (a gas at four times the reference
    pressure: J = u + 2 c / (gamma - 1) is above 5 sqrt(gamma R Tt), where
    both roots are negative) reports itself while the norms stay finite; a
    state that is not finite has NaN roots and NaN norms in the same step and
    reports the norms.  A good state then clears the status."""
    mesh = dg.Mesh(3, 2, 2, 2, 1, C.box_nodes(3, 2, 2, 1, 2.0, 1.0, 1.0), [C.IN_, C.OUT_, C.NS_, C.W_, C.P_, C.P_])
    prm = C.params(mu=1e-2, u=0.3)
    good = C.random_state(prm, mesh.nelem, mesh.nb, np.random.default_rng(1), 1e-3)
    hot = good.reshape(mesh.nelem, 5, mesh.nb).copy()
    hot[:, 4] *= 4.0
    broken = good.copy()
    broken[0] = np.nan
    with dg.Solver(mesh, prm, precision=precision) as s:
        s.set_step_form(form)
        for U, code in ((hot.ravel(), dg.ERR_BOUNDARY), (broken, dg.ERR_NONFINITE), (good, None)):
            s.set_state(U)
            if code is None:
                assert np.all(np.isfinite(s.step(dg.RK4, 1e-12, nsteps)))
                continue
            with pytest.raises(dg.DgbError) as ex:
                s.step(dg.RK4, 1e-12, nsteps)
            assert ex.value.code == code
