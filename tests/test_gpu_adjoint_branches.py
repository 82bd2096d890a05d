"""The adjoint's forward run takes the ENO branches that its reverse sweep
differentiates: those of the FP64 form, whatever the handle's advection."""
import numpy as np
import pytest

from stz_gb300 import _lib
from stz_gb300.adjoint import StepAdjoint
from stz_gb300.params import ADJOINT_DT, adjoint_shear
from stz_gb300.shear_sim import ShearSim

pytestmark = pytest.mark.gpu


def test_forward_is_the_fp64_form():
    P = adjoint_shear(48)
    rng = np.random.default_rng(2)
    chi = (600 + 30 * rng.standard_normal((48, 48))) / P.TZ
    tau = P.s_y * (1.4 + 0.05 * rng.standard_normal((50, 48)))
    out = []
    for advection in (_lib.ADV_AUTO, _lib.ADV_FP64):
        with ShearSim(P, chi, tol_mode=_lib.TOL_RELATIVE, tol=1e-13, advection=advection) as sim:
            sim.set("tau", tau)
            adj = StepAdjoint(sim, ADJOINT_DT, 6, 4)
            loss = adj.forward(np.full((48, 48), 2e-3))
            _, g = adj.backward()
            out.append((loss, g, sim.get("eps_pl"), sim.get("X")))
            # the handle's own steps keep its setting
            sim.steps(ADJOINT_DT, 1)
            out[-1] += (sim.get("X"),)
    (loss, g, eps, X, _), (loss1, g1, eps1, X1, _) = out
    assert loss == loss1
    np.testing.assert_array_equal(eps, eps1)
    np.testing.assert_array_equal(X, X1)
    # the reverse sweep adds atomically: equal up to the order, as two backward
    # calls are
    assert np.abs(g - g1).max() <= 1e-12 * np.abs(g).max()
    assert not np.array_equal(out[0][4], out[1][4])
