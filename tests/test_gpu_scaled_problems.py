"""FP64 solves over FP64's range.  Multiplying a right-hand side or the moduli
by a power of two is exact in every operation of the solver, so iterates,
residuals and cycle counts have to come out the same up to that power, bit for
bit, also where the numbers lie far outside of FP32's range."""
import numpy as np
import pytest

from stz_gb300 import _lib
from stz_gb300.params import ADJOINT_DT, adjoint_shear, simple_shear
from stz_gb300.shear_sim import ShearSim

pytestmark = pytest.mark.gpu

POWERS = [-400, -150, -100, 100, 150, 400]
# one launch for all levels, and with the wide levels as tiles
SIZES = [(64, 64), (30, 31), (256, 200)]


def _src(m, n):
    return np.random.default_rng(m + n).standard_normal((n + 1, m, 2))


def _sim(P, **kw):
    return ShearSim(P, precision=_lib.FP64, tol_mode=_lib.TOL_RELATIVE, tol=1e-12, **kw)


@pytest.mark.parametrize("m,n", SIZES)
@pytest.mark.parametrize("k", POWERS)
def test_right_hand_side(m, n, k):
    P, b, s = simple_shear(m, n, viscosity=0.02), _src(m, n), 2.0 ** k
    with _sim(P) as sim:
        z, cycles, _ = sim.mg_solve(0.01, b, 0 * b)
        zk, cyclesk, _ = sim.mg_solve(0.01, b * s, 0 * b)
        assert cyclesk == cycles
        np.testing.assert_array_equal(zk, z * s)
        # from a guess, and with the residual of another solve in between
        g = z * (1 + 1e-3 * b)
        w, _, _ = sim.mg_solve(0.01, b, g)
        wk, _, _ = sim.mg_solve(0.01, b * s, g * s)
        np.testing.assert_array_equal(wk, w * s)
        v, vk = sim.mg_vcycle(0.01, b, g), sim.mg_vcycle(0.01, b * s, g * s)
        np.testing.assert_array_equal(vk, v * s)


@pytest.mark.parametrize("m,n", SIZES)
@pytest.mark.parametrize("k", POWERS)
def test_moduli(m, n, k):
    P, b, s = simple_shear(m, n, viscosity=0.02), _src(m, n), 2.0 ** k
    Q = P.copy(mu=P.mu * s, K=P.K * s, viscosity=P.viscosity * s)
    with _sim(P) as sim, _sim(Q) as simk:
        z, cycles, _ = sim.mg_solve(0.01, b, 0 * b)
        zk, cyclesk, _ = simk.mg_solve(0.01, b, 0 * b)
        assert cyclesk == cycles
        np.testing.assert_array_equal(zk, z / s)


@pytest.mark.parametrize("m,n", SIZES)
def test_zero_right_hand_side(m, n):
    """From a guess to zero: the stopping rule asks for a residual whose squares
    vanish, 150 decades below the first one."""
    g = _src(m, n)
    with _sim(simple_shear(m, n, viscosity=0.02)) as sim:
        z, cycles, _ = sim.mg_solve(0.01, 0 * g, g)
        assert np.abs(z).max() < 1e-150 and cycles > 0


def test_reference_rule():
    """The absolute stopping rule, whose threshold follows the moduli."""
    P, b, s = simple_shear(64, 64, viscosity=0.02), _src(64, 64), 2.0 ** 200
    Q = P.copy(mu=P.mu * s, K=P.K * s, viscosity=P.viscosity * s)
    with ShearSim(P, tol=1e4) as sim, ShearSim(Q, tol=1e4) as simk:
        z, cycles, _ = sim.mg_solve(0.01, b, 0 * b)
        zk, cyclesk, _ = simk.mg_solve(0.01, b * s, 0 * b)
        assert cyclesk == cycles
        np.testing.assert_array_equal(zk, z)


@pytest.mark.parametrize("k", [-300, -120, 120, 300])
def test_adjoint_seed(k):
    """The gradients are linear in the loss's factor (atomic adds: equal up to
    their order)."""
    from stz_gb300.adjoint import StepAdjoint
    P = adjoint_shear(32)
    rng = np.random.default_rng(5)
    chi = (600 + 30 * rng.standard_normal((32, 32))) / P.TZ
    with ShearSim(P, chi, tol_mode=_lib.TOL_RELATIVE, tol=1e-13) as sim:
        sim.set("tau", np.full((34, 32), 1.4 * P.s_y))
        adj = StepAdjoint(sim, ADJOINT_DT, 6, 3)
        adj.forward(np.full((32, 32), 2e-3))
        g, c = adj.backward()
        gk, ck = adj.backward(2.0 ** k)
    assert np.abs(c).max() > 0
    np.testing.assert_allclose(gk / 2.0 ** k, g, rtol=1e-10)
    assert np.abs(ck / 2.0 ** k - c).max() <= 1e-10 * np.abs(c).max()
