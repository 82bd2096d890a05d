"""The advection and explicit-step kernels in 64-bit fixed point against the
FP64 form of the same step (STZG_ADV_FP64), from the same fields: sizes
around the 32 x 16 tile and its seam, rough fields, cells of one tile many
orders of magnitude apart, no velocity, plastic flow, and values that are not
finite (whose tiles the FP64 form takes)."""
import numpy as np
import pytest

from stz_gb300 import _lib
from stz_gb300.params import plastic_shear
from stz_gb300.shear_sim import ShearSim

pytestmark = pytest.mark.gpu

CELLS, NODES = ("p", "q", "s", "tau", "chi"), ("X", "Y", "u", "v")
EPS = 2.0 ** -53


def _state(P, kind, seed):
    g = np.random.default_rng(seed)
    m, n = P.m, P.n
    f = {k: P.s_y * 0.2 * g.standard_normal((n + 2, m)) for k in CELLS}
    f["chi"] = (600.0 + 30.0 * g.standard_normal((n + 2, m))) / P.TZ
    x = P.ax + (P.bx - P.ax) / m * np.arange(m)[None, :]
    y = np.linspace(P.ay, P.by, n + 1)[:, None]
    f["X"] = x + 0.01 * g.standard_normal((n + 1, m))
    f["Y"] = y + 0.01 * g.standard_normal((n + 1, m))
    f["u"] = P.u_bdry * np.linspace(-1, 1, n + 1)[:, None] + 0.1 * P.u_bdry * g.standard_normal((n + 1, m))
    f["v"] = 0.1 * P.u_bdry * g.standard_normal((n + 1, m))
    f["u"][0], f["u"][-1] = -P.u_bdry, P.u_bdry
    f["v"][0] = f["v"][-1] = 0
    if kind == "spread":
        for k in ("p", "q", "s", "tau"):
            f[k] *= 10.0 ** g.uniform(-14, 0, f[k].shape)
        f["v"] *= 10.0 ** g.uniform(-14, 0, f["v"].shape)
    elif kind == "still":
        f["u"][:] = f["v"][:] = 0
    elif kind == "plastic":
        f["tau"] += 1.02 * P.s_y
    elif kind == "nonfinite":
        f["q"][n // 2, m // 3] = np.nan
        f["chi"][1, m - 1] = np.inf
    return f


def _run(P, f, prec, advection, step):
    with ShearSim(P, precision=prec, advection=advection) as sim:
        for k in CELLS + NODES:
            sim.set(k, f[k])
        step(sim)
        out = {k: sim.get(k) for k in CELLS + NODES + ("eps_pl",)}
    out.update({k: out[k][1:-1] for k in CELLS})
    return out


def _compare(P, f, ref, got, dt, plastic):
    """An update is the old value and increments: at most four of ENO values
    times dt |velocity| / (2 dx) (below 4 max|f| h for each direction), the
    elastic rate and, in the explicit step, the force.  Each side rounds
    every operation at EPS of its operands, fewer than 64 of them; the fixed
    form's integers are cut at 2^-58 of the tile's largest value.  A plastic
    law adds the sensitivity of its exponentials (arguments up to 80)."""
    h = 0.5 * dt * max(P.m / (P.bx - P.ax), P.n / (P.by - P.ay))
    top = {k: np.nanmax(np.abs(np.where(np.isfinite(a), a, 0))) for k, a in f.items()}
    vel = max(top["u"], top["v"])
    stress = max(top[k] for k in ("p", "q", "s", "tau"))
    elastic = 8 * h * vel * (P.K + 2 * P.mu)
    grow = 1 + 8 * h * vel
    scale = {k: grow * top[k] + 8 * h * vel * stress + elastic for k in ("p", "q", "s", "tau")}
    scale["chi"] = grow * top["chi"]
    # the map is unwrapped by the period at the seam
    scale["X"] = scale["Y"] = grow * (max(top["X"], top["Y"]) + P.bx - P.ax)
    scale["u"] = scale["v"] = grow * vel + (12 * h * stress + 16 * P.viscosity * h * vel / dt * h) / P.mu
    scale["eps_pl"] = stress / P.mu
    tol = 64 * EPS * (80 if plastic else 1)
    for k, s in scale.items():
        a, b = ref[k], got[k]
        ok = np.isfinite(a)
        assert np.array_equal(ok, np.isfinite(b)), k
        assert np.array_equal(np.isnan(a), np.isnan(b)), k
        err = np.abs(a[ok] - b[ok]).max()
        assert err <= tol * s, (k, err, tol * s)


SIZES = [(8, 6), (30, 15), (32, 16), (34, 17), (62, 33), (64, 31), (66, 48), (128, 65)]


@pytest.mark.parametrize("kind", ["rough", "spread", "still", "plastic", "nonfinite"])
@pytest.mark.parametrize("m,n", SIZES)
def test_advection(m, n, kind):
    P = plastic_shear(m, n, u_bdry=1.0)
    f = _state(P, kind, 100 * m + n)
    dt = 0.2 * (P.bx - P.ax) / m
    step = lambda sim: sim.advection_step(dt)
    ref = _run(P, f, _lib.FP64, _lib.ADV_FP64, step)
    for prec in (_lib.FP64, _lib.MIXED):
        _compare(P, f, ref, _run(P, f, prec, _lib.ADV_AUTO, step), dt, kind == "plastic")
    if kind == "plastic":
        assert np.abs(ref["eps_pl"]).max() > 0


@pytest.mark.parametrize("kind", ["rough", "spread", "still", "plastic", "nonfinite"])
@pytest.mark.parametrize("m,n", SIZES)
def test_explicit_step(m, n, kind):
    P = plastic_shear(m, n, u_bdry=1.0, viscosity=0.02, chi_diff=1e-3)
    f = _state(P, kind, 100 * m + n + 1)
    dt = 0.5 * ((P.bx - P.ax) / m) ** 2
    step = lambda sim: sim.step_forward(dt)
    ref = _run(P, f, _lib.FP64, _lib.ADV_FP64, step)
    _compare(P, f, ref, _run(P, f, _lib.FP64, _lib.ADV_AUTO, step), dt, kind == "plastic")


@pytest.mark.parametrize("x", [10.0, 15.0, 19.9, 20.1])
def test_plastic_law_at_its_line(x):
    """The one-exponential form of the athermal law takes over where Omega
    eps0 sbar/theta is 20 (the form with tanh below it): that number at yield
    on both sides of the line, against the CPU oracle, to the gate of the
    explicit runs.  100 steps: past 200 the stiff sub-steps amplify the last
    bit of the inputs to 1e-3 in the oracle itself."""
    from oracle.bind import OracleSim
    from parity import group_errors
    from stz_gb300.shear_sim import random_chi
    N, M = 48, 40
    P = plastic_shear(N, M, u_bdry=4.0, s_y=0.2, viscosity=0.01)
    P.Omegaeps0 = x * P.theta / P.s_y
    chi = random_chi(N, M, 3, 600.0, 30.0, P.TZ, 21)
    dt = 0.5 * ((P.bx - P.ax) / N) ** 2
    o = OracleSim(P, chi)
    o.steps_direct(dt, 100)
    assert np.abs(o.eps_pl).max() > 0, "plastic-active case"
    for advection in (_lib.ADV_AUTO, _lib.ADV_FP64):
        with ShearSim(P, chi, advection=advection) as sim:
            sim.step_forward(dt, 100)
            err = group_errors(o.fields(), sim.fields(), M)
            assert max(err.values()) < 1e-10, (advection, err)
    o.close()
