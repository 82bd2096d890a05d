"""The fixed-point advection and explicit step against their FP64 form, cell by
cell: an updated value may differ by the rounding of the values that it is
computed from (those of its own stencil), not by that of larger ones elsewhere
in its tile."""
import numpy as np
import pytest

from stz_gb300 import _lib
from stz_gb300.params import plastic_shear
from stz_gb300.shear_sim import ShearSim
from test_gpu_fixed_point import CELLS, EPS, NODES, _run, _state

pytestmark = pytest.mark.gpu

STRESS = ("p", "q", "s", "tau")


def _neighbours(a, period=None):
    """Largest magnitude within two columns (periodic) or two rows of each entry."""
    top = np.abs(a)
    for k in (-2, -1, 1, 2):
        b = np.roll(a, -k, axis=1)
        if period is not None:
            b[:, slice(-k, None) if k > 0 else slice(0, -k)] += np.sign(k) * period
        top = np.maximum(top, np.abs(b))
        c = np.zeros_like(top)
        if k > 0:
            c[:-k] = np.abs(a[k:])
        else:
            c[-k:] = np.abs(a[:k])
        top = np.maximum(top, c)
    return top


def _spread(P, kind, seed):
    """Every field over 14 decades (the map, whose values carry the node's
    place, and chi, which must stay positive, over six), or large in one corner
    of the layer and small elsewhere."""
    f = _state(P, "rough", seed)
    g = np.random.default_rng(seed + 1)
    if kind == "cells":
        for k in STRESS + ("u", "v"):
            f[k] *= 10.0 ** g.uniform(-14, 0, f[k].shape)
        f["chi"] *= 10.0 ** g.uniform(-6, 0, f["chi"].shape)
        f["Y"] *= 10.0 ** g.uniform(-6, 0, f["Y"].shape)
    else:
        for k in STRESS + ("u", "v"):
            a = np.full(f[k].shape, 1e-9)
            a[: P.n // 2, : P.m // 3] = 1
            f[k] *= a
    f["u"][0], f["u"][-1] = -P.u_bdry, P.u_bdry
    f["v"][0] = f["v"][-1] = 0
    return f


def _corners(a):
    """Largest of a node array's four values around each cell."""
    b = np.maximum(np.abs(a), np.abs(np.roll(a, -1, axis=1)))
    return np.maximum(b[:-1], b[1:])


def _around(a):
    """Largest of the four cells (rows -1..n given) around each node."""
    b = np.maximum(np.abs(a), np.abs(np.roll(a, 1, axis=1)))
    return np.maximum(b[:-1], b[1:])


def _bounds(P, f, dt, explicit):
    """Per cell: the sum of the magnitudes that the update adds up.  An upwind
    increment is at most 8 L h v (L: the stencil's largest value, h v: dt
    |velocity| / (2 dx)), spin and elastic terms 8 h v times the stress or
    modulus, the force 16 h times the stresses around the node over mu, the
    viscous and diffusive terms 8 times their factors."""
    h = 0.5 * dt * max(P.m / (P.bx - P.ax), P.n / (P.by - P.ay))
    nv = np.maximum(np.abs(f["u"]), np.abs(f["v"]))
    cv = _corners(nv)
    d = 2 * h * h / dt
    out = {}
    for k in CELLS:
        out[k] = _neighbours(f[k])[1:-1] * (1 + 8 * h * cv)
    if explicit:
        out["chi"] += 8 * d * P.chi_diff * _neighbours(f["chi"])[1:-1]
        for k in STRESS:
            out[k] += 8 * h * cv * (P.K + 2 * P.mu)
    out["s"] = out["s"] + 8 * h * cv * np.abs(f["tau"][1:-1])
    out["tau"] = out["tau"] + 8 * h * cv * np.abs(f["s"][1:-1])
    for k in ("X", "Y"):
        out[k] = _neighbours(f[k], (P.bx - P.ax) if k == "X" else None) * (1 + 8 * h * nv)
    if explicit:
        force = 16 * h / P.mu * sum(_around(f[k]) for k in STRESS)
        for k in ("u", "v"):
            out[k] = _neighbours(f[k]) * (1 + 8 * h * nv + 8 * d * P.viscosity / P.mu) + force
    else:
        out["u"], out["v"] = np.abs(f["u"]), np.abs(f["v"])
    return out


def _check(P, f, ref, got, dt, explicit, roundings=64):
    """64 roundings of those magnitudes: the FP64 form makes fewer than 24, the
    fixed-point form is held to 32 and rounds the sum (mixed handles: eight
    times as many)."""
    for k, s in _bounds(P, f, dt, explicit).items():
        err = np.abs(ref[k] - got[k])
        bad = err > roundings * EPS * s + 1e-300
        assert not bad.any(), (k, int(bad.sum()), float((err[bad] / s[bad]).max() / EPS))


SIZES = [(30, 15), (34, 17), (64, 48), (130, 65)]


@pytest.mark.parametrize("kind", ["cells", "corner"])
@pytest.mark.parametrize("m,n", SIZES)
def test_advection(m, n, kind):
    P = plastic_shear(m, n, u_bdry=1.0)
    f = _spread(P, kind, 10 * m + n)
    dt = 0.2 * (P.bx - P.ax) / m
    step = lambda sim: sim.advection_step(dt)
    ref = _run(P, f, _lib.FP64, _lib.ADV_FP64, step)
    _check(P, f, ref, _run(P, f, _lib.FP64, _lib.ADV_AUTO, step), dt, False)
    _check(P, f, ref, _run(P, f, _lib.MIXED, _lib.ADV_AUTO, step), dt, False, 8 * 64)


@pytest.mark.parametrize("kind", ["cells", "corner"])
@pytest.mark.parametrize("m,n", SIZES)
def test_explicit_step(m, n, kind):
    P = plastic_shear(m, n, u_bdry=1.0, viscosity=0.02, chi_diff=1e-3)
    f = _spread(P, kind, 10 * m + n + 1)
    dt = 0.5 * ((P.bx - P.ax) / m) ** 2
    step = lambda sim: sim.step_forward(dt)
    ref = _run(P, f, _lib.FP64, _lib.ADV_FP64, step)
    _check(P, f, ref, _run(P, f, _lib.FP64, _lib.ADV_AUTO, step), dt, True)
