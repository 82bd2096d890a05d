"""The work this framework is used for, as cases that can be timed and checked.

A case is a dict of plain values; ``prepare`` makes from it and a seed what a
program has in hand (a simulation handle, host-side fields), ``run`` is one
pass through the public entry points and returns every result, ``work`` the
bytes and operations such a pass cannot do without, and ``exact`` the same
results from a plain 64-bit restatement in torch (Fourier transform along the
periodic direction and block elimination across it in place of multigrid).

A stepping pass restarts the handle from a saved state, as a program does that
resumes a run, sweeps parameters or holds the fields itself: the state goes up
from pinned host memory, the steps run, the new state comes down.  The states
are those of a layer under shear after the walls' ramp: a stress with a mean
and smooth fluctuations, an effective temperature with a given correlation
length, a sheared and slightly perturbed reference map.  Stresses, the two
maps and the velocity components come back as one array each, since single
components can vanish (simple shear leaves p, q and v at rounding level).
"""
import math

import numpy as np
import torch

from stz_gb300 import _lib
from stz_gb300.adjoint import StepAdjoint
from stz_gb300.batch import Batch
from stz_gb300.ct_sim import CtSim, transform_shear
from stz_gb300.params import ADJOINT_DT, adjoint_shear, default_dt, simple_shear
from stz_gb300.shear_sim import ShearSim
from stz_gb300.tgmg import PoissonFD, Predict, Tgmg

T0 = 1.5  # time of the saved states: past the walls' ramp
THETA = ("c0", "Omegaeps0", "chi_inf", "s_y")


def _qs(name, m, n, steps, **kw):
    c = {"name": name, "kind": "qs", "m": m, "n": n, "steps": steps, "mixed": True, "relative": True, "tol": 1e-10,
         "plastic": False, "host": False, "l": 4.0, "std": 30.0}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call of an interactive or coupled program: one step of a
        # small sample, where launches and round trips count
        _qs("step 64 mixed, one step", 64, 64, 1),
        # the reference-like small run (128 squared, FP64, relative residual 1e-10)
        _qs("steps 128 fp64", 128, 128, 20, mixed=False),
        # the default handle of a caller who switches over from the CPU class
        # (FP64, the reference's absolute stopping rule and predicted V-cycle
        # counts), a ragged rectangular grid, every cell near yield
        _qs("steps 190x131 default plastic", 190, 131, 8, mixed=False, relative=False, tol=1e4, plastic=True),
        # plastic flow at a production size in mixed precision
        _qs("steps 512 mixed plastic", 512, 512, 20, plastic=True),
        # the FP64 production run (1024 squared)
        _qs("steps 1024 fp64", 1024, 1024, 8, mixed=False, l=8.0),
        # fields that the caller keeps in host memory: the state travels both
        # ways around every step
        _qs("host steps 1024x768 mixed", 1024, 768, 4, host=True, l=8.0),
        # the headline run (2048 squared, mixed precision), one frame's steps
        _qs("steps 2048 mixed", 2048, 2048, 24, l=16.0, std=40.0),
        # the explicit step, which resolves the elastic waves
        {"name": "explicit 1024x768", "kind": "direct", "m": 1024, "n": 768, "steps": 20},
        # a parameter sweep: independent samples of uneven sizes in one call
        {"name": "batch of 24, 64 to 512", "kind": "batch", "count": 24, "steps": 8, "mixed": True},
        # calibration: the loss of a run and its gradients
        {"name": "adjoint 96", "kind": "adjoint", "m": 96, "n": 96, "steps": 12, "every": 4},
        # the same physics in coordinates that follow the shear (the frame of
        # the reference's other driver), y periodic
        {"name": "sheared frame 512x256", "kind": "ct", "m": 512, "n": 256, "steps": 4},
        # the general multigrid on its own: a Poisson problem, V-cycles with
        # the reference's predictor
        {"name": "poisson 1025", "kind": "poisson", "m": 1025, "n": 1025},
    ]


def _log(rng, lo, hi, even=False):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, v - (v & 1)) if even else v


def draw(rng):
    kind = rng.choice(["qs", "qs", "qs", "qs", "qs", "qs", "direct", "batch", "adjoint", "ct", "poisson"])
    if kind == "qs":
        m, n = _log(rng, 64, 2048, True), _log(rng, 64, 2048)
        mixed, plastic = rng.random() < 0.6, rng.random() < 0.4
        if not mixed:
            m, n = min(m, 1024), min(n, 1024)
        steps = max(1, min(24 if mixed else 16, int(rng.uniform(0.3, 1) * (1e8 if mixed else 1.2e7) / (m * n))))
        relative = mixed or rng.random() < 0.6
        host = rng.random() < 0.2
        c = _qs("", m, n, min(steps, 6) if host else steps, mixed=mixed, relative=relative,
                tol=1e-10 if relative else 1e4, plastic=plastic, host=host, l=round(rng.uniform(3, 16), 2),
                std=round(rng.uniform(10, 50), 1))
        del c["name"]
        return c
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(6, 32), "steps": rng.randint(2, 8), "mixed": rng.random() < 0.7}
    if kind == "adjoint":
        return {"kind": kind, "m": _log(rng, 32, 96, True), "n": _log(rng, 32, 96), "steps": rng.randint(4, 12),
                "every": rng.randint(2, 6)}
    if kind == "ct":
        # the reference's driver: nearly square cells, lines that halve evenly
        m = 32 * rng.randint(4, 16)
        return {"kind": kind, "m": m, "n": 32 * max(2, round(m / 64 * rng.uniform(0.8, 1.25))), "steps": rng.randint(1, 4)}
    if kind == "poisson":
        return {"kind": kind, "m": _log(rng, 65, 1025), "n": _log(rng, 65, 1025)}
    m, n = _log(rng, 64, 1024, True), _log(rng, 64, 768)
    return {"kind": "direct", "m": m, "n": n, "steps": rng.randint(4, 20)}


# ---- inputs ------------------------------------------------------------------

def _gen(seed, extra=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + extra)


def _smooth(g, count, n, m, l):
    """count fields of n x m with unit deviation and correlation length l (cells)."""
    w = torch.randn((count, n, m), generator=g, device="cuda", dtype=torch.float64)
    ky = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(m, device="cuda", dtype=torch.float64)[None, :]
    f = torch.exp(-2 * (math.pi * l) ** 2 * (kx * kx + ky * ky) / 2)
    w = torch.fft.irfft2(torch.fft.rfft2(w) * f, s=(n, m))
    return w / w.std(dim=(1, 2), keepdim=True)


def _ghosts(a):
    """Cell rows -1..n from the rows 0..n-1 by linear extrapolation at the walls."""
    return torch.cat([2 * a[..., :1, :] - a[..., 1:2, :], a, 2 * a[..., -1:, :] - a[..., -2:-1, :]], dim=-2)


def _params(c):
    if c["plastic"]:
        return simple_shear(c["m"], c["n"], u_bdry=0.04)
    return simple_shear(c["m"], c["n"])


def _state(P, seed, l, std, plastic, extra=0):
    """The saved state on the GPU: stress (4, n+2, m), chi (n+2, m), X and Y
    (2, n+1, m), vel (n+1, m, 2), eps_pl (n, m); time T0."""
    m, n, g = P.m, P.n, _gen(seed, extra)
    f = _smooth(g, 9, n + 1, m, l)
    # plastic: around 1.02 times the yield stress, so that most cells flow;
    # elastic: the stress that the reference-like walls build up per unit time
    stress = (0.01 * P.s_y if plastic else 5e-6) * f[:4, :n]
    stress[3] += 1.02 * P.s_y if plastic else 1e-4
    chi = (600.0 + std * f[4, :n]) / P.TZ
    y = torch.linspace(-1, 1, n + 1, device="cuda", dtype=torch.float64)[:, None]
    inside = torch.cos(0.5 * math.pi * y) ** 2
    inside[0] = inside[-1] = 0
    dx, dy = (P.bx - P.ax) / m, (P.by - P.ay) / n
    x = P.ax + dx * torch.arange(m, device="cuda", dtype=torch.float64)[None, :]
    maps = torch.stack([x - P.u_bdry * (T0 - 0.5) * y + 0.05 * dx * inside * f[5], y + 0.05 * dy * inside * f[6]])
    vel = torch.stack([P.u_bdry * y + 0.02 * P.u_bdry * inside * f[7], 0.02 * P.u_bdry * inside * f[8]], dim=-1)
    eps = 1e-3 * f[0, :n] ** 2 if plastic else torch.zeros((n, m), device="cuda", dtype=torch.float64)
    return {"stress": _ghosts(stress), "chi": _ghosts(chi), "map": maps, "vel": vel, "eps_pl": eps}


def _pinned(state):
    out = {}
    for k, v in state.items():
        out[k] = torch.empty(v.shape, dtype=torch.float64, pin_memory=True)
        out[k].copy_(v)
    torch.cuda.synchronize()
    return out


def _pointers(buf):
    """p, q, s, tau, chi, X, Y, vel, eps_pl of the bulk transfers."""
    at = [buf["stress"][k] for k in range(4)] + [buf["chi"], buf["map"][0], buf["map"][1], buf["vel"], buf["eps_pl"]]
    return [a.data_ptr() for a in at]


def _load(sim, up):
    """The saved state's wall speed is part of the handle, set once."""
    sim.set("u", up["vel"][..., 0].contiguous().numpy())


def _restart(sim, st, up):
    sim.time = T0
    if st["plastic"]:
        sim.set("eps_pl", up["eps_pl"].numpy())


def _batch_cases(c, seed):
    rng = np.random.default_rng(int(c["count"]) * 7919 + int(c["steps"]))
    sizes = [int(s) for s in rng.permutation(np.resize([64, 96, 128, 192, 256, 384, 512], c["count"]))]
    rng = np.random.default_rng(seed)
    return [(N, float(rng.uniform(0.2, 0.6)), float(rng.uniform(800.0, 1000.0)), float(rng.uniform(10.0, 50.0)))
            for N in sizes]


def _batch_states(c, seed):
    params, states = [], []
    for k, (N, c0, chi_inf, std) in enumerate(_batch_cases(c, seed)):
        P = simple_shear(N, c0=c0, chi_inf_K=chi_inf)
        params.append(P)
        states.append(_state(P, seed, 4.0, std, False, extra=k + 1))
    return params, states


def _direct_dt(P):
    return ((P.bx - P.ax) / P.m) ** 2 * 0.5  # the explicit driver's dt = dx^2 / 2


def _adjoint_inputs(c, seed):
    P = adjoint_shear(c["m"], c["n"])
    f = _smooth(_gen(seed), 3, P.n, P.m, 4.0)
    chi = (600.0 + 30.0 * f[0]) / P.TZ
    tau = _ghosts(P.s_y * (1.4 + 0.05 * f[1]))
    target = 2e-3 * (1 + 0.3 * f[2])
    return P, chi, tau, target


def _ct_inputs(c, seed):
    P = transform_shear(c["m"], c["n"])
    m, n = P.m, P.n
    f = _smooth(_gen(seed), 9, n, m, 4.0)
    dx, dy = (P.bx - P.ax) / m, (P.by - P.ay) / n
    x = P.ax + dx * torch.arange(m, device="cuda", dtype=torch.float64)[None, :]
    y = P.ay + dy * torch.arange(n, device="cuda", dtype=torch.float64)[:, None]
    h = {"u": 1e-5 * f[0], "v": 1e-5 * f[1], "p": 0.02 * f[2], "q": 0.02 * f[3], "s": 0.02 * f[4],
         "tau": 0.9 + 0.02 * f[5], "chi": (600.0 + 30.0 * f[6]) / P.TZ, "X": x + 0.05 * dx * f[7],
         "Y": y + 0.05 * dy * f[8]}
    out = {}
    for k, v in h.items():
        v = torch.cat([v, v[:1] + (P.by - P.ay if k == "Y" else 0)], dim=0)
        out[k] = np.ascontiguousarray(v.cpu().numpy())
    return P, out


CT_T0 = 50.0
CT_DT = 0.5 / 1e-3 / 600  # the reference driver's step


def _poisson_b(c, seed):
    """A sum of Gaussian sources, as the reference's timing program sets one up."""
    g = torch.Generator().manual_seed(1000003 * int(seed))
    x = torch.linspace(-1, 1, c["m"], device="cuda", dtype=torch.float64)[None, :]
    y = torch.linspace(-1, 1, c["n"], device="cuda", dtype=torch.float64)[:, None]
    b = torch.zeros((c["n"], c["m"]), device="cuda", dtype=torch.float64)
    for gx, gy, a, w in torch.rand((6, 4), generator=g, dtype=torch.float64).tolist():
        b += (2 * a - 1) * torch.exp(-((x - 1.2 * gx + 0.6) ** 2 + (y - 1.2 * gy + 0.6) ** 2) / (2 * (0.1 + 0.2 * w) ** 2))
    return b


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "qs":
        P = _params(c)
        sim = ShearSim(P, precision=_lib.MIXED if c["mixed"] else _lib.FP64,
                       tol_mode=_lib.TOL_RELATIVE if c["relative"] else _lib.TOL_REFERENCE, tol=c["tol"],
                       extrapolate=c["relative"])
        up = _pinned(_state(P, seed, c["l"], c["std"], c["plastic"]))
        down = _pinned(up)
        _load(sim, up)
        return {"case": c, "sim": sim, "up": up, "down": down, "plastic": c["plastic"], "dt": default_dt(c["m"])}
    if kind == "direct":
        P = simple_shear(c["m"], c["n"], u_bdry=0.04, viscosity=0.02)
        sim = ShearSim(P)
        up = _pinned(_state(P, seed, 6.0, 30.0, True))
        down = _pinned(up)
        _load(sim, up)
        return {"case": c, "sim": sim, "up": up, "down": down, "plastic": True, "dt": _direct_dt(P)}
    if kind == "batch":
        params, states = _batch_states(c, seed)
        batch = Batch(params, precision=_lib.MIXED if c["mixed"] else _lib.FP64)
        ups = [_pinned(s) for s in states]
        total = {k: sum(u[k].numel() for u in ups) for k in ups[0]}
        flat = {k: torch.empty(v, dtype=torch.float64, pin_memory=True) for k, v in total.items()}
        downs, at = [], dict.fromkeys(total, 0)
        for u in ups:
            d = {}
            for k, v in u.items():
                d[k] = flat[k][at[k]:at[k] + v.numel()].view(v.shape)
                at[k] += v.numel()
            downs.append(d)
        for k, u in enumerate(ups):
            _load(batch.sim(k), u)
        return {"case": c, "batch": batch, "ups": ups, "downs": downs, "flat": flat}
    if kind == "adjoint":
        P, chi, tau, target = _adjoint_inputs(c, seed)
        sim = ShearSim(P, tol_mode=_lib.TOL_RELATIVE, tol=1e-13)
        host = {k: np.ascontiguousarray(v.cpu().numpy()) for k, v in (("chi", chi), ("tau", tau), ("target", target))}
        return {"case": c, "sim": sim, "adj": StepAdjoint(sim, ADJOINT_DT, c["steps"], c["every"]), **host}
    if kind == "ct":
        P, fields = _ct_inputs(c, seed)
        return {"case": c, "sim": CtSim(P), "fields": fields}
    q = PoissonFD(c["m"], c["n"], -1.0, 1.0, -1.0, 1.0)
    q.b[...] = _poisson_b(c, seed).cpu().numpy()
    return {"case": c, "q": q, "solver": Tgmg(q), "predict": Predict()}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind in ("qs", "direct"):
        sim, up, down = state["sim"], state["up"], state["down"]
        _restart(sim, state, up)
        if kind == "qs" and c["host"]:
            ptr = _pointers(down)
            sim.step_host(state["dt"], _pointers(up), ptr)
            for _ in range(c["steps"] - 1):
                sim.step_host(state["dt"], ptr, ptr)
            return down
        sim.upload(_pointers(up))
        if kind == "qs":
            sim.steps(state["dt"], c["steps"])
        else:
            sim.step_forward(state["dt"], c["steps"])
        sim.download(_pointers(down))
        return down
    if kind == "batch":
        batch = state["batch"]
        for k, up in enumerate(state["ups"]):
            batch.sim(k).time = T0
            batch.sim(k).upload(_pointers(up))
        batch.run(default_dt(64), c["steps"])
        for k, down in enumerate(state["downs"]):
            batch.sim(k).download(_pointers(down))
        return state["flat"]
    if kind == "adjoint":
        sim, adj = state["sim"], state["adj"]
        sim.set_state(state["chi"])
        sim.set("tau", state["tau"])
        loss = adj.forward(state["target"])
        g_theta, g_chi = adj.backward()
        return {"loss": loss, "g_theta": g_theta, "g_chi": g_chi, "eps_pl": sim.get("eps_pl")}
    if kind == "ct":
        sim = state["sim"]
        sim.time = CT_T0
        for k, v in state["fields"].items():
            sim.set(k, v)
        sim.step_forward_quasistatic(CT_DT, c["steps"])
        return {"stress": np.stack([sim.get(k) for k in ("p", "q", "s", "tau")]), "chi": sim.get("chi"),
                "map": np.stack([sim.get("X"), sim.get("Y")]), "vel": np.stack([sim.get("u"), sim.get("v")])}
    q = state["q"]
    q.z[...] = 0
    state["solver"].solve_v_cycle(state["predict"])
    return q.z


def work(case):
    """Per cell and step: p, q, s, tau, chi, X, Y and the velocity read and
    written once (144 B); 14 ENO values and upwind products, the net force,
    one residual and one V-cycle of the projection, the stress correction
    (about 500 operations).  The state's way up and down once per pass."""
    c, kind = case, case["kind"]
    if kind == "batch":
        cells = sum(N * N for N, *_ in _batch_cases(c, 0))
    else:
        cells = c["m"] * c["n"]
    if kind == "poisson":
        # b in, z out; a few V-cycles of about 60 operations per point each
        return {"bytes": 16.0 * cells, "flops": 8 * 60.0 * cells}
    steps = c["steps"]
    if kind == "adjoint":
        # forward, recomputation and the reverse sweep
        return {"bytes": 3 * 144.0 * cells * steps, "flops": 4 * 500.0 * cells * steps}
    moved = 2 * 72.0 * cells * (steps if c.get("host") else 1)
    return {"bytes": 144.0 * cells * steps + moved, "flops": (300.0 if kind == "direct" else 500.0) * cells * steps}


# ---- 64-bit restatement --------------------------------------------------------

def _eno2(p0, p1, p2, p3):
    return torch.where((p0 - 2 * p1 + p2).abs() > (p1 - 2 * p2 + p3).abs(), 3 * p1 - 4 * p2 + p3, p0 - p2)


def _sx(a, k, period=None):
    """a at column i+k; a map gains the period beyond the seam."""
    r = torch.roll(a, -k, -1)
    if period is not None:
        e = torch.zeros(a.shape[-1], dtype=a.dtype, device=a.device)
        if k > 0:
            e[-k:] = period
        else:
            e[:-k] = -period
        r = r + e
    return r


def _ddx(a, u, period=None):
    """Upwind ENO2 difference along x (twice the derivative times dx)."""
    r, r2, l, l2 = (_sx(a, k, period) for k in (1, 2, -1, -2))
    return torch.where(u > 0, _eno2(r, a, l, l2), -_eno2(l, a, r, r2))


def _ddy(g, v, cells):
    """Along y.  cells: g holds rows -1..n, the result rows 0..n-1; nodes: g
    holds rows 0..n, the result rows 1..n-1.  One-sided next to a wall."""
    c, d, u = g[..., 1:-1, :], g[..., :-2, :], g[..., 2:, :]
    dd, uu = torch.roll(d, 1, -2), torch.roll(u, -1, -2)
    up, dn = _eno2(u, c, d, dd), -_eno2(d, c, u, uu)
    up = torch.cat([2 * (c - d)[..., :1, :], up[..., 1:, :]], dim=-2)
    dn = torch.cat([dn[..., :-1, :], -2 * (c - u)[..., -1:, :]], dim=-2)
    return torch.where(v > 0, up, dn)


def _dplastic(P, th, sbar, chi):
    c0, Om, _, s0 = th
    De, thinv, tau0 = P.Delta, 1 / P.theta, P.tau0
    bfac = torch.exp(-1 / chi)
    if P.stz_model == 0:
        sC1 = math.exp(-De * thinv)
        sC2 = torch.cosh(Om * sbar * thinv)
        sC, sT = sC1 * sC2, torch.tanh(Om * sbar * thinv)
        st = torch.clamp(sbar, min=1e-12)
        pM = 1 + st * sT / s0 + P.rho / (2 * sC2)
        M = s0 / (2 * st) * (pM - torch.sqrt(pM * pM - 4 * st * sT / s0))
        D = bfac * sC * (sT - M) / tau0
        return D, 2 * D * sbar / (s0 * c0), bfac * P.kappa * sC1 * P.rho / (tau0 * c0)
    on = sbar >= s0
    sb = torch.where(on, sbar, torch.ones_like(sbar))
    sC = 0.5 * (torch.exp((Om * sb - De) * thinv) + torch.exp((-Om * sb - De) * thinv))
    D = torch.where(on, bfac * sC * (torch.tanh(Om * sb * thinv) - s0 / sb) / tau0, torch.zeros_like(sb))
    return D, 2 * D * sb / (s0 * c0), torch.zeros_like(sb)


def _plastic(P, th, sbar, chi, dt):
    """Adaptive sub-steps of the plastic law: (stress drop, new chi)."""
    s, left, on = sbar, torch.full_like(sbar, dt), sbar >= 1e-12
    while bool(on.any()):
        D, d1, d2 = _dplastic(P, th, s, chi)
        D = 2 * P.t_scale * P.mu * D
        big = (left * D).abs() > P.adapt_fac
        adt = torch.where(big, P.adapt_fac / torch.where(big, D, torch.ones_like(D)).abs(), left)
        adt = torch.where(on, adt, torch.zeros_like(adt))
        s = s - adt * D
        chi = chi + (d1 * (th[2] - chi) - d2 * chi) * P.t_scale * adt
        left = left - adt
        on = on & big
    return sbar - s, chi


class _Solve:
    """(stencil) z = b on m x (n+1) nodes, x periodic, z given on the walls:
    rfft along x, then elimination of the 2 x 2 blocks across the rows."""

    def __init__(self, P, dt):
        m, n = P.m, P.n
        self.m, self.n = m, n
        xs, ys = m / (P.bx - P.ax), n / (P.by - P.ay)
        Kq, w = P.K + P.mu / 3, P.viscosity / dt
        Kmx, Kmy = (Kq + P.mu + w) * xs * xs, (Kq + P.mu + w) * ys * ys
        mx, my = (P.mu + w) * xs * xs, (P.mu + w) * ys * ys
        qK = 0.25 * Kq * xs * ys
        k = 2 * math.pi * torch.arange(m // 2 + 1, device="cuda", dtype=torch.float64) / m
        one, s = torch.ones_like(k), torch.sin(k)
        z = torch.zeros_like(k)

        def blocks(a, b, c, d):
            return torch.stack([torch.stack([a, b], -1), torch.stack([c, d], -1)], -2).to(torch.complex128)

        self.L = blocks(my * one, z, z, Kmy * one) - 2j * blocks(z, qK * s, qK * s, z)
        self.U = self.L.conj()
        C = blocks(-4 * Kmx * torch.sin(k / 2) ** 2 - 2 * my, z, z, -4 * mx * torch.sin(k / 2) ** 2 - 2 * Kmy)

        def inv(M):
            a, b, c, d = M[..., 0, 0], M[..., 0, 1], M[..., 1, 0], M[..., 1, 1]
            return torch.stack([torch.stack([d, -b], -1), torch.stack([-c, a], -1)], -2) / (a * d - b * c)[..., None, None]

        D, E = [inv(C)], [torch.zeros_like(C)]
        for _ in range(2, n):
            E.append(self.L @ D[-1])
            D.append(inv(C - E[-1] @ self.U))
        self.E, self.D = E, torch.stack(D)
        self.F = list(self.D @ self.U)

    def __call__(self, b, wall0, wall1):
        """b: (n-1, m, 2) of the interior rows; the walls' z (m, 2) each."""
        B = torch.fft.rfft(b, dim=1)[..., None]
        W0, W1 = torch.fft.rfft(wall0, dim=0)[..., None], torch.fft.rfft(wall1, dim=0)[..., None]
        rows = list(B)
        rows[0] = rows[0] - self.L @ W0
        rows[-1] = rows[-1] - self.U @ W1
        y = [rows[0]]
        for j in range(1, len(rows)):
            y.append(torch.baddbmm(rows[j], self.E[j], y[-1], alpha=-1))
        G = list(self.D @ torch.stack(y))
        x = [G[-1]]
        for j in range(len(rows) - 2, -1, -1):
            x.append(torch.baddbmm(G[j], self.F[j], x[-1], alpha=-1))
        z = torch.fft.irfft(torch.stack(x[::-1])[..., 0], n=self.m, dim=1)
        return torch.cat([wall0[None], z, wall1[None]])


def _wall(P, t):
    bv = P.u_bdry * min(t, 1.0)
    bp = P.u_bdry * (0.5 * t * t if t < 1 else t - 0.5)
    w = torch.zeros((P.m, 2), device="cuda", dtype=torch.float64)
    w[:, 0] = bv
    return -w, w, bp


def _averages(vel, dt, P):
    """Cell velocity and the differences (u_x, u_y, v_x, v_y) dt."""
    hx, hy = 0.5 * dt * P.m / (P.bx - P.ax), 0.5 * dt * P.n / (P.by - P.ay)
    a, b = vel[:-1], torch.roll(vel[:-1], -1, 1)
    c, d = vel[1:], torch.roll(vel[1:], -1, 1)
    mean, gx, gy = 0.25 * (a + b + c + d), hx * (b - a + d - c), hy * (c - a + d - b)
    return mean[..., 0], mean[..., 1], gx[..., 0], gy[..., 0], gx[..., 1], gy[..., 1]


def _force(S, xf, yf):
    """Net force at the nodes of rows 1..n-1 from cell stresses (4, n+2, m)."""
    p, q, s, t = S[:, 1:-1]
    A, B = p + q - s, p + q + s

    def dxs(a):
        d = a - torch.roll(a, 1, -1)
        return d[:-1] + d[1:]

    def dys(a):
        e = a + torch.roll(a, 1, -1)
        return e[1:] - e[:-1]

    return torch.stack([xf * dxs(A) - yf * dys(t), -xf * dxs(t) + yf * dys(B)], -1)


def _advect_map(M, vel, P, dt):
    hx, hy = 0.5 * dt * P.m / (P.bx - P.ax), 0.5 * dt * P.n / (P.by - P.ay)
    u, v = vel[1:-1, :, 0], vel[1:-1, :, 1]
    per = P.bx - P.ax
    X, Y = M
    cX = -u * hx * _ddx(X[1:-1], u, per) - v * hy * _ddy(X, v, False)
    cY = -u * hx * _ddx(Y[1:-1], u) - v * hy * _ddy(Y, v, False)
    return torch.stack([X[1:-1] + cX, Y[1:-1] + cY])


def _close_map(inner, P, bp):
    dx = (P.bx - P.ax) / P.m
    x = P.ax + dx * torch.arange(P.m, device="cuda", dtype=torch.float64)
    lo = torch.stack([x + bp, torch.full_like(x, P.ay)])[:, None]
    hi = torch.stack([x - bp, torch.full_like(x, P.by)])[:, None]
    return torch.cat([lo, inner, hi], dim=1)


def _step(P, th, S, time, dt, solve, explicit=False):
    """One step; S as _state's dict, time at its end."""
    hx, hy = 0.5 * dt * P.m / (P.bx - P.ax), 0.5 * dt * P.n / (P.by - P.ay)
    vel = S["vel"]
    uc, vc, ux, uy, vx, vy = _averages(vel, dt, P)
    spin = vx - uy
    F = torch.cat([S["stress"], S["chi"][None]])
    inc = -uc * hx * _ddx(F[:, 1:-1], uc) - vc * hy * _ddy(F, vc, True)
    p, q, s, t = S["stress"][:, 1:-1]
    sq = 3 * q * q + s * s + t * t
    sbar = torch.sqrt(torch.where(sq > 0, sq, torch.full_like(sq, 1e-300)))
    drop, chi = _plastic(P, th, sbar, S["chi"][1:-1] + inc[4], dt)
    fac = drop / sbar
    rate = [inc[0], inc[1] - fac * q, inc[2] + spin * t - fac * s, inc[3] - spin * s - fac * t]
    eps = S["eps_pl"] + drop / (2 * P.mu)
    maps = _advect_map(S["map"], vel, P, dt)
    w0, w1, bp = _wall(P, time)
    stress = torch.stack([a + r for a, r in zip((p, q, s, t), rate)])
    if explicit:
        xs, ys, nu = P.m / (P.bx - P.ax), P.n / (P.by - P.ay), P.viscosity
        c, u, v = vel[1:-1], vel[1:-1, :, 0], vel[1:-1, :, 1]
        comp = torch.stack([vel[..., 0], vel[..., 1]])
        adv = -u * hx * _ddx(comp[:, 1:-1], u) - v * hy * _ddy(comp, v, False)
        lap = dt * nu * (xs * xs * (torch.roll(c, 1, 1) + torch.roll(c, -1, 1) - 2 * c) +
                         ys * ys * (vel[2:] + vel[:-2] - 2 * c))
        new = c + torch.stack([adv[0], adv[1]], -1) + (lap - _force(S["stress"], hx, hy)) / P.mu
        vel = torch.cat([w0[None], new, w1[None]])
        sg = 1.0
    else:
        b = _force(_ghosts(stress), 0.5 / dt * P.m / (P.bx - P.ax), 0.5 / dt * P.n / (P.by - P.ay))
        vel = solve(b, w0, w1)
        _, _, ux, uy, vx, vy = _averages(vel, dt, P)
        sg = 1.0
    div = ux + vy
    stress = stress + sg * torch.stack([-P.K * div, -P.mu / 3 * div, P.mu * (ux - vy), P.mu * (uy + vx)])
    return {"stress": _ghosts(stress), "chi": _ghosts(chi), "map": _close_map(maps, P, bp), "vel": vel, "eps_pl": eps}


def _theta(P):
    return [getattr(P, k) for k in THETA]


def _exact_run(P, S, time, dt, steps, explicit=False):
    solve = None if explicit else _Solve(P, dt)
    for _ in range(steps):
        time += dt
        S = _step(P, _theta(P), S, time, dt, solve, explicit)
    return S


def exact(case, seed):
    """None for the sheared frame: with y periodic the projection fixes the
    velocity only up to a translation, which the advection then carries into
    every field, so no value of it is the exact one."""
    c, kind = case, case["kind"]
    if kind == "ct":
        return None
    if kind == "qs":
        P = _params(c)
        S = _state(P, seed, c["l"], c["std"], c["plastic"])
        return _exact_run(P, S, T0, default_dt(c["m"]), c["steps"])
    if kind == "direct":
        P = simple_shear(c["m"], c["n"], u_bdry=0.04, viscosity=0.02)
        return _exact_run(P, _state(P, seed, 6.0, 30.0, True), T0, _direct_dt(P), c["steps"], True)
    if kind == "batch":
        got = [_exact_run(P, S, T0, default_dt(64), c["steps"]) for P, S in zip(*_batch_states(c, seed))]
        return {k: torch.cat([g[k].reshape(-1) for g in got]) for k in got[0]}
    if kind == "adjoint":
        P, chi, tau, target = _adjoint_inputs(c, seed)
        m, n = P.m, P.n
        th = torch.tensor(_theta(P), device="cuda", dtype=torch.float64, requires_grad=True)
        chi.requires_grad_(True)
        zero = torch.zeros((3, n + 2, m), device="cuda", dtype=torch.float64)
        y = torch.linspace(P.ay, P.by, n + 1, device="cuda", dtype=torch.float64)[:, None]
        x = P.ax + (P.bx - P.ax) / m * torch.arange(m, device="cuda", dtype=torch.float64)[None, :]
        S = {"stress": torch.cat([zero, tau[None]]), "chi": _ghosts(chi),
             "map": torch.stack([x.expand(n + 1, m), y.expand(n + 1, m)]),
             "vel": torch.zeros((n + 1, m, 2), device="cuda", dtype=torch.float64),
             "eps_pl": torch.zeros((n, m), device="cuda", dtype=torch.float64)}
        solve, time = _Solve(P, ADJOINT_DT), 0.0
        for _ in range(c["steps"]):
            time += ADJOINT_DT
            S = _step(P, list(th), S, time, ADJOINT_DT, solve)
        loss = (P.bx - P.ax) / m * (P.by - P.ay) / n * ((S["eps_pl"] - target) ** 2).sum()
        g_theta, g_chi = torch.autograd.grad(loss, [th, chi])
        return {"loss": float(loss), "g_theta": g_theta, "g_chi": g_chi, "eps_pl": S["eps_pl"].detach()}
    b = _poisson_b(c, seed)
    m, n = c["m"], c["n"]
    hx, hy = 2.0 / (m - 1), 2.0 / (n - 1)
    hcc = -2 / hx ** 2 - 2 / hy ** 2
    z = b / hcc  # the edge points' own equation
    f = b[1:-1, 1:-1].clone()
    f[:, 0] -= z[1:-1, 0] / hx ** 2
    f[:, -1] -= z[1:-1, -1] / hx ** 2
    f[0] -= z[0, 1:-1] / hy ** 2
    f[-1] -= z[-1, 1:-1] / hy ** 2

    def sines(k):
        j = torch.arange(1, k, device="cuda", dtype=torch.int64)
        return math.sqrt(2 / k) * torch.sin(math.pi / k * ((j[:, None] * j[None, :]) % (2 * k)).double())

    sx, sy = sines(m - 1), sines(n - 1)
    ex = -4 / hx ** 2 * torch.sin(0.5 * math.pi / (m - 1) * torch.arange(1, m - 1, device="cuda").double()) ** 2
    ey = -4 / hy ** 2 * torch.sin(0.5 * math.pi / (n - 1) * torch.arange(1, n - 1, device="cuda").double()) ** 2
    z[1:-1, 1:-1] = sy @ ((sy @ f @ sx) / (ey[:, None] + ex[None, :])) @ sx
    return z
