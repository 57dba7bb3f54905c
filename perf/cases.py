"""Performance cases of the package: the calls a program makes, over their real range.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges,
``prepare(case, seed)`` forms what a program holds before the call, ``run(state)`` is one pass
through the public entry points, ``work(case)`` states the bytes and floating-point operations
a pass cannot do without, and ``exact(case, seed)`` gives the outputs in plain FP64 torch
(the formulas only, none of this package's code).

Kinds of case:

* ``evolve`` -- ``solve_bk`` with K2+Kf by scrambled Sobol points; ``vegas`` -- ``solve_bk`` with
  ``BKConfig``'s default integrator; ``dndy`` -- ``compute_dndy``; ``batch`` -- ``solve_bk_batch``.
* ``lo`` / ``sigma_r`` -- ``structure_functions`` of many points; ``f2`` -- one ``F2``; ``fixed`` --
  ``gbw_qg_fixed_sobol``; ``points`` -- the nested qqbar-g integrands at given points.

The mixed-precision DIS calls hand back double tensors that carry single-precision integrands;
a program that asks for that build keeps them as float32 beside its other data, and so do the
cases.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from nlo_bk_optimized_b200 import MV, BKConfig, compute_dndy, solve_bk
from nlo_bk_optimized_b200.bk.batch import solve_bk_batch
from nlo_bk_optimized_b200.bk.config import IntegrationMethod
from nlo_bk_optimized_b200.dipole import GBW, BKDipole
from nlo_bk_optimized_b200.dipole.table import DipoleTable
from nlo_bk_optimized_b200.dis import (
    F2,
    DISConfig,
    DISOrder,
    Polarization,
    Quark,
    QuarkType,
    integrand_qg_nested_massive,
    structure_functions,
)
from nlo_bk_optimized_b200.dis.fixed_sobol import gbw_qg_fixed_sobol

SQRT_S = 318.0
LIGHT = 0.14  # GeV, the light-quark mass of the benchmark's DIS workload


def listed() -> list[dict]:
    return [
        # the headline evolution (400 r, 2^20 points, RK4 h = 0.1), its first five steps: the
        # first is launched, the others replay
        {"name": "bk_headline", "kind": "evolve", "points": 399, "minr": 1e-7, "maxr": 1e2, "samples": 1 << 20,
         "stepper": "rk4", "step": 0.1, "steps": 5, "precision": "mixed"},
        # the plain evolution of a scan over parameters: 200 r, 2^14 points, RK4 h = 0.2 to Y = 4
        {"name": "bk_plain", "kind": "evolve", "points": 199, "minr": 1e-6, "maxr": 1e2, "samples": 1 << 14,
         "stepper": "rk4", "step": 0.2, "steps": 20, "precision": "mixed"},
        # the all-FP64 build that checks the mixed one, on an odd grid and budget
        {"name": "bk_fp64", "kind": "evolve", "points": 86, "minr": 1e-6, "maxr": 30.0, "samples": 5001,
         "stepper": "rk3", "step": 0.2, "steps": 1, "precision": "fp64"},
        # BKConfig() as it stands: 101 r, Vegas per parent with 1e5 points, RK3 h = 0.2
        {"name": "bk_default", "kind": "vegas", "points": 100, "minr": 1e-6, "maxr": 30.0, "samples": 100_000,
         "steps": 2},
        # one right-hand side at a small budget (the smallest BK call)
        {"name": "bk_dndy_small", "kind": "dndy", "points": 62, "minr": 1e-6, "maxr": 1e2, "samples": 1000,
         "precision": "mixed"},
        # parameter sets of uneven budgets evolved together
        {"name": "bk_batch", "kind": "batch", "points": 199, "minr": 1e-6, "maxr": 1e2, "sets": 24,
         "low": 1 << 16, "high": 1 << 18, "steps": 2},
        # NLO sigma_r of many points on a BK table, 50 bins (the DIS workload at a quarter of its
        # samples and half its iterations)
        {"name": "dis_sigma_r", "kind": "sigma_r", "count": 24, "samples": 1 << 16, "iterations": 5, "bins": 50,
         "charm": False},
        # one NLO F2 with the default quarks at a modest budget: a fit's inner call
        {"name": "dis_f2", "kind": "f2", "maxeval": 100_000, "charm": True},
        # the fixed-Sobol qqbar-g benchmark (GBW, charm), both polarisations
        {"name": "dis_fixed", "kind": "fixed", "mass": 1.4, "q2": 9.0},
        # the nested integrands at a program's own points (its own integrator)
        {"name": "dis_points", "kind": "points", "count": 1 << 17, "inner": 48, "mass": LIGHT, "term": "I3"},
        # LO structure functions of a kinematic grid in FP64 (the smallest DIS call)
        {"name": "dis_lo", "kind": "lo", "count": 64, "order": 24},
    ]


def _log_int(rng, low: float, high: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    kind = rng.choice(["evolve", "evolve", "evolve", "dndy", "vegas", "batch", "sigma_r", "f2", "fixed", "points",
                       "points", "lo"])
    if kind in ("evolve", "dndy"):
        fp64 = rng.random() < 0.2
        case = {"kind": kind, "points": _log_int(rng, 40, 200 if fp64 else 520),
                "minr": 10 ** rng.uniform(-7, -5), "maxr": rng.choice([30.0, 1e2]),
                "samples": _log_int(rng, 1 << 10, 1 << (13 if fp64 else 18)), "precision": "fp64" if fp64 else "mixed"}
        if kind == "evolve":
            case |= {"stepper": rng.choice(["rk3", "rk4", "euler"]), "step": rng.choice([0.1, 0.2]),
                     "steps": rng.randint(1, 2 if fp64 else 6)}
        return case
    if kind == "vegas":
        return {"kind": kind, "points": _log_int(rng, 50, 200), "minr": 1e-6, "maxr": rng.choice([30.0, 1e2]),
                "samples": _log_int(rng, 5_000, 200_000), "steps": 1}
    if kind == "batch":
        low = _log_int(rng, 1 << 12, 1 << 16)
        return {"kind": kind, "points": _log_int(rng, 60, 260), "minr": 1e-6, "maxr": 1e2, "sets": rng.randint(3, 32),
                "low": low, "high": 3 * low, "steps": rng.randint(1, 2)}
    if kind == "sigma_r":
        return {"kind": kind, "count": rng.randint(2, 24), "samples": _log_int(rng, 1 << 12, 1 << 16),
                "iterations": rng.randint(3, 5), "bins": rng.choice([32, 50]), "charm": rng.random() < 0.3}
    if kind == "f2":
        return {"kind": kind, "maxeval": _log_int(rng, 20_000, 200_000), "charm": rng.random() < 0.5}
    if kind == "fixed":
        return {"kind": kind, "mass": round(rng.choice([LIGHT, 1.4]) * rng.uniform(0.9, 1.1), 4),
                "q2": round(rng.uniform(2.0, 30.0), 3)}
    if kind == "points":
        return {"kind": kind, "count": _log_int(rng, 200, 1 << 17), "inner": rng.choice([16, 24, 33, 48, 48, 64]),
                "mass": rng.choice([LIGHT, 1.4]), "term": rng.choice(["I2", "I3"])}
    return {"kind": kind, "count": _log_int(rng, 4, 200), "order": rng.choice([12, 24, 32])}


# ------------------------------------------------------------------------------- inputs


def _uniform(seed: int, salt: int, shape, low: float, high: float) -> torch.Tensor:
    g = torch.Generator().manual_seed(1_000_003 * salt + seed)
    return low + (high - low) * torch.rand(shape, generator=g, dtype=torch.float64)


def _bk_config(case: dict) -> BKConfig:
    common = dict(RPOINTS=case["points"], MINR=case["minr"], MAXR=case["maxr"])
    if case["kind"] == "vegas":
        return BKConfig(MCINTPOINTS=case["samples"], **common)
    if case["kind"] == "batch":
        return BKConfig(INTMETHOD_NLO=IntegrationMethod.SOBOL, STEPPER="rk4", ALPHA_S_CAP=0.7, **common)
    extra = {k: v for k, v in (("STEPPER", case.get("stepper")), ("DE_SOLVER_STEP", case.get("step"))) if v}
    return BKConfig(INTMETHOD_NLO=IntegrationMethod.SOBOL, MCINTPOINTS=case["samples"],
                    PRECISION=case["precision"], **common, **extra)


def _qs0(seed: int, count: int = 1) -> list[float]:
    return _uniform(seed, 1, (count,), 0.1, 0.4).tolist()


def _budgets(case: dict, seed: int) -> list[int]:
    e = _uniform(seed, 2, (case["sets"],), math.log(case["low"]), math.log(case["high"]))
    return [int(v) for v in e.exp().round().tolist()]


def _kinematics(seed: int, count: int) -> tuple[torch.Tensor, torch.Tensor]:
    """Q^2 in [1, 50] GeV^2 and x_Bj in [1e-5, 1e-2], log-uniform."""
    return (_uniform(seed, 3, (count,), 0.0, math.log(50.0)).exp(),
            _uniform(seed, 4, (count,), math.log(1e-5), math.log(1e-2)).exp())


def _table(seed: int) -> DipoleTable:
    """A table of the shape an evolution to Y = 11 leaves: 400 r, step 0.1, MV rows whose
    saturation scale grows with the rapidity."""
    r = 1e-7 * torch.pow(torch.tensor(1e9, dtype=torch.float64), torch.arange(400, dtype=torch.float64) / 399)
    y = 0.1 * torch.arange(111, dtype=torch.float64)
    qs2 = _qs0(seed)[0] * torch.exp(0.2 * y)[:, None]
    e = 0.25 * torch.pow(r * r * qs2, 0.95) * torch.log(1 / (0.241 * r) + math.e)
    return DipoleTable(r=r.cuda(), y=y.cuda(), N=(-torch.expm1(-e)).cuda(), x0=0.01)


def _unit_points(case: dict, seed: int) -> torch.Tensor:
    return _uniform(seed, 5, (case["count"], 5), 1e-3, 1 - 1e-3).float()


def _gbw(seed: int) -> GBW:
    return GBW(Qs0sqr=_qs0(seed)[0], lambda_=0.29, gamma=1.0, x0=0.01)


def _quarks(case: dict) -> tuple[Quark, ...]:
    light = Quark(QuarkType.LIGHT, LIGHT)
    return (light, Quark(QuarkType.C, 1.4)) if case["charm"] else (light,)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    state = {"case": case, "seed": seed}
    if kind in ("evolve", "vegas", "dndy"):
        # the number of active parents, and so the shape of compute_dndy's rows, follows from Qs0
        state |= {"ic": MV(qs0sqr=0.2 if kind == "dndy" else _qs0(seed)[0]), "config": _bk_config(case),
                  "dtype": torch.float64 if case.get("precision") == "fp64" else torch.float32}
    elif kind == "batch":
        state |= {"ics": [MV(qs0sqr=q) for q in _qs0(seed, case["sets"])], "config": _bk_config(case),
                  "budgets": _budgets(case, seed)}
    elif kind == "sigma_r":
        q2, x = _kinematics(seed, case["count"])
        config = DISConfig(order=DISOrder.NLO, quarks=_quarks(case), transverse_area=16 * 2.56819,
                           vegas_bins=case["bins"])
        state |= {"q2": q2, "x": x, "dipole": BKDipole(_table(seed)), "config": config}
    elif kind == "f2":
        q2, x = _kinematics(seed, 1)
        config = DISConfig(order=DISOrder.NLO, quarks=_quarks(case), maxeval=case["maxeval"])
        state |= {"q2": q2[0], "x": x[0], "dipole": BKDipole(_table(seed)), "config": config}
    elif kind == "lo":
        q2, x = _kinematics(seed, case["count"])
        state |= {"q2": q2, "x": x, "dipole": _gbw(seed), "config": DISConfig(precision="fp64")}
    elif kind == "fixed":
        q2 = torch.tensor(case["q2"], dtype=torch.float32, device="cuda")
        state |= {"q2": q2, "x": torch.tensor(1e-3, dtype=torch.float32, device="cuda"), "dipole": _fixed_gbw(seed),
                  "quark": Quark(QuarkType.C, case["mass"]),
                  "config": DISConfig(maxr=5.0, nf_alphas=1, quarks=(Quark(QuarkType.C, case["mass"]),))}
    else:
        q2, x = _kinematics(seed, 1)
        quark = Quark(QuarkType.LIGHT, case["mass"])
        state |= {"q2": q2[0], "x": x[0], "points": _unit_points(case, seed).cuda(), "dipole": _gbw(seed),
                  "quark": quark, "config": DISConfig(quarks=(quark,), cuda_nested_points=case["inner"])}
    return state


def _fixed_gbw(seed: int) -> GBW:
    return GBW(Qs0sqr=_uniform(seed, 6, (1,), 0.5, 1.5).item(), lambda_=0.3, gamma=1.0, x0=1.0)


# ------------------------------------------------------------------------------- a pass


def _table_out(t: DipoleTable) -> dict:
    return {"r": t.r, "y": t.y, "N": t.N}


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind in ("evolve", "vegas"):
        step = state["config"].DE_SOLVER_STEP
        return _table_out(solve_bk(state["ic"], step * case["steps"], state["config"], dtype=state["dtype"],
                                   seed=state["seed"]))
    if kind == "dndy":
        d = compute_dndy(state["ic"], state["config"], dtype=state["dtype"], seed=state["seed"])
        return {"r": d.r, "K1": d.K1, "K2_Kf": d.K2_Kf, "N": d.N}
    if kind == "batch":
        tables = solve_bk_batch(state["ics"], state["config"].DE_SOLVER_STEP * case["steps"], state["config"],
                                samples=state["budgets"], seed=state["seed"], waves=4)
        return [_table_out(t)["N"] for t in tables]
    if kind == "sigma_r":
        out = structure_functions(state["q2"], state["x"], state["dipole"], state["config"], sqrt_s=SQRT_S,
                                  seed=state["seed"], vegas_samples=case["samples"],
                                  vegas_iterations=case["iterations"], vegas_min_iterations=case["iterations"])
        return {k: v.float() for k, v in out.items()}
    if kind == "f2":
        r = F2(state["q2"], state["x"], state["dipole"], state["config"], seed=state["seed"])
        return {"value": r.value.float(), "error": r.error.float()}
    if kind == "lo":
        return structure_functions(state["q2"], state["x"], state["dipole"], state["config"], sqrt_s=SQRT_S,
                                   quadrature_points=case["order"])
    if kind == "fixed":
        results = [gbw_qg_fixed_sobol(state["q2"], state["x"], pol, state["quark"], state["dipole"], state["config"],
                                      seed=state["seed"]) for pol in (Polarization.T, Polarization.L)]
        parts = [p for r in results for p in (*r.contributions, r.total)]
        return {"value": torch.stack([p.value for p in parts]).float(),
                "error": torch.stack([p.error for p in parts]).float()}
    return [integrand_qg_nested_massive(state["points"], state["q2"], state["x"], pol, state["quark"], case["term"],
                                        state["dipole"], state["config"]) for pol in (Polarization.T, Polarization.L)]


# ------------------------------------------------------------------------------- work

# operations of the formulas: a K2+Kf evaluation (and its share of a sample), a K1 evaluation, an
# outer sample of the nested qqbar-g terms per inner node, and of the other DIS terms
_K2_OPS, _SAMPLE_OPS, _K1_OPS, _NODE_OPS, _DIS_OPS = 148.0, 61.0, 120.0, 265.0, 400.0
_STAGES = {"rk4": 4, "rk3": 3, "euler": 1}


def _rhs_flops(points: int, samples: float) -> float:
    return samples * (0.9 * points * _K2_OPS + _SAMPLE_OPS) + 0.9 * points * points * 192 * _K1_OPS


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("evolve", "dndy", "vegas"):
        n = case["points"] + 1
        stages = 1 if kind == "dndy" else case["steps"] * _STAGES[case.get("stepper", "rk3")]
        if kind == "vegas":  # the warm-up and two iterations of every parent, each with its own points
            per_rhs = 0.9 * n * 2.05 * case["samples"] * (_K2_OPS + _SAMPLE_OPS) + 0.9 * n * n * 192 * _K1_OPS
        else:
            per_rhs = _rhs_flops(n, case["samples"])
        return {"bytes": 8.0 * n * (stages + 2), "flops": stages * per_rhs}
    if kind == "batch":
        n = case["points"] + 1
        mean = (case["high"] - case["low"]) / math.log(case["high"] / case["low"])
        return {"bytes": 8.0 * n * case["sets"] * (case["steps"] + 2),
                "flops": 4 * case["steps"] * case["sets"] * _rhs_flops(n, mean)}
    if kind == "sigma_r":
        jobs = 2 * case["count"] * (2 if case["charm"] else 1)
        per_job = case["samples"] * case["iterations"] * (2 * 48 * _NODE_OPS + 3 * _DIS_OPS)
        return {"bytes": 8.0 * (400 * 111 * 4 + 16 * case["count"]), "flops": jobs * per_job}
    if kind == "f2":
        quarks = 2 if case["charm"] else 1
        per_job = case["maxeval"] * 3 / 8 * (2 * 48 * _NODE_OPS + _DIS_OPS + 20 * _DIS_OPS)
        return {"bytes": 8.0 * 400 * 111 * 4, "flops": 2 * quarks * per_job}
    if kind == "fixed":
        return {"bytes": 8.0 * 64, "flops": 2 * 851_968.0 * (48 * _NODE_OPS + 3 * _DIS_OPS)}
    if kind == "points":
        return {"bytes": 2 * 4.0 * 6 * case["count"], "flops": 2.0 * case["count"] * (case["inner"] * _NODE_OPS + _DIS_OPS)}
    nodes = case["order"] ** 2 + (case["order"] // 2) ** 2
    return {"bytes": 8.0 * 11 * case["count"], "flops": 2.0 * case["count"] * nodes * 60}


# ------------------------------------------------------------------------------- 64-bit values

_B0 = (11 * 3.0 - 2 * 3.0) / (12 * math.pi)
_LEFT = 10 * math.log(2.5)
_LOG_SC = math.log(4 / 0.241**2)


class _Spline:
    """Natural cubic spline on log r, with given values below and above the grid."""

    def __init__(self, x: torch.Tensor, y: torch.Tensor):
        n = x.numel()
        h = x.diff()
        slope = y.diff() / h
        m = torch.zeros_like(y)
        if n > 2:
            a = torch.diag(2 * (h[1:] + h[:-1])) + torch.diag(h[1:-1], 1) + torch.diag(h[1:-1], -1)
            m[1:-1] = torch.linalg.solve(a, 6 * slope.diff())
        self.x, self.a, self.b = x, y, slope - h * (2 * m[:-1] + m[1:]) / 6
        self.c, self.d = m[:-1] / 2, m.diff() / (6 * h)

    def __call__(self, lx: torch.Tensor) -> torch.Tensor:
        lx = lx.clamp(float(self.x[0]), float(self.x[-1]))
        i = (torch.searchsorted(self.x, lx, right=True) - 1).clamp(0, self.x.numel() - 2)
        t = lx - self.x[i]
        return self.a[i] + t * (self.b[i] + t * (self.c[i] + t * self.d[i]))


def _alpha(log_d: torch.Tensor, cap: float) -> torch.Tensor:
    right = 5 * (_LOG_SC - 2 * log_d)
    a = 1 / (0.2 * _B0 * torch.logaddexp(torch.full_like(right, _LEFT), right))
    return a.clamp_max(cap) if cap > 0 else a


def _dlog_factor(v: torch.Tensor) -> torch.Tensor:
    """sum_k v^k / (k! (k+1)!): J1(t)/(t/2) for v < 0 and I1(t)/(t/2) for v > 0, t = 2 sqrt|v|."""
    term, out = torch.ones_like(v), torch.ones_like(v)
    w = v.clamp_min(-4.0)
    for k in range(1, 70):
        term = term * w / (k * (k + 1))
        out = out + term
    t = 2 * torch.sqrt(v.abs().clamp_min(4.0))
    j1 = torch.zeros_like(v)
    for k in range(64):  # J1(t) = 1/pi int_0^pi cos(q - t sin q) dq, spectrally exact here
        q = math.pi * (k + 0.5) / 64
        j1 = j1 + torch.cos(q - t * math.sin(q))
    return torch.where(v < -4.0, 2 * (j1 / 64) / t, out)


def _k1(r, N, act, x, n_spline, minr, cap) -> torch.Tensor:
    gx8, gw8 = (torch.from_numpy(v).to(r) for v in np.polynomial.legendre.leggauss(8))
    gx24, gw24 = (torch.from_numpy(v).to(r) for v in np.polynomial.legendre.leggauss(24))
    hw = 0.5 * x.diff()
    lz = (0.5 * (x[1:] + x[:-1])[:, None] + hw[:, None] * gx8).reshape(1, -1, 1)
    wz = (hw[:, None] * gw8).reshape(1, -1, 1)
    v = 0.5 * (gx24 + 1)
    sh2 = torch.sin(0.5 * math.pi * v * v).square().reshape(1, 1, -1)
    wa = (gw24 * math.pi * v).reshape(1, 1, -1)
    z = torch.exp(lz)
    out = torch.zeros_like(r)

    def amp(l):
        val = torch.exp(n_spline(l)).clamp_max(1.0)
        val = torch.where(l < x[0], torch.zeros_like(val), val)
        return torch.where(l > x[-1], torch.ones_like(val), val)

    NY, aY = amp(lz), _alpha(lz, cap)
    for part in act.split(max(1, int(4e6 / (lz.numel() * 24)))):
        R, LR = r[part].reshape(-1, 1, 1), x[part].reshape(-1, 1, 1)
        dY = lz - LR
        rho = torch.exp(dY)
        xr2 = (1 - rho).square() + 4 * rho * sh2
        dX = 0.5 * torch.log(xr2)
        Xsq, Ysq = xr2 * R * R, z * z
        aX, ar = _alpha(LR + dX, cap), _alpha(LR, cap)
        XmY = R * (R - 2 * z * (1 - 2 * sh2))
        if cap > 0:
            da = aY - aX
        else:  # alpha_Y - alpha_X without the cancellation of two logarithms
            right = 5 * (_LOG_SC - 2 * lz)
            s = 1 / (1 + torch.exp(_LEFT - right))
            delta = -5 * torch.log1p(XmY / Ysq)
            u = s * torch.expm1(delta)
            shift = torch.where(u > -0.5, torch.log1p(u.clamp_min(-0.6)),
                                torch.log(1 / (1 + torch.exp(right - _LEFT)) + s * torch.exp(delta)))
            da = aX * aY * 0.2 * _B0 * shift
        pref = 3.0 / (2 * math.pi**2)
        lo = pref * ar * (R * R + da * (aY * XmY + Ysq * da) / (aX * aY)) / (Xsq * Ysq)
        amin = torch.where((dX <= dY) & (dX <= 0), aX, torch.where(dY <= 0, aY, ar))
        NX = amp(LR + dX)
        NR = N[part].reshape(-1, 1, 1)
        dip = NX + NY - NR - NX * NY
        abar = amin * 3.0 / math.pi
        dlog = _dlog_factor(-abar * 4 * dX * dY) if bool((R > 1.01 * minr).any()) else torch.ones_like(dX)
        dlog = torch.where(R > 1.01 * minr, dlog, torch.ones_like(dlog))
        slog = -abar * (11 / 12) * (math.log(0.65) - 2 * torch.minimum(dX, dY)).abs()
        single = pref * ar * R * R / (Xsq * Ysq)
        fin = lo * ar * 3.0 / (4 * math.pi) * (67 / 9 - math.pi**2 / 3 - 10 / 9)
        val = (dlog * torch.exp(slog) * lo - single * slog + fin) * dip * wa * (2 * z * z * wz)
        out[part] = torch.nan_to_num(val, 0.0, 0.0, 0.0).sum((1, 2))
    return out


def _atanh_ratio_m1(t2: torch.Tensor) -> torch.Tensor:
    s = torch.zeros_like(t2)
    for k in range(30, 0, -1):
        s = s * t2 + 1 / (2 * k + 1)
    return s * t2


def _k2kf(r, act, x, s_spline, samples, seed, cap) -> torch.Tensor:
    """Mean of the K2 + Kf integrand over the first `samples` scrambled Sobol points."""
    unit = torch.quasirandom.SobolEngine(4, scramble=True, seed=seed).draw(samples, dtype=torch.float64).to(r.device)
    lo, hi = math.log(0.5 * float(r[0])), math.log(2 * float(r[-1]))
    scale = (hi - lo) ** 2 * (2 * math.pi) ** 2 * 9 / (8 * math.pi**4)

    def amp(l):
        p = s_spline(l)
        below, above = l < x[0], l > x[-1]
        p = torch.where(below, torch.zeros_like(p), torch.where(above, torch.full_like(p, -torch.inf), p))
        return p, torch.exp(p)

    def ndiff(a, b):  # N_a - N_b = S_b - S_a
        d = b[0] - a[0]
        near = torch.where(d <= 0, a[1] * torch.expm1(d.clamp_max(0.0)), -b[1] * torch.expm1(-d.clamp_min(0.0)))
        return torch.where(d.abs() < 1, near, b[1] - a[1])

    total = torch.zeros(act.numel(), dtype=r.dtype, device=r.device)
    R, LR = r[act][:, None], x[act][:, None]
    for u in unit.split(max(1, int(4e6 / max(1, act.numel())))):
        lz, lw = lo + (hi - lo) * u[:, 0], lo + (hi - lo) * u[:, 1]
        th, ph = 2 * math.pi * u[:, 2], 2 * math.pi * u[:, 3]
        z, w = torch.exp(lz), torch.exp(lw)
        c1, c2, c12 = torch.cos(th), torch.cos(ph), torch.cos(th - ph)
        zz = (z - w).square() + 4 * z * w * torch.sin(0.5 * (th - ph)).square()
        lzz = 0.5 * torch.log(zz)
        Y, W, Z = amp(lz), amp(lw), amp(lzz)
        NZ = -torch.expm1(Z[0])
        dN = ndiff(W, Y)
        D1, D2 = Y[1] * NZ + Z[1] * dN, W[1] * NZ - Z[1] * dN
        q, cpt = 1 / zz, scale * torch.exp(2 * lz + 2 * lw)
        Xs = (R - z).square() + 4 * R * z * torch.sin(0.5 * th).square()
        Ws = (R - w).square() + 4 * R * w * torch.sin(0.5 * ph).square()
        lX, lW = torch.log(Xs), torch.log(Ws)
        vX, vW = amp(0.5 * lX), amp(0.5 * lW)
        a, b = Xs * w * w, Ws * z * z
        t = R * (R * (w - z) * (w + z) - 2 * z * w * (w * c1 - z * c2)) / (a + b)
        small = t * t < 0.25
        hm1 = torch.where(small, _atanh_ratio_m1(torch.where(small, t * t, torch.zeros_like(t))),
                          (lX - lW + 2 * (lw - lz)) / (2 * t) - 1)
        L = 2 * (1 + hm1) / (a + b)
        fq2, g = 2 * hm1 * q * q, R * R * L * q
        k2 = fq2 - 4 * g + g * 2 * R * (R * (w - z * c12) + z * (z * c2 - w * c1)) / (Xs * w)
        k2s = fq2 - 4 * g + g * 2 * R * (R * (z - w * c12) + w * (w * c1 - z * c2)) / (Ws * z)
        val = 0.5 * (k2 * vX[1] * D1 + k2s * vW[1] * D2) - 0.5 * (g - fq2) * ndiff(vX, vW) * dN
        smallest = torch.minimum(torch.minimum(torch.minimum(lz, lw), lzz), torch.minimum(LR, 0.5 * torch.minimum(lX, lW)))
        val = val * _alpha(smallest, cap).square() * cpt
        total += torch.nan_to_num(val, 0.0, 0.0, 0.0).sum(1)
    return total / samples


def _bk_rhs(r, N, minr, samples, seed, cap):
    x = torch.log(r)
    floor = torch.full_like(N, -40.0)  # the tables' value where the logarithm does not exist
    n_spline = _Spline(x, torch.where(N > 0, torch.log(N.clamp_max(1.0)), floor))
    s_spline = _Spline(x, torch.where(N < 1, torch.log1p(-N.clamp_min(0.0)), floor))
    act = torch.nonzero((torch.arange(r.numel(), device=r.device) > 0) & (N <= 0.99999))[:, 0]
    k1 = _k1(r, N, act, x, n_spline, minr, cap)
    k2 = torch.zeros_like(r)
    k2[act] = _k2kf(r, act, x, s_spline, samples, seed, cap)
    return k1, k2, act


def _bk_start(case: dict, qs0: float):
    n = case["points"]
    r = case["minr"] * torch.pow(torch.tensor(case["maxr"] / case["minr"], dtype=torch.float64) ** (1 / n),
                                 torch.arange(n + 1, dtype=torch.float64)).cuda()
    e = r * r * qs0 / 4 * torch.log(1 / (0.241 * r) + 2.7182818)
    return r, torch.where(e < 1e-5, e, 1 - torch.exp(-e))


def _bk_rows(case: dict, qs0: float, samples: int, seed: int, stepper: str, h: float, cap: float) -> dict:
    r, N = _bk_start(case, qs0)

    def f(v):
        k1, k2, _ = _bk_rhs(r, v, case["minr"], samples, seed, cap)
        return k1 + k2

    rows, ys = [N], [0.0]
    for _ in range(case["steps"]):
        k1 = f(N)
        if stepper == "rk4":
            k2 = f(N + 0.5 * h * k1)
            k3 = f(N + 0.5 * h * k2)
            N = N + h / 6 * (k1 + 2 * k2 + 2 * k3 + f(N + h * k3))
        elif stepper == "rk3":
            k2 = f(N + 0.5 * h * k1)
            N = N + h / 6 * (k1 + 4 * k2 + f(N + h * (2 * k2 - k1)))
        else:
            N = N + h * k1
        N = N.clamp(0.0, 1.0)
        rows.append(N)
        ys.append(ys[-1] + h)
    return {"r": r, "y": torch.tensor(ys, dtype=torch.float64), "N": torch.stack(rows)}


def _bessel(x: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    return torch.special.modified_bessel_k0(x), torch.special.modified_bessel_k1(x)


class _QG:
    """The qqbar-g terms at points of the unit cube for the GBW dipole (FP64)."""

    def __init__(self, x, q2, xbj, mass, transverse, gbw: GBW, config: DISConfig):
        rule = np.polynomial.legendre.leggauss(config.cuda_nested_points)
        t = 0.5 * (rule[0] + 1)
        self.nodes, self.weights = (t**3).tolist(), (0.5 * rule[1] * 3 * t * t).tolist()
        self.q2, self.m2, self.transverse = q2, mass * mass, transverse
        w2 = q2 / xbj
        zmin = 1 / w2
        z1 = (1 - zmin) * x[:, 0]
        z2 = (1 - z1 - zmin) * x[:, 1] + zmin
        a, b, phi = config.maxr * x[:, 2], config.maxr * x[:, 3], 2 * math.pi * x[:, 4]
        d2 = (a * a + b * b - 2 * a * b * torch.cos(phi)).clamp_min(0.0)
        Y = torch.log(w2 * z2)

        def S(rsq):
            y = Y.clamp_min(math.log(1 / gbw.x0))
            e = 0.25 * torch.pow(rsq * gbw.Qs0sqr * torch.exp(gbw.lambda_ * y), gbw.gamma)
            return torch.exp(-e)

        s01, s02, s12 = S(a * a), S(b * b), S(d2)
        cf = 4 / 3
        self.n01, self.n012 = 1 - s01, 1 - 3 / (2 * cf) * (s02 * s12 - s01 / 9)
        small = torch.minimum(a, torch.minimum(b, torch.sqrt(d2)))
        log_arg = _LOG_SC - 2 * torch.log(small)
        alpha = 1 / ((33 - 2 * config.active_flavors) / (12 * math.pi) * log_arg)
        alpha = torch.where((alpha > config.max_alpha_s_freeze) | (log_arg < 0),
                            torch.full_like(alpha, config.max_alpha_s_freeze), alpha)
        jac = (1 - zmin) * (1 - z1 - zmin) * a * b * config.maxr**2 * 2 * math.pi
        self.scale = torch.where(Y >= 0, alpha * cf / math.pi * jac / z2, torch.zeros_like(Y))
        z0 = 1 - z1 - z2
        self.z0, self.z1, self.z2, self.zj, self.zk = z0, z1, z2, z0 + z2, z1 + z2
        self.a2, dot = a * a, -0.5 * (a * a - d2 - b * b)
        fj, fk = z0 / self.zj, z1 / self.zk
        self.dot, self.x2 = dot, (b * b, d2)
        self.x3 = (fj * fj * b * b + d2 - 2 * fj * dot, fk * fk * d2 + b * b - 2 * fk * dot)
        self.om = (z0 * z2 / (z1 * self.zj**2), z1 * z2 / (z0 * self.zk**2))
        self.lam = (z1 * z2 / z0, z0 * z2 / z1)
        self.M2 = (q2 * z1 * (1 - z1) + self.m2, q2 * z0 * (1 - z0) + self.m2)
        self.jj, self.kk = dot - fj * b * b, -dot + fk * d2
        self.jk, self.kj = -b * b + fk * dot, d2 - fj * dot
        self.x33 = fj * b * b + fk * d2 - (1 + fj * fk) * dot
        self.X2 = tuple(self.x3[s] + self.om[s] * self.x2[s] for s in (0, 1))
        self.P = tuple((2 * u * v + z2 * z2) / (v * v) for u, v in ((z0, self.zj), (z1, self.zk)))
        self.A = (1 - 2 * z1 * (1 - z1), 1 - 2 * z0 * (1 - z0))
        self.sing = [self._singular(s) for s in (0, 1)]
        self.F = (z2 * (z0 - z1) ** 2 * (self.jj * self.kk - self.kj * self.jk)
                  - (z1 * self.zj + z0 * self.zk) * (z0 * self.zj + z1 * self.zk) * dot * self.x33)
        self.c2 = (2 * z0 + z2) * (2 * z1 + z2) + z2 * z2

    def _singular(self, s):
        k0, k1 = _bessel(torch.sqrt(self.M2[s] * self.X2[s]))
        mh = self.M2[s] + self.m2 * self.lam[s]
        h = 4 * torch.sqrt(mh / self.X2[s]) * _bessel(torch.sqrt(mh * self.X2[s]))[1]
        return k0, k1, torch.sqrt(self.M2[s] / self.X2[s]) * k1 / self.x2[s], k0 / self.x2[s], h

    def moments(self):
        G = {k: [0.0, 0.0] for k in ("22", "12", "21", "11")}
        for y, w in zip(self.nodes, self.weights):
            for s in (0, 1):
                B, om = y * self.x3[s] + self.om[s] * self.x2[s], self.om[s]
                Al = y * self.lam[s] * self.m2 + self.M2[s]
                al, a0 = torch.sqrt(Al * B / y), torch.sqrt(self.M2[s] * B / y)
                (l0, l1), (s0, s1) = _bessel(al), _bessel(a0)
                G["22"][s] = G["22"][s] + w * 8 / y * om * (Al / B * (l0 + 2 * l1 / al)
                                                            - self.M2[s] / B * (s0 + 2 * s1 / a0))
                G["12"][s] = G["12"][s] + w * 4 / y**1.5 * om * (torch.sqrt(Al / B) * l1
                                                                 - torch.sqrt(self.M2[s] / B) * s1)
                G["21"][s] = G["21"][s] + w * 4 / math.sqrt(y) * torch.sqrt(Al / B) * l1
                G["11"][s] = G["11"][s] + w * 2 / y * l0
        return G["22"], G["12"], G["21"], G["11"]

    def i1(self):
        z0, z1, z2, zj, zk, m2 = self.z0, self.z1, self.z2, self.zj, self.zk, self.m2
        eg = math.exp(0.5772156649015329)
        uv, jk = 0.0, 0.0
        for s in (0, 1):
            d0, d1 = _bessel(torch.sqrt(self.a2 * self.M2[s]))
            damp = torch.exp(-self.x2[s] / (self.a2 * eg)) / self.x2[s]
            k0, k1 = self.sing[s][0], self.sing[s][1]
            if self.transverse:
                uv = uv - self.P[s] * damp * (self.A[s] * self.M2[s] * d1 * d1 + m2 * d0 * d0)
                jk = jk + self.P[s] / self.x2[s] * (self.A[s] * self.M2[s] * self.x3[s] / self.X2[s] * k1 * k1
                                                    + m2 * k0 * k0)
            else:
                u, v = (z1, z0) if s == 0 else (z0, z1)
                uv = uv - u * u * (2 * v * (v + z2) + z2 * z2) * damp * d0 * d0
                jk = jk + u * u * (2 * v * (v + z2) + z2 * z2) / self.x2[s] * k0 * k0
        (b0, _, ga, ea, ha), (b1, _, gb, eb, hb) = self.sing
        if not self.transverse:
            jk = jk - 2 * z0 * z1 * (z0 * (1 - z0) + z1 * (1 - z1)) * self.dot / (self.x2[0] * self.x2[1]) * b0 * b1
            return (self.n01 * uv + self.n012 * jk) * 4 * self.q2 * self.scale
        F = 0.5 * (4 / (zj * zk) * self.F * ga * gb - zj * z1 * z2 / zk**2 * self.jj * hb * ga
                   + zk * z0 * z2 / zj**2 * self.kk * ha * gb - z0 * z0 * z1 * z2 / zj**3 * self.jj * ha * ga
                   + z1 * z1 * z0 * z2 / zk**3 * self.kk * hb * gb + (z0 * z2) ** 2 / (8 * zj**4) * ha * ha
                   + (z1 * z2) ** 2 / (8 * zk**4) * hb * hb)
        return (self.n01 * uv + self.n012 * (jk + F - m2 * self.c2 * self.dot * ea * eb / (zj * zk))) * self.scale

    def i2(self, G):
        g22, g12, g21, g11 = G
        z0, z1, z2, zj, zk, m2 = self.z0, self.z1, self.z2, self.zj, self.zk, self.m2
        (b0, k1a, ga, ea, ha), (b1, k1b, gb, eb, hb) = self.sing
        if not self.transverse:
            v = (z1 * z1 * (2 * z0 * zj + z2 * z2) * g12[0] * b0 + z0 * z0 * (2 * z1 * zk + z2 * z2) * g12[1] * b1
                 - z0 * z1 * (z0 * (1 - z0) + z1 * (1 - z1)) * self.dot * (g12[0] * b1 / self.x2[1]
                                                                          + g12[1] * b0 / self.x2[0]))
            return v * self.q2 * self.n012 * self.scale
        jk = sum(self.P[s] * self.A[s] * g22[s] * self.x3[s] / 8 * torch.sqrt(self.M2[s] / self.X2[s]) * self.sing[s][1]
                 + m2 * self.P[s] * g12[s] / 4 * self.sing[s][0] for s in (0, 1))
        F = 0.5 * (self.F / (4 * zj * zk) * (g22[1] * ga + g22[0] * gb)
                   - zj * z1 * z2 / (16 * zk**2) * self.jj * hb * g22[0]
                   + zk * z0 * z2 / (16 * zj**2) * self.kk * ha * g22[1]
                   - z0 * z0 * z1 * z2 / (16 * zj**3) * self.jj * ha * g22[0]
                   + z1 * z1 * z0 * z2 / (16 * zk**3) * self.kk * hb * g22[1])
        zz, w = z2 * z2, z0 * z1 * z2 * z2
        Fm = 0.5 * m2 * (-w / (2 * zj**3) * self.jj * g21[0] * ea + w / (2 * zk**3) * self.kk * g21[1] * eb
                         - self.c2 * self.dot / (4 * zj * zk) * (g12[1] * ea + g12[0] * eb)
                         - (z0 * z2) ** 2 / (2 * zj * zk**2) * self.jk * g21[1] * ea
                         + (z1 * z2) ** 2 / (2 * zj**2 * zk) * self.kj * g21[0] * eb
                         - w / zj**3 * self.jj * g11[0] * ga + w / zk**3 * self.kk * g11[1] * gb
                         - zj * zz / zk**2 * self.jj * g11[1] * ga + zk * zz / zj**2 * self.kk * g11[0] * gb
                         + z0 * zz * z2 / (4 * zj**4) * ha * g11[0] + z1 * zz * z2 / (4 * zk**4) * hb * g11[1])
        return (jk + F + Fm) * self.n012 * self.scale

    def i3(self, G):
        g22, g12, g21, g11 = G
        z0, z1, z2, zj, zk, m2 = self.z0, self.z1, self.z2, self.zj, self.zk, self.m2
        z4 = z2**4
        if not self.transverse:
            a, c = z1 / zj, z0 / zk
            v = (z1 * z1 * (2 * z0 * zj + z2 * z2) * self.x2[0] / 64 * g12[0] ** 2
                 + z0 * z0 * (2 * z1 * zk + z2 * z2) * self.x2[1] / 64 * g12[1] ** 2
                 - z1 * z0 * (z1 * (1 - z1) + z0 * (1 - z0)) * self.dot / 32 * g12[0] * g12[1]
                 + m2 / 16 * z4 * (a * g11[0] - c * g11[1]) ** 2)
            return 4 * self.q2 * v * self.n012 * self.scale
        jk = sum(self.P[s] * self.x2[s] * (m2 / 64 * g12[s] ** 2 + self.A[s] * self.x3[s] / 256 * g22[s] ** 2)
                 for s in (0, 1))
        F = 0.5 * g22[0] * g22[1] / (64 * zj * zk) * self.F
        w = z0 * z1 * z2 * z2
        Fm = 0.5 * m2 * (z4 / (64 * zj**4) * (4 * z1 * (z1 - 1) + 2) * self.x3[0] * g21[0] ** 2
                         + z4 / (64 * zk**4) * (4 * z0 * (z0 - 1) + 2) * self.x3[1] * g21[1] ** 2
                         - w / (16 * zj**3) * self.jj * (g12[0] * g21[0] + g11[0] * g22[0])
                         + w / (16 * zk**3) * self.kk * (g12[1] * g21[1] + g11[1] * g22[1])
                         - self.c2 * self.dot / (32 * zj * zk) * g12[0] * g12[1]
                         + z4 / (32 * zj**2 * zk**2) * self.c2 * self.x33 * g21[0] * g21[1]
                         + m2 / 8 * (z2 / zj) ** 4 * g11[0] ** 2 + m2 / 8 * (z2 / zk) ** 4 * g11[1] ** 2
                         - (z0 * z2) ** 2 / (16 * zj * zk**2) * self.jk * g12[0] * g21[1]
                         + (z1 * z2) ** 2 / (16 * zk * zj**2) * self.kj * g12[1] * g21[0]
                         - zj * z2**2 / (16 * zk**2) * self.jj * g11[1] * g22[0]
                         + zk * z2**2 / (16 * zj**2) * self.kk * g11[0] * g22[1])
        return (jk + F + Fm) * self.n012 * self.scale


def _endpoints(src: torch.Tensor, maxr: float):
    """The two weighted points of the nearer-end split of the gluon plane, angle folded."""
    parent, radial, af = maxr * src[:, 2], src[:, 3], 0.5 * src[:, 4]
    c, s = torch.cos(2 * math.pi * af), torch.sin(2 * math.pi * af)
    closer = torch.where(c > 0, parent / (2 * c.clamp_min(1e-300)), torch.full_like(c, torch.inf))
    lim = closer.clamp_max(maxr)
    first, second = src.clone(), src.clone()
    first[:, 3], first[:, 4] = radial * lim / maxr, af
    disk = parent * c + torch.sqrt((maxr * maxr - parent.square() * s.square()).clamp_min(0.0))
    lim2 = torch.minimum(disk, closer).clamp_min(0.0)
    sr = radial * lim2
    gx, gy = parent - sr * c, sr * s
    gr = torch.sqrt(gx * gx + gy * gy)
    second[:, 3], second[:, 4] = gr / maxr, torch.atan2(gy, gx).remainder(2 * math.pi) / (2 * math.pi)
    return first, lim / maxr, second, sr * lim2 / (gr.clamp_min(1e-300) * maxr)


def _fixed_exact(case: dict, seed: int, transverse: bool) -> tuple[torch.Tensor, torch.Tensor]:
    config = DISConfig(maxr=5.0, nf_alphas=1)
    q2 = float(torch.tensor(case["q2"], dtype=torch.float32))
    xbj = float(torch.tensor(1e-3, dtype=torch.float32))
    bins = 32
    edges = torch.linspace(0, 1, bins + 1, dtype=torch.float64).expand(5, -1).clone().cuda()

    def values(sobol_seed, n):
        u = torch.quasirandom.SobolEngine(5, scramble=True, seed=sobol_seed).draw(n, dtype=torch.float32).double().cuda()
        k = (u * bins).floor().long().clamp_max(bins - 1)
        left, right = edges.gather(1, k.T).T, edges.gather(1, k.T + 1).T
        src, inv = left + (right - left) * (u * bins - k), (bins * (right - left)).prod(1)
        first, fw, second, sw = _endpoints(src, config.maxr)
        out = 0.0
        for p, w in ((first, fw), (second, sw)):
            q = _QG(p, q2, xbj, case["mass"], transverse, _fixed_gbw(seed), config)
            G = q.moments()
            v = torch.stack([q.i1(), q.i2(G), q.i3(G)], 1)
            out = out + torch.nan_to_num(v, 0.0, 0.0, 0.0) * w[:, None]
        return out * inv[:, None], k

    for round_ in range(3):
        v, k = values(seed + round_, 65_536)
        score = (v.abs() / v.abs().mean(0)).sum(1)
        for d in range(5):
            imp = torch.zeros(bins, dtype=torch.float64, device="cuda").scatter_add_(0, k[:, d], score)
            imp = imp / torch.bincount(k[:, d], minlength=bins).clamp_min(1)
            pad = torch.cat((imp[:1], imp, imp[-1:]))
            sm = (pad[:-2] + pad[1:-1] + pad[2:]) / 3
            sm[0], sm[-1] = (imp[0] + imp[1]) / 2, (imp[-2] + imp[-1]) / 2
            sm = sm + 2.220446049250313e-16
            cum = torch.cat((sm.new_zeros(1), sm.cumsum(0)))
            target = torch.linspace(0, 1, bins + 1, dtype=torch.float64, device="cuda") * cum[-1]
            i = (torch.searchsorted(cum, target, right=True) - 1).clamp(0, bins - 1)
            row = edges[d, i] + (target - cum[i]) / sm[i] * (edges[d, i + 1] - edges[d, i])
            row[0], row[-1] = 0.0, 1.0
            edges[d] = row
    est = torch.stack([values(seed + 10_000 + j, 32_768)[0].mean(0) for j in range(7)])
    est = torch.cat((est, est.sum(1, keepdim=True)), 1)
    return est.mean(0), est.std(0, unbiased=True) / math.sqrt(7)


def _lo_exact(case: dict, seed: int) -> dict:
    q2, x = _kinematics(seed, case["count"])
    gbw, config = _gbw(seed), DISConfig()
    n = case["order"]

    def cross_section(Q2, xb, transverse, nodes):
        t, w = np.polynomial.legendre.leggauss(nodes)
        t, w = torch.from_numpy(0.5 * (t + 1)), torch.from_numpy(0.5 * w)
        z, r = t[:, None].clone(), config.maxr * t[None, :]
        total = 0.0
        for q in config.quarks:
            eps = torch.sqrt(Q2 * z * (1 - z) + q.mass**2)
            arg = r * eps
            k0, k1 = _bessel(arg)
            v = ((1 - 2 * z + 2 * z * z) * eps**2 * k1 * k1 + q.mass**2 * k0 * k0 if transverse
                 else 4 * Q2 * (z * (1 - z)) ** 2 * k0 * k0)
            total = total + q.charge**2 * torch.where((arg >= 1e-7) & (arg <= 5e2), v, torch.zeros_like(v))
        y = max(math.log(gbw.x0 / xb), math.log(1 / gbw.x0))
        e = 0.25 * (r * r * gbw.Qs0sqr * math.exp(gbw.lambda_ * y))
        N = torch.where(e < 1e-7, e, 1 - torch.exp(-e))
        return float((w[:, None] * w[None, :] * 2 * math.pi * r * config.maxr * total * N).sum())

    alpha = 1 / 137.035999
    out = {k: [] for k in ("FT", "FL")}
    for Q2, xb in zip(q2.tolist(), x.tolist()):
        factor = 4 * alpha * 3 / (2 * math.pi) ** 2 * Q2 / (4 * math.pi**2 * alpha)
        for name, t in (("FT", True), ("FL", False)):
            out[name].append(factor * cross_section(Q2, xb, t, n))
    FT, FL = (torch.tensor(out[k], dtype=torch.float64) for k in ("FT", "FL"))
    y = q2 / (SQRT_S**2 * x)
    # the errors are differences of two rules near each other: no 64-bit value of their own
    return {"FT": FT, "FL": FL, "F2": FT + FL, "sigma_r": FT + (1 - y * y / (1 + (1 - y) ** 2)) * FL, "FT_error": None,
            "FL_error": None, "F2_error": None, "sigma_r_error": None}


@torch.no_grad()
def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "evolve":
        return _bk_rows(case, _qs0(seed)[0], case["samples"], seed, case["stepper"], case["step"], 0.0)
    if kind == "dndy":
        r, N = _bk_start(case, 0.2)
        k1, k2, act = _bk_rhs(r, N, case["minr"], case["samples"], seed, 0.0)
        return {"r": r[act], "K1": k1[act], "K2_Kf": k2[act], "N": N[act]}
    if kind == "batch":
        return [_bk_rows(case, q, s, seed, "rk4", 0.2, 0.7)["N"]
                for q, s in zip(_qs0(seed, case["sets"]), _budgets(case, seed))]
    if kind == "lo":
        return _lo_exact(case, seed)
    if kind == "fixed":
        parts = [_fixed_exact(case, seed, t) for t in (True, False)]
        return {"value": torch.cat([p[0] for p in parts]), "error": torch.cat([p[1] for p in parts])}
    if kind == "points":
        q2, x = _kinematics(seed, 1)
        pts = _unit_points(case, seed).double().cuda()
        config = DISConfig(quarks=(Quark(QuarkType.LIGHT, case["mass"]),), cuda_nested_points=case["inner"])
        out = []
        for transverse in (True, False):
            q = _QG(pts, float(q2[0]), float(x[0]), case["mass"], transverse, _gbw(seed), config)
            G = q.moments()
            out.append(torch.nan_to_num(q.i2(G) if case["term"] == "I2" else q.i3(G), 0.0, 0.0, 0.0))
        return out
    # vegas, sigma_r, f2: combinations of dozens to hundreds of adaptive integrals, whose grids and
    # stopping rounds a 64-bit run chooses anew; their integrands are those of the cases above
    return None
