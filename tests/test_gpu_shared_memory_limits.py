"""Launches whose shared memory crosses the 48 KB that need no opt-in, counting the kernel's own
(static) part: sizes on both sides of the line, ascending in a process of their own, where no larger
launch has raised a limit before.

* the nested mixed DIS terms: 27,904 B static + 420 B a bin cross at 51 bins; 118 bins cross by the
  dynamic part alone; 256 is the largest number;
* the spline refit: 56 B a knot, crossing at 878 knots (a static part of 144 B once made it 876);
* the BK Vegas rounds: 1,328 B + 368 B a bin + the tables, crossing at 903 knots with 32 bins in FP64
  (dynamic alone at 936) and at 129 bins with 24 knots in FP32 (133); grids long enough to cross
  at 32 bins in FP32 exceed the shared memory of K1.

Each result is compared with a value: FP64 nested terms at the same points (FP32 moments, 1e-5 of
the norm, and the grid's points in FP64: 1e-4), the oracle's spline (1e-9 of the largest
coefficient, as for the other refits) and the oracle's Vegas (1e-10 in FP64; in FP32 1e-4 of the
value and its error, as for the mixed build elsewhere)."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]


def _fresh(code: str) -> None:
    result = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert result.returncode == 0, result.stdout + result.stderr[-3000:]


def test_nested_dis_terms():
    _fresh("""
import torch
from nlo_bk_optimized_b200 import _native
from nlo_bk_optimized_b200.dipole import GBW
from nlo_bk_optimized_b200.dis import DISConfig, Polarization, Quark, QuarkType
from nlo_bk_optimized_b200.dis.observables import kinematics
from nlo_bk_optimized_b200.numerics.integration import VegasOptions, state_results, vegas_terms
quark = Quark(QuarkType.LIGHT, 0.14)
config = DISConfig(quarks=(quark,))
kins = [kinematics(q, 1e-3, Polarization.T, config, quark) for q in (2.0, 8.0)]
dipole = GBW(Qs0sqr=0.25, lambda_=0.29).native()
for bins in (50, 51, 64, 117, 118, 256):
    for term in ("I2N", "I3N"):
        options = VegasOptions(samples_per_iteration=4096, max_iterations=1, min_iterations=1, bins=bins, epsrel=0.0)
        number = _native.DIS_TERMS[term]
        got = [state_results(vegas_terms(number, kins, dipole, options, [1, 2], precision=p,
                                         device=torch.device("cuda")), number, bins)["value"]
               for p in (_native.PRECISION_MIXED, _native.PRECISION_FP64)]
        assert bool((got[1] != 0).all()), (bins, term)
        torch.testing.assert_close(got[0], got[1], rtol=1e-4, atol=0)
""")


def test_spline_refit():
    _fresh("""
import numpy as np, torch, oracle
from nlo_bk_optimized_b200 import MV, BKConfig, kernels
from nlo_bk_optimized_b200.bk.config import IntegrationMethod
from nlo_bk_optimized_b200.bk.evolution import _r_grid, rhs
for points in (875, 876, 877, 878):
    config = BKConfig(RPOINTS=points - 1, MINR=1e-5, MAXR=30.0, MCINTPOINTS=32, INTMETHOD_NLO=IntegrationMethod.SOBOL)
    r = _r_grid(config, device="cuda", dtype=torch.float64)
    N = MV(qs0sqr=0.2).dipole_amplitude(r)
    assert r.numel() == points
    got = kernels.splines(r, N)["s"].cpu().numpy()
    ref = oracle.loglog_spline(r.cpu().numpy(), N.cpu().numpy(), 1)
    for k, want in enumerate((ref.a, ref.b, ref.c, ref.d)):
        assert np.max(np.abs(got[:, k] - want)) <= 1e-9 * np.max(np.abs(want)), (points, k)
    dndy, k1, k2kf = rhs(N, r, config, seed=1)
    assert bool(torch.isfinite(dndy).all()) and bool((k1 != 0).any()) and bool((k2kf != 0).any())
""")


def test_bk_vegas_rounds_fp64():
    _fresh("""
import numpy as np, torch, oracle
from nlo_bk_optimized_b200 import MV, BKConfig
from nlo_bk_optimized_b200.bk.evolution import _r_grid, rhs
for points in (902, 903, 935, 936):
    config = BKConfig(RPOINTS=points - 1, MINR=1e-5, MAXR=30.0, MCINTPOINTS=256, PRECISION="fp64")
    r = _r_grid(config, device="cuda", dtype=torch.float64)
    N = MV(qs0sqr=0.2).dipole_amplitude(r)
    assert r.numel() == points
    _, _, k2kf = rhs(N, r, config, seed=1)
    rn, Nn = r.cpu().numpy(), N.cpu().numpy()
    spline = oracle.loglog_spline(rn, Nn, 1)
    for i in (points // 2, 2 * points // 3):
        ref = oracle.vegas_k2kf(float(rn[i]), spline, oracle.physics(config), oracle.nlo_box(rn), 1, samples=256,
                                warmup=max(2, 256 // 5))
        assert abs(float(k2kf[i]) - ref.value) <= 1e-10 * abs(ref.value), (points, i, float(k2kf[i]), ref)
""")


def test_bk_vegas_rounds_mixed():
    _fresh("""
import sys
sys.path.insert(0, "tests")
import oracle
from test_gpu_bk_vegas_mixed import _device, _setup
s = _setup()
assert s.r.numel() == 24
for bins in (128, 129, 132, 133, 256):
    got = _device(s, bins=bins, samples=1024)[0]
    for i in s.active[[3, 10, 15]]:
        ref = oracle.vegas_k2kf(float(s.rn[i]), s.spline, s.phys, s.box, 0, samples=1024, warmup=0, bins=bins,
                                max_iterations=1, min_iterations=1, epsrel=0.0, f32_points=True)
        assert abs(got[i] - ref.value) <= 1e-4 * (abs(ref.value) + ref.error), (bins, i, got[i], ref)
""")
