"""The launches of this library's kernels in an evolution, counted on the device by the profiler, against
the number per RK4 step that the bench multiplies: launched one by one (96 points) and replayed from
a recorded step (200 points)."""

from __future__ import annotations

import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [96, 200])
def test_launches_per_step(points, monkeypatch):
    from torch.profiler import ProfilerActivity, profile

    from nlo_bk_optimized_b200 import MV, BKConfig, solve_bk
    from nlo_bk_optimized_b200.bk.config import IntegrationMethod

    monkeypatch.syspath_prepend(str(Path(__file__).resolve().parents[1]))
    import bench

    config = BKConfig(RPOINTS=points - 1, MINR=1e-6, MAXR=1e2, MCINTPOINTS=4096, DE_SOLVER_STEP=0.1, STEPPER="rk4",
                      INTMETHOD_NLO=IntegrationMethod.SOBOL)

    def launches(steps: int) -> int:
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
            solve_bk(MV(qs0sqr=0.2), 0.1 * steps, config, device="cuda", seed=0)
            torch.cuda.synchronize()
        return sum(event.device_type.name == "CUDA" and "nlo::" in event.name for event in prof.events())

    if launches(1) == 0:
        pytest.skip("the profiler records no kernels here (another tool holds it)")
    few, more = launches(3), launches(7)
    assert more - few == 4 * bench.LAUNCHES_PER_RK4_STEP, (few, more)
