"""The multi-set K2+Kf kernel where its shares of parents and samples are ragged."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rpoints", [30, 32, 255, 449, 895])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_ragged_shares(rpoints, dtype):
    """One step of sets of 1, 31, 33 and 20,001 samples over grids of a partial group of 32
    parents, one group and a point, exactly eight groups, a parent tile and two points and
    exactly two parent tiles, against each set alone: the same points, the same FP32 sums of 32
    samples, and FP64 sums of at most 20,001 / 32 partials and 296 CTAs in another order
    (1e-12 relative, as for every batch)."""
    from nlo_bk_optimized_b200 import MV, BKConfig, solve_bk
    from nlo_bk_optimized_b200.bk.batch import solve_bk_batch
    from nlo_bk_optimized_b200.bk.config import IntegrationMethod

    base = dict(RPOINTS=rpoints, MINR=1e-6, MAXR=1e2, DE_SOLVER_STEP=0.2, STEPPER="euler",
                INTMETHOD_NLO=IntegrationMethod.SOBOL)
    budgets = [1, 31, 33, 20001]
    ics = [MV(qs0sqr=0.1 + 0.1 * k) for k in range(len(budgets))]
    for waves in (1, 3):
        tables = solve_bk_batch(ics, 0.2, BKConfig(MCINTPOINTS=64, **base), samples=budgets, device="cuda",
                                dtype=dtype, waves=waves)
        for ic, budget, table in zip(ics, budgets, tables):
            alone = solve_bk(ic, 0.2, BKConfig(MCINTPOINTS=budget, **base), device="cuda", dtype=dtype, seed=0)
            torch.testing.assert_close(table.N.double(), alone.N.double(), rtol=1e-12, atol=0)
