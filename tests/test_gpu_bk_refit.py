"""The spline refit's warp scans and the K2+Kf tiles at their edges, through the FP64 right-hand side
against the oracle's (1e-10 of the largest value, as in the FP64 parity tests): knot numbers around
the 32 stretches of a warp (one interior knot, one per lane and one more, stretches longer than the
factorisation's run-in), budgets around the tiles of a launch (one sample, a tile less one and
plus one, a share of several tiles)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,samples", [(2, 64), (3, 64), (32, 64), (33, 64), (34, 64), (65, 64), (400, 64),
                                            (600, 32), (20, 1), (20, 31), (20, 33), (20, 4095), (130, 18945),
                                            (20, 150001)])
def test_rhs_vs_oracle(points, samples):
    from nlo_bk_optimized_b200 import MV, BKConfig
    from nlo_bk_optimized_b200.bk.config import IntegrationMethod
    from nlo_bk_optimized_b200.bk.evolution import _r_grid, rhs

    config = BKConfig(RPOINTS=points, MINR=1e-5, MAXR=30.0, MCINTPOINTS=samples, PRECISION="fp64",
                      INTMETHOD_NLO=IntegrationMethod.SOBOL)
    r = _r_grid(config, device="cuda", dtype=torch.float64)
    N = MV(qs0sqr=0.2).dipole_amplitude(r)
    _, k1, k2kf = rhs(N, r, config, seed=2)
    state, shift = oracle.sobol_state(4, 2)
    ref = oracle.derivative(N.cpu().numpy(), r.cpu().numpy(), oracle.physics(config),
                            oracle.sobol(state, shift, 0, samples, as_f32=False), False)
    for got, want in ((k1, ref.K1), (k2kf, ref.K2 + ref.Kf)):
        assert np.max(np.abs(got.cpu().numpy() - want)) <= 1e-10 * np.max(np.abs(want))
