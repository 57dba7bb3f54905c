"""The end of a Vegas round of the DIS terms: the thread that combines the iteration sets the
convergence flag that every thread of the CTA has tested, so a round that converges has to re-bin
and store as one that does not.  Bit-equal states but for the flag: the same points and sums."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("term", ["DIP1", "I1"])
@pytest.mark.parametrize("bins", [2, 32, 50])
def test_converging_round_stores_everything(term, bins):
    from nlo_bk_optimized_b200 import _native
    from nlo_bk_optimized_b200.dipole import GBW
    from nlo_bk_optimized_b200.dis import DISConfig, Polarization, Quark, QuarkType
    from nlo_bk_optimized_b200.dis.observables import kinematics
    from nlo_bk_optimized_b200.numerics.integration import VegasOptions, vegas_terms

    quark = Quark(QuarkType.LIGHT, 0.14)
    config = DISConfig(quarks=(quark,))
    kins = [kinematics(2.0 + 0.1 * k, 1e-3, Polarization.T, config, quark) for k in range(64)]
    dipole, number = GBW(Qs0sqr=0.25, lambda_=0.29).native(), _native.DIS_TERMS[term]

    def state(**kw):
        options = VegasOptions(samples_per_iteration=2000, min_iterations=1, bins=bins, **kw)
        return vegas_terms(number, kins, dipole, options, list(range(64)), precision=_native.PRECISION_MIXED,
                           device=torch.device("cuda")).cpu()

    base = _native.DIS_DIMS[number] * (bins + 1)
    one = state(max_iterations=1, epsrel=0.0)
    converged = state(max_iterations=4, epsrel=0.0, epsabs=1e30)
    flag = base + _native.VEGAS_CONVERGED
    assert bool((converged[:, flag] == 1).all()) and bool((one[:, flag] == 0).all())
    assert bool((one[:, base + _native.VEGAS_EVALS] == 2000).all())
    converged[:, flag] = 0
    assert torch.equal(one, converged)
