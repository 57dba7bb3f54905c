"""The FP32 moments of the nested qqbar-g terms (one warp per 32 samples, lanes on the nodes of the
inner rule) against the oracle's FP64 integrand at the same points.

Sizes where the mapping can go wrong: rules shorter than a half-warp, one node off its
multiples, the largest; one sample, partial warps, a partial CTA.  Masses: 0.02 GeV keeps every
segment in the series of the lambda-difference, 0.14 mixes the forms, 4.5 takes the direct
one nearly everywhere.  Tolerance: the FP32 chain from the amplitudes (6e-8 of N ~ 1) to the
impact factor rounds some 10 times at 6e-8 and its terms cancel to about 1/20, so the vector of
values carries about 1e-5 of its norm at most."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import dis as od

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inner,count", [(8, 33), (15, 1), (16, 31), (17, 100), (33, 129), (48, 257), (128, 64)])
@pytest.mark.parametrize("mass", [0.02, 0.14, 4.5])
def test_moments_vs_oracle(inner, count, mass):
    from nlo_bk_optimized_b200.dipole import GBW
    from nlo_bk_optimized_b200.dis import DISConfig, Polarization, Quark, QuarkType, integrand_qg_nested_massive

    x = np.random.default_rng(inner).uniform(0.02, 0.98, (count, 5)).astype(np.float32).astype(np.float64)
    quark = Quark(QuarkType.LIGHT, mass)
    config = DISConfig(quarks=(quark,), cuda_nested_points=inner)
    points = torch.tensor(x, dtype=torch.float32, device="cuda")
    Q2, xbj = torch.tensor(8.0), torch.tensor(1e-3)
    for pol in (Polarization.T, Polarization.L):
        kin = od.Kinematics(Q2=8.0, xbj=float(xbj), mf=mass, transverse=pol is Polarization.T,
                            active_flavors=config.active_flavors)
        for term in ("I2", "I3"):
            got = integrand_qg_nested_massive(points, Q2, xbj, pol, quark, term, GBW(Qs0sqr=0.25, lambda_=0.29),
                                              config).double().cpu().numpy()
            ref = od.qg_integrand(x, kin, term + "n", od.GBWDipole(qs0sqr=0.25, lam=0.29), points=inner)
            floor = np.sqrt(count) * np.finfo(np.float32).tiny  # the device flushes what FP32 cannot hold
            assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref) + floor, (pol, term)
