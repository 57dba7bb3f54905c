"""The nested FP32 integrands where the number of points per warp changes: one to 32, doubling at
16 points per SM and warp slot, against the oracle in FP64.  Tolerance as for the moments: the FP32
chain rounds some 10 times at 6e-8 and its terms cancel to about 1/20, 1e-5 of the norm."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import dis as od

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_warp,extra", [(1, 0), (1, 1), (2, 1), (4, 1), (8, 1), (16, 0), (16, 1)])
def test_points_per_warp(per_warp, extra):
    from nlo_bk_optimized_b200.dipole import GBW
    from nlo_bk_optimized_b200.dis import DISConfig, Polarization, Quark, QuarkType, integrand_qg_nested_massive

    count = 16 * torch.cuda.get_device_properties(0).multi_processor_count * per_warp + extra
    x = np.random.default_rng(per_warp).uniform(0.02, 0.98, (count, 5)).astype(np.float32).astype(np.float64)
    quark = Quark(QuarkType.LIGHT, 0.14)
    config = DISConfig(quarks=(quark,), cuda_nested_points=9)
    Q2, xbj = torch.tensor(8.0), torch.tensor(1e-3)
    kin = od.Kinematics(Q2=8.0, xbj=float(xbj), mf=0.14, transverse=True, active_flavors=config.active_flavors)
    got = integrand_qg_nested_massive(torch.tensor(x, dtype=torch.float32, device="cuda"), Q2, xbj, Polarization.T,
                                      quark, "I3", GBW(Qs0sqr=0.25, lambda_=0.29), config).double().cpu().numpy()
    ref = od.qg_integrand(x, kin, "I3n", od.GBWDipole(qs0sqr=0.25, lam=0.29), points=9)
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
    # every point has its own value, the last ones too
    tail = slice(-64, None)
    assert np.linalg.norm(got[tail] - ref[tail]) <= 1e-4 * np.linalg.norm(ref[tail])


@pytest.mark.parametrize("inner", [8, 17, 48])
def test_values_repeat(inner):
    """The half-warps of a pair take their sums' place in the rows that both have read: the same bits
    on every call, at rules that leave lanes without a node and at more points than one pass takes."""
    from nlo_bk_optimized_b200.dipole import GBW
    from nlo_bk_optimized_b200.dis import DISConfig, Polarization, Quark, QuarkType, integrand_qg_nested_massive

    quark = Quark(QuarkType.LIGHT, 0.14)
    config = DISConfig(quarks=(quark,), cuda_nested_points=inner)
    x = torch.rand((90001, 5), generator=torch.Generator().manual_seed(inner)).clamp(0.02, 0.98).cuda()
    call = lambda: integrand_qg_nested_massive(x, torch.tensor(8.0), torch.tensor(1e-3), Polarization.L, quark, "I2",  # noqa: E731
                                               GBW(Qs0sqr=0.25, lambda_=0.29), config)
    first = call()
    assert all(torch.equal(first, call()) for _ in range(4))
