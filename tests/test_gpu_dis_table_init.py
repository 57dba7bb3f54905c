"""The BK table's initialised interpolation: spline and saturation search on the device."""

import numpy as np
import pytest
import torch

from oracle import dis as od

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("knots", [9, 33, 257, 1500])
@pytest.mark.parametrize("scale", [0.0005, 1.0, 20.0, 100.0])
def test_initialised_table(knots, scale):
    """Tables 1 - exp(-(r/scale)^2) up to r = 200: saturated at the search's first radius, after
    a few steps, in the second 32 radii of its first step, and not within its 41 steps; from
    the fewest knots a table may have.  The radius found is the oracle's (the same sums of
    steps: 1e-12), and so are the amplitudes: FP64 splines of values up to 1 whose overshoot
    on coarse knots stays below 1e3, a few tens of roundings each (1e-11)."""
    from nlo_bk_optimized_b200.dipole import BKDipole, DipoleTable

    r = np.geomspace(1e-5, 200.0, knots)
    y = np.array([0.0, 1.0, 2.5])
    N = np.array([-np.expm1(-((r / scale) ** 2) * np.exp(0.1 * v)) for v in y])
    N = np.minimum(N, 1.0)
    tab = BKDipole(DipoleTable(torch.as_tensor(r).cuda(), torch.as_tensor(y).cuda(), torch.as_tensor(N).cuda(), 1.0))
    ref = od.TableDipole(r, y, N)
    tab.initialize_interpolation(1.3)
    ref.initialize(1.3)
    assert tab.maxr_interpolate == pytest.approx(ref.maxr_interpolate, rel=1e-12)
    at = np.concatenate([r, np.geomspace(1.1e-5, 199.0, 777)])
    got = tab.dipole_amplitude(torch.as_tensor(at).cuda(), torch.full((at.size,), 1.3, dtype=torch.float64,
                                                                     device="cuda")).cpu().numpy()
    np.testing.assert_allclose(got, ref(at, np.full_like(at, 1.3)), rtol=0, atol=1e-11)
