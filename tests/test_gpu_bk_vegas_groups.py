"""Replica refinement on grids so long that the replicas do not fit one launch."""

import ctypes

import pytest
import torch

from nlo_bk_optimized_b200 import MV, BKConfig, _native
from nlo_bk_optimized_b200.bk.evolution import (
    VEGAS_REPLICAS,
    _r_grid,
    nlo_box,
    params_of,
    vegas_options_of,
    vegas_state,
    workspace,
)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [682, 683, 820])
def test_replica_groups(points):
    """Six replicas in groups of six, of five and one, and of four and two, against six calls with one
    replica each: a refined parent's value is the mean of its integrals, so 7 v - main equals the
    sum of 2 v_k - main, to a few roundings of seven of the largest term (7e-13 of it)."""
    config = BKConfig(RPOINTS=points - 1, MINR=1e-6, MAXR=1e2, MCINTPOINTS=512, PRECISION="fp64")
    r = _r_grid(config, device="cuda", dtype=torch.float64)
    N = MV(qs0sqr=0.2).dipole_amplitude(r).unsqueeze(0).contiguous()
    assert r.numel() == points
    lib, params = _native.load(), params_of(config, _native.PRECISION_FP64)
    box = _native.box(*nlo_box(float(r[0]), float(r[-1])))

    def call(seeds):
        opts = vegas_options_of(config)
        opts.replicas = len(seeds) - 1
        dirs = (_native.SobolDirs * len(seeds))(*[_native.sobol_dirs(4, s) for s in seeds])
        out = [torch.zeros(points, dtype=torch.float64, device="cuda") for _ in range(3)]
        grids = vegas_state(r.device, points)
        ws = workspace(r.device, points, opts)
        _native.check(lib.nlo_bk_rhs_vegas(params, r.data_ptr(), points, None, N.data_ptr(), 1, 0, 1,
                                           ctypes.byref(opts), dirs, box, grids.data_ptr(), out[0].data_ptr(),
                                           out[1].data_ptr(), out[2].data_ptr(), ws.data_ptr(), ws.numel(),
                                           _native.stream_handle(r.device)))
        return out[2]

    seeds = [1000 * k for k in range(1, VEGAS_REPLICAS + 1)]
    main, every = call([0]), call([0, *seeds])
    refined = every != main
    assert 8 < int(refined.sum()) < points
    singles = torch.stack([2 * call([0, s]) - main for s in seeds])
    scale = torch.maximum(main.abs(), singles.abs().amax(0))[refined]
    got, want = (7 * every - main)[refined], singles.sum(0)[refined]
    assert float(((got - want).abs() / scale).max()) <= 1e-13 * 7
