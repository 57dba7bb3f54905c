"""The Vegas rounds' warp sampling at its edges, through the K2+Kf integrals against the oracle.

Bin numbers around the 32 points of a warp's block (one conflict-free histogram phase for 32 and 64,
several for 31, 33 and 50), warm-ups that leave the next round starting inside a block of 32, a
partial last block, one and several CTAs per parent; and direction numbers that are no digital
net, which take the lane-serial histogram.  FP64 build: the oracle's driver on the same points,
whose histograms add in another order (1e-16 a sum), so 1e-10 as in the Vegas parity tests."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins,samples,reverse", [(32, 1005, False), (31, 2035, False), (33, 1005, False),
                                                  (50, 5003, False), (64, 2035, False), (32, 1005, True)])
def test_rounds_vs_oracle(bins, samples, reverse, monkeypatch):
    from nlo_bk_optimized_b200 import MV, BKConfig, _native
    from nlo_bk_optimized_b200.bk import evolution as ev

    config = BKConfig(RPOINTS=12, MINR=1e-4, MAXR=30.0, MCINTPOINTS=samples, PRECISION="fp64")
    r = ev._r_grid(config, device="cuda", dtype=torch.float64)
    N = MV(qs0sqr=0.2).dipole_amplitude(r)
    points, lib = r.numel(), _native.load()
    opts = ev.vegas_options_of(config)
    opts.bins = bins
    state_, shift = oracle.sobol_state(4, 3)
    dirs = _native.sobol_dirs(4, 3)
    if reverse:
        state_ = np.ascontiguousarray(np.asarray(state_).reshape(4, 30)[:, ::-1])
        for d in range(4):
            for j in range(30):
                dirs.state[d][j] = int(state_[d, j])
    monkeypatch.setattr(oracle, "sobol_state", lambda dims, seed: (state_, shift))
    grids = torch.zeros(int(lib.nlo_bk_vegas_state_doubles(points, bins)), dtype=torch.float64, device="cuda")
    ws = torch.empty(int(lib.nlo_bk_vegas_workspace_bytes(points, opts)), dtype=torch.uint8, device="cuda")
    dndy, k1, k2kf = (torch.empty_like(N) for _ in range(3))
    box = ev.nlo_box(float(r[0]), float(r[-1]))
    _native.check(lib.nlo_bk_rhs_vegas(ev.params_of(config, _native.PRECISION_FP64), r.data_ptr(), points, None,
                                       N.data_ptr(), 1, 0, 1, opts, dirs, _native.box(*box), grids.data_ptr(),
                                       dndy.data_ptr(), k1.data_ptr(), k2kf.data_ptr(), ws.data_ptr(), ws.numel(),
                                       _native.stream_handle(r.device)))
    rn, Nn = r.cpu().numpy(), N.cpu().numpy()
    edges = grids.cpu().numpy().reshape(points, -1)[:, : 4 * (bins + 1)].reshape(points, 4, bins + 1)
    spline, phys = oracle.loglog_spline(rn, Nn, 1), oracle.physics(config)
    for i in (1, 4, 7):
        ref = oracle.vegas_k2kf(float(rn[i]), spline, phys, tuple(np.array(v) for v in box), 3, samples=samples,
                                warmup=opts.warmup_samples, bins=bins)
        assert abs(float(k2kf[i]) - ref.value) <= 1e-10 * abs(ref.value)
        assert np.max(np.abs(edges[i] - ref.edges)) <= 1e-10
