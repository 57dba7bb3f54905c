"""The mixed build's Vegas rounds of K2+Kf (two packed blocks of 32 samples a pass) against the
oracle in FP64 on the same points."""

from __future__ import annotations

import ctypes
from types import SimpleNamespace

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _setup(points=24, minr=1e-5, maxr=30.0, qs0sqr=0.2, **kw):
    from nlo_bk_optimized_b200 import MV, BKConfig
    from nlo_bk_optimized_b200.bk import evolution as ev

    config = BKConfig(RPOINTS=points - 1, MINR=minr, MAXR=maxr, MCINTPOINTS=1024, PRECISION="mixed", **kw)
    r = ev._r_grid(config, device="cuda", dtype=torch.float64)
    N = MV(qs0sqr=qs0sqr).dipole_amplitude(r)
    rn, Nn = r.cpu().numpy(), N.cpu().numpy()
    active = np.nonzero((np.arange(rn.size) > 0) & (Nn <= 0.99999))[0]
    return SimpleNamespace(config=config, r=r, N=N, rn=rn, active=active, spline=oracle.loglog_spline(rn, Nn, 1),
                           phys=oracle.physics(config), box=oracle.nlo_box(rn))


def _device(s, *, bins, samples, warmup=0, iterations=1, epsrel=0.0, edges=None, seed=0):
    """Values, edges, slots and workspace of one right-hand side; `edges` [points, 4 (bins + 1)]: kept grids."""
    from nlo_bk_optimized_b200 import _native
    from nlo_bk_optimized_b200.bk import evolution as ev

    lib, points = _native.load(), s.r.numel()
    options = ev.vegas_options_of(s.config)
    options.bins, options.samples_per_iteration, options.warmup_samples = bins, samples, warmup
    options.max_iterations, options.min_iterations, options.epsrel = iterations, iterations, epsrel
    options.replicas = 0
    grids = torch.zeros(int(lib.nlo_bk_vegas_state_doubles(points, bins)), dtype=torch.float64, device="cuda")
    base = 4 * (bins + 1)
    if edges is not None:
        rows = grids.reshape(points, -1)
        rows[:, :base] = torch.as_tensor(edges)
        rows[:, base + 9] = 1.0  # the parent has a grid
    ws = torch.empty(int(lib.nlo_bk_vegas_workspace_bytes(points, options)), dtype=torch.uint8, device="cuda")
    dndy, k1, k2kf = (torch.empty_like(s.N) for _ in range(3))
    lower, width = ev.nlo_box(float(s.r[0]), float(s.r[-1]))
    _native.check(lib.nlo_bk_rhs_vegas(ev.params_of(s.config, _native.PRECISION_MIXED), s.r.data_ptr(), points, None,
                                       s.N.data_ptr(), 1, 0, 1, ctypes.byref(options), _native.sobol_dirs(4, seed),
                                       _native.box(lower, width), grids.data_ptr(), dndy.data_ptr(), k1.data_ptr(),
                                       k2kf.data_ptr(), ws.data_ptr(), ws.numel(), _native.stream_handle(s.r.device)))
    rows = grids.cpu().numpy().reshape(points, -1)
    return k2kf.cpu().numpy(), rows[:, :base].reshape(points, 4, bins + 1), rows[:, base:], ws


@pytest.mark.parametrize("bins,samples", [(32, 1005), (64, 1005), (96, 2035), (31, 1005), (33, 1005)])
def test_histograms_keep_every_sample(bins, samples):
    """A warp adds its blocks of 32 samples to the same rows one after the other, two blocks a pass (in
    one conflict-free phase at 32, 64 and 96 bins).  Every sample's |w| goes once into each
    dimension's histogram, so the four of a partial row have one sum: FP64 sums of at most 2,035
    positive terms in other orders, 2,035 x 1.1e-16 of it."""
    from nlo_bk_optimized_b200 import _native

    s = _setup()
    _, edges, slots, ws = _device(s, bins=bins, samples=samples)
    assert np.array_equal(edges, _device(s, bins=bins, samples=samples)[1])
    # up to 2,048 samples one CTA per parent: its partial row begins the workspace's Vegas part
    keys, points = 4 + 4 * bins, s.r.numel()
    start = int(_native.load().nlo_bk_rhs_workspace_bytes(points))
    rows = ws[start : start + 8 * keys * points].view(torch.float64).cpu().numpy().reshape(points, keys)[s.active]
    sums = rows[:, 2 : 2 + 4 * bins].reshape(-1, 4, bins).sum(2)
    assert np.all(slots[s.active, 4] == samples) and np.all(sums > 0)
    assert np.all(sums.max(1) - sums.min(1) <= 2.3e-13 * sums.max(1))
    assert np.all(sums.min(1) >= np.abs(rows[:, 0]) * (1 - 2.3e-13))


@pytest.mark.parametrize("points,maxr,qs0sqr,samples,symmetrize", [(119, 100.0, 0.948, 36068, True),
                                                                   (88, 100.0, 0.621, 12421, True),
                                                                   (77, 100.0, 2.585, 16178, False)])
def test_error_on_adapted_grids(points, maxr, qs0sqr, samples, symmetrize):
    """One iteration on grids adapted by a warm-up and two iterations in FP64 (the oracle's), whose
    samples gather where the integrand cancels: the vector of values over the parents keeps the
    single-precision bound of 2e-5 (the scalar evaluation with knot-relative amplitudes keeps
    1e-5 on average; positions rounded to FP32 in units of the grid gave up to 7e-5)."""
    s = _setup(points, minr=1e-6, maxr=maxr, qs0sqr=qs0sqr, SYMMETRIZE_Z_Z2_INTEGRATION=symmetrize)
    edges = np.tile(np.linspace(0, 1, 33), (points, 4, 1))
    want = np.zeros(points)
    for i in s.active:
        grid = oracle.VegasGrid(None)
        run = dict(min_iterations=1, epsrel=0.0, f32_points=True, state=grid)
        oracle.vegas_k2kf(float(s.rn[i]), s.spline, s.phys, s.box, 0, samples=samples, warmup=samples // 5,
                          max_iterations=2, **run | {"min_iterations": 2})
        edges[i] = grid.edges
        want[i] = oracle.vegas_k2kf(float(s.rn[i]), s.spline, s.phys, s.box, 0, samples=samples, warmup=0,
                                    max_iterations=1, **run).value
    got = _device(s, bins=32, samples=samples, edges=edges.reshape(points, -1))[0]
    error = np.linalg.norm(got[s.active] - want[s.active]) / np.linalg.norm(want[s.active])
    assert error <= 2e-5, error


def _couplings():
    from nlo_bk_optimized_b200.bk.config import RunningCouplingLO as LO, RunningCouplingNLO as NLO

    return {"smooth": {}, "capped": {"ALPHA_S_CAP": 0.3}, "fixed": {"RC_LO": LO.FIXED_LO, "RC_NLO": NLO.FIXED_NLO},
            "thresholds": {"NF": 5}, "parent": {"RC_NLO": NLO.PARENT_NLO}, "gluons": {"NF": 0}}


@pytest.mark.parametrize("symmetrize", [True, False])
@pytest.mark.parametrize("coupling,bins,warmup,samples", [("smooth", 32, 13, 4096), ("capped", 31, 45, 2035),
                                                          ("fixed", 33, 1005, 4099), ("thresholds", 50, 31, 5003),
                                                          ("parent", 64, 77, 2035), ("gluons", 2, 2, 33)])
def test_ragged_rounds_of_every_variant(symmetrize, coupling, bins, warmup, samples, monkeypatch):
    """Every instantiation of the packed evaluation, in an iteration that starts inside a block of 32
    points (after the warm-up) and ends in one.  The grid of the iteration is the device's own (a
    first call whose one iteration takes the warm-up's points leaves the same one), so that the
    oracle evaluates at the same points.  Tolerance: a sample's FP32 error is a few roundings of
    z over its distance to the parent, 4 x 6e-8 / (X/r) of it, and among the 1e5 evaluations of a case
    X/r reaches down to some 5e-4: 5e-4 of such a sample, which weighs no more than the value and
    its statistical error."""
    s = _setup(SYMMETRIZE_Z_Z2_INTEGRATION=symmetrize, **_couplings()[coupling])
    edges = _device(s, bins=bins, samples=warmup)[1]
    got, _, slots, _ = _device(s, bins=bins, samples=samples, warmup=warmup)
    draw = oracle.sobol
    monkeypatch.setattr(oracle, "sobol", lambda state, shift, offset, n, **kw: draw(state, shift, offset + warmup, n,
                                                                                    **kw))
    want, scale, parts = (np.zeros(s.r.numel()) for _ in range(3))
    for i in s.active:
        ref = oracle.vegas_k2kf(float(s.rn[i]), s.spline, s.phys, s.box, 0, samples=samples, warmup=0, bins=bins,
                                max_iterations=1, min_iterations=1, epsrel=0.0, f32_points=True,
                                state=oracle.VegasGrid(edges[i].copy()))
        want[i], scale[i], parts[i] = ref.value, abs(ref.value) + ref.error, ref.components[0]
        assert slots[i, 4] == warmup + samples
    a = s.active
    assert np.linalg.norm(got[a] - want[a]) <= 5e-4 * np.linalg.norm(scale[a])
    assert np.linalg.norm(slots[a, 13] / slots[a, 1] - parts[a]) <= 5e-4 * np.linalg.norm(scale[a])
