"""Sobol directions in the structure that the kernels take: the engine's numbers for every dimension
that it holds, and no dimension beyond it."""

from __future__ import annotations

import pytest
import torch

from nlo_bk_optimized_b200 import _native


@pytest.mark.parametrize("dims", [1, 4, 5, 8])
@pytest.mark.parametrize("seed", [0, 7, 123456789])
def test_directions_are_the_engines(dims, seed):
    dirs = _native.sobol_dirs(dims, seed)
    engine = torch.quasirandom.SobolEngine(dims, scramble=True, seed=seed)
    assert dirs.dims == dims
    assert [list(dirs.state[d]) for d in range(dims)] == engine.sobolstate.tolist()
    assert list(dirs.shift[:dims]) == engine.shift.tolist()
    assert all(not any(dirs.state[d]) and dirs.shift[d] == 0 for d in range(dims, 8))


@pytest.mark.parametrize("dims,error", [(0, ValueError), (9, IndexError), (64, IndexError)])
def test_other_dimensions_are_refused(dims, error):
    with pytest.raises(error):
        _native.sobol_dirs(dims, 1)
