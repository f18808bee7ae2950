"""The plan's forms by batch size (several CTAs per row, a CTA per row, a lane
per tree over row tiles, a lane per row for depths 9 and 10) against the oracle's
bin-space walk, bit for bit: batches around each form's edge and a tile's, tree
counts around a group's 32, a block's 1,024 and a row's 4,096, wide planes."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_predict import _bins, _ensemble, random_plane

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 64, 65, 1_024, 1_025, 1_480, 9_473, 75_777])
@pytest.mark.parametrize("trees,depth", [(1, 8), (33, 5)])
def test_batches(bb, orc, n, trees, depth):
    rng = np.random.Generator(np.random.PCG64(n + trees))
    nb = _bins(rng, 28)
    plane, codes = random_plane(bb, rng, n, nb)
    ens = _ensemble(rng, nb, trees, depth)
    plan = bb.PredictPlan(plane, ens, 0.3, 0.05)
    want = orc.predict_binned(codes, nb, ens, 0.3, 0.05)
    assert np.array_equal(plan.run(plane).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("n", [3, 200, 1_100])
@pytest.mark.parametrize("trees", [31, 32, 1_025, 4_097])
def test_tree_counts(bb, orc, n, trees):
    rng = np.random.Generator(np.random.PCG64(trees))
    nb = _bins(rng, 5)
    plane, codes = random_plane(bb, rng, n, nb)
    ens = _ensemble(rng, nb, trees, 3)
    plan = bb.PredictPlan(plane, ens, -0.5, 0.1)
    for k in (0, trees - 1):
        if k == 0 or trees > 1:
            want = orc.predict_binned(codes, nb, ens[:k] if k else ens, -0.5, 0.1)
            assert np.array_equal(plan.run(plane, n_trees=k).view(np.uint32),
                                  want.view(np.uint32))


@pytest.mark.parametrize("F,depth", [(256, 8), (70, 8), (28, 9), (28, 10)])
@pytest.mark.parametrize("n", [2, 500, 3_001])
def test_wide_and_deep(bb, orc, F, depth, n):
    rng = np.random.Generator(np.random.PCG64(F + depth + n))
    nb = _bins(rng, F)
    plane, codes = random_plane(bb, rng, n, nb)
    ens = _ensemble(rng, nb, 40, depth)
    plan = bb.PredictPlan(plane, ens, 0.0, 1.0)
    want = orc.predict_binned(codes, nb, ens, 0.0, 1.0)
    assert np.array_equal(plan.run(plane).view(np.uint32), want.view(np.uint32))
