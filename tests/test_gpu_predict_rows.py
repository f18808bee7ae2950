"""Batches that fill the lane-per-row form's passes, where shallow ensembles
take it, against the lane-per-tree form (the same rows in smaller batches) and
the oracle's bin-space walk, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_predict import _bins, _ensemble, random_plane

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F,codes16", [(5, False), (28, False), (54, False), (14, True)])
@pytest.mark.parametrize("trees,depth", [(1, 1), (31, 2), (33, 3), (100, 4), (129, 5), (160, 6), (100, 7), (137, 8)])
def test_full_passes(bb, orc, F, codes16, trees, depth):
    n = 303_104 - 37
    rng = np.random.Generator(np.random.PCG64(F * 100 + depth))
    nb = _bins(rng, F)
    if codes16:
        nb[0] = 300
    plane, codes = random_plane(bb, rng, n, nb)
    ens = _ensemble(rng, nb, trees, depth)
    plan = bb.PredictPlan(plane, ens, 0.3, 0.05)
    got = plan.run(plane)
    some = np.r_[0:600, n - 1200:n]
    want = orc.predict_binned(np.ascontiguousarray(codes[:, some]), nb, ens, 0.3, 0.05)
    assert np.array_equal(got[some].view(np.uint32), want.view(np.uint32))
    k = max(1, trees - 1)
    want = orc.predict_binned(np.ascontiguousarray(codes[:, some]), nb, ens[:k], 0.3, 0.05)
    assert np.array_equal(plan.run(plane, n_trees=k)[some].view(np.uint32), want.view(np.uint32))
