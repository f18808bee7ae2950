"""Batches around the edges of the CTA-per-row form -- where its CTAs give up half
their threads (two and four rows an SM), and its last batch (eight rows an SM,
sixteen with more than 500 trees) -- against the oracle's bin-space walk, bit for
bit."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_predict import _bins, _ensemble, random_plane

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm", [2, 4, 8, 16])
@pytest.mark.parametrize("past", [0, 1])
@pytest.mark.parametrize("trees", [500, 501])
def test_row_batches(bb, orc, per_sm, past, trees):
    import torch
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + past
    rng = np.random.Generator(np.random.PCG64(n + trees))
    nb = _bins(rng, 13)
    plane, codes = random_plane(bb, rng, n, nb)
    ens = _ensemble(rng, nb, trees, 4)
    plan = bb.PredictPlan(plane, ens, 0.2, 0.1)
    want = orc.predict_binned(codes, nb, ens, 0.2, 0.1)
    assert np.array_equal(plan.run(plane).view(np.uint32), want.view(np.uint32))
