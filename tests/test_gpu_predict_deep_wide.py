"""Plans of depth 9 and 10 over planes of one to eight mirror tiles (up to 256 u8
or 128 u16 features): a batch of any size scores as the oracle's bin-space walk,
bit for bit, around the batch sizes where the rows' passes and the trees' split
change."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_predict import _bins, _ensemble, random_plane

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F,top,depth", [(28, 256, 10), (65, 256, 9), (97, 256, 9), (128, 256, 10),
                                         (256, 256, 10), (49, 700, 9), (128, 700, 10)])
@pytest.mark.parametrize("n", [1, 2, 500, 4_097, 37_889, 100_000])
def test_any_batch(bb, orc, F, top, depth, n):
    rng = np.random.Generator(np.random.PCG64(F + depth + n))
    nb = _bins(rng, F, top)
    plane, codes = random_plane(bb, rng, n, nb)
    ens = _ensemble(rng, nb, 24, depth)
    plan = bb.PredictPlan(plane, ens, 0.1, 0.5)
    assert plan.depth == depth
    for k in (0, 7):
        want = orc.predict_binned(codes, nb, ens[:k] if k else ens, 0.1, 0.5)
        assert np.array_equal(plan.run(plane, n_trees=k).view(np.uint32), want.view(np.uint32))
