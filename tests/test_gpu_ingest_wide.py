"""Bin application where its form changes with the values rather than the rows: wide
planes of few rows on both sides of the border, and tables beside which shared
memory holds one tile of values, over several row tiles a CTA, against the
oracle's transform."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_ingest_forms import _matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,F,nb", [
    # 352 and 336 feature slots a row: 1,117 / 1,118 and 1,170 / 1,171 rows
    (1_117, 333, 255), (1_118, 333, 255), (1_170, 333, 300), (1_171, 333, 300),
    (195, 2_000, 60), (196, 2_000, 60), (700, 2_000, 60),
    # 39,647 cuts a tile leave room for two tiles of values, 48,863 for one
    (40_001, 32, 1_240), (100_003, 32, 1_250), (90_000, 33, 1_500), (14_000, 32, 1_540),
])
def test_codes(bb, orc, n, F, nb):
    rng = np.random.Generator(np.random.PCG64(n + F + nb))
    X, cuts, off = _matrix(rng, n, F, nb)
    want = orc.transform(X, cuts, off)
    import torch
    plane = bb.Plane.from_device(torch.as_tensor(X, device="cuda"), cuts, off)
    assert np.array_equal(plane.bins(), want)
    # the mirror, through the counts of a histogram build, which reads it
    ones = np.ones(n, np.float32)
    cells = bb.populate(plane, bb.TrainParams(hist_mode="exact", max_depth=1), ones, ones)
    count = np.concatenate([np.bincount(want[f], minlength=off[f + 1] - off[f])
                            for f in range(F)])
    assert np.array_equal(cells[:, 1], count)
