"""Cuts of the longest sample bb_fit_cuts takes, 2^32 - 1 rows: the last tile's keys
are counted and placed as every other's."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_the_longest_column(bb):
    import torch
    n = (1 << 32) - 1
    if torch.cuda.mem_get_info()[0] < 90 << 30:  # 17 GB of values, 52 of scratch
        pytest.skip("less than 90 GB free")
    X = torch.arange(7, device="cuda").float().sub_(3).repeat(n // 7 + 1)[:n]
    cuts, off = bb.fit_cuts_device(X[:, None], n_samples=n)
    want = np.array([-3, -2, -1, 0, 1, 2, 3, np.finfo(np.float32).max, np.inf], np.float32)
    assert np.array_equal(cuts, want) and off.tolist() == [0, len(want)]
    del X
    torch.cuda.empty_cache()
