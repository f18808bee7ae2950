"""The device cut fit's sort and scans at its tiles' edges against the host fit:
rows around a tile's 8,192 keys and a warp's run, columns of repeated, sorted,
signed-zero, infinite and missing values, budgets around a block's 1,024."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 511, 513, 8_191, 8_192, 8_193, 16_385, 70_001])
@pytest.mark.parametrize("max_bin", [3, 255, 1_026, 2_051])
def test_cuts_equal_the_host_fit(bb, n, max_bin):
    rng = np.random.Generator(np.random.PCG64(n + max_bin))
    x = rng.normal(0, 1, n).astype(np.float32)
    cols = [x, np.sort(x), np.round(x, 2), np.where(rng.random(n) < 0.4, np.float32(0), x),
            np.full(n, np.nan, np.float32), np.where(rng.random(n) < 0.5, np.nan, x * 1e30),
            rng.integers(-3, 3, n) * np.float32(-0.0), rng.integers(0, 5, n),
            np.where(rng.random(n) < 0.2, np.inf, -x), (x * 1e-40)]
    X = np.stack(cols, 1).astype(np.float32)
    want, woff = bb.fit_cuts(X, max_bin=max_bin)
    got, off = bb.fit_cuts_device(X, max_bin=max_bin)
    assert np.array_equal(off, woff)
    assert np.array_equal(got, want)
    if n >= 2_048:
        # below that the host fit keeps numpy's order of the two zeros, which
        # are one value; the device always puts -0.0 first
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
