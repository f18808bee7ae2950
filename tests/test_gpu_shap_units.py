"""TreeSHAP of small batches of deep trees, whose subtrees go to different warps
(their roots at level 1, 2 or 3 by the number of trees), against the numpy path
form: features split on again above and below a subtree's root, leaves above it,
trees of one leaf, batches around a row tile and the last one that takes units.

Both sides are FP64 sums in another order; 1e-9 relative to the largest
contribution leaves room for about 1e-12 of rounding."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_shap_trees import _check, _tree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 32, 33, 255])
@pytest.mark.parametrize("trees,depth,stop", [
    (1, 8, 0.0), (3, 5, 0.0), (30, 8, 0.2), (40, 6, 0.3),  # level 3 (2 up to depth 6)
    (500, 7, 0.5),                                          # level 2
    (1_000, 7, 0.6), (1_300, 6, 0.6),                       # level 1
])
@pytest.mark.parametrize("F,nb", [(2, 255), (20, 300)])
def test_units(bb, n, trees, depth, stop, F, nb):
    rng = np.random.Generator(np.random.PCG64(n + trees + F))
    mk = [lambda n_bins: _tree(bb, rng, n_bins, depth, stop=0.0)]
    mk += [lambda n_bins: _tree(bb, rng, n_bins, depth, stop=stop)] * (trees - 1)
    mk += [lambda n_bins: _tree(bb, rng, n_bins, 0), lambda n_bins: _tree(bb, rng, n_bins, 1)]
    _check(bb, rng, n, F, nb, mk, check=2)


def test_many_features(bb):
    rng = np.random.Generator(np.random.PCG64(5))
    mk = [lambda n_bins: _tree(bb, rng, n_bins, 8, stop=0.1)] * 12
    for n in (1, 64):
        _check(bb, rng, n, 128, 255, mk, check=2)
