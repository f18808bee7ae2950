"""Boosters, plans and planes of different bin counts side by side: a kernel's
shared-memory limit is one per process, so the one made last must not lower it
under the ones made before."""

import numpy as np
import pytest

import bonsai_b200 as bb

pytestmark = pytest.mark.gpu


def _data(seed, n, max_bin):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, 6)).astype(np.float32)
    y = (X[:, 0] * 2 + np.sin(X[:, 1] * 3)).astype(np.float32)
    cuts, off = bb.fit_cuts(X, max_bin=max_bin)
    return bb.Plane(X, cuts, off), y


def _trees(b):
    return [(t.feature, t.value, t.covers) for t in b.trees()]


@pytest.mark.parametrize("grower", ["depthwise", "levelwise", "leafwise"])
@pytest.mark.parametrize("hist", ["exact", "int8"])
@pytest.mark.parametrize("max_bin", [255, 1000])
def test_a_smaller_booster_between(grower, hist, max_bin):
    big, yb = _data(0, 6000, max_bin)
    small, ys = _data(1, 40, 3)
    p = bb.TrainParams(grower=grower, hist_mode=hist, max_depth=4, max_leaves=16)
    alone = bb.Booster(big, yb, p, max_trees=3)
    alone.update(3)
    want = _trees(alone)
    alone.close()
    first = bb.Booster(big, yb, p, max_trees=3)
    second = bb.Booster(small, ys, p, max_trees=3)
    second.update(1)
    first.update(3)
    for s, t in zip(want, _trees(first)):
        assert all(np.array_equal(x, y) for x, y in zip(s, t))
    first.close()
    second.close()
