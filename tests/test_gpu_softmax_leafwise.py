"""Softmax fits with leafwise trees: every class's tree is grown from that class's
gradients and, with a feature fraction, from that class's feature sample, below
the root too. A leafwise fit with max_depth d and 2^d leaves grows until the
depth cap stops it, so its trees hold the splits of the depthwise fit of the
same depth (whatever the order of the nodes), and its training scores are the
same."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LEAF = 0xFFFFFFFF


def _fit(bb, plane, y, grower, mode, fraction, rounds):
    p = bb.TrainParams(objective="softmax", n_classes=4, grower=grower, max_depth=4,
                       max_leaves=16, hist_mode=mode, seed=3, learning_rate=0.3,
                       feature_fraction=fraction, feature_seed=11)
    b = bb.Booster(plane, y, p, max_trees=rounds)
    b.update(rounds)
    trees, scores = b.trees(), b.scores()
    b.close()
    return trees, scores


def _splits(t):
    inner = t.feature != LEAF
    return sorted(zip(t.feature[inner].tolist(), t.split_bin[inner].tolist(),
                      t.default_left[inner].tolist(), t.covers[inner].tolist(),
                      t.gains[inner].tolist()))


@pytest.mark.parametrize("mode", ["exact", "int8", "int16"])
@pytest.mark.parametrize("fraction", [1.0, 0.5])
@pytest.mark.parametrize("max_bin", [255, 300])
def test_every_class_grows_its_own_tree(bb, mode, fraction, max_bin):
    rng = np.random.Generator(np.random.PCG64(21))
    n, F, K = 6_000, 40, 4
    X = rng.standard_normal((n, F)).astype(np.float32)
    X[rng.random((n, F)) < 0.05] = np.nan
    y = np.argmax(np.nan_to_num(X[:, :K]) + 0.5 * rng.standard_normal((n, K)), axis=1)
    cuts, off = bb.fit_cuts(X, max_bin=max_bin)
    plane = bb.Plane(X, cuts, off)
    y = y.astype(np.float32)
    # the exact form's scores are equal bit for bit over rounds; the quantised
    # leaves are renewed by sums in another order, so only the first round's
    # splits compare
    rounds = 3 if mode == "exact" else 1
    mine, scores = _fit(bb, plane, y, "leafwise", mode, fraction, rounds)
    want, ref = _fit(bb, plane, y, "depthwise", mode, fraction, rounds)
    for t in range(rounds * K):
        assert _splits(mine[t]) == _splits(want[t]), t
    if mode == "exact":
        assert np.array_equal(scores.view(np.uint32), ref.view(np.uint32))
    else:
        np.testing.assert_allclose(scores, ref, rtol=1e-6, atol=1e-6)
