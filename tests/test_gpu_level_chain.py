"""The quantised level chain (subtraction, split choice and plan in the find's
blocks, trees opened beside their quantisation) against the general path: a
booster's first tree, which takes it, and grow_tree's, which does not, have the
same splits, children and covers -- feature counts around the find's eight
warps, one and many chunks, depths to the last level, missing values, demoted
and empty frontiers, monotone and interaction constraints, 8 and 16-bit codes."""

import numpy as np
import pytest

import bonsai_b200 as bb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,F,max_bin,kw", [
    (1, 1, 15, {}),
    (39, 3, 15, {}),
    (40, 3, 15, {"max_depth": 1}),
    (200, 7, 3, {"max_depth": 8, "min_data_in_leaf": 1}),
    (4096, 8, 255, {"max_depth": 8}),
    (4097, 9, 255, {"max_depth": 5, "min_child_hess": 50.0}),
    (20011, 33, 63, {"max_depth": 8, "min_data_in_leaf": 1}),
    (20011, 28, 255, {"monotone": [1, -1, 0, 1]}),
    (20011, 12, 255, {"interaction_constraints": [[0, 1, 2], [2, 3], [5, 6, 7, 8]], "max_depth": 7}),
    (20011, 12, 700, {"max_depth": 6}),
    (60000, 65, 31, {"max_depth": 7, "lambda_l1": 2.0}),
    (5000, 4, 63, {"min_gain_to_split": 1e9}),
    (5000, 4, 63, {"max_depth": 0}),
])
@pytest.mark.parametrize("mode", ["int8", "int16"])
@pytest.mark.parametrize("grower", ["depthwise", "levelwise"])
def test_chain_equals_general(n, F, max_bin, kw, mode, grower):
    if grower == "levelwise" and ("monotone" in kw or "interaction_constraints" in kw):
        pytest.skip("refused by the levelwise grower")
    rng = np.random.default_rng(n + F)
    X = rng.standard_normal((n, F)).astype(np.float32)
    X[:, F // 2] = np.round(X[:, F // 2])
    X[rng.random((n, F)) < 0.1] = np.nan
    y = (np.nan_to_num(X[:, 0]) * 2 + np.sin(3 * np.nan_to_num(X[:, F - 1]))).astype(np.float32)
    cuts, off = bb.fit_cuts(X, max_bin=max_bin)
    plane = bb.Plane(X, cuts, off)
    p = bb.TrainParams(hist_mode=mode, grower=grower, **kw)
    b = bb.Booster(plane, y, p, max_trees=2)
    g = (np.full(n, np.float32(b.init_score)) - y).astype(np.float32)
    b.update(2)
    got = b.trees()[0]
    b.close()
    want = bb.grow_tree(plane, p, g, np.ones(n, np.float32))[0]
    for k in ("feature", "split_bin", "left", "right", "default_left", "covers", "gains"):
        assert np.array_equal(getattr(got, k), getattr(want, k)), k
    assert (got.depth, got.n_leaves) == (want.depth, want.n_leaves)
    plane.close()
