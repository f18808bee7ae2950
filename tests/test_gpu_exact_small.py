"""Small exact fits, whose sorts split a tile's features over several CTAs and
whose subtractions split a node's cells, against the oracle's grower: feature
counts around the parts of four, around a tile and two, 8 and 16-bit codes, one
and many chunks."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,F,max_bin", [(500, 3, 255), (500, 4, 255), (2049, 5, 255),
                                         (6000, 28, 255), (6000, 33, 63), (9000, 65, 255),
                                         (6000, 18, 700), (40_000, 28, 255)])
def test_cells_equal_the_serial_sums(bb, n, F, max_bin):
    rng = np.random.default_rng(n + F)
    X = rng.standard_normal((n, F)).astype(np.float32)
    X[rng.random((n, F)) < 0.05] = np.nan
    cuts, off = bb.fit_cuts(X, max_bin=max_bin)
    plane = bb.Plane(X, cuts, off)
    codes = plane.bins()
    g = rng.standard_normal(n).astype(np.float32)
    h = rng.random(n).astype(np.float32)
    got = np.asarray(bb.populate(plane, bb.TrainParams(), g, h)).reshape(-1, 2)
    for f in range(F):
        want = np.zeros((off[f + 1] - off[f], 2), np.float32)
        np.add.at(want[:, 0], codes[f], g)  # float adds in row order
        np.add.at(want[:, 1], codes[f], h)
        assert np.array_equal(got[off[f]:off[f + 1]], want.astype(np.float64))


@pytest.mark.parametrize("F,max_bin", [(3, 255), (28, 255), (40, 63), (9, 2000)])
def test_totals_of_the_children(bb, F, max_bin):
    # leaf values come from the children's totals: -G / (H + l2) of their rows
    n = 7001
    rng = np.random.default_rng(F)
    X = rng.standard_normal((n, F)).astype(np.float32)
    y = (X[:, 0] + X[:, F // 2] ** 2).astype(np.float32)
    cuts, off = bb.fit_cuts(X, max_bin=max_bin)
    plane = bb.Plane(X, cuts, off)
    g, h = -y, np.ones(n, np.float32)
    p = bb.TrainParams(max_depth=5)
    tree, values, ids = bb.grow_tree(plane, p, g, h)
    l2 = float(np.float32(p.lambda_l2))
    for leaf in np.unique(ids):
        rows = ids == leaf
        want = -g[rows].astype(np.float64).sum() / (rows.sum() + l2)
        # float cells: each of up to n adds rounds at 2^-24 of the running sum
        bound = 2.0 ** -24 * n * np.abs(g).max() / (rows.sum() + l2) + 1e-6
        assert abs(tree.value[leaf] - want) <= bound
