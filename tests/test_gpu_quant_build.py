"""The quantised histograms against integer sums in numpy: with integer
gradients whose largest is the quantisation range the codes are the gradients
themselves, so a populated root's cells and every split's gain in a grown tree
are exact -- row counts around a chunk's 2,048 and a CTA's share, feature counts
around a tile's 32, few and many bins, missing values, row subsets."""

import numpy as np
import pytest

import bonsai_b200 as bb

pytestmark = pytest.mark.gpu


def _data(seed, n, F, max_bin):
    rng = np.random.default_rng(seed)
    nb = rng.integers(2, max_bin + 2, F)
    nb[0] = max_bin + 1
    codes = np.empty((F, n), np.uint8)
    for f in range(F):
        codes[f] = np.minimum(np.abs(rng.standard_normal(n)) * nb[f] / 2, nb[f] - 1)
        codes[f, rng.random(n) < 0.05] = nb[f] - 1
    off = np.concatenate([[0], np.cumsum(nb)]).astype(np.uint32)
    g = rng.integers(-127, 128, n).astype(np.float32)
    h = rng.integers(0, 128, n).astype(np.float32)
    g[0], h[0] = 127, 127
    plane = bb.Plane.from_bins(codes, np.arange(off[-1], dtype=np.float32), off)
    return plane, off, codes.astype(np.int64), g, h


@pytest.mark.parametrize("n,F,max_bin", [(1, 1, 3), (2047, 3, 255), (2048, 31, 255),
                                         (2049, 32, 63), (4097, 33, 255), (20011, 70, 255),
                                         (148 * 4096 + 5, 5, 255)])
@pytest.mark.parametrize("subset", [False, True])
def test_root_cells(n, F, max_bin, subset):
    plane, off, codes, g, h = _data(n + F, n, F, max_bin)
    rows = np.sort(np.random.default_rng(1).choice(n, (n + 1) // 2, replace=False)) if subset \
        else np.arange(n)
    p = bb.TrainParams(hist_mode="int8")
    got = bb.populate(plane, p, g, h, rows.astype(np.uint32) if subset else None)
    got = np.asarray(got, np.float64).reshape(-1, 2)
    for f in range(F):
        w = off[f + 1] - off[f]
        for k, v in ((0, g), (1, h)):
            want = np.bincount(codes[f, rows], weights=v[rows].astype(np.float64), minlength=w)
            assert np.array_equal(got[off[f]:off[f + 1], k], want)


@pytest.mark.parametrize("n,F,depth", [(5000, 6, 6), (70001, 33, 8), (400_003, 4, 7)])
def test_every_split(n, F, depth):
    plane, off, codes, g, h = _data(n, n, F, 255)
    p = bb.TrainParams(hist_mode="int8", max_depth=depth)
    tree = bb.grow_tree(plane, p, g, h)[0]

    def score(G, H):
        return G * G / (H + float(np.float32(p.lambda_l2)))

    todo, seen = [(0, np.arange(n))], 0
    while todo:
        i, rows = todo.pop()
        if tree.feature[i] == 0xFFFFFFFF or tree.left[i] == 0:
            continue
        f = int(tree.feature[i])
        c, last = codes[f, rows], off[f + 1] - off[f] - 1
        left = np.where(c == last, tree.default_left[i] == 1, c <= tree.split_bin[i])
        G, H = g[rows].astype(np.float64), h[rows].astype(np.float64)
        gain = score(G[left].sum(), H[left].sum()) + score(G[~left].sum(), H[~left].sum()) \
            - score(G.sum(), H.sum())
        assert abs(gain - tree.gains[i]) <= 1e-5 * max(1.0, abs(gain))
        assert tree.covers[i] == len(rows)
        todo += [(int(tree.left[i]), rows[left]), (int(tree.right[i]), rows[~left])]
        seen += 1
    assert seen > 20
