"""Bin application and the row mirror over the forms they take (a thread per
value for small batches and very long cut tables; row tiles with padded or whole
tables), against the oracle's transform: features around a tile's and a vector's
edges, rows around a tile's and the forms' border, tables of 2 to 1,500 cuts,
values on the cuts, beyond them, infinite and missing."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(rng, n, F, nb):
    """Cut tables of nb - 3 .. nb cuts (the last two FLT_MAX and inf), and values."""
    cuts, off = [], [0]
    for f in range(F):
        k = max(2, nb - int(rng.integers(0, 4)))
        c = np.unique(rng.normal(0, 1, 4 * k).astype(np.float32))[:k - 2]
        c = np.concatenate([c, [np.finfo(np.float32).max, np.inf]]).astype(np.float32)
        cuts.append(c)
        off.append(off[-1] + len(c))
    X = rng.normal(0, 1.2, (n, F)).astype(np.float32)
    for f in range(F):  # values on the cuts
        at = rng.integers(0, n, n // 4 + 1)
        X[at, f] = rng.choice(cuts[f][:-1], len(at))
    X[rng.random((n, F)) < 0.03] = np.nan
    X[rng.random((n, F)) < 0.01] = np.inf
    X[rng.random((n, F)) < 0.01] = -np.inf
    return X, np.concatenate(cuts), np.array(off, np.uint32)


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("n,F,nb", [
    (1, 1, 255), (255, 3, 2), (256, 28, 255), (257, 33, 256), (16_384, 32, 100),
    (16_385, 28, 255), (16_641, 13, 40), (20_000, 37, 256), (17_000, 65, 9),
    (16_400, 33, 300), (16_399, 5, 1_500), (16_500, 34, 1_300),
])
def test_codes_and_scores(bb, orc, n, F, nb, device):
    rng = np.random.Generator(np.random.PCG64(n + F + nb))
    X, cuts, off = _matrix(rng, n, F, nb)
    want = orc.transform(X, cuts, off)
    if device:
        import torch
        plane = bb.Plane.from_device(torch.as_tensor(X, device="cuda"), cuts, off)
    else:
        plane = bb.Plane(X, cuts, off)
    assert np.array_equal(plane.bins(), want)
    # the mirror: every feature a one-split tree's, scored from the mirror's codes
    n_bins = np.diff(off)
    trees = []
    for f in range(F):
        s = int(rng.integers(0, n_bins[f] - 1))
        trees.append(bb.Tree(feature=np.array([f, bb.LEAF, bb.LEAF], np.uint32),
                             value=np.array([0, 1, 2 + f], np.float32),
                             left=np.array([1, 0, 0], np.uint32),
                             right=np.array([2, 0, 0], np.uint32),
                             default_left=np.array([f & 1, 0, 0], np.uint8),
                             gains=np.zeros(3, np.float32), covers=np.zeros(3, np.float32),
                             split_bin=np.array([s, 0, 0], np.uint32)))
    got = bb.predict(plane, trees, 0.0, 1.0)
    score = np.zeros(n, np.float32)
    for f, t in enumerate(trees):
        c = want[f]
        left = np.where(c == n_bins[f] - 1, f & 1, c <= t.split_bin[0])
        score = score + np.where(left, np.float32(1), np.float32(2 + f)).astype(np.float32)
    assert np.array_equal(got, score)


def test_tables_past_a_tiles_memory_are_refused(bb):
    F, nb = 32, 1_700
    cuts = np.concatenate([np.append(np.arange(nb - 1), np.inf)] * F).astype(np.float32)
    with pytest.raises(bb.ConfigError):
        bb.Plane(np.zeros((10, F), np.float32), cuts, (np.arange(F + 1) * nb).astype(np.uint32))
