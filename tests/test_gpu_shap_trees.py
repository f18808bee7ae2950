"""TreeSHAP's tree form (ensembles of depth at most 8 whose covers add up)
against the numpy path form: depths around each kernel's, features split on
again below (and missing codes), leaves at every level, batches around a row
tile's, the tree splits' and the cluster sizes' edges, wide planes; and the
ensembles that keep the path form: deeper ones, and covers that do not add up.

Both sides are FP64 sums in another order; 1e-9 relative to the largest
contribution leaves room for about 1e-12 of rounding."""

from __future__ import annotations

import numpy as np
import pytest
from test_shap import LEAF, shap_numpy

pytestmark = pytest.mark.gpu


def _tree(bb, rng, n_bins, depth, additive=True, stop=0.2):
    """A random tree: covers add up (unless additive is False)."""
    rec = []

    def node(level, cover):
        i = len(rec)
        rec.append(None)
        if level == depth or cover < 2 or (level > 0 and rng.random() < stop):
            rec[i] = (LEAF, rng.normal(), 0, 0, 0, cover, 0)
            return i
        f = int(rng.integers(0, len(n_bins)))
        s = int(rng.integers(0, n_bins[f] - 1))
        cl = int(rng.integers(1, cover))
        left = node(level + 1, cl)
        right = node(level + 1, cover - cl + (0 if additive else 1))
        rec[i] = (f, 0.0, left, right, int(rng.integers(0, 2)), cover, s)
        return i

    node(0, 1000)
    c = list(zip(*rec))
    return bb.Tree(feature=np.array(c[0], np.uint32), value=np.array(c[1], np.float32),
                   left=np.array(c[2], np.uint32), right=np.array(c[3], np.uint32),
                   default_left=np.array(c[4], np.uint8), gains=np.zeros(len(rec), np.float32),
                   covers=np.array(c[5], np.float32), split_bin=np.array(c[6], np.uint32))


def _plane(bb, rng, n, F, nb):
    n_bins = rng.integers(3, nb + 1, F)
    n_bins[0] = nb
    bins = np.stack([rng.integers(0, k, n) for k in n_bins])
    cuts = np.concatenate([np.append(np.arange(k - 1), np.inf) for k in n_bins])
    off = np.concatenate([[0], np.cumsum(n_bins)]).astype(np.uint32)
    dt = np.uint8 if nb <= 256 else np.uint16
    return bb.Plane.from_bins(bins.astype(dt), cuts.astype(np.float32), off), bins.T, n_bins


def _check(bb, rng, n, F, nb, trees, check=24):
    plane, bins, n_bins = _plane(bb, rng, n, F, nb)
    ens = [t(n_bins) for t in trees]
    got = bb.ShapPlan(plane, ens, 0.5, 0.1).run(plane)
    # the rows at the tiles' ends, and some between
    rows = np.unique(np.concatenate([np.arange(min(n, 3)), np.arange(max(0, n - 3), n),
                                     rng.integers(0, n, check)]))
    want = shap_numpy(bins[rows], n_bins - 1, ens, 0.5, 0.1)
    np.testing.assert_allclose(got[rows], want, rtol=0, atol=1e-9 * np.abs(want).max())
    assert np.array_equal(got, bb.ShapPlan(plane, ens, 0.5, 0.1).run(plane))


@pytest.mark.parametrize("depth", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("n,F", [(1, 2), (33, 9)])
def test_depths_and_repeated_features(bb, depth, n, F):
    rng = np.random.Generator(np.random.PCG64(depth * 100 + n))
    mk = [lambda nb, d=depth, s=s: _tree(bb, rng, nb, d, stop=s) for s in (0.0, 0.3, 0.5)]
    _check(bb, rng, n, F, 255, mk)


@pytest.mark.parametrize("n", [31, 32, 255, 256, 257, 600, 2_400, 4_740, 9_500, 20_011])
def test_batches(bb, n):
    rng = np.random.Generator(np.random.PCG64(n))
    mk = [lambda nb: _tree(bb, rng, nb, 5)] * 40 + [lambda nb: _tree(bb, rng, nb, 0)]
    _check(bb, rng, n, 7, 200, mk, check=6)


@pytest.mark.parametrize("F,nb", [(128, 255), (54, 300), (100, 1_000)])
def test_wide_planes(bb, F, nb):
    rng = np.random.Generator(np.random.PCG64(F))
    mk = [lambda n_bins: _tree(bb, rng, n_bins, 8, stop=0.05)] * 6
    _check(bb, rng, 300, F, nb, mk, check=6)


def test_ensembles_that_keep_the_path_form(bb):
    rng = np.random.Generator(np.random.PCG64(9))
    _check(bb, rng, 50, 12, 255, [lambda nb: _tree(bb, rng, nb, 9, stop=0.0)] * 2, check=4)
    _check(bb, rng, 300, 6, 255, [lambda nb: _tree(bb, rng, nb, 4, additive=False)] * 5)
    _check(bb, rng, 3, 6, 255, [lambda nb: _tree(bb, rng, nb, 0)] * 2)
