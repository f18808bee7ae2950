"""Leafwise trees whose root does not split, first in their grower and in
memory that other fits have written: the loop's body runs once without a pop and
must leave everything as it is."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(bb, seed, n, nf):
    g = np.random.default_rng(seed)
    X = g.standard_normal((n, nf)).astype(np.float32)
    cuts, off = bb.fit_cuts(X, max_bin=255)
    return X, bb.Plane(X, cuts, off)


def _wide_fit(bb, X, plane, mode):
    p = bb.TrainParams(grower="leafwise", hist_mode=mode, max_depth=8, max_leaves=100,
                       min_data_in_leaf=5)
    b = bb.Booster(plane, (1e3 * X[:, 0] + X[:, 1]).astype(np.float32), p, max_trees=2)
    b.update(2)
    out = [t.value.tobytes() + t.left.tobytes() for t in b.trees()]
    b.close()
    return out


@pytest.mark.parametrize("mode", ["exact", "int8", "int16"])
@pytest.mark.parametrize("stop", [{"min_data_in_leaf": 100}, {"max_leaves": 1}, {"max_depth": 0},
                                  {"min_gain_to_split": 1e30}])
def test_a_lone_root_in_used_memory(bb, mode, stop):
    X, holder = _data(bb, 1, 30_000, 40)  # holds the memory that its fits give back
    before = _wide_fit(bb, X, holder, mode)
    for n, nf in ((11, 3), (150, 1), (197, 33)):
        _, plane = _data(bb, n, n, nf)
        g = np.random.default_rng(n + 1)
        grad = g.standard_normal(n).astype(np.float32)
        hess = g.uniform(0.5, 1.0, n).astype(np.float32)
        kw = {"max_depth": 4, "max_leaves": 16, "hist_mode": mode, "lambda_l2": 1.0} | stop
        t, v, leaf = bb.grow_tree(plane, bb.TrainParams(grower="leafwise", **kw), grad, hess)
        assert len(t.feature) == 1 and t.covers[0] == n
        want = -grad.astype(np.float64).sum() / (hess.astype(np.float64).sum() + 1.0)
        # float sums of a bin's rows, each within n roundings
        np.testing.assert_allclose(v, want, rtol=0, atol=n * 6e-8 * np.abs(grad).sum())
        assert not leaf.any()
        plane.close()
    assert _wide_fit(bb, X, holder, mode) == before
    holder.close()
