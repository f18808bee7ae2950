"""The nodes that a demoted split leaves in a quantised tree: unreachable, of
cover 0 and of no rows, so of value zero whatever trees this one's or another
booster's memory held before."""

from __future__ import annotations

import numpy as np
import pytest
from conftest import TREE_FIELDS

pytestmark = pytest.mark.gpu


def _fit(bb, plane, y, **params):
    p = bb.TrainParams(max_depth=5, min_child_hess=0.0, learning_rate=0.2, **params)
    b = bb.Booster(plane, y.astype(np.float32), p, max_trees=6)
    b.update(6)
    trees = b.trees()
    b.close()
    return trees


@pytest.mark.parametrize("mode", ["int8", "int16"])
def test_demoted_children_hold_zero_after_any_other_fit(bb, mode):
    """A monotone direction against the data's and a min_data_in_leaf of 0.4 rows
    leave splits of gain by rounding alone, with an empty side; fits with wide
    bounds on every node come between the two that have to agree."""
    demoted = 0
    for seed in (227, 234, 247, 257):
        g = np.random.default_rng(seed)
        n, nf = int(g.integers(100, 400)), int(g.integers(1, 4))
        X = g.standard_normal((n, nf)).astype(np.float32)
        X[g.random((n, nf)) < 0.1] = np.nan
        cuts, off = bb.fit_cuts(X, max_bin=63)
        plane = bb.Plane(X, cuts, off)
        mono = [int(v) for v in g.choice([-1, 1], nf)]
        Z = np.nan_to_num(X)
        y = sum(-mono[k] * Z[:, k] for k in range(nf)) + 0.1 * g.standard_normal(n)
        common = {"hist_mode": mode, "monotone": mono}
        rare = {"min_data_in_leaf": int(0.4 * n), "lambda_l2": 10.0} | common
        first = _fit(bb, plane, y, **rare)
        demoted += sum(int((t.covers == 0).sum()) for t in first)
        for s in range(3):
            _fit(bb, plane, 100 * Z[:, s % nf] + 50 * g.standard_normal(n),
                 min_data_in_leaf=1, lambda_l2=0.1, **common)
        again = _fit(bb, plane, y, **rare)
        for a, b in zip(first, again):
            for t in (a, b):
                np.testing.assert_array_equal(t.value[t.covers == 0], 0.0)
            for k in TREE_FIELDS:
                assert getattr(a, k).tobytes() == getattr(b, k).tobytes(), k
        plane.close()
    assert demoted > 0
