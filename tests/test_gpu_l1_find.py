"""The quantised find where every candidate's gradient sum lies a few parts in ten
million above lambda_l1: what is left after the threshold is smaller than the
sums' rounding to float, and the split taken has to be the FP64 rule's all the
same. Gradients and hessians are whole numbers with the code range as their
maximum, so the scales are 1 and the integer sums are the sums."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
L1 = float(1 << 25)


def _close_rows(qmax):
    """(bin, g, h) rows of a column: bin 0 holds a sum of L1 exactly, bin 1 adds 6
    and bin 2 adds 3 more and enough hessian that (L1 + 6) beats (L1 + 9) if both
    are rounded to a multiple of 4 first; bin 3 takes the total back under L1."""
    whole = int(L1) // qmax
    rest = int(L1) - whole * qmax
    rows = [(0, qmax, 1)] * whole + [(0, rest, 1)]
    rows += [(1, 6, 1)]
    rows += [(2, 1, min(qmax, whole // 16))] * 3
    rows += [(3, -109, qmax)]
    return np.array(rows, np.int64)


def _plane(bb, cols, nb):
    bins = np.stack(cols).astype(np.uint8)
    F = len(cols)
    cuts = np.concatenate([np.append(np.arange(nb - 1), np.inf)] * F).astype(np.float32)
    return bb.Plane.from_bins(bins, cuts, (np.arange(F + 1) * nb).astype(np.uint32))


def _params(bb, grower, mode, depth):
    extra = {"max_leaves": 1 << depth} if grower == "leafwise" else {}
    return bb.TrainParams(hist_mode=mode, seed=5, max_depth=depth, min_data_in_leaf=1,
                          grower=grower, lambda_l1=L1, lambda_l2=0.0, min_child_hess=0.0, **extra)


@pytest.mark.parametrize("mode,qmax", [("int8", 127), ("int16", 32767)])
@pytest.mark.parametrize("grower", ["depthwise", "leafwise"])
def test_the_root_takes_the_larger_gain(bb, grower, mode, qmax):
    r = _close_rows(qmax)
    order = np.random.Generator(np.random.PCG64(1)).permutation(len(r))
    b, g, h = r[order].T
    plane = _plane(bb, [b], 5)
    tree, _, _ = bb.grow_tree(plane, _params(bb, grower, mode, 1), g.astype(np.float32),
                              h.astype(np.float32))
    h0 = float(r[r[:, 0] <= 1][:, 2].sum())
    h1 = float(r[r[:, 0] <= 2][:, 2].sum())
    assert 36.0 / h0 < 81.0 / h1  # the rule's own gains of bins 1 and 2
    assert (int(tree.feature[0]), int(tree.split_bin[0])) == (0, 2)
    assert tree.gains[0] == np.float32(81.0 / h1)


@pytest.mark.parametrize("mode,qmax", [("int8", 127), ("int16", 32767)])
@pytest.mark.parametrize("grower", ["depthwise", "leafwise"])
def test_a_child_takes_the_larger_gain(bb, grower, mode, qmax):
    """Column 0 parts those rows from others whose sum is -4 L1; the child that
    holds them splits on column 1 at bin 2."""
    r = _close_rows(qmax)
    m = 4 * int(L1) // qmax
    far = np.array([(3, -qmax, 1)] * m, np.int64)
    rows = np.concatenate([r, far])
    side = np.concatenate([np.zeros(len(r), np.int64), np.ones(m, np.int64)])
    order = np.random.Generator(np.random.PCG64(2)).permutation(len(rows))
    b, g, h = rows[order].T
    plane = _plane(bb, [side[order], b], 5)
    tree, _, _ = bb.grow_tree(plane, _params(bb, grower, mode, 2), g.astype(np.float32),
                              h.astype(np.float32))
    h1 = float(r[r[:, 0] <= 2][:, 2].sum())
    assert (int(tree.feature[0]), int(tree.split_bin[0])) == (0, 0)
    child = int(tree.left[0])
    assert (int(tree.feature[child]), int(tree.split_bin[child])) == (1, 2)
    assert tree.gains[child] == np.float32(81.0 / h1)
