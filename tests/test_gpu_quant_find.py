"""The quantised find (float approximation, then the FP64 rule for the close
candidates) against the rule on every candidate, recomputed here from the
integer histograms of the root: the chosen feature, bin, direction and gain of
a depth-1 tree, equal bit for bit -- bin counts around a lane's eight bins and a
group's 256, with and without missing rows, empty bins, L1 and L2 zero or
large, child-hessian bounds that cut candidates off, ties between features and
bins, and both cell widths."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rule(cells, off, scale, p):
    """The serial scan: the first strictly larger gain over features, bins and
    directions (missing left first), in FP64."""
    best = (0.0, None)
    q = np.rint(cells / scale).astype(np.int64)

    def score(g, h):
        t = g - p.lambda_l1 if g > p.lambda_l1 else (g + p.lambda_l1 if g < -p.lambda_l1 else 0.0)
        d = h + float(np.float32(p.lambda_l2))
        return (t * t) / d if d > 0.0 else 0.0

    for f in range(len(off) - 1):
        c = q[off[f]:off[f + 1]]
        T, m = c.sum(0), c[-1]
        node = score(float(T[0]) * scale[0], float(T[1]) * scale[1])
        rg, rh = float(T[0] - m[0]) * scale[0], float(T[1] - m[1]) * scale[1]
        mg, mh = float(m[0]) * scale[0], float(m[1]) * scale[1]
        pre = np.cumsum(c, 0)
        for b in range(len(c) - 2):
            lg, lh = float(pre[b, 0]) * scale[0], float(pre[b, 1]) * scale[1]
            for d in range(1 if m[0] == 0 and m[1] == 0 else 2):
                gl, hl = lg + (mg if d == 0 else 0.0), lh + (mh if d == 0 else 0.0)
                gr, hr = (rg - lg) + (mg if d else 0.0), (rh - lh) + (mh if d else 0.0)
                mch = float(np.float32(p.min_child_hess))
                if hl < mch or hr < mch:
                    continue
                gain = (score(gl, hl) + score(gr, hr)) - node
                if gain > best[0] and gain >= float(np.float32(p.min_gain_to_split)):
                    best = (gain, (f, b, d == 0))
    return best


@pytest.mark.parametrize("grower", ["depthwise", "leafwise"])
@pytest.mark.parametrize("nb,n,mode,kw", [
    (3, 50, "int8", {}), (9, 400, "int8", {"lambda_l2": 0.0, "min_child_hess": 0.0}),
    (10, 4_000, "int16", {"lambda_l1": 3.0}), (255, 3_000, "int8", {"min_child_hess": 40.0}),
    (256, 900, "int8", {"lambda_l2": 1e4}), (257, 5_000, "int8", {}),
    (300, 5_000, "int16", {"min_gain_to_split": 0.5}), (700, 2_000, "int8", {"lambda_l1": 0.5}),
])
def test_root_split_is_the_serial_scans(bb, grower, nb, n, mode, kw):
    rng = np.random.Generator(np.random.PCG64(nb * 7 + n))
    F = 11
    cols = [rng.integers(0, nb, n) for _ in range(F)]
    cols[1] = np.where(rng.random(n) < 0.9, nb - 1, cols[1])  # mostly missing
    cols[2] = cols[2] % max(1, nb - 1)                         # no missing
    cols[3] = (cols[3] // 5) * 5 % nb                          # empty bins
    cols[4] = cols[0]                                          # a tie between features
    bins = np.stack(cols).astype(np.uint8 if nb <= 256 else np.uint16)
    cuts = np.concatenate([np.append(np.arange(nb - 1), np.inf)] * F).astype(np.float32)
    off = (np.arange(F + 1) * nb).astype(np.uint32)
    plane = bb.Plane.from_bins(bins, cuts, off)
    g = (rng.normal(0, 1, n) + 0.3 * np.sin(bins[0])).astype(np.float32)
    h = rng.uniform(0.1, 1.0, n).astype(np.float32)
    extra = {"max_leaves": 2} if grower == "leafwise" else {}
    p = bb.TrainParams(hist_mode=mode, seed=5, max_depth=1, min_data_in_leaf=1, grower=grower,
                       **extra, **kw)
    cells = bb.populate(plane, p, g, h)
    qmax = 127.0 if mode == "int8" else 32767.0
    scale = (np.float64(np.abs(g).max()) / qmax, np.float64(h.max()) / qmax)
    gain, want = _rule(cells, off, np.array(scale), p)
    tree, _, _ = bb.grow_tree(plane, p, g, h)
    if want is None:
        assert tree.n_leaves == 1
        return
    got = (int(tree.feature[0]), int(tree.split_bin[0]), bool(tree.default_left[0]))
    assert got == want
    assert tree.gains[0] == np.float32(gain)
