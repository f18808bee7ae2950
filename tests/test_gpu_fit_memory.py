"""A fit's arrays come from one pool per device: fits that share it must not
meet in it, and the last plane to go gives it back."""

import os
import pathlib
import subprocess
import sys
import threading

import numpy as np
import pytest

import bonsai_b200 as bb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
HERE = pathlib.Path(__file__).resolve().parent


def _data(seed, n):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, 6)).astype(np.float32)
    y = (X[:, 0] * 2 + np.sin(X[:, 1] * 3)).astype(np.float32)
    cuts, off = bb.fit_cuts(X, max_bin=63)
    return bb.Plane(X, cuts, off), y


def _fit(plane, y, hist):
    p = bb.TrainParams(max_depth=5, hist_mode=hist)
    b = bb.Booster(plane, y, p, max_trees=6)
    b.update(6)
    trees, scores = b.trees(), b.scores()
    b.close()
    return [(t.feature, t.value, t.covers) for t in trees], scores


def _same(a, b):
    assert all(np.array_equal(x, y) for s, t in zip(a[0], b[0]) for x, y in zip(s, t))
    assert np.array_equal(a[1], b[1])


@pytest.mark.parametrize("hist", ["exact", "int8"])
def test_fits_in_threads_share_the_pool(hist):
    sizes = [1, 257, 4099, 20011]
    data = [_data(s, n) for s, n in enumerate(sizes)]
    alone = [_fit(p, y, hist) for p, y in data]
    got = [[None] * 4 for _ in sizes]

    def work(k):
        for r in range(4):
            got[k][r] = _fit(*data[k], hist)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(len(sizes)):
        for r in range(4):
            _same(got[k][r], alone[k])
    for p, _ in data:
        p.close()


def _bounds():
    plane, y = _data(0, 4099)
    _fit(plane, y, "int8")
    plane.close()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    big, yb = _data(1, 600_000)
    plane, y = _data(2, 4099)
    fits = [bb.Booster(big, yb, bb.TrainParams(max_depth=8), max_trees=4) for _ in range(24)]
    for b in fits:
        b.update(1)
    for b in fits:
        b.close()
    first = _fit(plane, y, "int8")
    big.close()
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= (1 << 30) + (64 << 20)
    _same(_fit(plane, y, "int8"), first)
    plane.close()
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= 64 << 20


def test_the_pool_is_bounded_and_given_back():
    # a process of its own: planes that other tests left open hold the pool
    code = f"import sys; sys.path.insert(0, {str(HERE)!r}); " \
           "import test_gpu_fit_memory as t; t._bounds()"
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, cwd=HERE.parent,
                   env={**os.environ, "PYTHONPATH": str(HERE.parent)})
