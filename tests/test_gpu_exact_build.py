"""The exact form's histogram build (sort and chain kernels) against the oracle's
serial fill, bit for bit, at the sizes where it can go wrong: rows around a
warp's, a chunk's and a ring's edges, bin counts around a ballot width's and a
bin group's, codes spread evenly, nearly all in one bin, sorted, and constant."""

from __future__ import annotations

import numpy as np
import pytest
from oracle import orc_fill

pytestmark = pytest.mark.gpu


def _plane(bb, n, nb, F, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    cols = []
    for f in range(F):
        c = rng.integers(0, nb, n)
        if f % 5 == 1:
            c = np.where(rng.random(n) < 0.95, nb - 1, c)  # as missing values are
        elif f % 5 == 2:
            c = np.sort(c)
        elif f % 5 == 3:
            c = np.full(n, f % nb)
        cols.append(c)
    bins = np.stack(cols).astype(np.uint8 if nb <= 256 else np.uint16)
    cuts = np.concatenate([np.append(np.arange(nb - 1), np.inf)] * F).astype(np.float32)
    off = (np.arange(F + 1) * nb).astype(np.uint32)
    g = rng.normal(0.0, 1.0, n).astype(np.float32)
    g[rng.random(n) < 0.1] = -0.0
    h = rng.uniform(0.0, 0.25, n).astype(np.float32)
    return bb.Plane.from_bins(bins, cuts, off), bins, np.diff(off), g, h


@pytest.mark.parametrize("n,nb,F", [
    (1, 255, 3), (31, 3, 33), (33, 16, 5), (513, 17, 7), (2047, 255, 28), (2048, 256, 28),
    (2049, 256, 32), (4097, 255, 35), (12_289, 31, 64), (50_001, 255, 9), (70_000, 2, 5),
    (2049, 257, 5), (30_001, 300, 17), (9_000, 3_000, 6), (9_000, 3_679, 6),
])
def test_cells_are_the_serial_fill(bb, orc, n, nb, F):
    plane, bins, n_bins, g, h = _plane(bb, n, nb, F, n + nb)
    got = bb.populate(plane, bb.TrainParams(), g, h)
    want = orc_fill(orc, bins, n_bins, g, h)
    assert np.array_equal(got.astype(np.float32), want)
    # a row sample, and a feature selection that leaves tiles out
    rows = np.flatnonzero(np.random.Generator(np.random.PCG64(n)).random(n) < 0.5)
    sel = list(range(0, F, 2))
    if len(rows):
        got = bb.populate(plane, bb.TrainParams(selected=sel), g, h, rows=rows)
        want = orc_fill(orc, bins, n_bins, g, h, rows=rows, selected=sel)
        assert np.array_equal(got.astype(np.float32), want)


def test_bins_past_the_exact_forms_ceiling_are_refused(bb):
    plane, _, _, g, h = _plane(bb, 100, 3_680, 2, 1)
    with pytest.raises(bb.ConfigError):
        bb.populate(plane, bb.TrainParams(), g, h)
