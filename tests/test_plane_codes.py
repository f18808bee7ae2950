"""bb_plane_from_bins refuses a code at or past its feature's bin count, wherever it
lies, before it asks for a device (CPU)."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("n", [1, 63, 257])
@pytest.mark.parametrize("f,at", [(0, 0), (1, -1), (2, 0), (2, -1)])
def test_a_code_past_the_bins_is_refused(dtype, n, f, at):
    from bonsai_b200._lib import lib, ptr
    nb = [3, 200, 17]
    bins = np.zeros((3, n), dtype)
    bins[f, at] = nb[f]
    off = np.concatenate([[0], np.cumsum(nb)]).astype(np.uint32)
    cuts = np.arange(off[-1], dtype=np.float32)
    plane = C.c_void_p()
    rc = lib().bb_plane_from_bins(ptr(bins), int(dtype is np.uint8), n, 3, ptr(cuts), ptr(off),
                                  C.byref(plane))
    assert rc != 0 and plane.value is None
    assert "not below its bin count" in lib().bb_last_error().decode()
