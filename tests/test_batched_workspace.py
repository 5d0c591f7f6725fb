"""Workspace of the batched targets: as large as their precision matrices, not the
largest ones that a target may have. Host arithmetic only."""
import ctypes

import pytest

from flowmc_gb300 import _lib
from flowmc_gb300 import batched  # noqa: F401  (declares the entry points)

pytestmark = pytest.mark.skipif(not _lib.LIB_PATH.exists(), reason="libflowmc.so not built")


def _size(dims, chains):
    n, nb = len(dims), ctypes.c_size_t()
    _lib.check(_lib.lib().fmc_batched_dense_workspace_size((ctypes.c_int32 * n)(*dims), (ctypes.c_int32 * n)(*chains), n,
                                                           ctypes.byref(nb)))
    return nb.value


def test_small_targets_need_little():
    assert _size([8] * 1000, [20] * 1000) < 2 << 20   # a padded 8 x 32 matrix and a table entry each
    assert _size([256], [32]) >= 4 * 256 * 256


def test_any_dimension_covers_every_one():
    dims, chains = [1, 8, 9, 31, 32, 33, 200, 255, 256], [1, 31, 32, 33, 64, 500, 7, 384, 385]
    nb = ctypes.c_size_t()
    _lib.check(_lib.lib().fmc_batched_workspace_size(len(dims), sum(chains), ctypes.byref(nb)))
    assert _size(dims, chains) <= nb.value
