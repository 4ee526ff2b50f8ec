"""The counting pass of the shared-memory finish (k_msd_local) where its bins
are laid out a second time over the keys' own range: chunks of one bucket
whose rows sit in a small part of it."""
import numpy as np
import pytest

import visondf_b200 as vdf
from test_msd_gpu import run_sort
from visondf_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.int64, np.uint64])
@pytest.mark.parametrize("rows", [65, 1000, 2047])
@pytest.mark.parametrize("spread", [1 << 6, 1 << 20, 1 << 40])
@pytest.mark.parametrize("two", [False, True])
def test_clustered_buckets(dt, rows, spread, two):
    rng = np.random.default_rng(rows + spread % 1009)
    n = 400_000  # two top digits: the buckets share their top 16 bits
    tops = rng.choice(1 << 16, size=n // rows + 1, replace=False).astype(np.uint64)
    top = np.repeat(tops, rows)[:n]
    k = (top << np.uint64(48)) | (rng.integers(0, spread, n).astype(np.uint64) + np.uint64(12345))
    k = k[rng.permutation(n)].view(dt)
    keys = [k, rng.integers(-50, 50, n).astype(np.int32)] if two else [k]
    c = vdf.Context(0)
    try:
        c.set_sort_strategy(_lib.SORT_MSD, 0)
        for order in (vdf.ORDER_ASC, vdf.ORDER_DESC_STABLE, vdf.ORDER_DESC_REVERSE):
            used, fell = run_sort(c, keys, order)
            assert used == 1
            if not two:
                assert fell == 0
    finally:
        c.close()
