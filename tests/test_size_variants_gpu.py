"""The default pass variants by row count, and the per-warp digit match, at the
sizes where the choice changes and on digits that take either match."""
import numpy as np
import pytest

from visondf_b200 import _lib
from test_sort_gpu import dev, host

pytestmark = pytest.mark.gpu


def keys_of(kind, dtype, n, rng):
    info = np.iinfo(dtype)
    if kind == "uniform":
        return rng.integers(info.min, info.max, n, dtype=dtype, endpoint=True)
    if kind == "equal":
        return np.full(n, info.min + 1, dtype)
    if kind == "twelve":  # as many digits as the warp's few-digit bound, and one more in places
        v = rng.integers(info.min, info.max, 13, dtype=dtype, endpoint=True)
        return v[rng.integers(0, 12, n) + (np.arange(n) % 4099 == 0)]
    k = np.sort(rng.integers(info.min, info.max, n, dtype=dtype, endpoint=True))  # runs, then spread
    k[n // 2:] = rng.permutation(k[n // 2:])
    return k


@pytest.mark.parametrize("kind", ["uniform", "equal", "twelve", "half sorted"])
@pytest.mark.parametrize("dtype,n", [(np.int32, 749_999), (np.int32, 750_000), (np.int32, 2_999_999),
                                     (np.int32, 3_000_000), (np.int64, 749_999), (np.int64, 750_000)])
def test_size_edges(ctx, kind, dtype, n):
    rng = np.random.default_rng(n + len(kind))
    k = keys_of(kind, dtype, n, rng)
    strategy = ctx.get_sort_strategy()
    try:
        ctx.set_sort_strategy(_lib.SORT_LSD, 0)
        perm = ctx.argsort([dev(k)])
        ctx.check()
    finally:
        ctx.set_sort_strategy(*strategy)
    assert (host(perm).view(np.uint32) == np.argsort(k, kind="stable")).all()
