"""The MSD plan's optional third top digit (8-byte keys whose top digits are
clustered, as those of doubles are): taken, not taken and failing, in every
order, with a second key and through a row view."""
import ctypes as C

import numpy as np
import pytest

import visondf_b200 as vdf
from test_msd_gpu import run_sort
from visondf_b200 import datagen

pytestmark = pytest.mark.gpu

ORDERS = [vdf.ORDER_ASC, vdf.ORDER_DESC_STABLE, vdf.ORDER_DESC_REVERSE]


def keys_of(kind, n, rng):
    if kind == "normal":
        return rng.standard_normal(n)
    if kind == "lognormal":
        return np.exp(rng.standard_normal(n))
    if kind == "uniform01":
        return rng.random(n)
    if kind == "clustered":  # 40 top 16-bit values, the rest uniform
        top = rng.choice(1 << 16, 40, replace=False).astype(np.uint64)[rng.integers(0, 40, n)]
        return (top << np.uint64(48)) | rng.integers(0, 1 << 48, n).astype(np.uint64)
    if kind == "one hot bucket":  # too many rows under one 24-bit prefix
        k = rng.standard_normal(n)
        k[: n // 20] = 1.0 + rng.random(n // 20) * 1e-9
        return k[rng.permutation(n)]
    return datagen.keys_for("uniform", np.int64, n, rng)


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("kind", ["normal", "lognormal", "uniform01", "clustered", "one hot bucket", "uniform"])
@pytest.mark.parametrize("n", [1 << 20, 1_500_001])
def test_clustered_top_digits(ctx, kind, order, n):
    rng = np.random.default_rng(n + len(kind))
    k = keys_of(kind, n, rng)
    used, fell = run_sort(ctx, [k], order)
    assert used == 1
    assert fell == int(kind == "one hot bucket")


@pytest.mark.parametrize("kind", ["normal", "clustered"])
def test_second_key_and_row_view(ctx, kind):
    from test_groupby_gpu import _host_args
    rng = np.random.default_rng(len(kind))
    n = 1_200_003
    k = keys_of(kind, n, rng)
    k[1::2] = k[::2][: n // 2]  # ties
    assert run_sort(ctx, [k, rng.integers(-9, 9, n).astype(np.int32)]) == (1, 0)
    view = rng.permutation(n).astype(np.uint32)
    a, out = _host_args([k], [], [], n, perm_in=view)
    a.groupby = 0
    assert vdf.lib.vdf_sort_groupby_host(ctx.handle, C.byref(a), None) == 0
    assert (out["perm"] == view[np.argsort(k[view], kind="stable")]).all()
