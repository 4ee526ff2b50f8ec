"""The group-by of few distinct keys without a sort (calls that ask only for
the group table) against the CPU oracle: group counts at the edges of the
accumulator layouts, every key and value type, orders, keys the sample of
rows misses, and the hand-over to the sorted path past 256 values."""
import numpy as np
import pytest
import torch

import oracle_bind as ob
import visondf_b200 as vdf
from gpu_util import dev, host
from test_dict_gpu import pool_of
from visondf_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def actx():
    c = vdf.Context(0)
    c.set_sort_strategy(_lib.SORT_AUTO, 0)  # from two rows on
    yield c
    c.close()


def values(rng, n, dt):
    if np.dtype(dt).kind == "f":
        return rng.standard_normal(n).astype(dt)
    info = np.iinfo(dt)
    return rng.integers(info.min, info.max, n, dtype=dt, endpoint=True)


def check(c, key, vals, order=vdf.ORDER_ASC, taken=None):
    s0 = c.sort_stats()
    gr = c.sort_groupby([dev(key)], [dev(v) for v in vals], agg_cols=list(range(len(vals))), order=order,
                        want_perm=False, want_sorted_keys=False, want_payload=False)
    c.check()
    s1 = c.sort_stats()
    o = ob.groupby([key], vals)
    assert gr.n_groups == o.n_groups
    flip = (lambda a: a[::-1]) if order != vdf.ORDER_ASC else (lambda a: a)
    bits = lambda a: a.view(f"u{a.dtype.itemsize}")  # noqa: E731
    assert (bits(host(gr.keys[0])) == bits(np.ascontiguousarray(flip(o.keys[0])))).all()
    assert (host(gr.count) == flip(o.count)).all()
    for i, (v, a) in enumerate(zip(vals, gr.aggs)):
        assert (host(a.min) == flip(o.min[i])).all() and (host(a.max) == flip(o.max[i])).all()
        if np.dtype(v.dtype).kind == "f":
            # the sums' bar everywhere in this suite: 1e-12 of the rows' magnitudes
            tol = 1e-12 * np.maximum(flip(o.abs[i]), 1e-300)
            assert (np.abs(host(a.sum) - flip(o.sum[i])) <= tol).all()
            assert (np.abs(host(a.mean) - flip(o.sum[i]) / flip(o.count)) <= tol).all()
        else:
            assert (host(a.sum) == flip(o.sum[i])).all()
            assert (host(a.sum_hi) == flip(o.sum_hi[i])).all()
    if taken is not None:
        assert s1["dict_taken"] - s0["dict_taken"] == int(taken)


# copies per warp change at these group counts (two value columns: 32 copies
# up to about 23 groups, then 16, 8, 4, 2)
@pytest.mark.parametrize("d", [1, 2, 15, 16, 23, 24, 40, 90, 180, 255, 256, 257, 3000])
@pytest.mark.parametrize("n", [2, 127, 129, 5000, 300_001])
def test_group_counts(actx, d, n):
    rng = np.random.default_rng(d * 31 + n)
    key = pool_of(rng, d, np.int32)[rng.integers(0, d, n)]
    check(actx, key, [values(rng, n, np.float64), values(rng, n, np.int64)],
          taken=np.unique(key).size <= 256)


@pytest.mark.parametrize("kdt", [np.int32, np.int64, np.uint32, np.uint64, np.float64, np.float32])
@pytest.mark.parametrize("order", [vdf.ORDER_ASC, vdf.ORDER_DESC_STABLE, vdf.ORDER_DESC_REVERSE])
def test_types_and_orders(actx, kdt, order):
    rng = np.random.default_rng(order + np.dtype(kdt).itemsize)
    n = 40_001
    pool = pool_of(rng, 37, kdt)
    if np.dtype(kdt).kind == "f":
        pool = pool[2:]  # the oracle compares groups by value: one zero only
    key = pool[rng.integers(0, pool.size, n)]
    check(actx, key, [values(rng, n, dt) for dt in (np.int32, np.uint64, np.float32, np.uint32)], order, True)
    check(actx, key, [values(rng, n, np.float64)], order, True)
    check(actx, key, [], order, True)
    check(actx, key, [values(rng, n, dt) for dt in (np.float64, np.float64, np.int64)], order, True)


@pytest.mark.parametrize("d", [3, 200])
def test_hot_keys_and_sorted_rows(actx, d):
    rng = np.random.default_rng(d)
    n = 200_003
    key = pool_of(rng, d, np.int64)[np.minimum(rng.geometric(0.5, n) - 1, d - 1)]
    vals = [values(rng, n, np.float64), rng.integers(-5, 5, n).astype(np.int64)]
    check(actx, key, vals, taken=True)
    check(actx, np.sort(key), vals, taken=True)


def test_keys_the_sample_misses(actx):
    # one row in 32 is sampled by pieces of 128 rows: a value in one row of
    # another piece is found by the second, full collection
    n = 500_000
    key = np.full(n, 5, np.int32)
    key[129] = -7
    key[n - 1] = 9
    vals = [np.arange(n, dtype=np.float64), np.arange(n, dtype=np.int64)]
    check(actx, key, vals, taken=True)
    key[130:130 + 300] = np.arange(1000, 1300)  # ... which may also find too many
    check(actx, key, vals, taken=False)


def test_infinities_and_nan(actx):
    n = 10_000
    key = (np.arange(n) % 5).astype(np.int32)
    key[17] = 100  # a group of one row
    v = np.linspace(-1, 1, n)
    v[17] = np.inf
    v[key == 1] = np.nan
    v[22] = np.nan  # one NaN in group 2
    k, x = dev(key), dev(v)
    kw = dict(want_perm=False, want_sorted_keys=False, want_payload=False)
    got = actx.sort_groupby([k], [x], agg_cols=[0], **kw)
    exp = actx.sort_groupby([k], [x], agg_cols=[0])  # the sorted path
    for f in ("sum", "min", "max", "mean"):
        a, b = getattr(got.aggs[0], f), getattr(exp.aggs[0], f)
        nan = torch.isnan(b)
        assert (torch.isnan(a) == nan).all()
        assert (a[~nan] == b[~nan]).all() if f in ("min", "max") else torch.allclose(a[~nan], b[~nan], rtol=1e-12)
