"""Small frames sorted, gathered and grouped by one CTA (vdf_small.cu) against
the CPU oracle: sizes at the edges of its rows per thread and its limit, key
and value types, orders, one to three keys, group shapes, a row view, and
outputs over the inputs."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle_bind as ob
import visondf_b200 as vdf
from gpu_util import bits_equal, dev, host
from test_dictagg_gpu import values
from visondf_b200 import datagen

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 1000, 1023, 1024, 1025, 2049, 4095, 4096, 4097]
ORDERS = [vdf.ORDER_ASC, vdf.ORDER_DESC_STABLE, vdf.ORDER_DESC_REVERSE]


def check(ctx, keys, vals, order=vdf.ORDER_ASC):
    l0 = ctx.kernel_launches
    gr = ctx.sort_groupby([dev(k) for k in keys], [dev(v) for v in vals], agg_cols=list(range(min(4, len(vals)))),
                          order=order, want_row_group=True, want_group_start=True)
    ctx.check()
    n = keys[0].size
    assert (ctx.kernel_launches - l0 == 1) == (n <= 4096)
    perm = ob.argsort(keys, order)
    assert (host(gr.perm).view(np.uint32) == perm).all()
    for k, s in zip(keys, gr.sorted_keys):
        assert bits_equal(host(s), k[perm])
    for v, p in zip(vals, gr.payload):
        assert bits_equal(host(p), v[perm])
    sk = [k[perm].view(f"u{k.itemsize}") for k in keys]
    head = np.ones(n, bool)
    if n > 1:
        head[1:] = np.any([s[1:] != s[:-1] for s in sk], axis=0)
    start = np.flatnonzero(head)
    assert gr.n_groups == start.size
    assert (host(gr.group_start) == start).all()
    assert (host(gr.row_group) == np.cumsum(head) - 1).all()
    assert (host(gr.count) == np.diff(np.append(start, n))).all()
    for k, g in zip(keys, gr.keys):
        assert bits_equal(host(g), k[perm][start])
    for v, a in zip(vals, gr.aggs):
        sv = v[perm]
        assert (host(a.min) == np.minimum.reduceat(sv, start)).all()
        assert (host(a.max) == np.maximum.reduceat(sv, start)).all()
        if v.dtype.kind == "f":
            exact = np.add.reduceat(sv.astype(np.longdouble), start)
            mags = np.add.reduceat(np.abs(sv.astype(np.longdouble)), start)
            assert (np.abs(host(a.sum) - exact) <= 1e-12 * np.maximum(mags, 1e-300)).all()
        else:
            total = [sum(int(t) for t in sv[b:e]) for b, e in zip(start, np.append(start[1:], n))]
            assert [(int(h) << 64) + (int(s) & (2**64 - 1)) for h, s in zip(host(a.sum_hi), host(a.sum))] == total


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dist", ["uniform", "few", "equal", "zipf"])
def test_sizes_and_distributions(ctx, n, dist):
    rng = np.random.default_rng(n * 5 + len(dist))
    for kdt in (np.int32, np.int64):
        check(ctx, [datagen.keys_for(dist, kdt, n, rng)], [values(rng, n, np.float64), values(rng, n, np.int64)])


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("kdt", [np.int32, np.int64, np.uint32, np.uint64, np.float64, np.float32])
def test_types_and_orders(ctx, order, kdt):
    rng = np.random.default_rng(order * 7 + np.dtype(kdt).itemsize)
    for dist in ("uniform", "few"):
        key = datagen.keys_for(dist, kdt, 3001, rng)
        check(ctx, [key], [values(rng, 3001, t) for t in (np.float32, np.uint32, np.uint64, np.int32, np.float64)], order)


@pytest.mark.parametrize("order", ORDERS)
def test_several_keys(ctx, order):
    rng = np.random.default_rng(order)
    n = 2500
    keys = [datagen.keys_for("few", np.int64, n, rng), datagen.keys_for("small", np.uint32, n, rng),
            datagen.keys_for("uniform", np.float64, n, rng)]
    for m in (2, 3):
        check(ctx, keys[:m], [values(rng, n, np.float64)], order)
    check(ctx, [keys[1], keys[0]], [], order)


def test_row_view_and_sort_only(ctx):
    from test_groupby_gpu import _host_args
    rng = np.random.default_rng(5)
    n = 3333
    k = datagen.keys_for("few", np.int64, n, rng)
    view = rng.permutation(n).astype(np.uint32)
    a, out = _host_args([k], [], [], n, perm_in=view)
    a.groupby = 0
    assert vdf.lib.vdf_sort_groupby_host(ctx.handle, C.byref(a), None) == 0
    assert (out["perm"] == view[np.argsort(k[view], kind="stable")]).all()


def test_outputs_over_the_inputs(ctx):
    rng = np.random.default_rng(6)
    n = 4000
    keys = [datagen.keys_for("few", np.int32, n, rng), datagen.keys_for("small", np.int32, n, rng)]
    vals = [values(rng, n, np.float64), values(rng, n, np.int64)]
    dk, dv = [dev(k) for k in keys], [dev(v) for v in vals]
    o = ctx.alloc_sort_groupby_outputs(dk, dv, [0, 1])
    o["skeys"], o["pay"] = dk, dv
    gr = ctx.sort_groupby(dk, dv, agg_cols=[0, 1], outputs=o)
    perm = ob.argsort(keys)
    assert (host(gr.perm).view(np.uint32) == perm).all()
    for h, d in zip(keys + vals, dk + dv):
        assert bits_equal(host(d), h[perm])
    assert (host(gr.aggs[1].sum) == ob.groupby(keys, vals).sum[1]).all()
