"""The group-by emit where its ways of folding a group meet: groups of 32, 33,
256 and 257 rows (one thread, eight lanes, a warp), groups that start, end or
run through the 512-row tile and 2,048-row CTA edges, for zero to four value
columns."""
import numpy as np
import pytest

import oracle_bind as ob
from gpu_util import dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nvals", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("runs", [[32, 33], [256, 257], [1, 32, 1, 33, 1, 257], [511, 1], [2047, 1], [2048], [2049],
                                  [5000, 1, 1, 30], [1]])
@pytest.mark.parametrize("n", [2047, 2048, 2049, 20_001])
def test_group_lengths_at_tile_edges(ctx, nvals, runs, n):
    rng = np.random.default_rng(n + nvals)
    reps = np.tile(runs, n // sum(runs) + 1)
    key = np.repeat(np.arange(reps.size, dtype=np.int64) * 3 - 1000, reps)[:n]
    vals = [rng.standard_normal(n), rng.integers(-2**62, 2**62, n), rng.standard_normal(n).astype(np.float32),
            rng.integers(0, 2**32, n, dtype=np.uint32)][:nvals]
    gr = ctx.groupby_sorted([dev(key)], [dev(v) for v in vals], want_row_group=True, want_group_start=True)
    o = ob.groupby([key], vals)
    assert gr.n_groups == o.n_groups
    assert (host(gr.keys[0]) == o.keys[0]).all() and (host(gr.count) == o.count).all()
    start = np.flatnonzero(np.append(True, key[1:] != key[:-1]))
    assert (host(gr.group_start) == start).all()
    assert (host(gr.row_group) == np.searchsorted(start, np.arange(n), side="right") - 1).all()
    for i, (v, a) in enumerate(zip(vals, gr.aggs)):
        assert (host(a.min) == o.min[i]).all() and (host(a.max) == o.max[i]).all()
        if v.dtype.kind == "f":
            assert (np.abs(host(a.sum) - o.sum[i]) <= 1e-12 * np.maximum(o.abs[i], 1e-300)).all()
        else:
            assert (host(a.sum) == o.sum[i]).all() and (host(a.sum_hi) == o.sum_hi[i]).all()
    quiet = ctx.groupby_sorted([dev(key)], [dev(v) for v in vals])  # head-less CTAs return at once
    assert (host(quiet.count) == o.count).all()
