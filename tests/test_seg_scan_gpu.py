"""The scan of the group-by's tile aggregates at its edges: one CTA of 256
tiles of 512 rows, two, and more CTAs than the last one has threads; groups
that run across CTAs."""
import numpy as np
import pytest

from gpu_util import dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 300_000])
@pytest.mark.parametrize("n", [131_071, 131_072, 131_073, 262_145, 257 * 131_072 + 5])
def test_scan_edges(ctx, n, rows):
    rng = np.random.default_rng(n + rows)
    key = (np.arange(n) // rows).astype(np.int32)
    val = rng.integers(-2**40, 2**40, n)
    for _ in range(2):  # the counter starts afresh on every call
        gr = ctx.groupby_sorted([dev(key)], [dev(val)])
        start = np.arange(0, n, rows)
        assert gr.n_groups == start.size
        assert (host(gr.keys[0]) == np.arange(start.size)).all()
        assert (host(gr.count) == np.diff(np.append(start, n))).all()
        assert (host(gr.aggs[0].sum).view(np.int64) == np.add.reduceat(val, start)).all()
        assert (host(gr.aggs[0].min).view(np.int64) == np.minimum.reduceat(val, start)).all()
