"""Left-join matching by hash table (First, Last) where its buckets overflow
and repeated keys race for a slot: few and many repeats per right key, the key
values that an empty slot's bytes spell, and both key widths."""
import numpy as np
import pytest

import oracle_bind as ob
from gpu_util import dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("dt", [np.int32, np.uint64])
@pytest.mark.parametrize("n_right,distinct", [(1, 1), (2, 2), (5, 1), (1000, 1000), (100_000, 7), (100_000, 30_000),
                                              (300_001, 300_001)])
def test_first_and_last(ctx, method, dt, n_right, distinct):
    rng = np.random.default_rng(n_right + distinct + method)
    info = np.iinfo(dt)
    pool = np.concatenate([np.array([-1, 0, 1], np.int64).astype(dt),
                           rng.integers(info.min, info.max, distinct, dtype=dt, endpoint=True)])[:max(3, distinct)]
    right = pool[rng.integers(0, min(distinct, pool.size), n_right)]
    left = np.concatenate([pool, rng.integers(info.min, info.max, 1000, dtype=dt, endpoint=True),
                           right[rng.integers(0, n_right, 50_000)]])
    match, count = ctx.left_join_index(dev(left), dev(right), method=method)
    exp, matched = ob.left_join(left, right, method)
    assert (host(match).view(np.uint32) == exp).all()
    assert count == matched
