"""The bucket grid's k-nearest search with colours and queries that are not numbers, or infinite,
against the scan (which compares every entry): such colours sort behind all others, and a query
whose surroundings hold fewer than k numbers looks further."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("p,step", [(2048, 9), (2048, 40), (4000, 9), (4000, 1000), (8000, 40), (20000, 9), (3000, 1)])
def test_grid_equals_scan(ctx, p, step, bad):
    rng = np.random.default_rng(p + step)
    pal = np.concatenate([50 + rng.uniform(-30, 30, (p, 1)), rng.uniform(-40, 40, (p, 2))], 1).astype(np.float32)
    queries = np.concatenate([50 + rng.uniform(-30, 30, (4000, 1)), rng.uniform(-40, 40, (4000, 2))], 1).astype(np.float32)
    queries[::5] = queries[::5] * 0.2 + np.array([20, -40, -40], np.float32) * 0.8  # the corner of bucket 0
    pal[::step] = bad
    queries[::13] = bad
    queries[5::29, 1] = bad
    try:
        ctx.set_nearest_method(1)
        idx, dist = ctx.nearest_n(pal, queries, 100)
        ctx.set_nearest_method(2)
        gidx, gdist = ctx.nearest_n(pal, queries, 100)
    finally:
        ctx.set_nearest_method(0)
    assert np.array_equal(idx, gidx) and np.array_equal(dist.view(np.uint32), gdist.view(np.uint32))
