"""Greedy descent (no worse swap accepted) against the CPU replay, bit for bit, from the first windows,
where most accept something, to the last, which accept nothing and are settled in one pass: grids
where every proposal touches others, one-row grids, empty cells, a palette outside shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,gw,gh,iters,chains,empty", [
    (9, 2, 2, 400, 2, 0.0), (5, 1, 11, 1000, 2, 0.0), (9, 5, 4, 3000, 3, 0.2), (60, 12, 9, 20000, 2, 0.0),
    (300, 22, 16, 20001, 2, 0.1), (300, 60, 45, 6000, 2, 0.0), (20000, 20, 15, 5000, 2, 0.0), (50, 14, 10, 700, 200, 0.0)])
def test_greedy_descent(ctx, orc, p, gw, gh, iters, chains, empty):
    rng = np.random.default_rng(p + iters + gw)
    pal = np.concatenate([rng.uniform(0, 100, (p, 1)), rng.uniform(-90, 90, (p, 2))], 1).astype(np.float32)
    grid = rng.integers(0, p, (gh, gw)).astype(np.int32)
    grid[rng.random((gh, gw)) < empty] = -1
    _, _, per, cg = ctx.optimize(pal, grid, iterations=iters, chains=chains, seed=5 + iters, greedy_only=True)
    for c in (0, chains - 1):
        rg, res, cnt = orc.anneal(pal, grid, iters, seed=5 + iters, chain=c, greedy_only=True)
        assert np.array_equal(cg[c], rg), c
        got = np.array([per[c].initial_cost, per[c].final_cost, per[c].best_cost], np.float32)
        assert np.array_equal(got.view(np.uint32), np.array(res[:3], np.float32).view(np.uint32))
        assert (per[c].accepted_count, per[c].improved_count) == (cnt[0], cnt[1])
