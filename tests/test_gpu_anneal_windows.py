"""The annealing kernel's windows of 64 proposals against the CPU replay, bit for bit:
iteration counts around a window, grids so small that most proposals touch each other, grids
mostly empty, more chains than multiprocessors (two chains share one), the largest grid the
annealer takes (least room for the writers table), and colours so far apart that the weights
leave the range of the short square root and reciprocal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # p, gw, gh, iterations, chains, empty share, t0, decay, greedy, colour scale
    (9, 5, 4, 1, 1, 0.0, 100.0, 0.99995, False, 1.0), (9, 5, 4, 63, 2, 0.0, 100.0, 0.99995, False, 1.0),
    (9, 5, 4, 64, 2, 0.0, 0.02, 0.99, False, 1.0), (9, 5, 4, 65, 2, 0.0, 0.02, 0.99, True, 1.0),
    (6, 2, 1, 300, 2, 0.0, 1.0, 0.999, False, 1.0), (6, 1, 9, 257, 2, 0.0, 0.1, 0.999, False, 1.0),
    (40, 17, 13, 1000, 3, 0.9, 0.05, 0.999, False, 1.0), (40, 40, 30, 3000, 2, 0.3, 0.01, 0.9995, False, 1.0),
    (30, 20, 15, 200, 200, 0.05, 0.1, 0.99, False, 1.0), (20000, 20, 15, 200, 200, 0.0, 0.1, 0.99, False, 1.0),
    (500, 398, 256, 500, 1, 0.0, 0.05, 0.999, False, 1.0), (30, 12, 9, 500, 2, 0.0, 0.5, 0.999, False, 1e15),
    (30, 12, 9, 500, 2, 0.0, 0.5, 0.999, False, 3e18), (30, 12, 9, 500, 2, 0.0, 0.5, 0.999, False, 1e-17)]


@pytest.mark.parametrize("p,gw,gh,iters,chains,empty,t0,decay,greedy,scale", CASES)
def test_anneal_windows(ctx, orc, p, gw, gh, iters, chains, empty, t0, decay, greedy, scale):
    rng = np.random.default_rng(p + 31 * iters + gw)
    pal = np.concatenate([rng.uniform(0, 100, (p, 1)), rng.uniform(-90, 90, (p, 2))], 1).astype(np.float32)
    pal *= np.float32(scale)
    grid = rng.integers(0, p, (gh, gw)).astype(np.int32)
    grid[rng.random((gh, gw)) < empty] = -1
    _, _, per, cg = ctx.optimize(pal, grid, iterations=iters, t0=t0, decay=decay, chains=chains, seed=77 + iters,
                                 stream=3, greedy_only=greedy)
    for c in range(chains) if chains < 10 else (0, 1, chains // 2, chains - 1):
        rg, res, cnt = orc.anneal(pal, grid, iters, t0=t0, decay=decay, seed=77 + iters, stream=3, chain=c,
                                  greedy_only=greedy)
        assert np.array_equal(cg[c], rg), c
        got = np.array([per[c].initial_cost, per[c].final_cost, per[c].best_cost], np.float32)
        assert np.array_equal(got.view(np.uint32), np.array(res[:3], np.float32).view(np.uint32))
        assert (per[c].accepted_count, per[c].improved_count) == (cnt[0], cnt[1])
