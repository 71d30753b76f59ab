"""Chains whose temperature falls to nothing (or starts there, or is below zero) against the CPU
replay, bit for bit: the acceptance bounds on either side of 1e-30, in subnormals, at zero of both
signs, with colours so far apart that the weights' differences are at their smallest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t0,decay", [(100.0, 0.97), (1e-28, 0.9), (1e-30, 1.0), (9.9e-31, 1.0), (1e-38, 0.9), (0.0, 0.9),
                                      (-0.0, 0.9), (-1e-35, 0.9), (float("inf"), 0.5)])
@pytest.mark.parametrize("spread", [1.0, 1e-4, 3e17])
def test_frozen(ctx, orc, t0, decay, spread):
    rng = np.random.default_rng(3)
    pal = (np.concatenate([rng.uniform(0, 100, (40, 1)), rng.uniform(-90, 90, (40, 2))], 1) * spread).astype(np.float32)
    pal[7] = pal[5]
    grid = rng.integers(0, 40, (7, 10)).astype(np.int32)
    grid[2, 3] = -1
    _, _, per, cg = ctx.optimize(pal, grid, iterations=6000, t0=t0, decay=decay, chains=3, seed=9)
    for c in (0, 2):
        rg, res, cnt = orc.anneal(pal, grid, 6000, t0=t0, decay=decay, seed=9, chain=c)
        assert np.array_equal(cg[c], rg), c
        got = np.array([per[c].initial_cost, per[c].final_cost, per[c].best_cost], np.float32)
        assert np.array_equal(got.view(np.uint32), np.array(res[:3], np.float32).view(np.uint32))
        assert (per[c].accepted_count, per[c].improved_count) == (cnt[0], cnt[1])
