"""The greedy walk where the counters are reset every few cells, against the CPU oracle, bit for
bit: runs of cells decided from their records alone (after a reset, and all of a cap-1 walk), at
the lengths where they end -- the distance lists are made ahead, a warp of records, a row -- at the
palette sizes where the rules for lists and for the scouts' distance change, and in the ring form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # p, gw, gh, cap, weight, drift of the cells
    (2, 8, 30, 1, 0.25, 3.0), (5, 31, 20, 1, 0.25, 1.0), (11, 40, 30, 1, 0.0, 1.0), (13, 40, 30, 1, 0.25, 0.5),
    (6, 33, 30, 2, 0.25, 0.5), (32, 64, 20, 1, 0.25, 0.3), (33, 65, 20, 1, 1.0, 0.3), (60, 52, 34, 2, 0.25, 0.3),
    (128, 90, 40, 1, 0.25, 0.3), (160, 90, 40, 2, 0.25, 0.3), (511, 100, 60, 1, 0.25, 0.2), (512, 100, 60, 1, 0.25, 0.2),
    (40, 70, 50, 1, 30.0, 0.3), (7, 120, 90, 200, 0.25, 0.3), (50, 300, 280, 1, 0.25, 0.2)]


@pytest.mark.parametrize("p,gw,gh,cap,weight,drift", CASES)
def test_short_epochs(ctx, orc, p, gw, gh, cap, weight, drift):
    rng = np.random.default_rng(p * 31 + gw * 7 + cap)
    pal = np.concatenate([50 + rng.uniform(-20, 20, (p, 1)), rng.uniform(-40, 40, (p, 2))], 1).astype(np.float32)
    cells = np.cumsum(rng.normal(0, drift, (gw * gh, 3)), axis=0)
    cells = (np.array([50, 0, 0]) + (cells + 40) % 80 - 40).astype(np.float32)
    grid, resets = ctx.place_greedy(pal, cells, gw, gh, cap, weight)
    rgrid, rresets = orc.place_greedy(pal, cells, gw, gh, cap, weight)
    assert np.array_equal(grid, rgrid)
    assert resets == rresets
