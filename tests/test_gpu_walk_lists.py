"""The greedy walk's prepared lists against the CPU oracle, bit for bit, where they can go wrong:
counters at and beyond the seven bits of the packed word, palettes shorter than a list or a
record, rows shorter than the lists' lead, caps of 1 (a reset every few cells), penalty windows
that close inside a list, reach beyond it or span the whole row of candidates, equal colours
(ties), one-colour targets, and the ring form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # p, gw, gh, cap, weight, colour spread of the palette, drift of the cells
    (12, 40, 30, 125, 0.25, 90, 3.0), (12, 40, 30, 126, 0.25, 90, 3.0), (12, 40, 30, 127, 0.25, 90, 3.0),
    (12, 40, 30, 128, 0.25, 90, 3.0), (9, 60, 40, 1000, 0.25, 90, 0.0), (3, 20, 20, 5, 0.25, 90, 3.0),
    (8, 17, 30, 3, 1.0, 90, 3.0), (9, 17, 30, 3, 1.0, 90, 3.0), (33, 8, 40, 2, 0.25, 30, 3.0),
    (33, 9, 40, 1, 0.25, 30, 3.0), (34, 13, 30, 1, 5.0, 10, 2.0), (200, 33, 25, 2, 0.0, 30, 1.0),
    (3000, 90, 70, 3, 0.25, 20, 0.5), (3000, 61, 43, 2, 3.0, 20, 0.5), (3000, 61, 43, 4, 60.0, 20, 0.5),
    *[(9000 + i, 100, 75, 5, 0.25, 40, 0.5) for i in range(6)], (500, 80, 60, 3, 0.25, 0.0, 0.5), (400, 50, 40, 0, 0.25, 60, 3.0), (12000, 300, 120, 3, 0.25, 40, 0.2)]


@pytest.mark.parametrize("p,gw,gh,cap,weight,spread,drift", CASES)
def test_walk_lists(ctx, orc, p, gw, gh, cap, weight, spread, drift):
    rng = np.random.default_rng(p * 13 + gw * 7 + cap)
    pal = np.concatenate([50 + rng.uniform(-spread / 2, spread / 2, (p, 1)), rng.uniform(-spread, spread, (p, 2))],
                         1).astype(np.float32)
    pal[p // 3] = pal[0]  # equal colours: the lower index first
    cells = np.cumsum(rng.normal(0, drift, (gw * gh, 3)), axis=0)
    cells = (np.array([50, 0, 0]) + (cells - cells.mean(0)) % max(spread, 1.0) - max(spread, 1.0) / 2).astype(np.float32)
    grid, resets = ctx.place_greedy(pal, cells, gw, gh, cap, weight)
    rgrid, rresets = orc.place_greedy(pal, cells, gw, gh, cap, weight)
    assert np.array_equal(grid, rgrid)
    assert resets == rresets
