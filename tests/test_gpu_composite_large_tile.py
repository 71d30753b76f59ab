"""One tile of more than 2^31 bytes (an output row may hold 2^31 / 3 pixels), against the CPU oracle
on rows before, at and beyond that byte, and as a copy over all of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _available():
    with open("/proc/meminfo") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("MemAvailable")) << 10


@pytest.mark.parametrize("tw,th,strength", [(30000, 24000, 0.0), (30000, 24000, 0.4), (29999, 24001, 0.4)])
def test_tile_beyond_31_bits(ctx, orc, tw, th, strength):
    if _available() < 24 << 30:
        pytest.skip("not enough host memory")
    block = np.random.default_rng(tw).integers(0, 256, 1 << 24).astype(np.uint8)
    thumb = np.resize(block, (1, th, tw, 3))
    assert thumb.nbytes > 1 << 31
    grid = np.zeros((1, 1), np.int32)
    cell_rgb = np.array([[200, 40, 90]], np.uint8)
    out = ctx.composite(grid, thumb, cell_rgb, strength)
    if strength == 0.0:
        assert np.array_equal(out, thumb[0])
        return
    thumb_rgb = orc.avg_rgb(thumb[0]).reshape(1, 3)
    at = (1 << 31) // (3 * tw)
    for y0 in (0, at - 1, th - 3):
        rows = np.ascontiguousarray(thumb[:, y0:y0 + 3])
        want = orc.composite(grid, rows, cell_rgb, thumb_rgb, strength)
        assert np.array_equal(out[y0:y0 + 3], want), y0
