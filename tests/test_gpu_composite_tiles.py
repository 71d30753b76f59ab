"""The composite's packed arithmetic and its walk over a tile against the CPU oracle, byte for byte:
tiles of one pixel, of odd widths (a row's last pixel alone), narrower and wider than a CTA's
threads, more tiles than CTAs, empty cells, and colours where the hue, the saturation or a divisor
is zero (grey, black, white, one channel)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tw,th,gw,gh", [
    (1, 1, 70, 50), (2, 3, 41, 37), (3, 2, 9, 5), (4, 1, 33, 60), (5, 5, 60, 40), (8, 8, 61, 43), (25, 25, 7, 5),
    (33, 17, 5, 6), (64, 3, 4, 5), (100, 90, 3, 2), (129, 70, 2, 2), (260, 4, 2, 3)])
@pytest.mark.parametrize("strength", [0.4, 1.0])
def test_composite_tiles(ctx, orc, tw, th, gw, gh, strength):
    rng = np.random.default_rng(tw * 100 + th)
    p = 24
    thumbs = rng.integers(0, 256, (p, th, tw, 3)).astype(np.uint8)
    thumbs[0] = 0
    thumbs[1] = 255
    thumbs[2] = thumbs[2][..., :1]                # grey
    thumbs[3][..., 1:] = 0                        # one channel
    thumbs[4] = np.where(thumbs[4] > 127, 255, 0)  # saturated: every sector's edge
    thumbs[5] = 120 + thumbs[5] % 3               # nearly grey
    grid = rng.integers(-1, p, (gh, gw)).astype(np.int32)
    cell_rgb = rng.integers(0, 256, (gh * gw, 3)).astype(np.uint8)
    cell_rgb[::7] = cell_rgb[::7][:, :1]
    thumb_rgb = np.stack([orc.avg_rgb(t) for t in thumbs])
    out = ctx.composite(grid, thumbs, cell_rgb, strength)
    assert np.array_equal(out, orc.composite(grid, thumbs, cell_rgb, thumb_rgb, strength))
