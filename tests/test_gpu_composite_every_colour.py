"""The composite's two-pixel arithmetic for every byte triple in both of its halves, against the CPU
oracle, byte for byte: one tile holds all 2^24 colours in order, a second the same ones moved on by
one pixel, so that each colour is the first of a pair in one and the second in the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,strength", [((200, 40, 90), 0.4), ((20, 90, 230), 1.0), ((90, 120, 60), 1.0)])
def test_every_colour_in_both_halves(ctx, orc, cell, strength):
    v = np.arange(1 << 24, dtype=np.uint32)
    colours = np.stack([v >> 16, (v >> 8) & 255, v & 255], axis=-1).astype(np.uint8)
    thumbs = np.empty((2, 6144, 4096, 3), np.uint8)
    thumbs[:, 4096:] = [250, 60, 20]  # a mean with a hue, which the shift starts from
    thumbs[0, :4096] = colours.reshape(4096, 4096, 3)
    thumbs[1, :4096] = np.roll(colours, 1, axis=0).reshape(4096, 4096, 3)
    grid = np.array([[0, 1]], np.int32)
    cell_rgb = np.array([cell, cell], np.uint8)
    out = ctx.composite(grid, thumbs, cell_rgb, strength)
    thumb_rgb = np.stack([orc.avg_rgb(t) for t in thumbs])
    assert int(thumb_rgb[0].max()) - int(thumb_rgb[0].min()) > 60
    want = orc.composite(grid, thumbs, cell_rgb, thumb_rgb, strength)
    bad = np.flatnonzero(np.any(out != want, axis=-1).ravel())
    assert bad.size == 0, (bad.size, out.reshape(-1, 3)[bad[:3]], want.reshape(-1, 3)[bad[:3]])
