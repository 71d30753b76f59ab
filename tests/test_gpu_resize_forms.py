"""Lanczos3 resize against the CPU oracle, byte for byte, where its two forms can go wrong: a kept
width, height or both, enlarging, one pixel, rows that are no multiple of four pixels or bytes,
fewer output rows than a band, many bands, source rows in several chunks, and images that do not
fit in shared memory (the two-kernel form)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,dw,dh,pad", [
    (1, 1, 1, 1, 0), (1, 1, 9, 7, 0), (5, 3, 5, 3, 1), (64, 64, 64, 16, 0), (64, 64, 16, 64, 0), (7, 9, 31, 40, 2),
    (140, 140, 24, 24, 0), (141, 139, 24, 24, 0), (142, 97, 25, 31, 3), (143, 64, 8, 8, 5), (97, 131, 13, 5, 0),
    (33, 2500, 8, 5, 0), (2500, 33, 8, 5, 1), (300, 1200, 24, 24, 4), (401, 303, 100, 75, 7), (16, 12, 48, 48, 0),
    (4001, 31, 333, 29, 0), (9000, 40, 1200, 20, 0), (1024, 768, 400, 300, 0), (40, 3000, 300, 290, 0)])
def test_resize_forms(ctx, orc, w, h, dw, dh, pad):
    rng = np.random.default_rng(w * 3 + h * 5 + dw)
    full = rng.integers(0, 256, (h, 3 * w + pad), dtype=np.uint8)
    full[: h // 2] = np.where(full[: h // 2] > 127, 255, 0)  # overshoot: the clamp
    img = np.lib.stride_tricks.as_strided(full, (h, w, 3), (full.strides[0], 3, 1))
    assert np.array_equal(ctx.resize(img, dw, dh), orc.resize_lanczos3(np.ascontiguousarray(img), dw, dh))
