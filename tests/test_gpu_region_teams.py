"""Cell and material statistics against the CPU oracle, bit for bit, over the teams of threads a
region gets: parts of a warp (many small regions), a warp, several warps of a CTA (few regions) and
row chunks, with team counts that do not divide a CTA, and rows of 8-, 4- and 1-byte alignment."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,gw,gh,pad", [
    (16, 16, 16, 16, 0), (644, 313, 161, 78, 0), (600, 400, 100, 80, 0), (1, 1, 1, 1, 0), (7, 3, 2, 1, 5),
    (64, 64, 1, 1, 0), (90, 91, 1, 1, 0), (257, 129, 3, 5, 3), (512, 512, 8, 8, 0), (516, 500, 9, 7, 4),
    (1000, 700, 20, 14, 0), (1920, 1080, 80, 45, 0), (1920, 1080, 37, 29, 16), (640, 360, 2, 1, 8), (375, 333, 1, 2, 0)])
def test_cells(ctx, orc, w, h, gw, gh, pad):
    rng = np.random.default_rng(w * 7 + h + gw)
    full = rng.integers(0, 256, (h, w * 3 + pad), dtype=np.uint8)
    img = full[:, :w * 3].reshape(h, w, 3) if pad == 0 else np.lib.stride_tricks.as_strided(
        full, (h, w, 3), (full.strides[0], 3, 1))
    lab, rgb = ctx.cells_lab(img, gw, gh)
    cw, ch = w // gw, h // gh
    picks = {(0, 0), (gw - 1, gh - 1), (gw // 2, gh // 2), (gw - 1, 0), *((int(rng.integers(gw)), int(rng.integers(gh))) for _ in range(40))}
    for x, y in picks:
        cell = np.ascontiguousarray(img[y * ch:(y + 1) * ch, x * cw:(x + 1) * cw])
        assert np.array_equal(np.asarray(lab).reshape(gh * gw, -1)[y * gw + x, :3].view(np.uint32),
                              orc.lab_mean_spec(cell).view(np.uint32)), (x, y)
        assert np.array_equal(np.asarray(rgb).reshape(gh * gw, -1)[y * gw + x, :3], orc.avg_rgb(cell)), (x, y)


@pytest.mark.parametrize("count,lo,hi", [(3, 1, 200), (40, 60, 90), (300, 3, 40), (17, 90, 130)])
def test_images(ctx, orc, count, lo, hi):
    rng = np.random.default_rng(count)
    imgs = [rng.integers(0, 256, (int(rng.integers(lo, hi)), int(rng.integers(lo, hi)), 3), dtype=np.uint8)
            for _ in range(count)]
    lab, rgb = ctx.images_lab(imgs)
    for i, img in enumerate(imgs):
        assert np.array_equal(lab[i].view(np.uint32), orc.lab_mean_spec(img).view(np.uint32)), i
        assert np.array_equal(np.asarray(rgb)[i, :3], orc.avg_rgb(img)), i
