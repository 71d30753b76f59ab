"""The bucket search at its largest grid, where the list length decides the warps of a CTA and the
size of their buffers, against the oracle's brute force: queries inside the palette's gamut and
outside it (the list form), and runs of one colour."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 17, 63, 64, 65, 100])
@pytest.mark.parametrize("p,repeat", [(34000, 1), (35000, 1), (35000, 90), (60000, 1)])
def test_large_palettes(ctx, orc, p, repeat, k):
    rng = np.random.default_rng(p + repeat)
    pal = np.concatenate([50 + rng.uniform(-30, 30, (p, 1)), rng.uniform(-10, 10, (p, 2))], 1).astype(np.float32)
    pal = pal[np.arange(p) // repeat]
    rng.shuffle(pal, axis=0)
    q = np.concatenate([50 + rng.uniform(-45, 45, (90, 1)), rng.uniform(-60, 60, (90, 2))], 1).astype(np.float32)
    q[:45] = pal[:45] + rng.normal(0, 1, (45, 3)).astype(np.float32)
    idx, dist = orc.nearest_n(pal, q, k)
    q = np.tile(q, (90, 1))  # more than a CTA an SM
    gidx, gdist = ctx.nearest_n(pal, q, k)
    assert np.array_equal(gidx, np.tile(idx, (90, 1)))
    assert np.array_equal(gdist.view(np.uint32), np.tile(dist, (90, 1)).view(np.uint32))
