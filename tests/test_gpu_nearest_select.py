"""The k-nearest searches' selection against the oracle's brute force, the same indices and distance
bits: list lengths around the powers of two that the sorts take, and more equal distances at the
k-th place than a sort takes, or than the buffer holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nctx(built):
    from mosaic_gpu import _capi as capi

    c = capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("k", [1, 2, 31, 32, 33, 63, 64, 65, 99, 100])
@pytest.mark.parametrize("repeat", [1, 40, 150, 700])
def test_selection(nctx, orc, k, repeat):
    from mosaic_gpu import _capi as capi

    rng = np.random.default_rng(k * 7 + repeat)
    n = 2500
    base = np.stack([rng.uniform(0, 100, n), rng.uniform(-90, 90, n), rng.uniform(-90, 90, n)], 1).astype(np.float32)
    pal = base[np.arange(n) // repeat]  # runs of one colour: equal distances
    rng.shuffle(pal, axis=0)
    q = np.concatenate([pal[:40], pal[40:80] + rng.normal(0, 2, (40, 3)).astype(np.float32),
                        rng.uniform(-100, 120, (20, 3)).astype(np.float32)])
    ridx, rdist = orc.nearest_n(pal, q, k)
    for method in (capi.MG_NEAREST_GRID, capi.MG_NEAREST_SCAN):
        nctx.set_nearest_method(method)
        idx, dist = nctx.nearest_n(pal, q, k)
        assert np.array_equal(idx, ridx), method
        assert np.array_equal(dist.view(np.uint32), rdist.view(np.uint32)), method
