"""The greedy walk against the CPU oracle, bit for bit, while the warps that prepare its cells are
held back (mg_ctx_inject_walk_delay): the walker may decide a cell only from what is of that cell,
however late it comes.  Rows at the widths where the ring of records is tightest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WIDTHS = [17, 28, 29, 60, 61, 100]


def _check(ctx, orc, seed, p, gw, gh, cap, weight, drift, scout_ns, refiner_ns):
    from mosaic_gpu import _capi

    rng = np.random.default_rng(seed)
    pal = np.concatenate([50 + rng.uniform(-20, 20, (p, 1)), rng.uniform(-40, 40, (p, 2))], 1).astype(np.float32)
    cells = np.cumsum(rng.normal(0, drift, (gw * gh, 3)), axis=0)
    cells = (np.array([50, 0, 0]) + (cells + 40) % 80 - 40).astype(np.float32)
    assert ctx.lib.mg_ctx_inject_walk_delay(ctx.h, scout_ns, refiner_ns) == _capi.MG_OK
    try:
        grid, resets = ctx.place_greedy(pal, cells, gw, gh, cap, weight)
    finally:
        assert ctx.lib.mg_ctx_inject_walk_delay(ctx.h, 0, 0) == _capi.MG_OK
    want, want_resets = orc.place_greedy(pal, cells, gw, gh, cap, weight)
    assert np.array_equal(grid, want) and resets == want_resets


@pytest.mark.parametrize("scout_ns", [0, 700, 25000])
@pytest.mark.parametrize("p", [5, 20, 64, 300, 511])
@pytest.mark.parametrize("gw", WIDTHS)
def test_records_alone(ctx, orc, gw, p, scout_ns):
    """Cap 1, few materials: the walk goes by the records."""
    for seed in range(4):
        _check(ctx, orc, seed * 1009 + p, p, gw, 23, 1, [0.25, 0.25, 0.0, 3.0][seed], [0.3, 2.0, 0.3, 0.3][seed],
               scout_ns, 0)


@pytest.mark.parametrize("refiner_ns", [0, 500, 2000, 20000])
@pytest.mark.parametrize("p,cap", [(5, 2), (16, 2), (40, 2), (120, 2), (9, 3), (300, 2), (700, 1)])
@pytest.mark.parametrize("gw", [40, 100])
def test_late_lists(ctx, orc, gw, p, cap, refiner_ns):
    """Lists that come late, with resets within their lead of one another and beyond it."""
    for seed in range(4):
        _check(ctx, orc, seed * 1013 + p, p, gw, 20, cap, [0.25, 1.0, 0.0, 3.0][seed], [0.3, 1.0, 0.3, 0.05][seed],
               0 if seed < 2 else 900, refiner_ns)


@pytest.mark.parametrize("refiner_ns", [0, 300, 1000, 4000, 20000])
@pytest.mark.parametrize("p,cap", [(5, 2), (12, 2), (20, 3), (160, 2)])
@pytest.mark.parametrize("gw", WIDTHS)
def test_records_written_again(ctx, orc, gw, p, cap, refiner_ns):
    """Runs from records beside refiners that are late for theirs: at rows of 28 and 60 cells a
    slot of the ring is another cell's once the walker is four cells past it."""
    for seed in range(4):
        _check(ctx, orc, seed * 1019 + p, p, gw, 26, cap, [0.25, 1.0, 0.0, 3.0][seed], [0.3, 1.0, 0.3, 0.05][seed],
               0, refiner_ns)


@pytest.mark.parametrize("refiner_ns", [0, 4000])
@pytest.mark.parametrize("gw", [28, 60])
def test_tight_ring(ctx, orc, gw, refiner_ns):
    """A palette beside which only the smaller ring of records fits: they are made less far ahead."""
    for drift in (0.0, 0.05):
        _check(ctx, orc, gw, 40000 if gw == 28 else 30000, gw, 16, 1, 0.25, drift, 0, refiner_ns)


def test_delay_arguments(ctx):
    from mosaic_gpu import _capi

    for scout, refiner in [(-1, 0), (0, -1), (100001, 0), (0, 100001)]:
        assert ctx.lib.mg_ctx_inject_walk_delay(ctx.h, scout, refiner) == _capi.MG_ERR_ARG
    assert ctx.lib.mg_ctx_inject_walk_delay(None, 0, 0) == _capi.MG_ERR_ARG
    assert ctx.lib.mg_ctx_inject_walk_delay(ctx.h, 0, 0) == _capi.MG_OK
