"""Thumbnails that the device makes, against the CPU oracle, for numbers and sizes of images over
which the choice between the two forms of the resize and the number of bands changes, with the
images copied to the device (a plan) and read in place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side,tw,th", [
    (1, 300, 16, 12), (1, 300, 40, 31), (3, 120, 12, 9), (3, 200, 64, 48), (9, 300, 14, 10), (24, 90, 31, 30),
    (40, 150, 16, 12), (40, 64, 64, 64), (110, 80, 16, 12), (170, 70, 33, 25), (420, 60, 20, 15), (420, 50, 12, 7)])
def test_counts(ctx, orc, n, side, tw, th):
    from mosaic_gpu import job

    cfg = job.scaled(job.WORKLOADS["recommended"], target_w=160, target_h=120, n_materials=n, material_side=side, grid_w=8,
                     grid_h=6, tile_w=tw, tile_h=th, iterations=50, chains=1, seed=n, max_usage=3, aspect_tolerance=10.0)
    inp = job.make_inputs(cfg)
    m = inp.mats
    thumbs = np.stack([orc.resize_lanczos3(np.ascontiguousarray(m.buf[int(o):int(o) + 3 * int(w) * int(h)].reshape(int(h), int(w), 3)),
                                           tw, th) for o, w, h in zip(m.off, m.w, m.h)])
    ref = orc.generate(job.Inputs(cfg, inp.target, m, thumbs), threads=8)
    assert ref["p"] == n
    holder = job.RequestHolder(job.Inputs(cfg, inp.target, m, None))
    res, grid, image = job.generate(ctx, holder)
    assert np.array_equal(grid, ref["grid"]) and np.array_equal(image, ref["image"])
    plan = job.Plan(ctx, holder)
    plan.run()
    res, grid, image = plan.read()
    assert np.array_equal(grid, ref["grid"]) and np.array_equal(image, ref["image"])
    plan.close()
