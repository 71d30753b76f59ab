"""mg_generate from ordinary host memory, which the kernels read in place where the GPU can: buffers
at any byte alignment, a read-only file map, and one buffer refilled between calls (the second call
sees the second contents), against the CPU oracle."""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(seed):
    from mosaic_gpu import job

    cfg = job.scaled(job.WORKLOADS["recommended"], target_w=242, target_h=181, n_materials=60, material_side=37,
                     grid_w=12, grid_h=9, tile_w=9, tile_h=7, iterations=200, chains=2, seed=seed)
    return job.make_inputs(cfg)


def _moved(a, make):
    """The array's bytes in the memory that make(size) gives, same shape."""
    out = make(a.nbytes)
    out[:] = np.ascontiguousarray(a).reshape(-1).view(np.uint8)
    return out.reshape(a.shape)


def _check(ctx, orc, inp, device_thumbs):
    from mosaic_gpu import job

    ref_inp = inp if not device_thumbs else job.Inputs(inp.cfg, inp.target, inp.mats, None)
    res, grid, image = job.generate(ctx, job.RequestHolder(ref_inp))
    if device_thumbs:  # the resized thumbnails, for the oracle
        tw, th = inp.tile
        thumbs = np.stack([orc.resize_lanczos3(np.ascontiguousarray(inp.mats.buf[int(o):int(o) + 3 * int(w) * int(h)].reshape(int(h), int(w), 3)), tw, th)
                           for o, w, h in zip(inp.mats.off, inp.mats.w, inp.mats.h)])
        ref_inp = job.Inputs(inp.cfg, inp.target, inp.mats, thumbs)
    ref = orc.generate(ref_inp, threads=8)
    assert np.array_equal(grid, ref["grid"]) and np.array_equal(image, ref["image"])
    assert res.n_resets == ref["n_resets"]


@pytest.mark.parametrize("device_thumbs", [False, True])
@pytest.mark.parametrize("where", [0, 1, 2, 3, 7, "file"])
def test_unregistered_memory(ctx, orc, tmp_path, where, device_thumbs):
    inp = _inputs(3)

    def make(n):
        if where == "file":
            make.count += 1
            path = tmp_path / f"bytes{make.count}"
            path.write_bytes(bytes(n))
            return np.memmap(path, np.uint8, "r+", shape=(n,))
        block = np.zeros(n + 64 + where, np.uint8)
        start = (-block.ctypes.data) % 64 + where
        return block[start:start + n]

    make.count = 0
    mats = copy.copy(inp.mats)
    mats.buf = _moved(inp.mats.buf, make)
    from mosaic_gpu import job

    _check(ctx, orc, job.Inputs(inp.cfg, _moved(inp.target, make), mats, _moved(inp.thumbs, make)), device_thumbs)


def test_refilled_buffer(ctx, orc):
    a, b = _inputs(4), _inputs(5)
    a.mats.buf[:] = 255 - a.mats.buf
    _check(ctx, orc, a, True)
    a.mats.buf[:] = b.mats.buf[:a.mats.buf.size] if b.mats.buf.size >= a.mats.buf.size else a.mats.buf[::-1]
    a.target[:] = 255 - a.target
    _check(ctx, orc, a, True)
