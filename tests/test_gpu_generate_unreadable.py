"""mg_generate with inputs in memory that the GPU would read in place: a read-only file map gives the
oracle's result; memory that cannot be read -- a page without permission, the part of a file map
behind the file's end, an unmapped page -- is refused with MG_ERR_ARG before anything is given to
the GPU, and the context goes on."""
import copy
import ctypes
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIBC = ctypes.CDLL(None, use_errno=True)
PAGE = mmap.PAGESIZE


def _inputs():
    from mosaic_gpu import job

    cfg = job.scaled(job.WORKLOADS["recommended"], target_w=400, target_h=300, n_materials=60, material_side=61,
                     grid_w=12, grid_h=9, tile_w=33, tile_h=31, iterations=200, chains=2, seed=11)
    return job.make_inputs(cfg)


def _with(inp, field, data):
    from mosaic_gpu import job

    mats = copy.copy(inp.mats)
    target, thumbs = inp.target, inp.thumbs
    if field == "materials":
        mats.buf = data.reshape(inp.mats.buf.shape)
    elif field == "target":
        target = data.reshape(inp.target.shape)
    else:
        thumbs = data.reshape(inp.thumbs.shape)
    return job.Inputs(inp.cfg, target, mats, thumbs)


def _bytes(inp, field):
    a = {"materials": inp.mats.buf, "target": inp.target, "thumbnails": inp.thumbs}[field]
    return np.ascontiguousarray(a).reshape(-1).view(np.uint8)


def _expect(ctx, orc, inp):
    from mosaic_gpu import job

    res, grid, image = job.generate(ctx, job.RequestHolder(inp))
    ref = orc.generate(inp, threads=8)
    assert np.array_equal(grid, ref["grid"]) and np.array_equal(image, ref["image"])


@pytest.mark.parametrize("field", ["target", "materials", "thumbnails"])
def test_read_only_file_map(ctx, orc, tmp_path, field):
    inp = _inputs()
    path = tmp_path / "bytes"
    path.write_bytes(_bytes(inp, field).tobytes())
    _expect(ctx, orc, _with(inp, field, np.memmap(path, np.uint8, "r")))


@pytest.mark.parametrize("field", ["target", "materials", "thumbnails"])
@pytest.mark.parametrize("how", ["no permission", "file's end", "unmapped"])
def test_unreadable_memory_is_refused(ctx, orc, tmp_path, field, how):
    from mosaic_gpu import _capi, job

    inp = _inputs()
    data = _bytes(inp, field)
    assert data.size > 2 * PAGE
    size = (data.size + PAGE - 1) // PAGE * PAGE
    last = (data.size // PAGE - 1) * PAGE  # the last whole page
    if how == "file's end":
        path = tmp_path / "bytes"
        path.write_bytes(data.tobytes())
        block = np.memmap(path, np.uint8, "r+")
        with open(path, "r+b") as f:
            f.truncate(last)
        moved = block
    else:
        m = mmap.mmap(-1, size)
        block = np.frombuffer(m, np.uint8)
        block[:data.size] = data
        moved = block[:data.size]
        at = ctypes.c_void_p(block.ctypes.data + last)
        if how == "no permission":
            assert LIBC.mprotect(at, ctypes.c_size_t(PAGE), 0) == 0
        else:
            assert LIBC.munmap(at, ctypes.c_size_t(PAGE)) == 0
    with pytest.raises(_capi.MosaicError) as e:
        job.generate(ctx, job.RequestHolder(_with(inp, field, moved)))
    assert e.value.code == _capi.MG_ERR_ARG
    assert b"cannot be read" in ctx.lib.mg_last_error()
    _expect(ctx, orc, inp)
    if how == "unmapped":  # the hole is filled again before the object unmaps its range
        LIBC.mmap.restype = ctypes.c_void_p
        LIBC.mmap.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_long]
        LIBC.mmap(at, PAGE, mmap.PROT_READ | mmap.PROT_WRITE, mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS | 0x10, -1, 0)
