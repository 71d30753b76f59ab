"""Performance cases of the mosaic path: the calls a program makes, over the sizes and options it makes them with.

A case is a dict of plain values; "kind" says which public entry point it drives:

  generate        mg_generate, one job from host buffers to host buffers (uploads, whole pipeline, download)
  plan            mg_plan_run + mg_plan_read: the same job over inputs that already sit in device memory
  batch           mg_batch_run + mg_batch_read: uneven mosaics over one resident palette, targets on the device
  generate_batch  mg_generate_batch: the same from pinned host targets to pinned host results, one call
  served          mg_server: a burst of requests submitted to the request loop, every one waited for
  cells           mg_cells_lab_noalloc: the cell reduction alone on the caller's device buffers
  place           mg_place_greedy: candidate search and greedy placement from host Lab colours
  optimize        mg_optimize: annealing chains over a placed grid

Images are synthetic and seeded: targets are a uniform background with alpha-blended Gaussian blobs and +-8 noise,
materials a base colour with a linear gradient and +-16 noise (what bench.py's generator makes, here on the GPU).
"""
import ctypes as C
import math
import sys
import weakref
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path.cwd() / "mosaic-art-rust_gb300"))

from mosaic_gpu import _capi as capi  # noqa: E402
from mosaic_gpu import job, synth  # noqa: E402

K_CANDIDATES = 100  # candidates per cell the placement looks at


# ---- the cases ------------------------------------------------------------------------------------------------------
def _job(kind, target_w, target_h, blobs, materials, side, aspects, grid_w, grid_h, usage, strength, iterations, chains,
         tile_w=0, tile_h=0, weight=0.25, thumbs="device", pinned=False, scoring="cli", similarity=True, row_pad=0):
    """A whole generate_mosaic job.  aspects: materials drawn from {1:1, 4:3, 3:4} (the filter then keeps about a third)
    instead of all square.  thumbs: "host" (the caller resized them), "device" (Lanczos3) or "area".  pinned: the host
    buffers come from mg_host_alloc.  row_pad: extra bytes between target rows."""
    return {k: v for k, v in locals().items()}


def listed():
    named = {
        # A preview: a thumbnail-sized target, a folder of 90 small pictures, ordinary (pageable) memory.  Latency counts.
        "generate_tiny": _job("generate", 384, 288, 6, 90, 64, True, 16, 12, 3, 0.4, 300, 4, 12, 12, thumbs="host"),
        # The plain job on the crate's defaults: one chain, no colour adjustment, tiles of the cell's size, made on the device.
        "generate_small": _job("generate", 1024, 768, 8, 500, 128, False, 40, 30, 3, 0.0, 500, 1),
        # Sizes as photographs have them: nothing divides anything, rows are padded, the GUI's scoring, area thumbnails.
        "generate_ragged": _job("generate", 1531, 1147, 11, 333, 101, True, 61, 43, 2, 1.0, 1000, 3, 37, 29, weight=0.1,
                                thumbs="area", scoring="gui", similarity=False, row_pad=13),
        # The recommended settings, host to host through pinned buffers: the headline job as a program calls it.
        "generate_recommended": _job("generate", 3840, 2880, 32, 1500, 256, True, 80, 60, 3, 0.4, 2000, 32, 48, 48,
                                     thumbs="host", pinned=True),
        # The same job run again on resident inputs (a program that varies nothing but the seed, or benchmarks).
        "plan_recommended": _job("plan", 3840, 2880, 32, 1500, 256, True, 80, 60, 3, 0.4, 2000, 32, 48, 48,
                                 thumbs="host", pinned=True),
        # A poster: 24 000 cells, 5000 materials, long annealing.
        "plan_large": _job("plan", 7680, 5760, 128, 5000, 128, False, 179, 134, 8, 0.4, 100000, 64, 32, 32, pinned=True),
        # A render job over one resident library of 10 000 pictures: mosaics of 300 to 19 200 cells in one batch.
        "batch_uneven": {"kind": "batch", "mosaics": 64, "mix": 1, "cells_lo": 300, "cells_hi": 19200, "cell_px": 32,
                         "materials": 10000, "side": 128, "usage": 4, "strength": 0.4, "iterations": 5000, "chains": 8},
        # A handful of mosaics handed over in one call, host memory to host memory.
        "generate_batch": {"kind": "generate_batch", "mosaics": 12, "mix": 2, "cells_lo": 300, "cells_hi": 19200,
                           "cell_px": 32, "materials": 10000, "side": 128, "usage": 4, "strength": 0.4,
                           "iterations": 5000, "chains": 8},
        # A burst at the request loop, over 20 000 resident pictures.
        "served_burst": {"kind": "served", "mosaics": 32, "mix": 3, "cells_lo": 500, "cells_hi": 50000, "cell_px": 24,
                         "materials": 20000, "side": 128, "usage": 5, "strength": 0.4, "iterations": 2000, "chains": 4},
        # The colour statistics alone, for a host that owns its device memory (its pool, its stream).
        "cells_3840": {"kind": "cells", "target_w": 3840, "target_h": 2880, "blobs": 32, "grid_w": 80, "grid_h": 60},
        # Placement as a library call: colours known, no images, a library of 5000 pictures.
        "place_5000": {"kind": "place", "grid_w": 120, "grid_h": 90, "materials": 5000, "usage": 4, "weight": 0.25},
        # The optimiser as a library call on a placed grid.
        "optimize_80x60": {"kind": "optimize", "grid_w": 80, "grid_h": 60, "materials": 521, "iterations": 10000,
                           "chains": 16, "greedy_only": False},
    }
    return [{"name": name, **case} for name, case in named.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above; sizes spread over their logarithm, odd ones as likely as even ones."""
    kind = rng.choice(["generate"] * 5 + ["plan"] * 3 + ["batch", "generate_batch", "served", "cells", "cells", "place", "optimize"])
    if kind in ("generate", "plan"):
        gw = _log(rng, 12, 179)
        gh = max(6, int(gw * rng.uniform(0.6, 0.85)))
        px = _log(rng, 8, 48)
        side = _log(rng, 32, 256)
        aspects = rng.random() < 0.5
        # the filter keeps materials of the target's aspect: 4:3 ones need a 4:3 target, square ones any (the fallback)
        tw, th = gw * px + rng.randrange(px), 0
        th = int(tw * 0.75) if aspects else gh * px + rng.randrange(px)
        gh = min(gh, th)
        tile = _log(rng, 8, 48)
        return _job(kind, tw, th, rng.randrange(4, 65), _log(rng, 60, min(5000, 98304000 // (side * side))), side, aspects,
                    gw, gh, rng.randrange(1, 9), rng.choice([0.0, 0.4, 0.4, 1.0]), _log(rng, 100, 30000),
                    _log(rng, 1, 32), rng.choice([tile, tile + 1]), tile, rng.choice([0.0, 0.1, 0.25, 0.25]),
                    rng.choice(["host", "device", "area"]), rng.random() < 0.5, rng.choice(["cli", "cli", "gui"]),
                    rng.random() < 0.7, rng.choice([0, 0, 5, 16]))
    if kind in ("batch", "generate_batch", "served"):
        hi = _log(rng, 3000, 19200)
        return {"kind": kind, "mosaics": _log(rng, 2, 32 if kind == "batch" else 12), "mix": rng.randrange(1 << 20),
                "cells_lo": 300, "cells_hi": hi, "cell_px": rng.choice([16, 20, 24, 27, 32]),
                "materials": _log(rng, 400, 12000), "side": rng.choice([64, 96, 100, 128]), "usage": rng.randrange(2, 7),
                "strength": rng.choice([0.0, 0.4, 0.4, 1.0]), "iterations": _log(rng, 500, 5000), "chains": rng.randrange(1, 9)}
    if kind == "cells":
        gw, gh, px = _log(rng, 8, 179), _log(rng, 6, 134), _log(rng, 4, 64)
        px = max(1, min(px, 7680 // gw, 5760 // gh))
        return {"kind": kind, "target_w": gw * px + rng.randrange(px), "target_h": gh * px + rng.randrange(px),
                "blobs": rng.randrange(4, 65), "grid_w": gw, "grid_h": gh}
    if kind == "place":
        gw = _log(rng, 9, 220)
        return {"kind": kind, "grid_w": gw, "grid_h": max(5, int(gw * rng.uniform(0.6, 0.85))),
                "materials": _log(rng, 50, 20000), "usage": rng.randrange(1, 9), "weight": rng.choice([0.0, 0.1, 0.25])}
    gw = _log(rng, 12, 179)
    return {"kind": kind, "grid_w": gw, "grid_h": max(6, int(gw * 0.75)), "materials": _log(rng, 50, 5000),
            "iterations": _log(rng, 500, 50000), "chains": _log(rng, 1, 64), "greedy_only": rng.random() < 0.25}


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed & 0x7FFFFFFF)


def _target(w, h, blobs, g):
    """(h, w, 3) uint8 on the GPU."""
    r = torch.rand((blobs + 1, 6), generator=g, device="cuda").cpu().tolist()
    img = torch.empty((3, h, w), device="cuda")
    for c in range(3):
        img[c] = math.floor(256 * r[blobs][c])
    ys = torch.arange(h, device="cuda", dtype=torch.float32) + 0.5
    xs = torch.arange(w, device="cuda", dtype=torch.float32) + 0.5
    for b in range(blobs):
        cx, cy, sigma = r[b][0] * w, r[b][1] * h, 40.0 + 160.0 * r[b][2]
        x0, x1 = max(0, int(cx - 4 * sigma)), min(w, int(cx + 4 * sigma) + 1)
        y0, y1 = max(0, int(cy - 4 * sigma)), min(h, int(cy + 4 * sigma) + 1)
        if x1 <= x0 or y1 <= y0:
            continue
        a = torch.outer(torch.exp(-(ys[y0:y1] - cy) ** 2 / (2 * sigma * sigma)),
                        torch.exp(-(xs[x0:x1] - cx) ** 2 / (2 * sigma * sigma)))
        for c in range(3):
            img[c, y0:y1, x0:x1] += a * (math.floor(256 * r[b][3 + c]) - img[c, y0:y1, x0:x1])
    noise = torch.randint(-8, 9, (3, h, w), generator=g, device="cuda", dtype=torch.int8)
    return img.round_().add_(noise).clamp_(0, 255).to(torch.uint8).permute(1, 2, 0).contiguous()


def _host(t, pinned):
    """The GPU bytes as a host array: from mg_host_alloc or ordinary memory."""
    t = t.contiguous()
    if not pinned:
        return t.cpu().numpy()
    out = _pinned(t.numel()).reshape(t.shape)
    torch.from_numpy(out).copy_(t)
    return out


def _pinned(n):
    """n bytes of pinned memory, freed with the last array that looks at them."""
    lib = capi.load()
    addr = lib.mg_host_alloc(max(n, 16))
    if not addr:
        raise MemoryError("pinned allocation failed")
    buf = (C.c_uint8 * max(n, 16)).from_address(addr)
    weakref.finalize(buf, lib.mg_host_free, addr)
    return np.frombuffer(buf, np.uint8)[:n]


def _materials(n, side, aspects, g, pinned, thumb=None):
    """Packed host materials, and area thumbnails (n, th, tw, 3) when thumb = (tw, th)."""
    sel = torch.randint(0, 3, (n,), generator=g, device="cuda").cpu().numpy() if aspects else np.zeros(n, np.int64)
    w = np.where(sel == 2, side * 3 // 4, side).astype(np.int32)
    h = np.where(sel == 1, side * 3 // 4, side).astype(np.int32)
    off = np.zeros(n, np.int64)
    parts, thumbs, at = [], None, 0
    if thumb:
        thumbs = torch.empty((n, thumb[1], thumb[0], 3), dtype=torch.uint8, device="cuda")
    for s in range(3):
        ids = np.flatnonzero(sel == s)
        for j in range(0, len(ids), 1000):
            part = ids[j:j + 1000]
            m, pw, ph = len(part), int(w[part[0]]), int(h[part[0]])
            base = torch.randint(0, 256, (m, 3, 1, 1), generator=g, device="cuda").float()
            u = torch.rand((2, m, 1, 1, 1), generator=g, device="cuda")
            amp, ang = 32 * u[0], 2 * math.pi * u[1]
            xs = (torch.arange(pw, device="cuda") + 0.5 - pw / 2) / (max(pw, ph) / 2)
            ys = (torch.arange(ph, device="cuda") + 0.5 - ph / 2) / (max(pw, ph) / 2)
            img = base + amp * (torch.cos(ang) * xs + torch.sin(ang) * ys[:, None])
            noise = torch.randint(-16, 17, img.shape, generator=g, device="cuda", dtype=torch.int8)
            img = img.round_().add_(noise).clamp_(0, 255)
            if thumb:
                small = torch.nn.functional.adaptive_avg_pool2d(img, (thumb[1], thumb[0])).round_().to(torch.uint8)
                thumbs[torch.from_numpy(part).cuda()] = small.permute(0, 2, 3, 1)
            size = pw * ph * 3
            flat = torch.zeros((m, (size + 15) // 16 * 16), dtype=torch.uint8, device="cuda")
            flat[:, :size] = img.to(torch.uint8).permute(0, 2, 3, 1).reshape(m, size)
            off[part] = at + np.arange(m, dtype=np.int64) * flat.shape[1]
            at += flat.numel()
            parts.append(flat.reshape(-1))
    mats = synth.Materials(_host(torch.cat(parts), pinned), off, w, h)
    return mats, (_host(thumbs, pinned) if thumb else None)


def _lab(n, g):
    """Lab colours of n uniform sRGB colours, from ordinary float arithmetic (host array)."""
    rgb = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
    return _rgb_to_lab64(rgb).float().cpu().numpy()


def _rgb_to_lab64(v):
    """sRGB in [0, 1] to CIE 1976 Lab (D65), last dimension RGB, 64 bits."""
    lin = torch.where(v <= 0.04045, v / 12.92, ((v + 0.055) / 1.055) ** 2.4)
    prim = np.array([[0.64, 0.33], [0.30, 0.60], [0.15, 0.06]])
    white = np.array([0.95047, 1.0, 1.08883])
    xyz = np.stack([prim[:, 0] / prim[:, 1], np.ones(3), (1 - prim[:, 0] - prim[:, 1]) / prim[:, 1]])
    m = xyz * np.linalg.solve(xyz, white)[None, :] / white[:, None]
    t = lin @ torch.from_numpy(m.T.copy()).to(v)
    f = torch.where(t > 216 / 24389, t.clamp_min(1e-9) ** (1 / 3), (24389 / 27 * t + 16) / 116)
    return torch.stack([116 * f[..., 1] - 16, 500 * (f[..., 0] - f[..., 1]), 200 * (f[..., 1] - f[..., 2])], -1)


def _smooth_lab(gw, gh, g):
    """Cell colours of a smooth picture (a coarse random colour field enlarged, with a little noise)."""
    coarse = torch.rand((1, 3, max(2, gh // 12), max(2, gw // 12)), generator=g, device="cuda")
    field = torch.nn.functional.interpolate(coarse, size=(gh, gw), mode="bicubic", align_corners=False)[0]
    field = (field + 0.01 * torch.randn(field.shape, generator=g, device="cuda")).clamp(0, 1)
    return _rgb_to_lab64(field.permute(1, 2, 0).reshape(-1, 3).double()).float().cpu().numpy()


def _grids(case):
    """Grid widths and heights of a mix of mosaics: cells log-uniform, aspect 4:3."""
    rng = np.random.default_rng(case["mix"])
    cells = np.exp(rng.uniform(math.log(case["cells_lo"]), math.log(case["cells_hi"]), case["mosaics"]))
    gw = np.maximum(8, np.sqrt(cells * 4 / 3).round().astype(int))
    return [(int(a), max(1, int(round(a * 3 / 4)))) for a in gw]


class _State:
    """What a program holds between calls; closed in the order server / batch / plan, palette, context."""

    def __init__(self):
        self.closing = []

    def __del__(self):
        try:
            for obj in self.closing:
                obj.close()
        except Exception:
            pass


def _context(case):
    ctx = capi.Context(0)
    if case.get("scoring") == "gui":
        ctx.set_scoring(capi.MG_SCORING_GUI)
    if case.get("thumbs") == "area":
        capi.check(ctx.lib.mg_ctx_set_thumbnail_filter(ctx.h, capi.MG_THUMB_AREA))
    return ctx


def _prepare_job(case, seed, s, g):
    tw = case["tile_w"] or case["target_w"] // case["grid_w"]
    th = case["tile_h"] or case["target_h"] // case["grid_h"]
    t = _target(case["target_w"], case["target_h"], case["blobs"], g)
    stride = 3 * case["target_w"] + case["row_pad"]
    rows = torch.zeros((case["target_h"], stride), dtype=torch.uint8, device="cuda")
    rows[:, :3 * case["target_w"]] = t.reshape(case["target_h"], -1)
    target = _host(rows, case["pinned"])
    mats, thumbs = _materials(case["materials"], case["side"], case["aspects"], g, case["pinned"],
                              (tw, th) if case["thumbs"] == "host" else None)
    cfg = job.JobConfig(case["kind"], case["target_w"], case["target_h"], case["blobs"], case["materials"], case["side"],
                        int(case["aspects"]), case["grid_w"], case["grid_h"], case["usage"], case["weight"],
                        case["strength"], case["iterations"], case["chains"], case["tile_w"], case["tile_h"],
                        seed=seed, build_similarity=case["similarity"], device_thumbnails=case["thumbs"] != "host")
    s.holder = job.RequestHolder(job.Inputs(cfg, target, mats, thumbs))
    s.image = (_pinned(case["grid_h"] * th * case["grid_w"] * tw * 3) if case["pinned"]
               else np.zeros(case["grid_h"] * th * case["grid_w"] * tw * 3, np.uint8)).reshape(s.holder.out_shape())
    s.grid = np.zeros(case["grid_w"] * case["grid_h"], np.int32)
    s.ctx = _context(case)
    if case["kind"] == "plan":
        s.plan = job.Plan(s.ctx, s.holder)
        s.closing.append(s.plan)
    s.closing.append(s.ctx)


def _prepare_many(case, seed, s, g):
    px, grids = case["cell_px"], _grids(case)
    s.ctx = _context(case)
    mats, _ = _materials(case["materials"], case["side"], False, g, False)
    s.palette = job.Palette(s.ctx, mats, None, px, px, 1.0)
    on_host = case["kind"] != "batch"
    s.targets = [_target(gw * px, gh * px, 8, g) for gw, gh in grids]
    if on_host:
        s.targets = [_host(t, True) for t in s.targets]
    s.requests = [job.mosaic_request(t if on_host else t.data_ptr(), gw * px, gh * px, gw, gh, max_usage=case["usage"],
                                     strength=case["strength"], iterations=case["iterations"], chains=case["chains"],
                                     seed=seed, stream=i) for i, (t, (gw, gh)) in enumerate(zip(s.targets, grids))]
    cells = sum(gw * gh for gw, gh in grids)
    s.image = _pinned(cells * px * px * 3)
    s.grid = np.zeros(cells, np.int32)
    s.views, at = [], 0
    for gw, gh in grids:
        n = gw * gh
        s.views.append((s.grid[at:at + n], s.image[at * px * px * 3:(at + n) * px * px * 3].reshape(gh * px, gw * px, 3)))
        at += n
    if case["kind"] == "batch":
        torch.cuda.synchronize()  # the batch copies the targets on the context's own stream
        s.batch = job.Batch(s.ctx, s.palette, s.requests)
        s.closing.append(s.batch)
        s.targets = None
    elif case["kind"] == "served":
        s.server = job.Server(s.ctx, s.palette)
        s.closing.append(s.server)
    s.closing += [s.palette, s.ctx]


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    g = _generator(seed)
    if s.kind in ("generate", "plan"):
        _prepare_job(case, seed, s, g)
    elif s.kind in ("batch", "generate_batch", "served"):
        _prepare_many(case, seed, s, g)
    elif s.kind == "cells":
        s.w, s.h, s.gw, s.gh = case["target_w"], case["target_h"], case["grid_w"], case["grid_h"]
        s.img = _target(s.w, s.h, case["blobs"], g)
        s.lab = torch.zeros((s.gw * s.gh, 4), device="cuda")
        s.rgb = torch.zeros((s.gw * s.gh, 4), dtype=torch.uint8, device="cuda")
        s.lib = capi.load()
    elif s.kind == "place":
        s.ctx = _context(case)
        s.closing.append(s.ctx)
        s.palette_lab = _lab(case["materials"], g)
        s.cell_lab = _smooth_lab(case["grid_w"], case["grid_h"], g)
        s.case = case
    else:
        s.ctx = _context(case)
        s.closing.append(s.ctx)
        s.palette_lab = _lab(case["materials"], g)
        # a placed grid: each cell holds one of the 8 materials nearest its colour
        near = torch.cdist(torch.from_numpy(_smooth_lab(case["grid_w"], case["grid_h"], g)).cuda(),
                           torch.from_numpy(s.palette_lab).cuda()).topk(min(8, case["materials"]), largest=False).indices
        pick = torch.randint(0, near.shape[1], (near.shape[0], 1), generator=g, device="cuda")
        s.start = near.gather(1, pick).reshape(case["grid_h"], case["grid_w"]).to(torch.int32).cpu().numpy()
        s.case, s.seed = case, seed
    return s


# ---- one pass -------------------------------------------------------------------------------------------------------
def _numbers(r):
    return [r.palette_size, r.n_resets, r.best_chain, r.initial_cost, r.final_cost, r.best_cost, r.accepted_count,
            r.improved_count]


def _summary(results):
    """The scalar results of several mosaics, one array per field."""
    rows = [_numbers(r) for r in results]
    return [np.array(col, np.float32 if isinstance(col[0], float) else np.int64) for col in zip(*rows)]


def run(s):
    if s.kind == "generate":
        res, grid, image = job.generate(s.ctx, s.holder, s.image, s.grid)
        return {"grid": grid, "image": image, "result": _numbers(res)}
    if s.kind == "plan":
        s.plan.run()
        res, grid, image = s.plan.read(s.image, s.grid)
        return {"grid": grid, "image": image, "result": _numbers(res)}
    if s.kind == "batch":
        s.batch.run()
        results = []
        for i, (grid, image) in enumerate(s.views):
            r = capi.Result()
            r.grid, r.image = capi.ptr(grid, C.c_int32), capi.ptr(image, C.c_uint8)
            capi.check(s.ctx.lib.mg_batch_read(s.batch.h, i, C.byref(r)))
            results.append(r)
        return {"grid": s.grid, "image": s.image, "result": _summary(results)}
    if s.kind == "generate_batch":
        results, _, _ = job.generate_batch(s.ctx, s.palette, s.requests, s.views)
        return {"grid": s.grid, "image": s.image, "result": _summary(results)}
    if s.kind == "served":
        tickets = [s.server.submit(m, grid, image) for m, (grid, image) in zip(s.requests, s.views)]
        results = []
        for t in tickets:
            status, r, _ = s.server.wait(t)
            capi.check(status)
            results.append(r)
        return {"grid": s.grid, "image": s.image, "result": _summary(results)}
    if s.kind == "cells":
        capi.check(s.lib.mg_cells_lab_noalloc(s.img.data_ptr(), s.w, s.h, 3 * s.w, s.gw, s.gh, s.lab.data_ptr(),
                                              s.rgb.data_ptr(), torch.cuda.current_stream().cuda_stream))
        return {"lab": s.lab, "rgb": s.rgb}
    if s.kind == "place":
        grid, resets = s.ctx.place_greedy(s.palette_lab, s.cell_lab, s.case["grid_w"], s.case["grid_h"], s.case["usage"],
                                          s.case["weight"])
        return {"grid": grid, "resets": resets}
    grid, best, per, grids = s.ctx.optimize(s.palette_lab, s.start, s.case["iterations"], chains=s.case["chains"],
                                            seed=s.seed, greedy_only=s.case["greedy_only"])
    rows = [[r.initial_cost, r.final_cost, r.best_cost] for r in [best] + per]
    counts = [[r.improved_count, r.accepted_count, r.iterations, r.best_chain] for r in [best] + per]
    return {"grid": grid, "chain_grids": grids, "costs": np.array(rows, np.float32), "counts": np.array(counts, np.int64)}


def exact(case, seed):
    """The cell Lab means in 64 bits.  The other kinds return whole numbers and bytes, and costs that follow from a
    sequence of accept / reject decisions and have no value of their own in other arithmetic."""
    if case["kind"] != "cells":
        return None
    img = _target(case["target_w"], case["target_h"], case["blobs"], _generator(seed))
    gw, gh = case["grid_w"], case["grid_h"]
    cw, ch = case["target_w"] // gw, case["target_h"] // gh
    out = torch.zeros((gh, gw, 4), dtype=torch.float64, device="cuda")
    for y in range(gh):
        rows = img[y * ch:(y + 1) * ch, :gw * cw].double() / 255
        out[y, :, :3] = _rgb_to_lab64(rows).reshape(ch, gw, cw, 3).mean(dim=(0, 2))
    return {"lab": out.reshape(-1, 4), "rgb": None}


# ---- the least a pass moves and computes ----------------------------------------------------------------------------
def work(case):
    """Bytes: each input read once, each output written once.  Operations: about 60 a pixel for sRGB -> Lab, 60 an
    adjusted output pixel, 8 a candidate looked at, 100 an annealing proposal."""
    kind = case["kind"]
    if kind == "cells":
        n = case["grid_w"] * case["grid_h"]
        px = (case["target_w"] // case["grid_w"]) * (case["target_h"] // case["grid_h"]) * n
        return {"bytes": 3 * px + 20 * n, "flops": 60 * px}
    if kind == "place":
        n = case["grid_w"] * case["grid_h"]
        return {"bytes": 12 * (n + case["materials"]) + 4 * n, "flops": 8 * n * min(K_CANDIDATES, case["materials"])}
    if kind == "optimize":
        n = case["grid_w"] * case["grid_h"]
        return {"bytes": 12 * case["materials"] + 4 * n * (2 + case["chains"]), "flops": 100 * case["iterations"] * case["chains"]}
    if kind in ("generate", "plan"):
        n = case["grid_w"] * case["grid_h"]
        tw = case["tile_w"] or case["target_w"] // case["grid_w"]
        th = case["tile_h"] or case["target_h"] // case["grid_h"]
        side = case["side"]
        kept, area = (case["materials"] / 3, side * (side * 3 // 4)) if case["aspects"] else (case["materials"], side * side)
        px = case["target_w"] * case["target_h"] + kept * area
        out = n * tw * th
        fixed = 3 * px + 3 * kept * tw * th
    else:
        n = sum(a * b for a, b in _grids(case))
        kept = case["materials"]
        px = out = n * case["cell_px"] ** 2
        fixed = 3 * px + 3 * min(kept, n) * case["cell_px"] ** 2
    jobs = case.get("mosaics", 1)
    adjusted = out if case["strength"] > 0 else 0
    return {"bytes": fixed + 3 * out + 4 * n,
            "flops": 60 * px + 60 * adjusted + 8 * n * min(K_CANDIDATES, kept) + 100 * case["iterations"] * case["chains"] * jobs}
