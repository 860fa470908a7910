"""Performance cases of the AV1 post-decode filter library, through its public
entry points.

A case is a dict of plain values:
  kind      "chain"   one frame, vaco_av1_postfilter_frame_dev, status read per call
            "stream"  `frames` frames back to back under deferred status, one flush
            "batch"   `frames` frames of the mix in one vaco_av1_postfilter_batch_dev
            "host"    one frame from page-locked host memory and back,
                      vaco_av1_postfilter_frame_host
            "stages"  one frame function by function: deblock_picture, cdef_picture,
                      restore_plane of every plane
            "grain"   film grain synthesis of one output frame
            "emit"    frame emission (u16 planes packed into an output frame)
  width, height, depth, upscaled, layout ("420", "422", "444", "400")
  lr        restoration: "all" planes, "luma" only, "none"
  lr_unit   restoration unit size
  deblock, level_map, frames, lag (film grain) where the kind uses them

Every output is whole samples of planes (AV1's filters are defined bit by
bit), so outputs compare for equality and there is no 64-bit value to give.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from vaco_b200 import abi, synth
from vaco_b200._lib import lib
from vaco_b200.frame import FrameInputs, picture_struct, pinned_copy
from vaco_b200.gpu import Context, DeviceFrame

LAYOUTS = {"420": (1, 1), "422": (1, 0), "444": (0, 0), "400": (1, 1)}


def _case(kind, width, height, depth, **more):
    c = {"kind": kind, "width": width, "height": height, "depth": depth, "upscaled": width, "layout": "420",
         "lr": "all", "lr_unit": 64, "deblock": True, "level_map": False, "frames": 1, "lag": 3}
    c.update(more)
    return c


def listed():
    cases = {
        # a thumbnail or conference tile, one call per frame: launch latency
        "chain_360p_8bit": _case("chain", 640, 360, 8),
        # a web rendition whose sides are no multiple of the 64-sample tile,
        # per-superblock filter levels, restoration on luma alone
        "chain_854x478_10bit_levels": _case("chain", 854, 478, 10, lr="luma", lr_unit=128, level_map=True),
        # ordinary HD HDR playback, one call per frame
        "chain_1080p_10bit": _case("chain", 1920, 1080, 10),
        # screen content and mezzanine files: full chroma, 12 bits, odd extents
        "chain_1365x767_12bit_444": _case("chain", 1365, 767, 12, layout="444", lr_unit=256),
        # CDEF as the only filter that is on
        "cdef_1080p_8bit": _case("chain", 1920, 1080, 8, lr="none", deblock=False),
        # super-resolution to 4K
        "superres_2880to3840_10bit": _case("chain", 2880, 2160, 10, upscaled=3840),
        # a transcoder's 4K frames, enqueued back to back
        "stream_4k_10bit": _case("stream", 3840, 2160, 10, frames=4),
        # a server's frames of many streams in one launch set
        "batch_mix_16": _case("batch", 3840, 2160, 10, frames=16),
        # the drop-in call of a decoder that keeps its frames in host memory
        "host_1080p_10bit": _case("host", 1920, 1080, 10),
        # a decoder that replaces its filters one function at a time
        "stages_1080p_10bit": _case("stages", 1920, 1080, 10),
        # film grain before display
        "grain_4k_10bit": _case("grain", 3840, 2160, 10),
        # the output frame of a 4K decode
        "emit_4k_10bit": _case("emit", 3840, 2160, 10),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def draw(rng):
    kind = rng.choice(["chain"] * 6 + ["stream", "batch", "host", "stages", "grain", "emit"])
    depth = rng.choice([8, 8, 10, 10, 10, 12])
    layout = rng.choice(["420"] * 5 + ["422", "444", "400"])
    top = {"batch": 1920, "stream": 2560, "host": 2560}.get(kind, 3840)
    width = int(round(math.exp(rng.uniform(math.log(320), math.log(top)))))
    height = max(176, int(round(width * rng.choice([9 / 16, 9 / 16, 3 / 4, 1 / 2.39]))) + rng.randint(-3, 3))
    if layout in ("420", "422", "400"):
        width &= ~1
    if layout in ("420", "400"):
        height &= ~1
    upscaled = width
    if kind in ("chain", "stream") and rng.random() < 0.2:
        upscaled = min(3840, int(width * rng.randint(9, 16) / 8)) & ~1
        upscaled = max(upscaled, width)
    return _case(kind, width, height, depth, upscaled=upscaled, layout=layout,
                 lr=rng.choice(["all", "all", "luma", "none"]), lr_unit=rng.choice([64, 64, 128, 256]),
                 deblock=rng.random() < 0.9, level_map=rng.random() < 0.4, lag=rng.choice([3, 3, 2, 1, 0]),
                 frames=rng.randint(2, 6) if kind == "stream" else rng.randint(4, 12) if kind == "batch" else 1)


# ---------------------------------------------------------------- inputs

def _content(gen, rows, cols, depth):
    """A plane of three sinusoids and N(0, 4) noise (in 8-bit units): the
    content model of vaco_b200.synth, drawn on the GPU."""
    dev = gen.device
    u = torch.rand(3, 4, generator=gen, device=dev).cpu().numpy().astype(np.float64)
    ys = torch.arange(rows, device=dev, dtype=torch.float32)[:, None]
    xs = torch.arange(cols, device=dev, dtype=torch.float32)[None, :]
    acc = torch.randn(rows, cols, generator=gen, device=dev).mul_(4.0).add_(128.0)
    amps = u[:, 0] / u[:, 0].sum() * 112.0
    for k in range(3):
        period, theta, phase = 32.0 + 480.0 * u[k, 1], math.pi * u[k, 2], 2 * math.pi * u[k, 3]
        fy, fx = 2 * math.pi * math.sin(theta) / period, 2 * math.pi * math.cos(theta) / period
        acc += float(amps[k]) * torch.sin(xs * fx + ys * fy + phase)
    top = (1 << depth) - 1
    return (acc * (top / 255.0)).round_().clamp_(0, top).to(torch.int16)


def _frame(c, seed):
    """One frame's inputs: reconstruction planes and the side information a
    decoder holds when it reaches the post-filters."""
    ssx, ssy = LAYOUTS[c["layout"]]
    mono = c["layout"] == "400"
    w, h = c["width"], c["height"]
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    mi_cols, mi_rows = 2 * ((w + 7) >> 3), 2 * ((h + 7) >> 3)
    planes = []
    for k in range(1 if mono else 3):
        sx, sy = (ssx, ssy) if k else (0, 0)
        planes.append(_content(gen, (mi_rows * 4) >> sy, (mi_cols * 4) >> sx, c["depth"]).cpu().numpy().view(np.uint16))
    tx_l, tx_c = synth.tx_maps(rng, mi_rows, mi_cols, ssx, ssy)
    skip8 = (rng.random((mi_rows // 2, mi_cols // 2)) < 0.2).astype(np.uint8)
    sb = ((mi_rows + 15) // 16, (mi_cols + 15) // 16)
    levels = [int(v) for v in rng.integers(1, 64, 4)] if c["deblock"] else [0, 0, 0, 0]
    lvl_map = None
    if c["level_map"]:
        per_sb = np.clip(np.array(levels)[None, None, :] + rng.integers(-8, 9, size=(*sb, 1)), 0, 63)
        lvl_map = np.repeat(np.repeat(per_sb, 16, 0), 16, 1)[:mi_rows, :mi_cols].astype(np.uint8).copy()
    f = FrameInputs(
        bit_depth=c["depth"], coded_width=w, coded_height=h, upscaled_width=c["upscaled"], planes=planes,
        tx_luma=tx_l, tx_chroma=tx_c, skip=np.repeat(np.repeat(skip8, 2, 0), 2, 1).copy(),
        cdef_idx=rng.integers(0, 8, size=sb).astype(np.int32), subsampling_x=ssx, subsampling_y=ssy, monochrome=mono,
        lvl_map=lvl_map, deblock_levels=levels, sharpness=int(rng.integers(0, 8)), cdef=synth.cdef_settings(rng))
    on = [c["lr"] == "all" or (c["lr"] == "luma" and k == 0) for k in range(3)]
    f.lr_type = tuple(abi.FRAME_LR_SWITCHABLE if v else abi.FRAME_LR_NONE for v in on)
    f.lr_unit_size = (c["lr_unit"],) * 3
    f.lr_units = []
    for k in range(f.num_planes):
        rows, cols = f.output_shape(k)
        f.lr_units.append(synth.lr_units(rng, cols, rows, c["lr_unit"], k > 0) if on[k] else None)
    return f


def _frame_cases(c):
    """The single frames of a case.  A batch takes the server mix in turn: the
    case's own size, then half, a third and a sixth of it."""
    if c["kind"] != "batch":
        return [c] * c["frames"]
    got = []
    for i in range(c["frames"]):
        d = (1, 2, 3, 6)[i % 4]
        s = dict(c, width=max(64, c["width"] // d) & ~1, height=max(64, c["height"] // d) & ~1)
        s["upscaled"] = s["width"]
        s["depth"] = c["depth"] if i % 4 < 2 else 8
        got.append(s)
    return got


def _grain_params(c, rng):
    """Parameters as an encoder's grain table has them: 8 luma and 4 + 4
    chroma points, small auto-regression taps, overlap on."""
    p = abi.FilmGrainParams()
    p.apply_grain, p.grain_seed, p.overlap_flag = 1, int(rng.integers(1, 65536)), 1
    for n, v, sc in ((8, p.point_y_value, p.point_y_scaling), (4, p.point_cb_value, p.point_cb_scaling),
                     (4, p.point_cr_value, p.point_cr_scaling)):
        for i, x in enumerate(np.sort(rng.choice(256, n, replace=False))):
            v[i], sc[i] = int(x), int(rng.integers(16, 128))
    p.num_y_points, p.num_cb_points, p.num_cr_points = 8, 4, 4
    p.grain_scaling_minus_8, p.ar_coeff_lag, p.ar_coeff_shift_minus_6 = 3, c["lag"], 1
    for arr, n in ((p.ar_coeffs_y_plus_128, 24), (p.ar_coeffs_cb_plus_128, 25), (p.ar_coeffs_cr_plus_128, 25)):
        for i in range(n):
            arr[i] = int(np.clip(128 + rng.normal(0, 12), 0, 255))
    p.cb_mult, p.cb_luma_mult, p.cb_offset = 128, 192, 256
    p.cr_mult, p.cr_luma_mult, p.cr_offset = 128, 192, 256
    return p


@functools.lru_cache(maxsize=None)
def _context(deferred):
    """The program's library handles: one that reads each call's status, one
    that enqueues frames and reads the status at the flush."""
    ctx = Context(torch.cuda.current_device())
    if deferred:
        ctx.set_deferred_status(True)
    return ctx


def _picture(tensors):
    return picture_struct([t.data_ptr() for t in tensors], [tuple(t.shape) for t in tensors])


def prepare(case, seed):
    c = case
    if c["kind"] in ("grain", "emit"):
        ssx, ssy = LAYOUTS[c["layout"]]
        mono = c["layout"] == "400"
        w, h = c["upscaled"], c["height"]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        info = abi.FrameInfo()
        info.bit_depth, info.subsampling_x, info.subsampling_y, info.monochrome = c["depth"], ssx, ssy, int(mono)
        info.coded_width = info.upscaled_width = w
        info.coded_height = h
        info.mi_cols, info.mi_rows = 2 * ((w + 7) >> 3), 2 * ((h + 7) >> 3)
        # a decoder's picture: rows padded to 64 samples
        shapes = [(h, w)] + ([] if mono else [((h + ssy) >> ssy, (w + ssx) >> ssx)] * 2)
        src = [_content(gen, r, (k + 63) // 64 * 64, c["depth"]) for r, k in shapes]
        pin = picture_struct([t.data_ptr() for t in src], shapes, [t.shape[1] for t in src])
        s = {"case": c, "ctx": _context(False), "info": info, "src": src, "pin": pin}
        if c["kind"] == "grain":
            rng = np.random.Generator(np.random.PCG64(seed))
            s["params"] = _grain_params(c, rng)
            s["gauss"] = np.clip(np.rint(rng.normal(0, 512, 2048)), -2048, 2047).astype(np.int16)
            s["out"] = [torch.zeros_like(t) for t in src]
            s["pout"] = picture_struct([t.data_ptr() for t in s["out"]], shapes, [t.shape[1] for t in src])
        else:
            size = 2 if c["depth"] > 8 else 1
            s["out"] = [torch.zeros(r, (k * size + 63) // 64 * 64, dtype=torch.uint8, device="cuda") for r, k in shapes]
            fb = abi.FrameBuffer()
            for k, t in enumerate(s["out"]):
                fb.planes[k], fb.linesize[k] = t.data_ptr(), t.shape[1]
            s["frame"] = fb
        return s
    frames = [_frame(fc, seed * 64 + i) for i, fc in enumerate(_frame_cases(c))]
    if c["kind"] == "host":
        pf, outs, job = _pinned(frames[0])
        return {"case": c, "ctx": _context(False), "frame": pf, "out": outs, "job": job}
    dev = [DeviceFrame(f, torch.cuda.current_device()) for f in frames]
    s = {"case": c, "ctx": _context(c["kind"] == "stream"), "dev": dev}
    if c["kind"] == "batch":
        s["jobs"] = s["ctx"].batch_jobs(dev)
    if c["kind"] == "stages":
        s["deblocked"] = [torch.empty_like(t) for t in dev[0].planes]
        s["cdef"] = [torch.empty_like(t) for t in dev[0].planes]
    return s


def _pinned(f):
    """pinned_copy() of a frame some of whose planes have no units."""
    units = f.lr_units
    f.lr_units = [u if u is not None else np.zeros(1, abi.lr_unit_dtype()) for u in units]
    return pinned_copy(f)


# ---------------------------------------------------------------- one pass

def _ok(status, msg):
    if status != abi.OK:
        raise RuntimeError(abi.MESSAGES.get(msg.value, "failed"))


def _run_stages(s):
    """decode_frame's filter tail, one library function per filter."""
    ctx, d, l, m = s["ctx"], s["dev"][0], lib(), C.c_int32()
    f, job = d.f, d.job
    before, after = _picture(s["deblocked"]), _picture(s["cdef"])
    info, db, cdef = job.info, job.deblock, job.cdef
    _ok(l.vaco_av1_deblock_picture_dev(ctx.handle, None, C.byref(job.src), C.byref(before), C.byref(info), job.tx_luma,
                                       job.tx_chroma, job.lvl_map, C.byref(db), C.byref(m)), m)
    _ok(l.vaco_av1_cdef_picture_dev(ctx.handle, None, C.byref(before), C.byref(after), C.byref(info), job.skip,
                                    job.cdef_idx, job.cdef_stride, job.cdef_count, C.byref(cdef), C.byref(m)), m)
    for k in range(f.num_planes):
        if job.lr_type[k] == abi.FRAME_LR_NONE:
            continue
        rows, cols = f.output_shape(k)
        p, q, o = s["deblocked"][k], s["cdef"][k], d.outputs[k]
        cfg = abi.LrPlaneConfig(cols, rows, f.bit_depth, job.lr_unit_size[k], f.plane_sub(k)[1])
        _ok(l.vaco_av1_restore_plane_dev(ctx.handle, None, p.data_ptr(), p.shape[1], p.shape[0], p.shape[1],
                                         q.data_ptr(), q.shape[1], q.shape[0], q.shape[1], C.byref(cfg),
                                         job.lr_units[k], job.lr_unit_count[k], o.data_ptr(), o.shape[1],
                                         C.byref(m)), m)
    return [s["deblocked"], s["cdef"], d.outputs]


def run(state):
    s = state
    kind, ctx, m = s["case"]["kind"], s["ctx"], C.c_int32()
    if kind == "chain":
        ctx.postfilter_frame_dev(s["dev"][0])
        return s["dev"][0].outputs
    if kind == "stream":
        for d in s["dev"]:
            ctx.postfilter_frame_dev(d)
        ctx.flush()
        return [d.outputs for d in s["dev"]]
    if kind == "batch":
        statuses, _ = ctx.postfilter_batch_dev(s["dev"], jobs=s["jobs"])
        if any(statuses):
            raise RuntimeError("a frame of the batch failed")
        return [d.outputs for d in s["dev"]]
    if kind == "host":
        _ok(lib().vaco_av1_postfilter_frame_host(ctx.handle, C.byref(s["job"]), C.byref(m)), m)
        return s["out"]
    if kind == "stages":
        return _run_stages(s)
    if kind == "grain":
        _ok(lib().vaco_av1_film_grain_dev(ctx.handle, None, C.byref(s["pin"]), C.byref(s["pout"]), C.byref(s["info"]),
                                          C.byref(s["params"]), s["gauss"].ctypes.data, C.byref(m)), m)
        return s["out"]
    _ok(lib().vaco_av1_emit_frame_dev(ctx.handle, None, C.byref(s["pin"]), C.byref(s["info"]), C.byref(s["frame"]),
                                      C.byref(m)), m)
    return s["out"]


# ---------------------------------------------------------------- what a pass cannot do without

def _samples(c, width, padded):
    ssx, ssy = LAYOUTS[c["layout"]]
    h = c["height"]
    if padded:
        width, h = (width + 7) // 8 * 8, (h + 7) // 8 * 8
    chroma = 0 if c["layout"] == "400" else 2 * ((width + ssx) >> ssx) * ((h + ssy) >> ssy)
    return width * h + chroma


def _side_bytes(c):
    """Transform sizes, levels and skip flags per 4x4 cell, restoration units."""
    ssx, ssy = LAYOUTS[c["layout"]]
    cells = 4 * ((c["width"] + 7) // 8) * ((c["height"] + 7) // 8)
    n = cells * 2
    if c["layout"] != "400":
        n += cells >> (ssx + ssy)
    if c["level_map"]:
        n += 4 * cells
    if c["lr"] != "none":
        n += 20 * (_samples(c, c["upscaled"], False) // c["lr_unit"] ** 2)
    return n


def work(case):
    """Input planes and side information read once, outputs written once (the
    function-by-function form: each function's).  The arithmetic is integer
    throughout; it is not counted as floating-point operations."""
    c = case
    out = 2 * _samples(c, c["upscaled"], False)
    if c["kind"] == "grain":
        return {"bytes": 2 * out, "flops": 0}
    if c["kind"] == "emit":
        return {"bytes": out + (out if c["depth"] > 8 else out // 2), "flops": 0}
    total = 0
    for f in _frame_cases(c):
        total += 2 * _samples(f, f["width"], True) + 2 * _samples(f, f["upscaled"], False) + _side_bytes(f)
    if c["kind"] == "stages":
        padded = 2 * _samples(c, c["width"], True)
        total = 4 * padded + _side_bytes(c)
        if c["lr"] != "none":
            total += padded + out
    return {"bytes": total, "flops": 0}
