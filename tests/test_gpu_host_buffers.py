"""The synchronous host call by the caller's buffers: page-locked frames in as
many bands as their size gives, with copies in, filters and copies out truly at
once, and pageable ones in one band.  The bands are counted by the launches of a
frame without restoration, one a band that completes a row of tiles."""
import ctypes as C

import numpy as np
import pytest

import oracle
from vaco_b200 import abi, synth
from vaco_b200._lib import lib
from vaco_b200.frame import alloc_outputs, host_job
from vaco_b200.gpu import Context

pytestmark = pytest.mark.gpu


def pinned(shape, stride=None):
    import torch

    t = torch.zeros(shape[0], stride or shape[1], dtype=torch.int16, pin_memory=True)
    return t.numpy().view(np.uint16)[:, : shape[1]]


class HostFrame:
    """A frame's host job; `pin`: which sides are page-locked, `pad`: samples
    by which rows are longer than the planes are wide."""

    def __init__(self, f, pin="both", pad=0):
        self.f, self.outs = f, alloc_outputs(f)
        self.job = host_job(f, self.outs)
        self.keep = []
        if pin in ("both", "src"):
            for k in range(f.num_planes):
                a = pinned(f.planes[k].shape, f.planes[k].shape[1] + pad)
                a[:] = f.planes[k]
                self.keep.append(a)
                self.job.src.planes[k], self.job.src.stride[k] = a.ctypes.data, a.strides[0] // 2
        if pin in ("both", "dst"):
            self.outs = [pinned(o.shape, o.shape[1] + pad) for o in self.outs]
            for k, o in enumerate(self.outs):
                self.job.dst.planes[k], self.job.dst.stride[k] = o.ctypes.data, o.strides[0] // 2

    def run(self, ctx):
        """Status, message and the kernels launched."""
        m, before = C.c_int32(), ctx.launches
        for o in self.outs:
            o[:] = 0xABCD
        st = lib().vaco_av1_postfilter_frame_host(ctx.handle, C.byref(self.job), C.byref(m))
        return st, m.value, ctx.launches - before

    def check(self, ctx, threads):
        want, m = oracle.postfilter_frame(self.f, threads=threads)
        assert m == 0
        st, m, launches = self.run(ctx)
        assert (st, m) == (abi.OK, 0)
        for k, (g, w) in enumerate(zip(self.outs, want)):
            assert np.array_equal(g, w), f"plane {k}: {int((g != w).sum())} samples differ"
        return launches


def no_restoration(f):
    f.lr_type, f.lr_units = (abi.FRAME_LR_NONE,) * 3, []
    return f


def filter_launches(f):
    """The bands that complete a row of 64x64 tiles: one band per 2.5 MB of
    input, 5 and the tile rows at most, each a smaller share of the rows."""
    rows = -(-f.mi_rows // 16)
    size = sum(2 * p.size for p in f.planes[: f.num_planes])
    bands = min(size // (5 << 19) + 1, 5, rows)
    n = start = done = 0
    for b in range(bands):
        rest = (bands - 1 - b) ** 2
        start = min(max(start + 1, rows - rows * rest // bands**2), rows - (bands - 1 - b))
        to = rows if b == bands - 1 else start - 1
        n, done = n + (to > done), max(done, to)
    return n


# 4:2:0 in 2, 3, 4 and 5 bands, in one a tile row (3), then in 3 at 8 and 12 bits
SIZES = [(1600, 902, 10), (1918, 1078, 10), (2046, 1370, 10), (2562, 1438, 10), (20000, 130, 10), (1922, 1082, 8),
         (1366, 1534, 12)]


@pytest.mark.parametrize("size", SIZES, ids=lambda s: f"{s[0]}x{s[1]}-{s[2]}")
@pytest.mark.parametrize("pad", [0, 24])
def test_page_locked_frames_in_bands(ctx, size, pad, oracle_threads):
    f = synth.make_small(7, *size, lr_unit=64 if pad else 128, with_lvl_map=True)
    HostFrame(f, pad=pad).check(ctx, oracle_threads)
    f.lr_type, f.lr_units = (abi.FRAME_LR_SWITCHABLE, abi.FRAME_LR_NONE, abi.FRAME_LR_NONE), f.lr_units[:1]
    HostFrame(f, pad=pad).check(ctx, oracle_threads)
    want = filter_launches(f)
    assert want > 1
    assert HostFrame(no_restoration(f), pad=pad).check(ctx, oracle_threads) == want


@pytest.mark.parametrize("layout", [(1, 0, False), (0, 0, False), (1, 1, True)], ids=["422", "444", "mono"])
@pytest.mark.parametrize("bd", [8, 12])
def test_page_locked_layouts_in_bands(ctx, layout, bd, oracle_threads):
    f = synth.make_small(8, 1918, 1434, bd, lr_unit=32, subsampling=layout[:2], monochrome=layout[2])
    HostFrame(f).check(ctx, oracle_threads)
    assert HostFrame(no_restoration(f)).check(ctx, oracle_threads) == filter_launches(f) > 1


@pytest.mark.parametrize("deferred", [False, True])
def test_different_frames_in_turn(deferred, oracle_threads):
    """Nothing of a frame is left in the next one's buffers, also after one
    that is refused, whichever band holds its bad sample."""
    ctx = Context(0)
    ctx.set_deferred_status(deferred)
    good = [HostFrame(synth.make_small(60 + i, w, h, 10, lr_unit=u, with_lvl_map=i == 1))
            for i, (w, h, u) in enumerate([(2562, 1438, 64), (1918, 1078, 32), (2562, 1438, 256)])]
    f = synth.make_small(70, 2562, 1438, 10)
    f.planes[0][5, 7] = 1 << 10
    bad_first = HostFrame(f)
    f = synth.make_small(71, 2562, 1438, 10)
    f.planes[2][-1, -1] = 1 << 10
    bad_last = HostFrame(f)
    for h in (good[0], good[1], bad_last, good[2], good[0], bad_first, good[1]):
        if h in good:
            h.check(ctx, oracle_threads)
        else:
            assert h.run(ctx)[:2] == (abi.INVALID_DATA, abi.MSG["DB_SAMPLE"])
    ctx.set_deferred_status(False)
    ctx.close()


@pytest.mark.parametrize("pin", ["none", "src", "dst"])
def test_pageable_frames_in_one_band(ctx, pin, oracle_threads):
    f = synth.make_small(9, 1918, 1078, 10, with_lvl_map=True)
    assert HostFrame(f, pin=pin).check(ctx, oracle_threads) == 2  # the fused kernel and restoration
    assert HostFrame(no_restoration(f), pin=pin).check(ctx, oracle_threads) == 1
