"""The per-stage device entry points on both of their routes: the fused kernel
alone as one filter, and the per-stage kernels that in-place calls, odd cell
counts and pictures it objects to still take."""
import ctypes as C

import numpy as np
import pytest

import oracle
from vaco_b200 import abi, synth
from vaco_b200._lib import lib
from vaco_b200.frame import picture_struct
from vaco_b200.gpu import DeviceFrame

pytestmark = pytest.mark.gpu

LAYOUTS = [(1, 1, False), (1, 0, False), (0, 0, False), (1, 1, True)]
SIZES = [(60, 44), (64, 64), (200, 136), (328, 200)]


def picture(tensors):
    return picture_struct([t.data_ptr() for t in tensors], [tuple(t.shape) for t in tensors],
                          [t.stride(0) for t in tensors])


def out_like(planes, pad):
    """Zeroed planes of the same extents, rows `pad` samples longer."""
    import torch

    return [torch.zeros(p.shape[0], p.shape[1] + pad, dtype=p.dtype, device=p.device)[:, : p.shape[1]] for p in planes]


def deblock(ctx, d, dst):
    j, m = d.job, C.c_int32()
    st = lib().vaco_av1_deblock_picture_dev(ctx.handle, None, C.byref(j.src), C.byref(picture(dst)), C.byref(j.info),
                                            j.tx_luma, j.tx_chroma, j.lvl_map, C.byref(j.deblock), C.byref(m))
    return st, m.value


def cdef(ctx, d, dst):
    j, m = d.job, C.c_int32()
    st = lib().vaco_av1_cdef_picture_dev(ctx.handle, None, C.byref(j.src), C.byref(picture(dst)), C.byref(j.info),
                                         j.skip, j.cdef_idx, j.cdef_stride, j.cdef_count, C.byref(j.cdef), C.byref(m))
    return st, m.value


def check(dst, want, what):
    for k, (t, w) in enumerate(zip(dst, want)):
        assert np.array_equal(t.cpu().numpy().view(np.uint16), w), f"{what} plane {k}"


@pytest.mark.parametrize("layout", LAYOUTS, ids=["420", "422", "444", "mono"])
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("bd", [8, 12])
def test_deblock_and_cdef_routes(ctx, size, bd, layout, oracle_threads):
    f = synth.make_small(91, *size, bd, subsampling=layout[:2], monochrome=layout[2], with_lvl_map=True, sharpness=2)
    d = DeviceFrame(f)
    want, m = oracle.deblock_picture(f, threads=oracle_threads)
    assert m == 0
    for pad in (0, 2, 3):  # vector rows, word rows, rows only the per-stage kernels take
        dst = out_like(d.planes, pad)
        assert deblock(ctx, d, dst) == (abi.OK, 0)
        check(dst, want, f"deblock pad {pad}")
    want_cdef, m = oracle.cdef_picture(f, threads=oracle_threads)
    assert m == 0
    for pad in (0, 2, 3):
        dst = out_like(d.planes, pad)
        assert cdef(ctx, d, dst) == (abi.OK, 0)
        check(dst, want_cdef, f"cdef pad {pad}")
    assert deblock(ctx, d, d.planes) == (abi.OK, 0)  # in place
    check(d.planes, want, "deblock in place")


def test_cdef_ignores_bad_samples_outside_filtered_blocks(ctx, oracle_threads):
    f = synth.make_small(92, 200, 136, 10)
    f.skip[:] = 0
    f.skip[16:, :] = 1  # only the first 64 rows are filtered
    f.planes[0][120, 100] = 4000
    want, m = oracle.cdef_picture(f, threads=oracle_threads)
    assert m == 0
    d = DeviceFrame(f)
    dst = out_like(d.planes, 0)
    assert cdef(ctx, d, dst) == (abi.OK, 0)
    check(dst, want, "cdef")
    f.planes[0][30, 100] = 4000
    _, m = oracle.cdef_picture(f, threads=oracle_threads)
    assert m != 0
    assert cdef(ctx, DeviceFrame(f), dst) == (abi.INVALID_DATA, m)
    f.planes[0][30, 100] = 0  # the context is clean again
    assert cdef(ctx, DeviceFrame(f), dst) == (abi.OK, 0)


@pytest.mark.parametrize("where", ["before", "after", "unit"])
def test_restore_plane_errors_leave_the_output(ctx, where):
    import torch

    w, h = 203, 75
    rng = np.random.default_rng(5)
    before = rng.integers(0, 1024, (h, 208)).astype(np.uint16)
    after = rng.integers(0, 1024, (h, 205)).astype(np.uint16)
    units = synth.lr_units(rng, w, h, 64, False)
    if where == "unit":
        units["type"][-1], units["vertical"][-1] = abi.LR_WIENER, (50, 0, 0)
    else:
        (before if where == "before" else after)[h - 1, w - 1] = 1024
    t = [torch.from_numpy(a.view(np.int16)).cuda() for a in (before, after)]
    u = torch.from_numpy(units.view(np.uint8)).cuda()
    out = torch.full((h, w), 77, dtype=torch.int16, device="cuda")
    cfg, m = abi.LrPlaneConfig(w, h, 10, 64, 0), C.c_int32()
    st = lib().vaco_av1_restore_plane_dev(ctx.handle, None, t[0].data_ptr(), 208, h, 208, t[1].data_ptr(), 205, h, 205,
                                          C.byref(cfg), u.data_ptr(), len(units), out.data_ptr(), w, C.byref(m))
    assert st == abi.INVALID_DATA
    assert m.value == (abi.MSG["LR_COEFFICIENT"] if where == "unit" else abi.MSG["LR_SAMPLE"])
    assert bool((out == 77).all())
