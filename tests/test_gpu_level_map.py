"""Level maps with values above 63, which every entry point that takes a map
refuses, and which must not reach the fused kernel's segment lists (a list
entry has 6 bits for a level, next to the segment's offset)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from vaco_b200 import abi, synth
from vaco_b200._lib import lib
from vaco_b200.frame import picture_struct
from vaco_b200.gpu import DeviceFrame, VacoError

pytestmark = pytest.mark.gpu


def deblock_picture(ctx, d):
    j, m, dst = d.job, C.c_int32(), [p.clone() for p in d.planes]
    pic = picture_struct([t.data_ptr() for t in dst], [tuple(t.shape) for t in dst])
    st = lib().vaco_av1_deblock_picture_dev(ctx.handle, None, C.byref(j.src), C.byref(pic), C.byref(j.info), j.tx_luma,
                                            j.tx_chroma, j.lvl_map, C.byref(j.deblock), C.byref(m))
    return st, m.value


@pytest.mark.parametrize("level", [64, 128, 192, 255])
@pytest.mark.parametrize("bd", [8, 12])
@pytest.mark.parametrize("where", ["corner", "all"])
def test_levels_above_63_are_refused(ctx, level, bd, where, oracle_threads):
    f = synth.make_small(17, 200, 136, bd, with_lvl_map=True)
    good, levels = DeviceFrame(f), f.lvl_map
    f.lvl_map = levels.copy()
    f.lvl_map[(slice(None),) * 2 if where == "all" else (-1, -1)] = level
    _, m = oracle.postfilter_frame(f, threads=oracle_threads)
    assert m == abi.MSG["DB_PARAMS"]
    bad = DeviceFrame(f)
    with pytest.raises(VacoError) as e:
        ctx.postfilter_frame_dev(bad)
    assert (e.value.status, e.value.msg) == (abi.INVALID_DATA, m)
    assert ctx.postfilter_batch_dev([good, bad]) == ([abi.OK, abi.INVALID_DATA], [0, m])
    assert deblock_picture(ctx, bad) == (abi.INVALID_DATA, m)
    f.lvl_map = levels
    want, m = oracle.postfilter_frame(f, threads=oracle_threads)
    assert m == 0
    ctx.postfilter_frame_dev(good)
    for k, (g, w) in enumerate(zip(good.outputs_numpy(), want)):
        assert np.array_equal(g, w), f"plane {k}"
