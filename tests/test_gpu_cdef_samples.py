"""cdef_picture on pictures with samples above the bit depth: refused with the
oracle's message where a filtered block or its taps' reach holds one, accepted
where none does, and in either case in one launch."""
import ctypes as C

import numpy as np
import pytest

import oracle
from vaco_b200 import abi, synth
from vaco_b200._lib import lib
from vaco_b200.frame import picture_struct
from vaco_b200.gpu import DeviceFrame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [(1, 1, False), (1, 0, False), (0, 0, False), (1, 1, True)],
                         ids=["420", "422", "444", "mono"])
@pytest.mark.parametrize("bd", [8, 10, 12])
def test_samples_above_the_depth(ctx, bd, layout, oracle_threads):
    rng = np.random.default_rng(bd + 100 * layout[0] + 10 * layout[1])
    seen = set()
    for i in range(40):
        f = synth.make_small(300 + i, 136, 88, bd, subsampling=layout[:2], monochrome=layout[2])
        skip8 = rng.random((f.skip.shape[0] // 2, f.skip.shape[1] // 2)) < 0.8
        f.skip = np.repeat(np.repeat(skip8, 2, 0), 2, 1).astype(np.uint8)
        if i % 5 == 4:  # a strength index that does not exist
            f.cdef_idx[rng.integers(f.cdef_idx.shape[0]), rng.integers(f.cdef_idx.shape[1])] = 9
        for _ in range(rng.integers(1, 4)):
            p = f.planes[rng.integers(f.num_planes)]
            p[rng.integers(p.shape[0]), rng.integers(p.shape[1])] = rng.choice([1 << bd, 0x8000, 0xFFFF])
        want, m = oracle.cdef_picture(f, planes=f.planes[: f.num_planes], threads=oracle_threads)
        seen.add(m)
        d, msg = DeviceFrame(f), C.c_int32()
        dst = [p.clone() for p in d.planes]
        pic = picture_struct([t.data_ptr() for t in dst], [tuple(t.shape) for t in dst])
        j, before = d.job, ctx.launches
        st = lib().vaco_av1_cdef_picture_dev(ctx.handle, None, C.byref(j.src), C.byref(pic), C.byref(j.info), j.skip,
                                             j.cdef_idx, j.cdef_stride, j.cdef_count, C.byref(j.cdef), C.byref(msg))
        assert (st, msg.value) == (abi.INVALID_DATA if m else abi.OK, m), i
        assert ctx.launches == before + 1
        for k in range(0 if m else f.num_planes):
            assert np.array_equal(dst[k].cpu().numpy().view(np.uint16), want[k]), f"{i}: plane {k}"
    assert {0, abi.MSG["CDEF_BLOCK_PARAMS"]} <= seen  # in every layout and depth
