"""The chain through the device entry point, which launches a frame's tiles at
once, on both sides of the line between the fused kernel's bodies: up to two
tiles per SM (296 on 148 SMs) at 512 threads a tile, more at 256, in every
chroma layout, depth class and with restoration and without, where the planes
are written directly.  (The host entry point cuts frames of this size into
launches of fewer tiles.)"""
import numpy as np
import pytest

import oracle
from vaco_b200 import abi, synth
from vaco_b200.gpu import DeviceFrame

pytestmark = pytest.mark.gpu


def check(ctx, f, threads):
    want, m = oracle.postfilter_frame(f, threads=threads)
    assert m == 0
    d, before = DeviceFrame(f), ctx.launches
    ctx.postfilter_frame_dev(d)
    for k, (g, w) in enumerate(zip(d.outputs_numpy(), want)):
        assert np.array_equal(g, w), f"plane {k}: {int((g != w).sum())} samples differ"
    return ctx.launches - before


@pytest.mark.parametrize("layout", [(1, 1, False), (1, 0, False), (0, 0, False), (1, 1, True)],
                         ids=["420", "422", "444", "mono"])
@pytest.mark.parametrize("size", [(2366, 510), (1430, 806)], ids=["296", "299"])
@pytest.mark.parametrize("bd", [8, 10, 12])
def test_bodies_at_the_line(ctx, size, bd, layout, oracle_threads):
    f = synth.make_small(5, *size, bd, subsampling=layout[:2], monochrome=layout[2], with_lvl_map=True)
    assert check(ctx, f, oracle_threads) == 2
    f.lr_type, f.lr_units = (abi.FRAME_LR_NONE,) * 3, []
    # rows of an odd count of samples are copied by a second kernel
    odd = any(f.output_shape(k)[1] & 1 for k in range(f.num_planes))
    assert check(ctx, f, oracle_threads) == 1 + odd


@pytest.mark.parametrize("bd", [8, 12])
def test_cdef_only_full_hd(ctx, bd, oracle_threads):
    """No deblocking, no restoration: 510 tiles written directly."""
    assert check(ctx, synth.make_small(11, 1920, 1080, bd, chain=False), oracle_threads) == 1
