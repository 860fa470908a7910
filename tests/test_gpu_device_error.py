"""Calls that fail because the device refuses something: here scratch that no
GPU has room for, in a superres frame 2^30 samples wide."""
import ctypes as C

import numpy as np
import pytest

import oracle
from vaco_b200 import abi, synth
from vaco_b200._lib import lib
from vaco_b200.frame import picture_struct
from vaco_b200.gpu import Context, DeviceFrame, VacoError

pytestmark = pytest.mark.gpu


@pytest.fixture
def own_ctx():
    c = Context(0)
    yield c
    c.close()


def too_wide(f):
    """The frame's device job, upscaled to 292 GB of luma; its output is never reached."""
    d = DeviceFrame(f)
    d.job.info.upscaled_width = 1 << 30
    for k in range(3):
        d.job.dst.width[k] = d.job.dst.stride[k] = (1 << 30) >> (k > 0)
    return d


def same(got, want, what):
    for k, (g, w) in enumerate(zip(got, want)):
        assert np.array_equal(g, w), f"{what} plane {k}"


@pytest.mark.parametrize("batch", [False, True])
def test_device_error_is_reported_once(own_ctx, batch, oracle_threads):
    """The next call, one whose launches are checked by the thread's last
    error (in place: the per-stage kernels), and torch know nothing of it."""
    import torch

    f = synth.make_small(31, 200, 136, 10)
    want, m = oracle.deblock_picture(f, threads=oracle_threads)
    assert m == 0
    bad = too_wide(f)
    with pytest.raises(VacoError) as e:
        if batch:
            own_ctx.postfilter_batch_dev([bad])
        else:
            own_ctx.postfilter_frame_dev(bad)
    assert e.value.status == abi.DEVICE_ERROR
    d, msg = DeviceFrame(f), C.c_int32()
    j = d.job
    pic = picture_struct([t.data_ptr() for t in d.planes], [tuple(t.shape) for t in d.planes])
    assert lib().vaco_av1_deblock_picture_dev(own_ctx.handle, None, C.byref(j.src), C.byref(pic), C.byref(j.info),
                                              j.tx_luma, j.tx_chroma, j.lvl_map, C.byref(j.deblock),
                                              C.byref(msg)) == abi.OK
    torch.cuda.synchronize()
    same([t.cpu().numpy().view(np.uint16) for t in d.planes], want, "deblock")


def test_call_that_failed_half_way_leaves_the_next_one_alone(own_ctx, oracle_threads):
    """A frame with a bad sample fails while its first kernel is still queued
    behind other work.  What that kernel reports later is not the next call's error."""
    import torch

    f = synth.make_small(31, 200, 136, 10)
    want, m = oracle.postfilter_frame(f, threads=oracle_threads)
    assert m == 0
    good = DeviceFrame(f)
    own_ctx.postfilter_frame_dev(good)  # the scratch both calls share is there
    f.planes[0][40, 33] = 1 << 10
    bad = too_wide(f)
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # about 0.1 s on the stream of both calls
    with pytest.raises(VacoError) as e:
        own_ctx.postfilter_frame_dev(bad)
    assert e.value.status == abi.DEVICE_ERROR
    own_ctx.postfilter_frame_dev(good)
    same(good.outputs_numpy(), want, "next frame")
