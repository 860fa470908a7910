"""A context's status word over runs of good and bad frames: a kernel raises
the host flag with the first report only, and the calls reset the word only
where it can hold one, so no report may be lost and none may last."""
import pytest

import oracle
from vaco_b200 import abi, synth
from vaco_b200.gpu import Context, DeviceFrame, VacoError

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def frames(oracle_threads):
    """A good frame and two bad ones, with the oracle's messages: every sample
    above the depth, one unit's coefficient out of range."""
    def frame():
        return synth.make_small(44, 200, 136, 10)

    samples, unit = frame(), frame()
    for p in samples.planes:
        p[:] = 1024
    unit.lr_units[0]["type"][0], unit.lr_units[0]["set"][0] = abi.LR_SGRPROJ, 16
    got = [(f, oracle.postfilter_frame(f, threads=oracle_threads)[1]) for f in (frame(), samples, unit)]
    assert [m for _, m in got] == [0, abi.MSG["DB_SAMPLE"], abi.MSG["LR_COEFFICIENT"]]
    return [(DeviceFrame(f), m) for f, m in got]


@pytest.fixture
def own_ctx():
    c = Context(0)
    yield c
    c.close()


def call(ctx, d):
    try:
        ctx.postfilter_frame_dev(d)
    except VacoError as e:
        assert e.status == abi.INVALID_DATA
        return e.msg
    return 0


ORDER = (0, 1, 1, 2, 0, 2, 1, 0, 0, 2)


@pytest.mark.parametrize("flush", [False, True])
def test_each_call_reports_its_own_frame(own_ctx, frames, flush):
    for i in ORDER:
        d, m = frames[i]
        assert call(own_ctx, d) == m
        if flush:  # of a context that does not defer: nothing is left to report
            own_ctx.flush()


def test_each_flush_reports_its_own_frames(own_ctx, frames):
    own_ctx.set_deferred_status(True)
    for group in ((0, 0), (1, 0), (2, 1), (0,), (2, 2, 0), (1,), (0, 2)):
        for i in group:
            assert call(own_ctx, frames[i][0]) == 0
        want = [frames[i][1] for i in group if i]
        try:
            own_ctx.flush()
            got = 0
        except VacoError as e:
            got = e.msg
        # deblocking's checks come before restoration's
        assert got == (min(want, key=lambda m: m != abi.MSG["DB_SAMPLE"]) if want else 0)
    own_ctx.set_deferred_status(False)
    for i in ORDER:
        assert call(own_ctx, frames[i][0]) == frames[i][1]


def test_each_batch_reports_its_own_frames(own_ctx, frames):
    for group in ((0, 0), (1, 2, 0), (0, 1), (0,), (2, 2), (0, 0, 0)):
        status, msg = own_ctx.postfilter_batch_dev([frames[i][0] for i in group])
        assert msg == [frames[i][1] for i in group]
        assert [s != abi.OK for s in status] == [i != 0 for i in group]
