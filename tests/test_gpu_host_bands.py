"""The synchronous host call, which filters a large frame in bands of tile rows
while other bands are copied, against the oracle: band edges against
restoration units, stripes and planes without restoration, every layout, and
errors found in different bands."""
import numpy as np
import pytest

import oracle
from vaco_b200 import abi, synth
from vaco_b200.gpu import VacoError

pytestmark = pytest.mark.gpu

LAYOUTS = [(1, 1, False), (1, 0, False), (0, 0, False), (1, 1, True)]


def check(ctx, f, threads):
    want, m = oracle.postfilter_frame(f, threads=threads)
    assert m == 0
    for k, (g, w) in enumerate(zip(ctx.postfilter_frame(f), want)):
        assert np.array_equal(g, w), f"plane {k}: {int((g != w).sum())} samples differ"


@pytest.mark.parametrize("layout", LAYOUTS, ids=["420", "422", "444", "mono"])
@pytest.mark.parametrize("size", [(1600, 522), (1022, 1370), (4000, 202)])
@pytest.mark.parametrize("unit", [32, 64, 256])
def test_host_call_in_bands(ctx, layout, size, unit, oracle_threads):
    f = synth.make_small(61 + unit, *size, 10, lr_unit=unit, subsampling=layout[:2], monochrome=layout[2],
                         with_lvl_map=True)
    check(ctx, f, oracle_threads)
    f.lr_type = (abi.FRAME_LR_SWITCHABLE, abi.FRAME_LR_NONE, abi.FRAME_LR_NONE)
    f.lr_units = f.lr_units[:1]
    check(ctx, f, oracle_threads)
    f.lr_type, f.lr_units = (abi.FRAME_LR_NONE,) * 3, []
    check(ctx, f, oracle_threads)


@pytest.mark.parametrize("row", [0, 700, 1367])
def test_host_call_in_bands_errors(ctx, row, oracle_threads):
    f = synth.make_small(77, 1022, 1370, 10)
    good = f.planes[0][row, 5]
    f.planes[0][row, 5] = 1024
    _, m = oracle.postfilter_frame(f, threads=oracle_threads)
    with pytest.raises(VacoError) as e:
        ctx.postfilter_frame(f)
    assert e.value.msg == m
    f.planes[0][row, 5] = good
    units = f.lr_units[2]
    last = len(units) - 1 if row else 0
    keep = units[last].copy()
    units["type"][last], units["set"][last] = abi.LR_SGRPROJ, 16
    _, m = oracle.postfilter_frame(f, threads=oracle_threads)
    with pytest.raises(VacoError) as e:
        ctx.postfilter_frame(f)
    assert e.value.msg == m
    units[last] = keep
    check(ctx, f, oracle_threads)
