"""The fused kernel's CDEF taps against the oracle where their arithmetic is
tightest: samples at both ends of the range beside each other, every strength,
and shifts from 0 to past the sample width (damping 12 with strength 1)."""
import numpy as np
import pytest

import oracle
from vaco_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [(1, 1, False), (1, 0, False), (0, 0, False), (1, 1, True)],
                         ids=["420", "422", "444", "mono"])
@pytest.mark.parametrize("bd", [8, 10, 12])
@pytest.mark.parametrize("damping", [3, 6, 12])
def test_cdef_taps_at_the_range_ends(ctx, bd, damping, layout, oracle_threads):
    f = synth.make_small(71 + bd, 200, 136, bd, subsampling=layout[:2], monochrome=layout[2])
    rng = np.random.default_rng(bd * 100 + damping)
    top = (1 << bd) - 1
    for k, p in enumerate(f.planes):
        noise = rng.choice([0, 1, top // 2, top - 1, top], size=p.shape)
        f.planes[k] = np.where(rng.random(p.shape) < 0.5, noise, p).astype(np.uint16)
    f.deblock_levels = (0, 0, 0, 0)
    f.cdef.damping = damping - (bd - 8) if damping == 12 else damping
    f.cdef.y_primary, f.cdef.uv_primary = [0, 1, 2, 3, 5, 8, 14, 15], [15, 13, 8, 4, 3, 2, 1, 0]
    f.cdef.y_secondary, f.cdef.uv_secondary = [4, 0, 1, 2, 4, 1, 2, 4], [1, 2, 4, 0, 4, 2, 1, 4]
    f.cdef_idx = (np.arange(f.cdef_idx.size, dtype=np.int32) % 8).reshape(f.cdef_idx.shape)
    want, m = oracle.postfilter_frame(f, threads=oracle_threads)
    assert m == 0
    for k, (g, w) in enumerate(zip(ctx.postfilter_frame(f), want)):
        assert np.array_equal(g, w), f"plane {k}"
