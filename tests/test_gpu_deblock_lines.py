"""The fused kernel's deblocking against the oracle where its arithmetic is
tightest: samples at both ends of the range beside each other, flat areas one
step either side of the flatness bound, the lowest and highest levels and every
sharpness that changes the strengths, at every transform size."""
import numpy as np
import pytest

import oracle
from vaco_b200 import abi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [(1, 1, False), (1, 0, False), (0, 0, False), (1, 1, True)],
                         ids=["420", "422", "444", "mono"])
@pytest.mark.parametrize("bd", [8, 10, 12])
@pytest.mark.parametrize("levels", [(1, 63, 2, 62), (63, 63, 63, 63), (20, 40, 30, 10)])
def test_deblocking_lines(ctx, bd, levels, layout, oracle_threads):
    for sharpness in (0, 3, 7):
        f = synth.make_small(31 + sharpness, 264, 200, bd, subsampling=layout[:2], monochrome=layout[2],
                             sharpness=sharpness)
        rng = np.random.default_rng(bd * 10 + sharpness)
        top, step = (1 << bd) - 1, 1 << (bd - 8)
        for k, p in enumerate(f.planes):
            h, w = p.shape
            cells = rng.integers(0, 4, ((h + 7) // 8, (w + 7) // 8))
            kind = np.repeat(np.repeat(cells, 8, 0), 8, 1)[:h, :w]
            base = np.repeat(np.repeat(rng.integers(0, top + 1, cells.shape), 8, 0), 8, 1)[:h, :w]
            flat = np.clip(base + rng.integers(-step - 1, step + 2, (h, w)), 0, top)
            near = np.clip(top // 2 + rng.integers(-3 * step, 3 * step + 1, (h, w)), 0, top)
            ends = rng.choice([0, 1, top - 1, top], size=(h, w))
            f.planes[k] = np.choose(kind, [p, flat, near, ends]).astype(np.uint16)
        f.deblock_levels = levels
        f.cdef.enabled = False
        f.lr_type, f.lr_units = (abi.FRAME_LR_NONE,) * 3, []
        want, m = oracle.postfilter_frame(f, threads=oracle_threads)
        assert m == 0
        for k, (g, w) in enumerate(zip(ctx.postfilter_frame(f), want)):
            assert np.array_equal(g, w), f"sharpness {sharpness} plane {k}: {int((g != w).sum())} samples differ"
