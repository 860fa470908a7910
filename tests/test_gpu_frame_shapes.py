"""The chain on both sides of the line between the fused kernel's two shapes:
296 tiles (512 threads a tile on a 148-SM GPU) and 299 (256 threads), in every
chroma layout and at 8 and 12 bits."""
import numpy as np
import pytest

import oracle
from vaco_b200 import abi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [(1, 1, False), (1, 0, False), (0, 0, False), (1, 1, True)],
                         ids=["420", "422", "444", "mono"])
@pytest.mark.parametrize("size", [(2366, 510), (1430, 806)])
@pytest.mark.parametrize("bd", [8, 12])
@pytest.mark.parametrize("lr_off", [False, True], ids=["lr", "direct"])
def test_chain_tile_shapes(ctx, size, bd, layout, lr_off, oracle_threads):
    f = synth.make_small(5, *size, bd, subsampling=layout[:2], monochrome=layout[2], with_lvl_map=True)
    if lr_off:
        f.lr_type = (abi.FRAME_LR_NONE,) * 3
        f.lr_units = []
    want, m = oracle.postfilter_frame(f, threads=oracle_threads)
    assert m == 0
    for k, (g, w) in enumerate(zip(ctx.postfilter_frame(f), want)):
        assert np.array_equal(g, w), f"plane {k}"
