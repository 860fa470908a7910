"""Pictures with odd counts of mode-info cells, whose last 8x8 blocks reach past
the planes: the per-stage kernels take them, on the layouts, depths and sides
where a plane can end inside a block, against the oracle."""
import numpy as np
import pytest

import oracle
from vaco_b200 import synth
from vaco_b200.frame import FrameInputs

pytestmark = pytest.mark.gpu


class CellFrame(FrameInputs):
    """A frame of any count of cells (rows, cols)."""

    cells = (0, 0)
    mi_rows = property(lambda self: self.cells[0])
    mi_cols = property(lambda self: self.cells[1])


def cell_frame(seed, w, h, bd, cut, **kw):
    """synth.make_small()'s frame without its last rows and columns of cells."""
    f = synth.make_small(seed, w, h, bd, sharpness=2, **kw)
    o = CellFrame(**vars(f))
    o.cells = rows, cols = f.mi_rows - cut[0], f.mi_cols - cut[1]
    o.coded_width = o.upscaled_width = 4 * cols
    o.coded_height = 4 * rows
    sx, sy = f.subsampling_x, f.subsampling_y
    o.planes = [f.planes[k][: o.padded_shape(k)[0], : o.padded_shape(k)[1]].copy() for k in range(f.num_planes)]
    o.tx_luma, o.skip = f.tx_luma[:rows, :cols].copy(), f.skip[:rows, :cols].copy()
    o.tx_chroma = f.tx_chroma[: (rows + sy) >> sy, : (cols + sx) >> sx].copy()
    return o


LAYOUTS = [(1, 1, False), (1, 0, False), (0, 0, False), (1, 1, True)]


def same(got, want):
    for k, (g, w) in enumerate(zip(got, want)):
        assert np.array_equal(g, w), f"plane {k}: {int((g != w).sum())} samples differ"


@pytest.mark.parametrize("layout", LAYOUTS, ids=["420", "422", "444", "mono"])
@pytest.mark.parametrize("bd", [8, 10, 12])
@pytest.mark.parametrize("cut", [(1, 0), (0, 1), (1, 1)], ids=["rows", "cols", "both"])
@pytest.mark.parametrize("size", [(8, 8), (64, 72), (200, 136)])
def test_cdef(ctx, size, cut, bd, layout, oracle_threads):
    f = cell_frame(5, *size, bd, cut, subsampling=layout[:2], monochrome=layout[2])
    want, m = oracle.cdef_picture(f, threads=oracle_threads)
    assert m == 0
    same(ctx.cdef_picture(f), want)


@pytest.mark.parametrize("layout", LAYOUTS, ids=["420", "422", "444", "mono"])
@pytest.mark.parametrize("bd", [8, 10, 12])
@pytest.mark.parametrize("cut", [(1, 0), (0, 1), (1, 1)], ids=["rows", "cols", "both"])
def test_deblock(ctx, cut, bd, layout, oracle_threads):
    f = cell_frame(6, 200, 136, bd, cut, subsampling=layout[:2], monochrome=layout[2])
    want, m = oracle.deblock_picture(f, threads=oracle_threads)
    assert m == 0
    same(ctx.deblock_picture(f), want)


@pytest.mark.parametrize("layout", LAYOUTS, ids=["420", "422", "444", "mono"])
@pytest.mark.parametrize("cut", [(1, 0), (0, 1), (1, 1)], ids=["rows", "cols", "both"])
def test_deblock_with_a_level_map(ctx, cut, layout, oracle_threads):
    """A subsampled chroma cell's levels are those of its last luma cell, which
    the map's last cells have not: its last row and column stand in.  The map
    holds the frame's levels throughout, so the result is the one without it."""
    f = cell_frame(6, 200, 136, 10, cut, subsampling=layout[:2], monochrome=layout[2])
    f.deblock_levels = (30, 24, 41, 17)
    want, m = oracle.deblock_picture(f, threads=oracle_threads)
    assert m == 0
    f.lvl_map = np.tile(np.array(f.deblock_levels, np.uint8), (*f.cells, 1))
    same(ctx.deblock_picture(f), want)
