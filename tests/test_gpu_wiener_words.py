"""The Wiener filter's two-sample dot products at the ends of the coefficients'
ranges (centre tap 0 and 218), samples at both ends of theirs, and tiles of odd
and partial widths."""
import numpy as np
import pytest

import oracle
from vaco_b200 import abi

pytestmark = pytest.mark.gpu

ENDS = [(10, 8, 46), (-5, -23, -17), (-5, 8, -17), (10, -23, 46), (0, 0, 0), (0, 8, 46), (3, -7, 15)]
SIZES = [(1, 1), (5, 3), (7, 9), (62, 57), (66, 71), (131, 129)]


def content(kind, w, h, bd, rng):
    top = (1 << bd) - 1
    if kind == "random":
        return rng.integers(0, top + 1, (h, w)).astype(np.uint16)
    if kind == "extremes":  # single samples, both ends
        return (rng.integers(0, 2, (h, w)) * top).astype(np.uint16)
    cells = rng.integers(0, 2, ((h + 3) // 4, (w + 3) // 4)) * top  # 4x4 cells at both ends
    return np.repeat(np.repeat(cells, 4, 0), 4, 1)[:h, :w].astype(np.uint16)


@pytest.mark.parametrize("kind", ["random", "extremes", "cells"])
@pytest.mark.parametrize("bd", [8, 10, 12])
def test_wiener_matches_the_oracle(ctx, bd, kind, oracle_threads):
    rng = np.random.default_rng(100 * bd + len(kind))
    for w, h in SIZES:
        counts = max((w + 32) // 64, 1) * max((h + 32) // 64, 1)
        for i, ends in enumerate(ENDS):
            units = np.zeros(counts, abi.lr_unit_dtype())
            units["type"] = abi.LR_WIENER
            units["horizontal"] = [ends if k % 2 == 0 else ENDS[(i + k) % len(ENDS)] for k in range(counts)]
            units["vertical"] = [ENDS[(i + 2 * k + i % 3) % len(ENDS)] for k in range(counts)]
            before, after = (content(kind, w, h, bd, rng) for _ in range(2))
            want, m = oracle.restore_plane(before, after, w, h, bd, 64, False, units, threads=oracle_threads)
            assert m == 0
            got = ctx.restore_plane(before, after, w, h, bd, 64, False, units)
            np.testing.assert_array_equal(got, want, err_msg=f"{w}x{h} {ends}")
