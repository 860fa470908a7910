"""Film grain on the GPU against the oracle where the template wavefront and the
apply kernel's work items change shape: every layout and auto-regression lag
with taps over their whole range, frame extents on both sides of the 8-sample
chunk, the 32-sample block and the two-row item, and planes whose rows are not
16-byte aligned."""
import ctypes as C

import numpy as np
import pytest

import oracle
from test_film_grain import FORMATS, frame, gauss_table, random_params
from vaco_b200 import abi

pytestmark = pytest.mark.gpu


def grain_dev(ctx, planes, info, p, g):
    import torch

    from vaco_b200._lib import lib
    from vaco_b200.frame import picture_struct

    din = [torch.from_numpy(q.view(np.int16)).cuda() for q in planes]
    dout = [torch.zeros_like(t) for t in din]
    pin = picture_struct([t.data_ptr() for t in din], [q.shape for q in planes])
    pout = picture_struct([t.data_ptr() for t in dout], [q.shape for q in planes])
    msg = C.c_int32()
    st = lib().vaco_av1_film_grain_dev(ctx.handle, None, C.byref(pin), C.byref(pout), C.byref(info), C.byref(p),
                                       g.ctypes.data, C.byref(msg))
    assert st == abi.OK, abi.MESSAGES.get(msg.value)
    return [t.cpu().numpy().view(np.uint16) for t in dout]


@pytest.mark.parametrize("fmt", list(FORMATS))
@pytest.mark.parametrize("lag", [0, 1, 2, 3])
@pytest.mark.parametrize("size", [(31, 32), (64, 33), (129, 98)])
def test_film_grain_wavefront_and_items(ctx, fmt, lag, size):
    for bd in (8, 12):
        seed = 900 + 10 * lag + bd
        info, planes = frame(seed, *size, bd, fmt)
        p = random_params(seed, mono=FORMATS[fmt][2], num_y_points=8, overlap_flag=1, ar_coeff_lag=lag,
                          ar_coeff_shift_minus_6=lag, grain_scale_shift=0)
        rng = np.random.default_rng(seed)
        for arr in (p.ar_coeffs_y_plus_128, p.ar_coeffs_cb_plus_128, p.ar_coeffs_cr_plus_128):
            for i in range(24):
                arr[i] = int(rng.integers(0, 256))
        g = gauss_table(seed)
        want, m = oracle.film_grain(planes, info, p, g)
        assert m == 0
        for got in (ctx.film_grain(planes, info, p, g), grain_dev(ctx, planes, info, p, g)):
            for k, (a, b) in enumerate(zip(got, want)):
                assert np.array_equal(a, b), f"{bd}-bit plane {k}: {int((a != b).sum())} samples differ"
