"""GPU parity of the row-shift convolution on CTA pairs ("conv_pairs" 2 = wherever it fits), forward and backward-data, at the edges of
its tiles, slabs and classes: one position more or less than a tile, filters that leave the image on every side, partly filled
channel groups and filter tiles, both strides, splits of the reduction, accumulation into dx."""
import ctypes

import numpy as np
import pytest

from oracle import eddl_oracle as orc

pytestmark = pytest.mark.gpu
F = np.float32

CASES = [  # n, c, h, w, k, kernel, stride, pad
    (1, 16, 1, 1, 8, (1, 1), 1, 0), (1, 32, 15, 15, 32, (3, 3), 1, 1), (1, 33, 16, 16, 31, (3, 3), 1, 1), (4, 40, 7, 8, 129, (3, 3), 1, 1),
    (3, 64, 7, 7, 64, (3, 3), 1, 1), (2, 20, 21, 37, 36, (5, 5), 1, 2), (2, 17, 9, 10, 24, (2, 4), 1, 1), (2, 16, 6, 5, 16, (7, 7), 1, 3),
    (1, 512, 5, 5, 64, (3, 3), 1, 1), (1, 256, 14, 14, 32, (1, 1), 1, 0), (2, 24, 13, 13, 40, (3, 3), 2, 1), (2, 24, 14, 14, 40, (3, 3), 2, 0),
    (3, 32, 9, 12, 16, (1, 1), 2, 0), (2, 16, 11, 11, 16, (5, 5), 2, 2), (1, 16, 12, 12, 16, (3, 3), 1, 0), (1, 16, 10, 60, 16, (3, 3), 1, 2),
    (130, 16, 2, 2, 16, (3, 3), 1, 1), (5, 16, 100, 3, 70, (3, 1), 1, 0),
]


@pytest.fixture()
def pairs(lib):
    lib.call("set_option", b"conv_pairs", 2)
    yield lib
    lib.call("set_option", b"conv_pairs", 1)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)).replace(" ", ""))
@pytest.mark.parametrize("precision,limit", [(0, 1e-5), (1, 2e-3), (2, 1e-5)])
def test_forward_and_backward_data(pairs, case, precision, limit):
    L = pairs
    n, c, h, w, k, (kr, kc), s, p = case
    rng = np.random.default_rng(h * w + c)
    x, wt, b = rng.standard_normal((n, c, h, w)).astype(F), rng.standard_normal((k, c, kr, kc)).astype(F), rng.standard_normal(k).astype(F)
    pads = (p, p, p, p)
    want = orc.conv2d_fwd(x, wt, b, (s, s), pads)
    oh, ow = want.shape[2:]
    dy, dx0 = rng.standard_normal(want.shape).astype(F), rng.standard_normal(x.shape).astype(F)
    geo = (n, c, h, w, k, kr, kc, oh, ow, s, s, p, p, precision)
    dw_ = L.to_device(wt)
    y = L.to_device(np.full(want.shape, np.nan, F))
    L.call("conv2d_fwd", 0, L.to_device(x), dw_, L.to_device(b), y, *geo)
    # the limits are those of the precisions (fp32-equivalent 1e-5, plain TF32 with 11-bit factors) relative to the largest value
    assert np.max(np.abs(y.numpy() - want)) <= limit * np.max(np.abs(want))
    back = orc.conv2d_bwd_data(dy, wt, x.shape, dx0, (s, s), pads)
    dx = L.to_device(dx0)
    L.call("conv2d_bwd_data", 0, L.to_device(dy), dw_, dx, *geo)
    assert np.max(np.abs(dx.numpy() - back)) <= limit * np.max(np.abs(back))
    L.call("sync", 0)


@pytest.mark.parametrize("stride,kernel,pad", [(1, 3, 1), (2, 3, 1), (2, 1, 0)])
def test_zeros_owed_to_dx_are_stored_not_added(pairs, stride, kernel, pad):
    L = pairs
    n, c, h, k = 4, 32, 40, 32
    rng = np.random.default_rng(stride + kernel)
    oh = (h + 2 * pad - kernel) // stride + 1
    wt, dy = rng.standard_normal((k, c, kernel, kernel)).astype(F), rng.standard_normal((n, k, oh, oh)).astype(F)
    L.call("set_option", b"lazy_zero", 1)
    try:
        dx = L.empty((n, c, h, h))
        L.call("fill", 0, dx, dx.size, 3.0); L.call("fill", 0, dx, dx.size, 0.0)
        L.call("conv2d_bwd_data", 0, L.to_device(dy), L.to_device(wt), dx, n, c, h, h, k, kernel, kernel, oh, oh, stride, stride, pad, pad, 0)
        want = orc.conv2d_bwd_data(dy, wt, (n, c, h, h), None, (stride, stride), (pad,) * 4)
        assert np.max(np.abs(dx.numpy() - want)) <= 1e-5 * np.max(np.abs(want))
    finally:
        L.call("set_option", b"lazy_zero", 0)


def test_repeated_calls_give_the_same_bits(pairs):
    """Several tiles per CTA pair, slab and stage rings that wrap, split reductions: nothing depends on timing."""
    L = pairs
    rng = np.random.default_rng(7)
    for n, c, h, k, p in ((40, 64, 28, 96, 1), (2, 256, 7, 64, 1)):
        x, wt = L.to_device(rng.standard_normal((n, c, h, h)).astype(F)), L.to_device(rng.standard_normal((k, c, 3, 3)).astype(F))
        geo = (n, c, h, h, k, 3, 3, h, h, 1, 1, p, p, 0)
        y = L.empty((n, k, h, h))
        L.call("conv2d_fwd", 0, x, wt, None, y, *geo)
        first = y.numpy()
        for _ in range(3):
            L.call("conv2d_fwd", 0, x, wt, None, y, *geo)
            np.testing.assert_array_equal(y.numpy(), first)


# n, c, h, w, k, kernel, stride, pad, precision, pass: short reductions into a dx that holds values, slabs of several passes, two weight
# stages, a dx of which every fourth pixel is written
SLOWER_ON_PAIRS = [(35, 832, 21, 69, 16, 3, 1, 1, 2, "bwd_data"), (34, 704, 20, 49, 16, 3, 1, 0, 0, "bwd_data"), (31, 48, 18, 72, 247, 5, 1, 2, 0, "bwd_data"),
                   (27, 16, 70, 70, 208, 3, 1, 0, 2, "fwd"), (64, 256, 56, 56, 512, 1, 2, 0, 0, "bwd_data")]


@pytest.mark.parametrize("case", SLOWER_ON_PAIRS, ids=lambda c: "-".join(map(str, c)))
def test_layers_that_pairs_would_slow_down_stay_on_the_other_kernels(lib, case):
    """The default choice against the same call with CTA pairs off: these layers took 1.13 to 1.5 times as long on pairs (the bound leaves
    room for the spread of single launches, a few percent)."""
    L = lib
    n, c, h, w, k, r, s, p, precision, which = case
    oh, ow = (h + 2 * p - r) // s + 1, (w + 2 * p - r) // s + 1
    x, y, wt = L.zeros((n, c, h, w)), L.zeros((n, k, oh, ow)), L.zeros((k, c, r, r))
    geo = (n, c, h, w, k, r, r, oh, ow, s, s, p, p, precision)

    def us(pairs):
        L.call("set_option", b"conv_pairs", pairs)
        times = []
        for _ in range(25):
            L.call("timer_start", 0, 3)
            if which == "fwd":
                L.call("conv2d_fwd", 0, x, wt, None, y, *geo)
            else:
                L.call("conv2d_bwd_data", 0, y, wt, x, *geo)
            L.call("timer_stop", 0, 3)
            ms = ctypes.c_float()
            L.call("timer_elapsed_ms", 0, 3, ctypes.byref(ms))
            times.append(ms.value * 1e3)
        return float(np.median(times[5:]))
    try:
        off, default = us(0), us(1)
    finally:
        L.call("set_option", b"conv_pairs", 1)
    assert default <= 1.08 * off + 2
