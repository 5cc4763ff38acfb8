"""GPU parity of backward-weight on CTA pairs ("conv_pairs" 2 = wherever it fits) at the edges of its tiles: one channel or filter more
or less than a tile, a second CTA with nothing to do, planes that end inside a K-block, the widest slab, split and unsplit
reductions, accumulation into the gradient and the store into known zeros."""
import ctypes

import numpy as np
import pytest

from oracle import eddl_oracle as orc

pytestmark = pytest.mark.gpu
F = np.float32

CASES = [  # n, c, h, w, k, kernel
    (1, 14, 6, 6, 32, 3), (2, 15, 4, 57, 33, 3), (3, 28, 8, 8, 64, 3), (2, 29, 10, 10, 65, 3), (1, 43, 7, 8, 129, 3), (5, 32, 7, 7, 40, 3), (70, 16, 16, 16, 32, 3), (2, 17, 12, 3, 48, 3),
    (1, 32, 6, 6, 32, 1), (2, 33, 8, 9, 257, 1), (3, 300, 6, 6, 40, 1), (2, 256, 4, 8, 129, 1), (1, 255, 10, 10, 256, 1), (4, 64, 7, 7, 300, 1), (90, 48, 16, 16, 272, 1),
]


@pytest.fixture()
def pairs(lib):
    lib.call("set_option", b"conv_pairs", 2)
    yield lib
    lib.call("set_option", b"conv_pairs", 1)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
@pytest.mark.parametrize("precision,limit", [(0, 1e-5), (1, 2e-3)])
@pytest.mark.parametrize("zero", [False, True])
def test_backward_weight(pairs, case, precision, limit, zero):
    L = pairs
    n, c, h, w, k, kr = case
    p = kr // 2
    rng = np.random.default_rng(h * w + c)
    x, dy = rng.standard_normal((n, c, h, w)).astype(F), rng.standard_normal((n, k, h, w)).astype(F)
    gw0 = np.zeros((k, c, kr, kr), F) if zero else rng.standard_normal((k, c, kr, kr)).astype(F)
    want, _ = orc.conv2d_bwd_weight(x, dy, gw0, None, (1, 1), (p,) * 4, (kr, kr))
    L.call("set_option", b"lazy_zero", 1 if zero else 0)
    try:
        gw = L.to_device(np.full(gw0.shape, np.nan, F) if zero else gw0)
        if zero:
            L.call("fill", 0, gw, gw.size, 0.0)
        args = (0, L.to_device(x), L.to_device(dy))
        geo = (n, c, h, w, k, kr, kr, h, w, 1, 1, p, p, precision)
        L.call("conv2d_bwd_weight", *args, gw, None, *geo)
        # the limits are those of the precisions (fp32-equivalent 1e-5, plain TF32 with 11-bit factors) relative to the largest value
        got = gw.numpy()
        assert np.max(np.abs(got - want)) <= limit * np.max(np.abs(want))
        if zero:                                    # nothing depends on timing
            L.call("fill", 0, gw, gw.size, 0.0)
            L.call("conv2d_bwd_weight", *args, gw, None, *geo)
            np.testing.assert_array_equal(gw.numpy(), got)
        L.call("sync", 0)
    finally:
        L.call("set_option", b"lazy_zero", 0)


@pytest.mark.parametrize("case", [(1, 48, 10, 8, 720), (2, 16, 7, 8, 592)], ids=lambda c: "-".join(map(str, c)))
def test_accumulating_into_the_gradient_of_a_small_layer_is_not_slower_on_pairs(lib, case):
    """A reduction of a few K-blocks, so that adding to the gradient is most of the call: the default choice against the same call with
    CTA pairs off (1.8 times as long with one old value in flight per thread)."""
    L = lib
    n, c, h, w, k = case
    x, dy, gw = L.zeros((n, c, h, w)), L.zeros((n, k, h, w)), L.zeros((k, c, 3, 3))
    geo = (n, c, h, w, k, 3, 3, h, w, 1, 1, 1, 1, 0)

    def us(pairs):
        L.call("set_option", b"conv_pairs", pairs)
        times = []
        for _ in range(25):
            L.call("timer_start", 0, 3)
            L.call("conv2d_bwd_weight", 0, x, dy, gw, None, *geo)
            L.call("timer_stop", 0, 3)
            ms = ctypes.c_float()
            L.call("timer_elapsed_ms", 0, 3, ctypes.byref(ms))
            times.append(ms.value * 1e3)
        return float(np.median(times[5:]))
    try:
        off, default = us(0), us(1)
    finally:
        L.call("set_option", b"conv_pairs", 1)
    assert default <= 1.2 * off + 2
