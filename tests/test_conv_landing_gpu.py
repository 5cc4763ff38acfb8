"""The convolution kernels fed by TMA through a landing ring, called again and again on unchanged inputs: every call gives the bits of the
first, and the first agrees with the fp32 FMA kernel.  Large layers with several tiles per CTA whose activations are hot in L2
(backward-weight has just read dy), where a slot of the ring is refilled soonest after it has been read."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32
REPEATS = 50

LAYERS = [(64, 64, 56, 256, 1), (64, 256, 14, 1024, 1), (64, 1024, 14, 256, 1), (32, 64, 56, 64, 3), (16, 256, 28, 128, 3)]     # n, c, h = w, k, kernel


def _differs(L, a, b, work, rows):
    """Whether any element of a differs from b's: the rows of (a - b)^2 are summed on the device (a NaN counts as different)."""
    L.call("axpby", 0, 1.0, a, -1.0, b, work, 0, a.size)
    L.call("sqr", 0, work, work, a.size)
    L.call("reduce_sum2d", 0, work, rows, a.shape[0], a.size // a.shape[0], 1, 0)
    return bool(np.any(rows.numpy() != 0))


def _options(L, **values):
    for name, v in values.items():
        L.call("set_option", name.encode(), v)


@pytest.mark.parametrize("layer", LAYERS, ids=lambda l: "-".join(map(str, l)))
@pytest.mark.parametrize("precision,limit", [(0, 1e-5), (1, 2e-3)])
def test_every_call_gives_the_same_bits(lib, layer, precision, limit):
    L = lib
    n, c, h, k, r = layer
    rng = np.random.default_rng(c + k + h)
    x, w, dy, dx0 = (L.to_device(rng.standard_normal(s, dtype=F)) for s in ((n, c, h, h), (k, c, r, r), (n, k, h, h), (n, c, h, h)))
    y, dx, gw = L.empty((n, k, h, h)), L.empty((n, c, h, h)), L.empty((k, c, r, r))
    geo = (n, c, h, h, k, r, r, h, h, 1, 1, r // 2, r // 2, precision)

    def forward():
        L.call("fill", 0, y, y.size, 7.0)
        L.call("conv2d_fwd", 0, x, w, None, y, *geo)
        L.call("sync", 0)
        return y

    def backward(into):                                 # a delta that holds values, zeros, or zeros still owed
        _options(L, lazy_zero=1 if into == "owed" else 0)
        if into == "values":
            L.call("memcpy_d2d", 0, dx, dx0, dx.size * 4)
        else:
            L.call("fill", 0, dx, dx.size, 0.0)
        L.call("fill", 0, gw, gw.size, 0.0)
        L.call("conv2d_bwd_weight", 0, x, dy, gw, None, *geo)
        L.call("conv2d_bwd_data", 0, dy, w, dx, *geo)
        L.call("sync", 0)
        _options(L, lazy_zero=0)
        return dx
    passes = {"forward": forward, **{i: (lambda i=i: backward(i)) for i in ("values", "zeros", "owed")}}
    try:
        _options(L, conv_path=1)
        reference = {name: run().numpy() for name, run in passes.items()}
        _options(L, conv_path=0, conv_pairs=0)
        for name, run in passes.items():
            got = run()
            first, work, rows = L.empty(got.shape), L.empty(got.shape), L.empty((n,))
            L.call("memcpy_d2d", 0, first, got, got.size * 4)
            # the limits are those of the precisions (fp32-equivalent 1e-5, plain TF32 with 11-bit factors) relative to the largest value
            assert np.max(np.abs(first.numpy() - reference[name])) <= limit * np.max(np.abs(reference[name])), name
            assert sum(_differs(L, run(), first, work, rows) for _ in range(REPEATS)) == 0, name
    finally:
        _options(L, conv_path=0, conv_pairs=1, lazy_zero=0)
