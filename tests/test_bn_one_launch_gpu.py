"""GPU parity of BatchNorm where a channel is kept in the shared memory of a cluster, at the edges of its shares and block sizes, against
the restatement of the reference's arithmetic; the quotients by sigma against IEEE division; the ReLU backward pass folded in."""
import ctypes

import numpy as np
import pytest

from oracle import eddl_oracle as orc

pytestmark = pytest.mark.gpu
F = np.float32
SHAPES = [(1, 1, 1, 1), (2, 3, 1, 2), (5, 7, 7, 7), (3, 33, 2, 2), (4, 5, 9, 13), (64, 2, 28, 28), (3, 300, 10, 10), (16, 3, 64, 64), (2, 4, 113, 115), (129, 2, 100, 36), (40, 2, 256, 256), (112, 2, 64, 64)]


def launches(L):
    n = ctypes.c_ulonglong()
    L.call("launch_count", 0, ctypes.byref(n))
    return n.value


def _forward(L, x, g, b, relu=True):
    n, z, h, w = x.shape
    y, opa, r = L.empty(x.shape), L.empty(x.shape), L.empty(x.shape)
    gm, gv, me, va = L.to_device(np.full(z, 0.25, F)), L.to_device(np.full(z, 2.0, F)), L.empty((z,)), L.empty((z,))
    dg, db = L.to_device(g), L.to_device(b)
    L.call("bn_fwd", 0, n, z, h * w, L.to_device(x), y, opa, gm, gv, dg, db, me, va, 1, 1e-3, 0.99, r if relu else None)
    return y, opa, r, gm, gv, me, va, dg, db


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_forward_and_backward(lib, shape):
    L = lib
    n, z, h, w = shape
    rng = np.random.default_rng(h * w)
    x = (rng.standard_normal(shape) * 1.5 + 0.3).astype(F)
    g, b = rng.uniform(0.5, 1.5, z).astype(F), rng.standard_normal(z).astype(F)
    y, opa, r, gm, gv, me, va, dg, db = _forward(L, x, g, b)
    # statistics: fp32 sums of N terms in another order than the reference's, combined in double
    mean, sq = x.astype(np.float64).mean(axis=(0, 2, 3)), (x.astype(np.float64) ** 2).mean(axis=(0, 2, 3))
    np.testing.assert_allclose(me.numpy(), mean, rtol=1e-5, atol=1e-6)
    np.testing.assert_allclose(va.numpy(), np.sqrt(np.maximum(sq - mean ** 2, 0) + 1e-3), rtol=2e-5, atol=3e-4 if n * h * w == 1 else 1e-6)
    # given the statistics, every element is exact: the quotient is the correctly rounded one
    m, s = me.numpy()[None, :, None, None], va.numpy()[None, :, None, None]
    o = ((x - m).astype(F) / s).astype(F)
    np.testing.assert_array_equal(opa.numpy(), o)
    want = ((o * g[None, :, None, None]).astype(F) + b[None, :, None, None]).astype(F)
    np.testing.assert_array_equal(y.numpy(), want)
    np.testing.assert_array_equal(r.numpy(), np.where(want > 0, want, F(0)))
    delta, pd0 = rng.standard_normal(shape).astype(F), rng.standard_normal(shape).astype(F)
    gg0, gb0 = rng.standard_normal(z).astype(F), rng.standard_normal(z).astype(F)
    dd, pd, gg, gb, m1, m2 = L.to_device(delta), L.to_device(pd0), L.to_device(gg0), L.to_device(gb0), L.empty((z,)), L.empty((z,))
    L.call("bn_bwd", 0, n, z, h * w, dd, opa, pd, gg, gb, dg, va, m1, m2)
    back = orc.bn_bwd(delta, o, pd0, gg0, gb0, g, va.numpy())
    np.testing.assert_allclose(gg.numpy(), back["gg"], rtol=1e-4, atol=2e-5); np.testing.assert_allclose(gb.numpy(), back["gb"], rtol=1e-4, atol=2e-5)
    np.testing.assert_array_equal(dd.numpy(), (delta * g[None, :, None, None]).astype(F))
    a = (m1.numpy()[None, :, None, None] * o).astype(F) + m2.numpy()[None, :, None, None]
    np.testing.assert_array_equal(pd.numpy(), pd0 + ((dd.numpy() - a.astype(F)).astype(F) / s).astype(F))


def test_the_widest_share_is_one_launch(lib):
    """Sixteen blocks with all the shared memory that a share may have: the device is asked whether it holds such a cluster, and it does."""
    L = lib
    x = np.random.default_rng(6).standard_normal((112, 2, 64, 64)).astype(F)
    dx, y, opa, ones, zeros, me, va = L.to_device(x), L.empty(x.shape), L.empty(x.shape), L.to_device(np.ones(2, F)), L.zeros((2,)), L.empty((2,)), L.empty((2,))
    for _ in range(2):
        before = launches(L)
        L.call("bn_fwd", 0, 112, 2, 4096, dx, y, opa, zeros, ones, ones, zeros, me, va, 1, 1e-3, 0.0, None)
        assert launches(L) == before + 1


@pytest.mark.parametrize("shape", [(64, 4, 28, 28), (30, 50, 7, 7), (8, 2, 256, 256), (64, 300, 2, 2)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("own", [True, False])
def test_relu_backward_folded_in(lib, shape, own):
    """relu_bwd into a delta owed zeros followed by bn_bwd: the bits of the two calls on real zeros, whether ReLU tests the
    BatchNorm's own output (computed again), another tensor (read), or an output overwritten in between."""
    L = lib
    n, z, h, w = shape
    rng = np.random.default_rng(z)
    x = rng.standard_normal(shape).astype(F)
    g, b = rng.uniform(0.5, 1.5, z).astype(F), rng.standard_normal(z).astype(F)
    d, other = rng.standard_normal(shape).astype(F), rng.standard_normal(shape).astype(F)
    E = x.size

    def run(lazy, overwrite=False):
        L.call("set_option", b"lazy_zero", lazy)
        try:
            y, opa, r, gm, gv, me, va, dg, db = _forward(L, x, g, b)
            act = y if own else L.to_device(other)
            if overwrite:
                L.call("scale", 0, y, y, -1.0, E)
            dd, pd, gg, gb, m1, m2 = L.empty(shape), L.empty(shape), L.zeros((z,)), L.zeros((z,)), L.empty((z,)), L.empty((z,))
            for a in (dd, pd):
                L.call("fill", 0, a, E, 5.0); L.call("fill", 0, a, E, 0.0)
            src, before = L.to_device(d), launches(L)        # kept alive: releasing it would run the record
            L.call("relu_bwd", 0, src, act, dd, E)
            L.call("bn_bwd", 0, n, z, h * w, dd, opa, pd, gg, gb, dg, va, m1, m2)
            return launches(L) - before, [t.numpy() for t in (dd, pd, gg, gb, m1, m2)]
        finally:
            L.call("set_option", b"lazy_zero", 0)
    for overwrite in (False, True):
        (folded, got), (separate, want) = run(1, overwrite), run(0, overwrite)
        assert folded == separate - 1                       # relu_bwd was taken over
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("layout", [(8, 16, 1600), (16, 16, 800), (4, 32, 1600), (2, 8, 12800)], ids=lambda l: "x".join(map(str, l)))
def test_relu_backward_folded_in_under_another_layout(lib, layout):
    """bn_bwd over the buffers of an 8 x 32 x 800 forward pass, split into [batch, channels, pixels] in another way: what ReLU tests is the
    tensor as it was written, not gamma and beta of the new channels."""
    L = lib
    rng = np.random.default_rng(5)
    x = rng.standard_normal((8, 32, 20, 40)).astype(F)
    g, b = rng.uniform(0.5, 1.5, 32).astype(F), rng.standard_normal(32).astype(F)
    d, E = rng.standard_normal(x.shape).astype(F), x.size

    def run(lazy):
        L.call("set_option", b"lazy_zero", lazy)
        try:
            y, opa, r, gm, gv, me, va, dg, db = _forward(L, x, g, b)
            dd, pd, gg, gb, m1, m2 = L.empty(x.shape), L.empty(x.shape), L.zeros((32,)), L.zeros((32,)), L.zeros((32,)), L.zeros((32,))
            for a in (dd, pd):
                L.call("fill", 0, a, E, 5.0); L.call("fill", 0, a, E, 0.0)
            src, before = L.to_device(d), launches(L)        # kept alive: releasing it would run the record
            L.call("relu_bwd", 0, src, y, dd, E)
            L.call("bn_bwd", 0, *layout, dd, opa, pd, gg, gb, dg, va, m1, m2)
            return launches(L) - before, [t.numpy() for t in (dd, pd, gg, gb, m1, m2)]
        finally:
            L.call("set_option", b"lazy_zero", 0)
    (folded, got), (separate, want) = run(1), run(0)
    assert folded == separate - 1                           # relu_bwd was taken over
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("shape,folds", [((27, 53, 37, 41), False), ((6, 1866, 79, 11), False), ((125, 296, 2, 29), False), ((64, 1024, 7, 7), True), ((128, 512, 7, 7), True), ((8, 200, 25, 25), True), ((64, 64, 28, 28), True)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "")
@pytest.mark.parametrize("own", [True, False])
def test_relu_backward_is_folded_in_where_that_is_cheaper(lib, shape, folds, own):
    """Scalar two-pass planes in slices, long ones in one slice, short ones with few and with many channels, planes of one launch, 16-byte planes."""
    L = lib
    n, z, h, w = shape
    rng = np.random.default_rng(z)
    x, d, other = (rng.standard_normal(shape, dtype=F) for _ in range(3))
    g, b = rng.uniform(0.5, 1.5, z).astype(F), rng.standard_normal(z).astype(F)
    E = x.size

    def run(lazy):
        L.call("set_option", b"lazy_zero", lazy)
        try:
            y, opa, r, gm, gv, me, va, dg, db = _forward(L, x, g, b)
            act = y if own else L.to_device(other)
            dd, pd, gg, gb, m1, m2 = L.empty(shape), L.empty(shape), L.zeros((z,)), L.zeros((z,)), L.empty((z,)), L.empty((z,))
            for a in (dd, pd):
                L.call("fill", 0, a, E, 0.0)
            src, before = L.to_device(d), launches(L)
            L.call("relu_bwd", 0, src, act, dd, E)
            L.call("bn_bwd", 0, n, z, h * w, dd, opa, pd, gg, gb, dg, va, m1, m2)
            return launches(L) - before, [t.numpy() for t in (dd, pd, gg, gb, m1, m2)]
        finally:
            L.call("set_option", b"lazy_zero", 0)
    (launched, got), (separate, want) = run(1), run(0)
    assert launched == separate - (1 if folds else 0)
    for a, b in zip(got, want):
        np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-5)


def test_relu_backward_with_copies(lib):
    """relu_bwd whose result is added into one or two zero deltas next (LAdd): one kernel, the bits of the separate calls; and a
    record that nothing takes over is run by the next call."""
    L = lib
    n = 300001
    rng = np.random.default_rng(1)
    d, i = rng.standard_normal(n).astype(F), rng.standard_normal(n).astype(F)
    want = np.where(i > 0, d, F(0))
    L.call("set_option", b"lazy_zero", 1)
    try:
        for copies in (0, 1, 2, 3):
            dd, di = L.to_device(d), L.to_device(i)
            pd, c = L.empty((n,)), [L.empty((n,)) for _ in range(copies)]
            for a in [pd] + c:
                L.call("fill", 0, a, n, 5.0); L.call("fill", 0, a, n, 0.0)
            L.call("relu_bwd", 0, dd, di, pd, n)
            for a in c:
                L.call("axpby", 0, 1.0, pd, 1.0, a, a, 0, n)
            for a in c + [pd]:
                np.testing.assert_array_equal(a.numpy(), want)
    finally:
        L.call("set_option", b"lazy_zero", 0)


@pytest.mark.parametrize("which", ["d", "act"])
@pytest.mark.parametrize("shape", [(64, 4, 28, 28), (8, 2, 256, 256)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("then", ["bn_bwd", "axpby"])
def test_relu_backward_whose_input_lies_in_the_next_output(lib, which, shape, then):
    """relu_bwd reads d and act when it is called: what follows may write into their memory, half of which is part of its output here."""
    L = lib
    n, z, h, w = shape
    rng = np.random.default_rng(8)
    x, v, o = (rng.standard_normal(shape).astype(F) for _ in range(3))
    g, b = rng.uniform(0.5, 1.5, z).astype(F), rng.standard_normal(z).astype(F)
    E = x.size

    def run(lazy):
        L.call("set_option", b"lazy_zero", lazy)
        try:
            y, opa, r, gm, gv, me, va, dg, db = _forward(L, x, g, b)
            gg, gb, m1, m2, dd, other = L.zeros((z,)), L.zeros((z,)), L.empty((z,)), L.empty((z,)), L.empty(shape), L.to_device(o)
            arena = L.empty((E + E // 2,))
            low, high = arena.addr, arena.addr + 4 * (E // 2)        # the output; the input that reaches into it
            L.call("memcpy_h2d", 0, high, v.ctypes.data_as(ctypes.c_void_p), v.nbytes)
            L.call("fill", 0, dd, E, 5.0); L.call("fill", 0, dd, E, 0.0); L.call("fill", 0, low, E, 0.0)
            L.call("relu_bwd", 0, high if which == "d" else other, high if which == "act" else other, dd, E)
            if then == "bn_bwd":
                L.call("bn_bwd", 0, n, z, h * w, dd, opa, low, gg, gb, dg, va, m1, m2)
            else:
                L.call("axpby", 0, 1.0, dd, 1.0, low, low, 0, E)
            return [t.numpy() for t in (dd, arena, gg, gb)]
        finally:
            L.call("set_option", b"lazy_zero", 0)
    for got, want in zip(run(1), run(0)):
        np.testing.assert_array_equal(got, want)


def test_quotients_are_the_ieee_ones(lib):
    """Dividends of every magnitude (denormals, zeros, infinities and NaNs among them) by divisors with awkward mantissas: inference-mode
    BatchNorm with mean 0 computes x / sqrt(v + eps) per element."""
    L = lib
    rng = np.random.default_rng(2)
    z, rc = 64, 40000
    x = (rng.uniform(1, 2, (1, z, rc)) * np.exp2(rng.integers(-140, 120, (1, z, rc))) * rng.choice([-1, 1], (1, z, rc))).astype(F)
    x[0, :, :8] = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, 3e38, 1.0], F)
    half = rng.uniform(1, 2, (1, z, rc)).astype(F)
    x = np.where(rng.random(x.shape) < 0.7, half, x).astype(F)
    v = np.concatenate([rng.uniform(1e-6, 10, z - 4), [1e-18, 1e20, 0.25, 3.9999998]]).astype(F)
    y, opa, va = L.empty(x.shape), L.empty(x.shape), L.empty((z,))
    L.call("bn_fwd", 0, 1, z, rc, L.to_device(x), y, opa, L.zeros((z,)), L.to_device(v), None, None, None, va, 0, 0.0, 0.99, None)
    with np.errstate(all="ignore"):
        want = (x / va.numpy()[None, :, None]).astype(F)
    np.testing.assert_array_equal(y.numpy(), want)
