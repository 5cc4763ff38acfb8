"""GPU parity of the kernels for small calls: the cluster FMA GEMM at the edges of its tiles and slices, 2x2 pooling with and without
leftover rows, the sliced bias gradient, loss and metric in one launch, multi-tensor tables that repeat."""
import ctypes

import numpy as np
import pytest

from oracle import eddl_oracle as orc

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (64, 64, 32), (65, 63, 33), (100, 10, 576), (3, 1024, 129), (1024, 100, 2), (130, 70, 4096), (17, 5, 1000), (200, 1100, 31)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("inc", [0, 1])
def test_mult2d_tiles_and_slices(lib, m, n, k, ta, tb, inc):
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    A = rng.standard_normal((k, m) if ta else (m, k)).astype(F); B = rng.standard_normal((n, k) if tb else (k, n)).astype(F)
    C = rng.standard_normal((m, n)).astype(F)
    dc = lib.to_device(C)
    lib.call("mult2d", 0, lib.to_device(A), ta, lib.to_device(B), tb, dc, inc, m, n, k)
    a, b = (A.T if ta else A).astype(np.float64), (B.T if tb else B).astype(np.float64)
    want = a @ b + (C if inc else 0)
    # fp32 sums of k products in any order: |error| <= (k + 1) 2^-24 sum |a||b| (+ the rounding of the last add)
    bound = (k + 2) * 2.0 ** -24 * (np.abs(a) @ np.abs(b) + np.abs(C))
    assert np.all(np.abs(dc.numpy() - want) <= bound)


# both sides of the lines between the kernels: outer products of up to 16 terms over few and many tiles, k steps of a slice, few and many
# slices in memory, the tensor-core kernel from 2^26 multiply-adds on
@pytest.mark.parametrize("m,n,k", [(1100, 1000, 16), (1200, 1600, 16), (1200, 1600, 17), (1200, 1601, 1), (1, 2, 4097), (3, 2, 30001), (1, 64, 12544), (65, 10, 4096), (5, 520, 8200),
                                   (32, 1000, 1025), (8, 4096, 2100), (300, 1000, 1000), (64, 1000, 2048), (9600, 64, 70)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("inc", [0, 1])
def test_mult2d_routes(lib, m, n, k, ta, tb, inc):
    test_mult2d_tiles_and_slices(lib, m, n, k, ta, tb, inc)


def _us(lib, fn, reps=20):
    fn(); fn()
    best = 1e9
    for _ in range(3):
        lib.call("timer_start", 0, 3)
        for _ in range(reps):
            fn()
        lib.call("timer_stop", 0, 3)
        ms = ctypes.c_float()
        lib.call("timer_elapsed_ms", 0, 3, ctypes.byref(ms))
        best = min(best, ms.value * 1e3 / reps)
    return best


def test_a_long_reduction_is_spread_over_the_gpu(lib):
    """8 x 2 outputs: with an eighth of the reduction a call is bound by its launches, so eight times as many terms must cost less than five
    times as much (a fixed number of slices: eight times; measured 70 against 25 us)."""
    def us(k):
        a, b, c = lib.zeros((8, k)), lib.zeros((k, 2)), lib.empty((8, 2))
        return _us(lib, lambda: lib.call("mult2d", 0, a, 0, b, 0, c, 0, 8, 2, k))
    assert us(100000) < 5 * us(12500)


@pytest.mark.parametrize("shape", [(2, 3, 2, 2), (3, 5, 28, 28), (2, 4, 7, 7), (1, 2, 9, 12), (2, 2, 12, 10), (1, 3, 5, 6)])
@pytest.mark.parametrize("lazy", [0, 1])
def test_maxpool_2x2_stride_2(lib, shape, lazy):
    n, c, h, w = shape
    rng = np.random.default_rng(h * w)
    x = rng.integers(-3, 4, shape).astype(F)                   # ties on purpose: the first maximum wins
    oh, ow = h // 2, w // 2
    geo = (n, c, h, w, oh, ow, 2, 2, 2, 2, 0, 0)
    y, ix, iy = lib.empty((n, c, oh, ow)), lib.empty((n, c, oh, ow)), lib.empty((n, c, oh, ow))
    lib.call("maxpool2d_fwd", 0, lib.to_device(x), y, ix, iy, *geo)
    wy, wx, wi = orc.maxpool2d_fwd(x[:, :, :2 * oh, :2 * ow], (2, 2), (2, 2), (0, 0, 0, 0))
    np.testing.assert_array_equal(y.numpy(), wy); np.testing.assert_array_equal(ix.numpy(), wx); np.testing.assert_array_equal(iy.numpy(), wi)
    dy, d0 = rng.standard_normal((n, c, oh, ow)).astype(F), rng.standard_normal(shape).astype(F)
    dx = lib.to_device(d0)
    lib.call("maxpool2d_bwd", 0, lib.to_device(dy), ix, iy, dx, *geo)
    np.testing.assert_array_equal(dx.numpy(), orc.maxpool2d_bwd(dy, wx, wi, shape, d0))
    if lazy:
        big = lib.empty((40 * n, c * 64, h, w))                # large enough for a fill to be recorded: every element must be written
        lib.call("set_option", b"lazy_zero", 1)
        try:
            lib.call("fill", 0, big, big.size, 7.0); lib.call("fill", 0, big, big.size, 0.0)
            reps = (40, 64, 1, 1)
            t = [lib.to_device(np.tile(a, reps)) for a in (dy, wx, wi)]
            lib.call("maxpool2d_bwd", 0, *t, big, 40 * n, 64 * c, *geo[2:])
            np.testing.assert_array_equal(big.numpy(), np.tile(orc.maxpool2d_bwd(dy, wx, wi, shape), reps))
        finally:
            lib.call("set_option", b"lazy_zero", 0)


@pytest.mark.parametrize("n,k,hw", [(1, 1, 1), (2, 3, 45), (7, 16, 784), (3, 700, 49), (5, 33, 4096)])
def test_conv_bias_gradient_slices(lib, n, k, hw):
    rng = np.random.default_rng(k)
    dy, x, g0 = rng.standard_normal((n, k, hw, 1)).astype(F), rng.standard_normal((n, 1, hw, 1)).astype(F), rng.standard_normal(k).astype(F)
    for _ in range(2):                                         # the second call finds the arrival counters as the first left them
        gw, gb = lib.zeros((k, 1, 1, 1)), lib.to_device(g0)
        lib.call("conv2d_bwd_weight", 0, lib.to_device(x), lib.to_device(dy), gw, gb, n, 1, hw, 1, k, 1, 1, hw, 1, 1, 1, 0, 0, 0)
        want = g0 + dy.astype(np.float64).sum(axis=(0, 2, 3))
        assert np.all(np.abs(gb.numpy() - want) <= (n * hw + 2) * 2.0 ** -24 * (np.abs(dy).sum(axis=(0, 2, 3), dtype=np.float64) + np.abs(g0)))


@pytest.mark.parametrize("rows,cols", [(1, 1), (8, 10), (9, 3), (100, 10), (64, 1000), (3000, 7)])
def test_loss_and_metric(lib, rows, cols):
    rng = np.random.default_rng(rows)
    p = rng.random((rows, cols), dtype=F) + F(1e-3); p /= p.sum(axis=1, keepdims=True)
    y = np.eye(cols, dtype=F)[rng.integers(0, cols, rows)]
    dp, dyt = lib.to_device(p), lib.to_device(y)
    loss, hits = ctypes.c_float(), ctypes.c_int()
    for _ in range(2):
        lib.call("cce_value", 0, dyt, dp, rows, cols, ctypes.byref(loss)); lib.call("accuracy", 0, dyt, dp, rows, cols, ctypes.byref(hits))
        assert abs(loss.value - float(orc.cce_value(y, p))) <= 1e-5 * abs(float(orc.cce_value(y, p))) + 1e-6
        assert hits.value == orc.accuracy(y, p)
        p = np.roll(p, 1, axis=1)
        lib.call("memcpy_h2d", 0, dp, np.ascontiguousarray(p).ctypes.data_as(ctypes.c_void_p), p.nbytes)


def test_multi_tensor_tables_are_told_apart(lib):
    """More tensor lists than the library keeps tables for, each used twice: every call works on its own list."""
    rng = np.random.default_rng(0)
    lists = []
    for t in range(20):
        p, g, m = (rng.standard_normal(5 + 37 * t).astype(F) for _ in range(3))
        lists.append((p, g, m, lib.to_device(p), lib.to_device(g), lib.to_device(m)))
    for turn in range(2):
        for i, (p, g, m, dp, dg, dm) in enumerate(lists):
            arr = lambda d: (ctypes.c_void_p * 1)(d.addr)
            lib.call("sgd_momentum_multi", 0, arr(dp), arr(dg), arr(dm), (ctypes.c_size_t * 1)(dp.size), 1, 0.1, 0.9)
            wp, wm = orc.sgd_step(p, g, m, 0.1, 0.9)
            np.testing.assert_array_equal(dp.numpy(), wp); np.testing.assert_array_equal(dm.numpy(), wm)
            lists[i] = (wp, g, wm, dp, dg, dm)


@pytest.mark.parametrize("name,tensors", [("sgd_momentum_multi", 3), ("adam_multi", 4)])
def test_multi_tensor_calls_refuse_what_cannot_be(lib, name, tensors):
    """A list with a missing tensor or a size that no device holds is an error of the call, whatever its other sizes say, and no tensor
    of the list has been touched."""
    from eddl_b200 import capi
    more = (0.1, 0.9) if tensors == 3 else (0.1, 0.9, 0.999, 1e-8, 1)
    good = [lib.to_device(np.full(8, 1 + i, F)) for i in range(tensors)]
    for missing in range(-1, tensors):
        for size in (7, 2 ** 40, 2 ** 62, 2 ** 64 - 8):
            if missing < 0 and size == 7:
                continue
            lists = [(ctypes.c_void_p * 2)(a.addr, None if i == missing else a.addr) for i, a in enumerate(good)]
            with pytest.raises(capi.Error):
                lib.call(name, 0, *lists, (ctypes.c_size_t * 2)(8, size), 2, *more)
    for i, a in enumerate(good):
        np.testing.assert_array_equal(a.numpy(), np.full(8, 1 + i, F))


def test_a_reported_error_changes_nothing_for_the_calls_after_it(lib):
    """A copy that CUDA refuses (cudaErrorInvalidValue, the value 1) is reported once.  The kernels launched next run once, whatever
    route they take: statistics and deltas that are read, changed and written back show a second run."""
    from eddl_b200 import capi
    rng = np.random.default_rng(3)
    n, z, h = 8, 64, 14
    x, d, x0 = (rng.standard_normal((n, z, h, h)).astype(F) for _ in range(3))
    w, g, b = rng.standard_normal((z, z, 3, 3)).astype(F), rng.uniform(0.5, 1.5, z).astype(F), rng.standard_normal(z).astype(F)

    def run(refused):
        def after():
            if refused:
                with pytest.raises(capi.Error):
                    lib.call("memcpy_h2d", 0, None, x.ctypes.data_as(ctypes.c_void_p), 64)
        dx, dd, dg, db, dw = (lib.to_device(a) for a in (x, d, g, b, w))
        y, opa, me, va, m1, m2 = lib.empty(x.shape), lib.empty(x.shape), lib.empty((z,)), lib.empty((z,)), lib.empty((z,)), lib.empty((z,))
        gm, gv, gg, gb = lib.zeros((z,)), lib.zeros((z,)), lib.zeros((z,)), lib.zeros((z,))
        pd, cx, gw, c = lib.to_device(x0), lib.to_device(x0), lib.to_device(w), lib.to_device(x0[0, 0])
        geo = (n, z, h, h, z, 3, 3, h, h, 1, 1, 1, 1, 0)
        after(); lib.call("bn_fwd", 0, n, z, h * h, dx, y, opa, gm, gv, dg, db, me, va, 1, 1e-3, 0.9, None)
        after(); lib.call("conv2d_bwd_data", 0, dd, dw, cx, *geo)
        after(); lib.call("conv2d_bwd_weight", 0, dx, dd, gw, None, *geo)
        after(); lib.call("bn_bwd", 0, n, z, h * h, dd, opa, pd, gg, gb, dg, va, m1, m2)
        after(); lib.call("mult2d", 0, dx, 0, dx, 0, c, 1, h, h, h)
        return [t.numpy() for t in (y, gm, gv, cx, gw, dd, pd, gg, gb, c)]
    for got, want in zip(run(True), run(False)):
        np.testing.assert_array_equal(got, want)
