"""The work that users of eddl_b200 have it do, as measurable cases.

Everything goes through the public binding (``eddl_b200.capi``: the C ABI of ``include/eddl_b200.h``) with the calls, in the
order, that EDDL's own host code makes when a net is built on this backend: a training step zeroes the deltas and gradients in
one ``fill_multi``, runs the layers forward, reads loss and metric back, runs the layers backward (every layer ADDS into its
parent's delta and into its gradients) and ends with one multi-tensor optimizer call.  Deferred zero fills are on, as in EDDL.

Kinds of case: ``net`` (a whole training step or a prediction), ``conv`` (the three passes of one Conv2D layer) and ``bn``
(BatchNorm + ReLU, forward and backward).
"""
import ctypes
import math

import torch

from eddl_b200 import capi

DEV = 0


# ---- the cases -------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the small MNIST convnet of the 60-step training run: tiny layers, so launches and host work decide
        _net("cnn", 100, 28, 10, name="cnn_train_b100"),
        # the MNIST multi-layer perceptron with Adam: dense layers, forward and backward, at EDDL's example batch
        _net("mlp", 100, 28, 10, optimizer="adam", name="mlp_train_b100"),
        # VGG-16-BN on 32x32 images: ordinary 3x3 layers that shrink to 2x2 planes
        _net("vgg16bn", 128, 32, 10, name="vgg16bn_train_b128"),
        # ResNet-50 at the headline batch: the largest
        _net("resnet50", 64, 224, 1000, name="resnet50_train_b64"),
        # the same net answering one image: latency of some 170 small calls in a row
        _net("resnet50", 1, 224, 1000, mode="predict", name="resnet50_predict_b1"),
        # the Conv2D layers of the microbenchmark: the compute-bound 3x3, a bottleneck's 1x1, the three-channel stem, 7x7 planes
        _conv(64, 256, 56, 56, 256, 3, 1, 1, name="conv_256ch_56x56_k3"),
        _conv(64, 1024, 14, 14, 256, 1, 1, 0, name="conv_1024ch_14x14_k1"),
        _conv(64, 3, 224, 224, 64, 7, 2, 3, name="conv_stem_224x224_k7s2"),
        _conv(32, 512, 7, 7, 512, 3, 1, 1, name="conv_512ch_7x7_k3"),
        # odd everything: a user's own net on images that are no power of two, with bias and a 5x5 filter
        _conv(6, 20, 45, 37, 36, 5, 1, 2, bias=True, name="conv_odd_20ch_45x37_k5"),
        # the faster precision that a caller may choose (plain TF32), on a strided layer with bias
        _conv(32, 128, 56, 56, 128, 3, 2, 1, bias=True, precision=1, name="conv_tf32_128ch_56x56_k3s2"),
        # BatchNorm + ReLU of a middle stage, the memory-bound half of a residual net
        _bn(64, 512, 28, 28, name="bn_relu_512ch_28x28"),
    ]


def _net(net, batch, hw, classes, mode="train", optimizer="sgd", **more):
    return dict(more, kind="net", net=net, batch=batch, hw=hw, classes=classes, mode=mode, optimizer=optimizer)


def _conv(n, c, h, w, k, kernel, stride, pad, bias=False, precision=0, **more):
    return dict(more, kind="conv", n=n, c=c, h=h, w=w, k=k, kernel=kernel, stride=stride, pad=pad, bias=bias, precision=precision)


def _bn(b, z, h, w, **more):
    return dict(more, kind="bn", b=b, z=z, h=h, w=w)


def _log_int(rng, lo, hi):
    """A whole number whose logarithm is uniform over [lo, hi]: odd ones come as often as even ones."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges: nets at other batch and image sizes, layers of any geometry, BatchNorm of any plane."""
    what = rng.choice(["net", "net", "conv", "conv", "conv", "conv", "bn"])
    if what == "net":
        net = rng.choice(["cnn", "mlp", "vgg16bn", "resnet50"])
        mode = rng.choice(["train", "train", "predict"])
        optimizer = rng.choice(["sgd", "adam"]) if mode == "train" else "sgd"
        classes = _log_int(rng, 2, 1000)
        if net in ("cnn", "mlp"):
            return _net(net, _log_int(rng, 1, 512), rng.randint(16, 40), classes, mode, optimizer)
        if net == "vgg16bn":
            return _net(net, _log_int(rng, 1 if mode == "predict" else 8, 192), 32 * rng.randint(1, 2), classes, mode, optimizer)
        return _net(net, _log_int(rng, 1 if mode == "predict" else 8, 48), 32 * rng.randint(2, 7), classes, mode, optimizer)
    if what == "bn":
        while True:
            b, z, h, w = _log_int(rng, 1, 128), _log_int(rng, 8, 2048), _log_int(rng, 2, 112), _log_int(rng, 2, 112)
            if 64 <= b * h * w and 1 << 12 <= b * z * h * w <= 1 << 25:
                return _bn(b, z, h, w)
    def channels(lo, hi):
        # most layers of real nets have a multiple of 16 channels; the rest are anything
        n = _log_int(rng, lo, hi)
        return max(16, n // 16 * 16) if rng.random() < 0.6 else n
    while True:
        kernel, stride = rng.choice([1, 1, 3, 3, 3, 5, 7]), rng.choice([1, 1, 1, 2])
        pad = rng.choice([kernel // 2, kernel // 2, kernel // 2, 0])
        h = _log_int(rng, 7, 112)
        w = h if rng.random() < 0.6 else _log_int(rng, 7, 112)
        case = _conv(_log_int(rng, 1, 64), channels(1, 1024), h, w, channels(8, 1024), kernel, stride, pad,
                     rng.random() < 0.4, rng.choice([0, 0, 0, 0, 1, 2]))
        if 1e7 <= _conv_flops(case) <= 1e11 and case["n"] * max(case["c"], case["k"]) * h * w <= 1 << 26 and min(h, w) + 2 * pad >= kernel:
            return case


# ---- device memory -----------------------------------------------------------------------------------------------------------
class _View:
    """A buffer of the library as torch sees it; keeps the buffer alive."""

    def __init__(self, array, shape=None):
        self.array = array
        self.__cuda_array_interface__ = {"shape": tuple(shape or array.shape), "typestr": "<f4", "data": (array.ptr.value, False), "version": 2}


def _torch(array):
    return torch.as_tensor(_View(array), device="cuda:%d" % DEV)


def _library():
    L = capi.lib()
    L.call("init", DEV)
    L.call("set_option", b"lazy_zero", 1)
    return L


class _Random:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda:%d" % DEV)
        self.g.manual_seed(int(seed))

    def normal(self, array, scale=1.0, shift=0.0):
        _torch(array).normal_(shift, scale, generator=self.g)

    def uniform(self, array, lo=0.0, hi=1.0):
        _torch(array).uniform_(lo, hi, generator=self.g)

    def labels(self, array):
        rows, cols = array.shape
        t = _torch(array).zero_()
        t.scatter_(1, torch.randint(0, cols, (rows, 1), generator=self.g, device=t.device), 1.0)


class _Fills:
    """The zero fills of one step, one library call."""

    def __init__(self, L, arrays):
        n = len(arrays)
        self.L, self.n = L, n
        self.ptrs = (ctypes.c_void_p * n)(*[p for p, _ in arrays])
        self.sizes = (ctypes.c_size_t * n)(*[s for _, s in arrays])
        self.values = (ctypes.c_float * n)(*([0.0] * n))

    def run(self):
        self.L.call("fill_multi", DEV, self.ptrs, self.sizes, self.values, self.n)


# ---- nets --------------------------------------------------------------------------------------------------------------------
class _Param:
    def __init__(self, offset, size, init):
        self.offset, self.size, self.init = offset, size, init


class _Blob:
    """A layer's output and, when training, the delta that its consumers add into."""

    def __init__(self, L, shape, train):
        self.shape, self.out = shape, L.empty(shape, DEV)
        self.delta = L.empty(shape, DEV) if train else None
        self.size = self.out.size


class _Net:
    """A convnet as EDDL lays it out: one tensor per layer output, parameters in layer order."""

    def __init__(self, case, L):
        self.L, self.train = L, case["mode"] == "train"
        self.fwd, self.bwd, self.blobs, self.params, self.grads, self.keep, self.zeroed_forward = [], [], [], [], [], [], []
        self.total, self.flops, self.floats = 0, 0.0, 0.0
        n, hw, classes = case["batch"], case["hw"], case["classes"]
        channels = 1 if case["net"] in ("cnn", "mlp") else 3
        self.x = self.blob((n, channels, hw, hw))
        self.y = L.empty((n, classes), DEV)
        self.p = self.softmax(getattr(self, case["net"])(self.x, classes))

    # parameters live in flat buffers, every tensor on a 256-byte boundary; refs are resolved when the buffers exist
    def param(self, size, init, trainable=True):
        p = _Param(self.total, size, init)
        self.total += (size + 63) // 64 * 64
        self.params.append(p)
        if trainable:
            self.grads.append(p)
        return p

    def blob(self, shape):
        b = _Blob(self.L, shape, self.train)
        self.blobs.append(b)
        return b

    def temp(self, shape):
        t = self.L.empty(shape, DEV)
        self.keep.append(t)
        return t

    def f(self, name, *args):
        self.fwd.append((name, args))

    def b(self, *calls):
        self.bwd.append(calls)

    def conv(self, x, k, kernel, stride, pad, bias):
        n, c, h, w = x.shape
        oh, ow = (h + 2 * pad - kernel) // stride + 1, (w + 2 * pad - kernel) // stride + 1
        fan = c * kernel * kernel
        wt = self.param(k * fan, ("normal", math.sqrt(2.0 / fan)))
        bs = self.param(k, ("fill", 0.0)) if bias else None
        o = self.blob((n, k, oh, ow))
        geo = (n, c, h, w, k, kernel, kernel, oh, ow, stride, stride, pad, pad, 0)
        self.f("conv2d_fwd", x.out, ("p", wt), ("p", bs), o.out, *geo)
        self.b(("conv2d_bwd_weight", (x.out, o.delta, ("g", wt), ("g", bs)) + geo), ("conv2d_bwd_data", (o.delta, ("p", wt), x.delta) + geo))
        self.flops += 2.0 * n * k * fan * oh * ow * (3 if self.train else 1)
        self.floats += 2.0 * o.size
        return o

    def relu(self, x):
        o = self.blob(x.shape)
        self.f("relu_fwd", x.out, o.out, x.size)
        self.b(("relu_bwd", (o.delta, x.out, x.delta, x.size)))
        return o

    def bn(self, x, relu=True, last=False):
        # scales and shifts of a net that trains stably: the last BatchNorm of a residual branch starts small, and most units
        # are on (with He weights, scale 1 and shift 0 throughout, rounding alone moves a ResNet-50's gradients by percents)
        n, z, rc = x.shape[0], x.shape[1], x.shape[2] * x.shape[3]
        gamma, beta = self.param(z, ("fill", 0.2 if last else 1.0)), self.param(z, ("fill", 1.0 if relu else 0.0))
        mean, var = self.param(z, ("normal", 0.1), False), self.param(z, ("uniform", 0.5, 1.5), False)
        o, opa = self.blob(x.shape), self.temp(x.shape)
        bm, bv, m1, m2 = (self.temp((z,)) for _ in range(4))
        r = self.blob(x.shape) if relu else None
        self.f("bn_fwd", n, z, rc, x.out, o.out, opa, ("p", mean), ("p", var), ("p", gamma), ("p", beta), bm, bv, int(self.train), 1e-3, 0.99, r.out if relu else None)
        back = [("bn_bwd", (n, z, rc, o.delta, opa, x.delta, ("g", gamma), ("g", beta), ("p", gamma), bv, m1, m2))]
        if relu:
            back.insert(0, ("relu_bwd", (r.delta, o.out, o.delta, o.size)))
        self.b(*back)
        self.floats += 2.0 * x.size
        return r if relu else o

    def pool(self, x, kernel, stride, average=False):
        n, c, h, w = x.shape
        oh, ow = (h - kernel) // stride + 1, (w - kernel) // stride + 1
        o = self.blob((n, c, oh, ow))
        geo = (n, c, h, w, oh, ow, kernel, kernel, stride, stride, 0, 0)
        if average:
            self.f("avgpool2d_fwd", x.out, o.out, *geo)
            self.b(("avgpool2d_bwd", (o.delta, x.delta) + geo))
        else:
            ix, iy = self.temp(o.shape), self.temp(o.shape)
            self.f("maxpool2d_fwd", x.out, o.out, ix, iy, *geo)
            self.b(("maxpool2d_bwd", (o.delta, ix, iy, x.delta) + geo))
        self.floats += 2.0 * o.size
        return o

    def pad(self, x, p):
        n, c, h, w = x.shape
        o = self.blob((n, c, h + 2 * p, w + 2 * p))
        geo = (n, c, h, w, p, p, p, p)
        self.f("pad", x.out, o.out, *geo)
        self.b(("pad_bwd", (x.delta, o.delta) + geo))
        return o

    def add_relu(self, a, b):
        # LAdd: out = 0; out += a; out += b
        o = self.blob(a.shape)
        self.f("fill", o.out, o.size, 0.0)
        for t in (a, b):
            self.f("axpby", 1.0, t.out, 1.0, o.out, o.out, 0, o.size)
        self.b(*[("axpby", (1.0, o.delta, 1.0, t.delta, t.delta, 0, o.size)) for t in (a, b)])
        self.floats += 2.0 * o.size
        return self.relu(o)

    def dense(self, x, units):
        rows, cols = x.shape[0], x.size // x.shape[0]
        wt, bs = self.param(cols * units, ("normal", math.sqrt(2.0 / cols))), self.param(units, ("fill", 0.0))
        o = self.blob((rows, units))
        self.f("mult2d", x.out, 0, ("p", wt), 0, o.out, 0, rows, units, cols)
        self.f("sum2d_rowwise", o.out, ("p", bs), o.out, rows, units)
        self.b(("mult2d", (x.out, 1, o.delta, 0, ("g", wt), 1, cols, units, rows)), ("reduce_sum2d", (o.delta, ("g", bs), rows, units, 0, 1)),
               ("mult2d", (o.delta, 0, ("p", wt), 1, x.delta, 1, rows, cols, units)))
        self.flops += 2.0 * rows * cols * units * (3 if self.train else 1)
        self.floats += 2.0 * o.size
        return o

    def softmax(self, x):
        o = self.blob(x.shape)
        self.f("softmax_fwd", x.out, o.out, *x.shape)
        self.b(("softmax_bwd", (o.delta, o.out, x.delta) + tuple(x.shape)))
        return o

    # architectures
    def cnn(self, l, classes):
        for f in (16, 32, 64):
            l = self.pool(self.relu(self.conv(l, f, 3, 1, 1, True)), 2, 2)
        return self.dense(l, classes)

    def mlp(self, l, classes):
        for _ in range(3):
            l = self.relu(self.dense(l, 1024))
        return self.dense(l, classes)

    def vgg16bn(self, l, classes):
        for f in (64, 64, 0, 128, 128, 0, 256, 256, 256, 0, 512, 512, 512, 0, 512, 512, 512, 0):
            l = self.bn(self.conv(l, f, 3, 1, 1, False)) if f else self.pool(l, 2, 2)
        return self.dense(self.relu(self.dense(l, 512)), classes)

    def resnet50(self, l, classes):
        l = self.bn(self.conv(self.pad(l, 3), 64, 7, 2, 0, False))
        l = self.pool(self.pad(l, 1), 3, 2)
        for f, blocks in ((64, 3), (128, 4), (256, 6), (512, 3)):
            for i in range(blocks):
                half, x = f > 64 and i == 0, l
                l = self.bn(self.conv(l, f, 1, 1, 0, False))
                l = self.bn(self.conv(self.pad(l, 1), f, 3, 2, 0, False) if half else self.conv(l, f, 3, 1, 1, False))
                l = self.bn(self.conv(l, 4 * f, 1, 1, 0, False), relu=False, last=True)
                if i == 0:
                    x = self.bn(self.conv(x, 4 * f, 1, 2 if half else 1, 0, False), relu=False)
                l = self.add_relu(x, l)
        return self.dense(self.pool(l, l.shape[2], 1, average=True), classes)


class _NetState:
    def __init__(self, case, seed):
        L = self.L = _library()
        net = self.net = _Net(case, L)
        L.sync(DEV)
        rand = _Random(seed)
        self.adam = case["optimizer"] == "adam"
        self.P = L.empty((net.total,), DEV)
        flat = _torch(self.P).zero_()
        for p in net.params:
            t = flat[p.offset:p.offset + p.size]
            if p.init[0] == "normal":
                t.normal_(0.0, p.init[1], generator=rand.g)
            elif p.init[0] == "uniform":
                t.uniform_(p.init[1], p.init[2], generator=rand.g)
            else:
                t.fill_(p.init[1])
        if case["net"] in ("cnn", "mlp"):
            rand.uniform(net.x.out)
        else:
            rand.normal(net.x.out)
        rand.labels(net.y)
        for b in net.blobs[1:]:
            _torch(b.out).zero_()                 # the frames of padding layers stay zero
        self.fwd = self.bind(net.fwd)
        self.outputs = {"p": _torch(net.p.out)}
        if net.train:
            self.G, self.M = L.empty((net.total,), DEV), L.empty((net.total,), DEV)
            self.V = L.empty((net.total,), DEV) if self.adam else None
            for a in (self.G, self.M) + ((self.V,) if self.adam else ()):
                _torch(a).zero_()
            self.bwd = self.bind([call for calls in reversed(net.bwd) for call in calls])
            self.fills = _Fills(L, [(b.delta.ptr.value, b.size) for b in net.blobs] + [(self.G.ptr.value + 4 * p.offset, p.size) for p in net.grads])
            n = len(net.grads)
            table = [(ctypes.c_void_p * n)(*[a.ptr.value + 4 * p.offset for p in net.grads]) for a in (self.P, self.G, self.M) + ((self.V,) if self.adam else ())]
            sizes = (ctypes.c_size_t * n)(*[p.size for p in net.grads])
            self.step_args = (*table, sizes, n)
            self.step = 0
            self.loss, self.hits = ctypes.c_float(), ctypes.c_int()
            self.outputs.update(params=_torch(self.P), grads=_torch(self.G), m=_torch(self.M))
            if self.adam:
                self.outputs["v"] = _torch(self.V)
        torch.cuda.synchronize()

    def bind(self, calls):
        def arg(a):
            if not isinstance(a, tuple):
                return a
            base, p = a
            return None if p is None else (self.P if base == "p" else self.G).ptr.value + 4 * p.offset
        return [(name, (DEV,) + tuple(arg(a) for a in args)) for name, args in calls]

    def run(self):
        L, net = self.L, self.net
        if not net.train:
            for name, args in self.fwd:
                L.call(name, *args)
            return self.outputs
        self.fills.run()
        for name, args in self.fwd:
            L.call(name, *args)
        rows, cols = net.p.shape
        L.call("cce_value", DEV, net.y, net.p.out, rows, cols, ctypes.byref(self.loss))
        L.call("accuracy", DEV, net.y, net.p.out, rows, cols, ctypes.byref(self.hits))
        L.call("cce_delta", DEV, net.y, net.p.out, net.p.delta, net.p.size)
        for name, args in self.bwd:
            L.call(name, *args)
        self.step += 1                            # the learning rates are so small that every pass is the same step
        if self.adam:
            L.call("adam_multi", DEV, *self.step_args, 1e-8, 0.9, 0.999, 1e-6, self.step)
        else:
            L.call("sgd_momentum_multi", DEV, *self.step_args, 1e-9, 0.9)
        return dict(self.outputs, loss=self.loss.value, hits=float(self.hits.value))


# ---- single layers -----------------------------------------------------------------------------------------------------------
def _conv_out(c):
    return tuple((c[d] + 2 * c["pad"] - c["kernel"]) // c["stride"] + 1 for d in ("h", "w"))


def _conv_flops(c):
    oh, ow = _conv_out(c)
    return 2.0 * c["n"] * c["k"] * c["c"] * c["kernel"] ** 2 * max(oh, 0) * max(ow, 0)


class _ConvState:
    """Forward, backward-weight and backward-data of one Conv2D layer, with the zero fills of the step they belong to."""

    def __init__(self, c, seed):
        L = self.L = _library()
        oh, ow = _conv_out(c)
        shape_w = (c["k"], c["c"], c["kernel"], c["kernel"])
        self.x, self.w, self.dy = L.empty((c["n"], c["c"], c["h"], c["w"]), DEV), L.empty(shape_w, DEV), L.empty((c["n"], c["k"], oh, ow), DEV)
        self.y, self.gw, self.dx = L.empty(self.dy.shape, DEV), L.empty(shape_w, DEV), L.empty(self.x.shape, DEV)
        self.bias, self.gbias = (L.empty((c["k"],), DEV), L.empty((c["k"],), DEV)) if c["bias"] else (None, None)
        L.sync(DEV)
        rand = _Random(seed)
        for a, scale in ((self.x, 1.0), (self.w, 1.0), (self.dy, 1.0)) + (((self.bias, 1.0),) if c["bias"] else ()):
            rand.normal(a, scale)
        zero = [self.gw, self.dx] + ([self.gbias] if c["bias"] else [])
        self.fills = _Fills(L, [(a.ptr.value, a.size) for a in zero])
        self.geo = (c["n"], c["c"], c["h"], c["w"], c["k"], c["kernel"], c["kernel"], oh, ow, c["stride"], c["stride"], c["pad"], c["pad"], c["precision"])
        self.outputs = {"y": _torch(self.y), "gw": _torch(self.gw), "dx": _torch(self.dx)}
        if c["bias"]:
            self.outputs["gbias"] = _torch(self.gbias)
        torch.cuda.synchronize()

    def run(self):
        L = self.L
        self.fills.run()
        L.call("conv2d_fwd", DEV, self.x, self.w, self.bias, self.y, *self.geo)
        L.call("conv2d_bwd_weight", DEV, self.x, self.dy, self.gw, self.gbias, *self.geo)
        L.call("conv2d_bwd_data", DEV, self.dy, self.w, self.dx, *self.geo)
        return self.outputs


class _BnState:
    """BatchNorm + ReLU forward, then ReLU and BatchNorm backward.  What ReLU's backward pass tests is an input of its own: an
    output within rounding of zero would otherwise switch a whole delta on or off."""

    def __init__(self, c, seed):
        L = self.L = _library()
        shape, z = (c["b"], c["z"], c["h"], c["w"]), c["z"]
        names = "x y opa r dr act dy dx"
        for name in names.split():
            setattr(self, name, L.empty(shape, DEV))
        for name in "gamma beta gmean gvar mean var ggamma gbeta m1 m2".split():
            setattr(self, name, L.empty((z,), DEV))
        L.sync(DEV)
        rand = _Random(seed)
        rand.normal(self.x, 1.5, 0.3)
        rand.normal(self.dr, 1e-2)
        rand.normal(self.act, 1.0, 0.2)
        rand.uniform(self.gamma, 0.5, 1.5)
        rand.normal(self.beta, 0.5)
        rand.normal(self.gmean, 0.1)
        rand.uniform(self.gvar, 0.5, 1.5)
        self.fills = _Fills(L, [(a.ptr.value, a.size) for a in (self.dy, self.dx, self.ggamma, self.gbeta)])
        self.dims = (c["b"], z, c["h"] * c["w"])
        self.outputs = {k: _torch(getattr(self, k)) for k in ("y", "opa", "r", "dx", "ggamma", "gbeta", "gmean", "gvar")}
        torch.cuda.synchronize()

    def run(self):
        L = self.L
        self.fills.run()
        L.call("bn_fwd", DEV, *self.dims, self.x, self.y, self.opa, self.gmean, self.gvar, self.gamma, self.beta, self.mean, self.var, 1, 1e-3, 0.99, self.r)
        L.call("relu_bwd", DEV, self.dr, self.act, self.dy, self.act.size)
        L.call("bn_bwd", DEV, *self.dims, self.dy, self.opa, self.dx, self.ggamma, self.gbeta, self.gamma, self.var, self.m1, self.m2)
        return self.outputs


# ---- the interface -------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    return {"net": _NetState, "conv": _ConvState, "bn": _BnState}[case["kind"]](case, seed)


def run(state):
    return state.run()


class _Counter:
    """Stands in for the library where only the sizes of a net are wanted."""

    class Array:
        def __init__(self, shape):
            self.shape, self.size = shape, math.prod(shape)

    def empty(self, shape, dev=0):
        return self.Array(shape)


def work(case):
    if case["kind"] == "conv":
        oh, ow = _conv_out(case)
        x, y, w = case["n"] * case["c"] * case["h"] * case["w"], case["n"] * case["k"] * oh * ow, case["k"] * case["c"] * case["kernel"] ** 2
        # x, w, dy read once, y, gw, dx written once
        return {"bytes": 8.0 * (x + y + w), "flops": 3.0 * _conv_flops(case)}
    if case["kind"] == "bn":
        size = case["b"] * case["z"] * case["h"] * case["w"]
        # x, dr and act read; y, opa, r and dx written
        return {"bytes": 28.0 * size, "flops": 20.0 * size}
    net = _Net(case, _Counter())
    state = {"train": 7 if case["optimizer"] == "adam" else 5, "predict": 1}[case["mode"]]
    # parameters, gradients and moments, the input, and every layer's output written in the forward pass and (training) read
    # once in the backward pass
    floats = net.total * state + net.x.size + net.floats * (1.0 if case["mode"] == "train" else 0.5)
    return {"bytes": 4.0 * floats, "flops": net.flops}


def tolerance(case):
    if case["kind"] == "conv":
        # fp32-equivalent products (three-term split) and sums; plain TF32 keeps 10 bits of each factor
        return {"rel": 1e-3 if case["precision"] == 1 else 1e-5}
    if case["kind"] == "bn":
        return {"rel": 1e-5}
    if case["mode"] == "predict":
        return {"rel": 1e-4}
    # a ReLU or max-pool decision within rounding of a tie may go the other way (a few in ten million do), and its whole delta
    # with it: seen with kernels of the same precision that sum in another order, 2e-3 over BatchNorm nets
    return {"rel": 3e-3, "max": 0.5} if case["net"] in ("cnn", "mlp") else {"rel": 1e-2, "max": 0.9}
