"""The work that programs built on this library have it do, as cases whose time can be measured.

A case is one training-step piece issued through the exported entry points: a Conv2D layer, a depthwise-separable layer, a
Linear layer, an attention layer, a MobileBERT-style encoder block, a matrix product, or the whole residual network of
pulp-trainlib_b200/nets.  Tensors live in device memory (torch tensors handed over by address) unless the case says `host`.
"""
import ctypes
import importlib
import math
import os

import numpy as np
import torch

pkg = importlib.import_module("pulp-trainlib_b200")
lib = pkg.load()
if torch.cuda.is_available():
    torch.cuda.init()
    lib.trainlib_init(torch.cuda.current_device())

NET_PATH = os.path.join(os.path.dirname(pkg.LIB_PATH), "nets", "libresnet8_b200.so")


def _net():
    net = ctypes.CDLL(NET_PATH)
    net.resnet8_param_count.restype = ctypes.c_size_t
    net.resnet8_workspace_floats.restype = ctypes.c_size_t; net.resnet8_workspace_floats.argtypes = [ctypes.c_int]
    net.resnet8_init_params.argtypes = [ctypes.c_void_p, ctypes.c_uint]
    net.resnet8_bind.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]; net.resnet8_bind.restype = ctypes.c_int
    net.resnet8_forward.argtypes = [ctypes.c_void_p] * 3
    net.resnet8_update.argtypes = [ctypes.c_float]
    net.resnet8_logits.restype = ctypes.c_void_p
    net.resnet8_flops_per_stream.restype = ctypes.c_double
    return net


NET = _net()
ESIZE = {"fp32": 4, "fp16": 2}


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # One Conv2D layer's training step at batch 1 (configuration 1 of the benchmark): on-device learning of a small CNN,
        # the call sequence the code generator writes, with the tensors kept in device memory.
        dict(name="conv_layer", kind="conv", dtype="fp32", n=1, cin=16, h=32, w=32, cout=32, k=3, stride=1, bias=False, host=False),
        # The same step by a program that only relinks: its tensors are ordinary host arrays, every call stages them.
        dict(name="conv_layer_host", kind="conv", dtype="fp32", n=1, cin=16, h=32, w=32, cout=32, k=3, stride=1, bias=False, host=True),
        # A half-precision Conv2D layer over a batch of independent streams, planes that are no power of two.
        dict(name="conv_fp16_streams", kind="conv", dtype="fp16", n=128, cin=24, h=28, w=28, cout=48, k=3, stride=1, bias=True, host=False),
        # A depthwise-separable layer (depthwise 3x3, pointwise 1x1) over a batch of streams: mobile networks.
        dict(name="separable_streams", kind="separable", dtype="fp32", n=64, c=64, h=28, w=28, cout=128),
        # Linear layers at batch 1 (configuration 2): the smallest and one of the largest of its sweep.
        dict(name="linear_small", kind="linear", dtype="fp32", n=1, inn=256, out=256, bias=False),
        dict(name="linear_fp16_wide", kind="linear", dtype="fp16", n=1, inn=4096, out=1024, bias=False),
        # Multi-head self-attention forward and backward (configuration 3).
        dict(name="attention", kind="mhsa", dtype="fp32", L=256, E=256, F=256, heads=4),
        # MobileBERT-style encoder block in half precision (configuration 4), replayed as a recorded graph.
        dict(name="encoder_block_fp16", kind="block", dtype="fp16", L=128, H=512, B=128, heads=4, nffn=4, FF=512),
        # The matrix product on its own: a large square one in half precision, a ragged one in single precision with B transposed.
        dict(name="mm_fp16_4096", kind="mm", dtype="fp16", N=4096, K=4096, M=4096, trans_B=0),
        dict(name="mm_fp32_ragged", kind="mm", dtype="fp32", N=1000, K=600, M=1300, trans_B=1),
        # The residual network on many independent streams (configuration 5, replayed as a recorded graph) and on a few hundred
        # (the share of one GPU in a multi-GPU job is of that order), issued call by call.
        dict(name="resnet8_4096", kind="resnet", n=4096, replay=True),
        dict(name="resnet8_200", kind="resnet", n=200, replay=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["conv", "conv", "conv", "separable", "linear", "linear", "mhsa", "block", "mm", "mm", "resnet"])
    dtype = rng.choice(["fp32", "fp16"])
    if kind == "conv":
        while True:
            c = dict(kind=kind, dtype=dtype, n=1 if rng.random() < 0.4 else _log(rng, 2, 512), cin=_log(rng, 1, 64), h=rng.randint(6, 48), w=rng.randint(6, 48),
                     cout=_log(rng, 4, 96), k=rng.choice([1, 3, 3, 3, 5]), stride=rng.choice([1, 1, 1, 2]), bias=rng.random() < 0.5, host=False)
            c["host"] = c["n"] == 1 and rng.random() < 0.3
            if work(c)["flops"] < 4e10:
                return c
    if kind == "separable":
        return dict(kind=kind, dtype=dtype, n=_log(rng, 1, 128), c=_log(rng, 8, 96), h=rng.randint(7, 40), w=rng.randint(7, 40), cout=_log(rng, 8, 160))
    if kind == "linear":
        return dict(kind=kind, dtype=dtype, n=1 if rng.random() < 0.6 else _log(rng, 2, 512), inn=_log(rng, 16, 4096), out=_log(rng, 10, 4096), bias=rng.random() < 0.5)
    if kind == "mhsa":
        heads = rng.choice([1, 2, 4, 8])
        return dict(kind=kind, dtype=dtype, L=_log(rng, 24, 512), E=_log(rng, 24, 384), F=heads * rng.choice([8, 12, 16, 32, 40, 64]), heads=heads)
    if kind == "block":
        return dict(kind=kind, dtype=dtype, L=_log(rng, 32, 256), H=rng.choice([128, 256, 384, 512]), B=rng.choice([64, 96, 128]), heads=4, nffn=rng.randint(1, 4),
                    FF=rng.choice([128, 256, 512]))
    if kind == "mm":
        return dict(kind=kind, dtype=dtype, N=_log(rng, 16, 4096), K=_log(rng, 16, 4096), M=_log(rng, 16, 4096), trans_B=rng.randint(0, 1))
    return dict(kind="resnet", n=_log(rng, 1, 2048), replay=rng.random() < 0.5)


def _conv_out(c):
    pad = c["k"] // 2
    return (c["h"] - c["k"] + 2 * pad) // c["stride"] + 1, (c["w"] - c["k"] + 2 * pad) // c["stride"] + 1


def work(c):
    """Bytes with every input read once and every output written once; floating-point operations at two per multiply-add."""
    es, kind = ESIZE.get(c.get("dtype"), 4), c["kind"]
    if kind == "conv":
        ho, wo = _conv_out(c)
        x, y, wt = c["n"] * c["cin"] * c["h"] * c["w"], c["n"] * c["cout"] * ho * wo, c["cout"] * c["cin"] * c["k"] ** 2
        return {"bytes": es * (2 * x + 2 * y + 3 * wt), "flops": 6.0 * y * c["cin"] * c["k"] ** 2}
    if kind == "separable":
        px = c["n"] * c["h"] * c["w"]
        return {"bytes": es * (px * (4 * c["c"] + 2 * c["cout"]) + 2 * (9 * c["c"] + c["c"] * c["cout"])), "flops": 6.0 * px * c["c"] * (9 + c["cout"])}
    if kind == "linear":
        io = c["inn"] * c["out"]
        return {"bytes": es * (2 * io + 2 * c["n"] * (c["inn"] + c["out"])), "flops": 6.0 * c["n"] * io}
    if kind == "mhsa":
        L, E, F = c["L"], c["E"], c["F"]
        return {"bytes": es * (8 * E * F + 4 * E * L + 8 * F * L + 2 * c["heads"] * L * L), "flops": 6.0 * (3 * L * E * F + 2 * L * L * F + L * F * E)}
    if kind == "block":
        L, H, B, FF = c["L"], c["H"], c["B"], c["FF"]
        macs = L * H * B + 4 * L * B * B + 2 * L * L * B + c["nffn"] * 2 * L * B * FF + L * B * H
        return {"bytes": es * (2 * (2 * H * B + 4 * B * B + c["nffn"] * 2 * B * FF) + 3 * L * H), "flops": 6.0 * macs}
    if kind == "mm":
        return {"bytes": es * (c["N"] * c["K"] + c["K"] * c["M"] + c["N"] * c["M"]), "flops": 2.0 * c["N"] * c["K"] * c["M"]}
    return {"bytes": 4.0 * (c["n"] * (3 * 32 * 32 + 10 + 11) + 3 * NET.resnet8_param_count()), "flops": NET.resnet8_flops_per_stream() * c["n"]}


def tolerance(c):
    if c["kind"] == "resnet":
        # a pre-activation within rounding of zero flips its ReLU gate between two correct implementations, and the summed
        # gradients of the layers below it move by that stream's share
        return {"rel": 3e-3}
    if c.get("dtype") == "fp16":
        # eleven bits of mantissa; the attention layers also round q, k, v and the probabilities, a block some sixty tensors
        return {"rel": {"mhsa": 5e-3, "block": 1e-2}.get(c["kind"], 1e-3)}
    return {"rel": {"mhsa": 2e-5, "block": 5e-5}.get(c["kind"], 1e-5)}


# ------------------------------------------------------------------------------------------------ building blocks
class State(object):
    """Tensors of one program and the argument structs over them."""

    def __init__(self, case, seed):
        self.case = case
        self.half = case.get("dtype") == "fp16"
        self.host = bool(case.get("host"))
        self.dt = torch.float16 if self.half else torch.float32
        self.sfx = "_fp16" if self.half else ""
        self.p = "fp16" if self.half else "fp32"
        self.gen = torch.Generator("cuda").manual_seed(int(seed))
        self.keep = pkg.Keep()
        self.calls, self.out, self.graph = [], None, None

    def __del__(self):
        if self.graph:
            lib.trainlib_synchronize()
            lib.trainlib_graph_destroy(self.graph)

    def _own(self, t):
        t = t.to(self.dt)
        return t.cpu().numpy() if self.host else t

    def normal(self, *shape, scale=1.0):
        return self._own(torch.randn(shape, device="cuda", generator=self.gen) * scale)

    def uniform(self, *shape):
        return self._own(torch.rand(shape, device="cuda", generator=self.gen) * 2 - 1)

    def zeros(self, *shape):
        return self._own(torch.zeros(shape, device="cuda"))

    def ptr(self, t):
        if isinstance(t, torch.Tensor):
            self.keep.hold(t)
            return t.data_ptr()
        return t

    def blob(self, data, diff=None, C=1, H=1, W=1, dim=None):
        return pkg.make_blob(self.keep, self.ptr(data), self.ptr(diff), C=C, H=H, W=W, dim=dim, half=self.half)

    def flat(self, data, diff=None, dim=None):
        dim = int(math.prod(data.shape)) if dim is None else dim
        return self.blob(data, diff, W=dim, dim=dim)

    def args(self, struct, **fields):
        return pkg.make_args(self.keep, struct, **{k: self.ptr(v) for k, v in fields.items()})

    def call(self, name, args, into=None):
        """append one entry-point call to the program"""
        (self.calls if into is None else into).append((getattr(lib, name), ctypes.byref(args)))

    def zero(self, t, into=None):
        """append a clear of one device tensor (buffers that a backward pass adds to)"""
        f, p, n = lib.trainlib_memset, t.data_ptr(), t.numel() * t.element_size()
        (self.calls if into is None else into).append((lambda _: f(p, 0, n), None))


def _conv(s, c):
    n, cin, h, w, cout, k = (c[i] for i in ("n", "cin", "h", "w", "cout", "k"))
    ho, wo = _conv_out(c)
    x, wt, dy = s.uniform(n, cin, h, w), s.uniform(cout, cin, k, k), s.normal(n, cout, ho, wo, scale=1.0 / math.sqrt(n * ho * wo))
    y, dw, dx = s.zeros(n, cout, ho, wo), s.zeros(cout, cin, k, k), s.zeros(n, cin, h, w)
    b, db, one = s.normal(cout), s.zeros(cout), s.zeros(4)
    a = s.args("Conv2D_args" + s.sfx, input=s.blob(x, dx, cin, h, w), coeff=s.blob(wt, dw, cin, k, k, dim=cout * cin * k * k), bias=s.flat(b, db),
               output=s.blob(y, dy, cout, ho, wo), Lpad=k // 2, Rpad=k // 2, Upad=k // 2, Dpad=k // 2, stride_h=c["stride"], stride_w=c["stride"],
               i2c_buffer=one, bt_buffer=one, skip_wg_grad=0, skip_in_grad=0, HWC=0, opt_matmul_type_fw=0, opt_matmul_type_wg=0, opt_matmul_type_ig=0,
               USE_BIASES=1 if c["bias"] else 0, USE_IM2COL=0, USE_DMA_IM2COL=0)
    o = s.args("optim_args" + s.sfx, weights=s.flat(wt, dw), biases=s.flat(b, db), learning_rate=1e-3, weight_decay_lambda=0.0, use_biases=1 if c["bias"] else 0)
    for f in ("fw_cl", "bw_param_grads_cl", "bw_input_grads_cl"):
        s.call("pulp_conv2d_%s_%s" % (s.p, f), a)
    s.call("pulp_gradient_descent_%s" % s.p, o)
    s.out = [y, dw, dx, wt] + ([db, b] if c["bias"] else [])


def _separable(s, c):
    n, ch, h, w, cout = (c[i] for i in ("n", "c", "h", "w", "cout"))
    x, wd, wp = s.normal(n, ch, h, w), s.normal(ch, 3, 3, scale=1 / 3), s.normal(cout, ch, scale=1 / math.sqrt(ch))
    m, y, dy = s.zeros(n, ch, h, w), s.zeros(n, cout, h, w), s.normal(n, cout, h, w, scale=1 / math.sqrt(n * h * w))
    dx, dm, dwd, dwp, tr = s.zeros(n, ch, h, w), s.zeros(n, ch, h, w), s.zeros(ch, 3, 3), s.zeros(cout, ch), s.zeros(cout * ch + ch * h * w)
    strides = {} if s.half else dict(stride_h=1, stride_w=1)
    dwa = s.args("DepthWise_Conv_args" + s.sfx, input=s.blob(x, dx, ch, h, w), coeff=s.blob(wd, dwd, ch, 3, 3), output=s.blob(m, dm, ch, h, w),
                 Lpad=1, Rpad=1, Upad=1, Dpad=1, skip_wg_grad=0, skip_in_grad=0, HWC=0, **strides)
    pwa = s.args("PointWise_Conv_args" + s.sfx, input=s.blob(m, dm, ch, h, w), coeff=s.blob(wp, dwp, ch, 1, 1, dim=cout * ch), output=s.blob(y, dy, cout, h, w),
                 transpose_buffer=tr, skip_wg_grad=0, skip_in_grad=0, opt_matmul_type_fw=0, opt_matmul_type_wg=0, opt_matmul_type_ig=0, HWC=0)
    s.call("pulp_conv_dw_%s_fw_cl" % s.p, dwa)
    s.call("pulp_conv_pw_%s_fw_cl" % s.p, pwa)
    s.call("pulp_conv_pw_%s_bw_cl" % s.p, pwa)
    s.call("pulp_conv_dw_%s_bw_cl" % s.p, dwa)
    s.out = [m, y, dm, dwp, dx, dwd]


def _linear(s, c):
    n, inn, out = c["n"], c["inn"], c["out"]
    W, x, dy, b = s.normal(out, inn, scale=1 / math.sqrt(inn)), s.normal(n, inn), s.normal(n, out), s.normal(out)
    y, dW, dx, db = s.zeros(n, out), s.zeros(out, inn), s.zeros(n, inn), s.zeros(out)
    a = s.args("Linear_args" + s.sfx, input=s.flat(x, dx, inn), coeff=s.blob(W, dW, H=out, W=inn), bias=s.flat(b, db), output=s.flat(y, dy, out),
               skip_wg_grad=0, skip_in_grad=0, opt_matmul_type_fw=0, opt_matmul_type_wg=0, opt_matmul_type_ig=0, use_biases=1 if c["bias"] else 0)
    s.call("pulp_linear_%s_fw_cl" % s.p, a)
    s.call("pulp_linear_%s_bw_cl" % s.p, a)
    s.out = [y, dW, dx] + ([db] if c["bias"] else [])


def _mhsa(s, c):
    L, E, F, h = c["L"], c["E"], c["F"], c["heads"]
    x, dx, y, dy = s.normal(E, L), s.zeros(E, L), s.zeros(E, L), s.normal(E, L)
    ws, dws = [s.normal(E, F, scale=1 / math.sqrt(E)) for _ in range(4)], [s.zeros(F, E) for _ in range(3)] + [s.zeros(E, F)]
    bs, dbs = [s.zeros(F) for _ in range(3)], [s.zeros(F) for _ in range(3)]
    act, dact = [s.zeros(F, L) for _ in range(4)], [s.zeros(F, L) for _ in range(4)]
    sm, dsm = s.zeros(h, L, L), s.zeros(h, L, L)
    a = s.args("Mhsa_args" + s.sfx, input=s.blob(x, dx, 1, L, E), n_heads=h, output=s.blob(y, dy, 1, L, E),
               coeff_in_q=s.blob(ws[0], dws[0], 1, F, E), coeff_in_k=s.blob(ws[1], dws[1], 1, F, E), coeff_in_v=s.blob(ws[2], dws[2], 1, F, E),
               coeff_out=s.blob(ws[3], dws[3], 1, E, F), bias_in_q=s.flat(bs[0], dbs[0]), bias_in_k=s.flat(bs[1], dbs[1]), bias_in_v=s.flat(bs[2], dbs[2]),
               q=s.blob(act[0], dact[0], 1, L, F), k=s.blob(act[1], dact[1], 1, L, F), v=s.blob(act[2], dact[2], 1, L, F),
               attention_map=s.blob(act[3], dact[3], 1, L, F), temp_buffer=s.zeros(max(L * L, E * F, L * F, E * L)), grad=s.zeros(L * L),
               softmax_buffer=s.blob(sm, dsm, 1, h, L * L), maxes=s.zeros(L), sums=s.zeros(L),
               opt_matmul_type_fw=0, opt_matmul_type_wg=0, opt_matmul_type_ig=0)
    s.call("pulp_mhsa_%s_fw_cl" % s.p, a)
    s.zero(dx)                                    # the backward adds to the input gradient
    s.call("pulp_mhsa_%s_bw_cl" % s.p, a)
    s.out = [y, sm, dx] + act + dws


class _LnArgs(ctypes.Structure):
    """struct trainlib_layernorm_args"""
    _fields_ = [(n, ctypes.c_void_p) for n in ("x", "weight", "bias", "output", "eps")] + [("size", ctypes.c_int), ("step_size", ctypes.c_int)] + \
               [(n, ctypes.c_void_p) for n in ("dy", "dx", "dweight", "dbias")]


def _block(s, c):
    """x1 = LN(X Wbi); x = LN(x1 + MHSA(x1)); nffn times x = LN(x + GELU(x W1) W2); Y = LN(X + x Wbo); MSE against a target.
    Linear layers are matrix products and their backward two products and one transpose; backward calls run in reverse order."""
    L, H, B, FF, heads = c["L"], c["H"], c["B"], c["FF"], c["heads"]
    sfx, p = s.sfx, s.p
    fw, eps = s.calls, s.keep.hold(np.array([1e-3], np.float16 if s.half else np.float32))
    params = []

    def act(*shape):
        return s.zeros(*shape), s.zeros(*shape)

    def param(t):
        params.append((t, s.zeros(*t.shape)))
        return params[-1]

    def weight(*shape):
        return param(s.normal(*shape, scale=0.02))

    def product(into, A, Bm, C, n, k, m, trans):
        s.call("mm" + sfx, s.args("matMul_args" + sfx, A=A, B=Bm, C=C, N=n, K=k, M=m, trans_B=trans, USE_BIASES=0), into)

    def linear(x, w, y):
        (l, k), m, bw = x[0].shape, w[0].shape[1], []
        product(fw, x[0], w[0], y[0], l, k, m, 0)
        product(bw, y[1], w[0], x[1], l, m, k, 1)
        xt = s.zeros(k, l)
        s.call("transpose_matrix" + sfx, s.args("transp_args" + sfx, in_matrix=x[0], out_matrix=xt, N=l, M=k), bw)
        product(bw, xt, y[1], w[1], k, l, m, 0)
        return bw

    def norm(x, y):
        rows, width = x[0].shape
        w, b = param(1 + s.normal(width, scale=0.02)), weight(width)
        a = s.keep.hold(_LnArgs())
        a.x, a.weight, a.bias, a.output, a.eps = s.ptr(x[0]), s.ptr(w[0]), s.ptr(b[0]), s.ptr(y[0]), eps.ctypes.data
        a.size, a.step_size = rows * width, width
        a.dy, a.dx, a.dweight, a.dbias = s.ptr(y[1]), s.ptr(x[1]), s.ptr(w[1]), s.ptr(b[1])
        s.call("trainlib_layernorm_fp16_fw_cl" if s.half else "pulp_layerNorm_fp32_fw_cl", a)
        bw = []
        s.call("trainlib_layernorm_%s_bw_cl" % p, a, bw)
        return bw

    def gelu(x, y):
        a = s.args("act_args" + sfx, input=s.flat(*x), output=s.flat(*y), H=1, W=x[0].numel())
        s.call("pulp_gelu_fp16_fw_cl" if s.half else "pulp_gelu_tanh_approx_fp32_fw_cl", a)
        bw = []
        s.call("trainlib_gelu_%s_bw_cl" % p, a, bw)
        return bw

    def residual(skip, branch, out):
        a = s.args("SkipConn_args" + sfx, skip=s.flat(*skip), lout=s.flat(*branch), output=s.flat(*out), skip_in_grad=0)
        s.call("pulp_residualconn_%s_fw" % p, a)
        copy, add = [], []
        s.call("pulp_residualconn_%s_bw" % p, a, copy)
        s.call("pulp_sumnode_%s_bw" % p, a, add)
        return copy, add

    def attention(x, y):
        ws = [weight(B, B) for _ in range(4)]
        q, k, v, att = act(B, L), act(B, L), act(B, L), act(B, L)
        sm, zb = act(heads, L, L), act(B)
        b2 = lambda t, hh, ww: s.blob(t[0], t[1], 1, hh, ww)
        a = s.args("Mhsa_args" + sfx, input=b2(x, L, B), input_bn=s.blob(x[0], None, 1, L, B), n_heads=heads, output=b2(y, L, B),
                   coeff_in_q=b2(ws[0], B, B), coeff_in_k=b2(ws[1], B, B), coeff_in_v=b2(ws[2], B, B), coeff_out=b2(ws[3], B, B),
                   bias_in_q=s.flat(*zb), bias_in_k=s.flat(*zb), bias_in_v=s.flat(*zb), bias_out=s.flat(*zb),
                   q=b2(q, L, B), k=b2(k, L, B), v=b2(v, L, B), attention_map=b2(att, L, B), temp_buffer=s.zeros(max(L * L, B * B, L * B)), grad=s.zeros(L * L),
                   softmax_buffer=b2(sm, heads, L * L), maxes=s.zeros(L), sums=s.zeros(L), opt_matmul_type_fw=0, opt_matmul_type_wg=0, opt_matmul_type_ig=0)
        s.call("pulp_mhsa_mobilebert_inference_%s_fw_cl" % p, a)
        bw = []
        s.zero(x[1], bw)
        s.call("pulp_mhsa_mobilebert_inference_%s_bw_cl" % p, a, bw)
        return bw

    X, T = (s.normal(L, H), s.zeros(L, H)), s.normal(L, H)
    t0, x1, at, r1, x = (act(L, B) for _ in range(5))
    bw_bi = linear(X, weight(H, B), t0)
    bw_n1 = norm(t0, x1)
    bw_at = attention(x1, at)
    cp1, add1 = residual(x1, at, r1)
    bw_n2 = norm(r1, x)
    ffn = []
    for _ in range(c["nffn"]):
        hid, gl, o, r, nxt = act(L, FF), act(L, FF), act(L, B), act(L, B), act(L, B)
        b1 = linear(x, weight(B, FF), hid)
        bg = gelu(hid, gl)
        b2_ = linear(gl, weight(FF, B), o)
        cp, ad = residual(x, o, r)
        ffn.append(norm(r, nxt) + cp + b2_ + bg + b1 + ad)
        x = nxt
    t1, r2, Y = act(L, H), act(L, H), act(L, H)
    bw_bo = linear(x, weight(B, H), t1)
    cpo, addo = residual(X, t1, r2)
    bw_no = norm(r2, Y)
    loss = s.zeros(1)
    la = s.args("loss_args" + sfx, output=s.flat(*Y), target=T, wr_loss=loss)
    s.call("pulp_MSELoss" + sfx, la)
    s.call("pulp_MSELoss_backward" + sfx, la)
    # loss scaling, as half-precision training needs it
    s.call("pulp_scalar_mul_%s_cl" % p, s.args("scalar_mul_args" + sfx, input=Y[1], scalar=1024.0, dim=L * H))
    s.calls = s.calls + bw_no + cpo + bw_bo + sum(reversed(ffn), []) + bw_n2 + cp1 + bw_at + add1 + bw_n1 + bw_bi + addo
    s.out = [Y[0], loss, X[1]] + [g for _, g in params]
    _run_calls(s)                                 # once, so that the library's scratch has its final size
    lib.trainlib_graph_begin()
    _run_calls(s)
    s.graph = lib.trainlib_graph_end()
    pkg.check(lib)


def _mm(s, c):
    N, K, M = c["N"], c["K"], c["M"]
    A, B, C = s.normal(N, K, scale=1 / math.sqrt(K)), s.normal(*((M, K) if c["trans_B"] else (K, M))), s.zeros(N, M)
    s.call("mm" + s.sfx, s.args("matMul_args" + s.sfx, A=A, B=B, C=C, N=N, K=K, M=M, trans_B=c["trans_B"], USE_BIASES=0))
    s.out = [C]


def _resnet(s, c, seed):
    n, count = c["n"], NET.resnet8_param_count()
    host = np.zeros(count, np.float32)
    NET.resnet8_init_params(host.ctypes.data, int(seed) & 0x7fffffff)
    s.params, s.grads = torch.from_numpy(host).cuda(), torch.zeros(count, device="cuda")
    s.ws = torch.zeros(NET.resnet8_workspace_floats(n), device="cuda")
    s.img, s.loss = s.normal(n, 3, 32, 32), s.zeros(n)
    s.lab = torch.nn.functional.one_hot(torch.randint(0, 10, (n,), device="cuda", generator=s.gen), 10).float()
    _resnet_bind(s)
    at = (NET.resnet8_logits() - s.ws.data_ptr()) // 4
    s.out = [s.loss, s.ws[at:at + 10 * n].view(n, 10), s.grads, s.params]
    torch.cuda.synchronize()
    if c["replay"]:
        before = s.params.clone()
        _resnet_step(s)
        lib.trainlib_graph_begin()
        _resnet_step(s)
        s.graph = lib.trainlib_graph_end()
        pkg.check(lib)
        lib.trainlib_synchronize()
        s.params.copy_(before)


def _resnet_bind(s):
    NET.resnet8_bind(s.case["n"], s.params.data_ptr(), s.grads.data_ptr(), s.ws.data_ptr())


def _resnet_step(s):
    NET.resnet8_forward(s.img.data_ptr(), s.lab.data_ptr(), s.loss.data_ptr())
    NET.resnet8_backward()
    NET.resnet8_update(1e-2 / s.case["n"])        # the gradient is a sum over the streams


def _run_calls(s):
    for fn, a in s.calls:
        fn(a)


def prepare(case, seed):
    s = State(case, seed)
    lib.trainlib_set_streams(case.get("n", 1))
    if case["kind"] == "resnet":
        _resnet(s, case, seed)
    else:
        {"conv": _conv, "separable": _separable, "linear": _linear, "mhsa": _mhsa, "block": _block, "mm": _mm}[case["kind"]](s, case)
    torch.cuda.synchronize()
    return s


def run(s):
    if s.graph:
        lib.trainlib_graph_launch(s.graph)
    elif s.case["kind"] == "resnet":
        _resnet_bind(s)                           # the network keeps one set of buffers at a time
        _resnet_step(s)
    else:
        lib.trainlib_set_streams(s.case.get("n", 1))
        _run_calls(s)
    return s.out
