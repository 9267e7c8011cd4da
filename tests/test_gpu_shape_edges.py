"""Shapes at the edges of the kernels' tiles and dispatch rules (partial tiles, odd strides, several streams per tile, rows
longer than a tile, split contractions), fp32 and fp16, against the CPU oracle."""
import numpy as np
import pytest

from abi_runner import AbiRunner
from metrics import FP16_TOL, FP32_TOL, assert_close, seeded
from oracle_bind import geom, out_hw

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.fixture(params=[False, True], ids=["fp32", "fp16"])
def run(pkg, gpulib, request):
    gpulib.trainlib_set_streams(1)
    r = AbiRunner(pkg, gpulib, device=True, half=request.param)
    yield r
    r.close()
    gpulib.trainlib_set_streams(1)


def rounded(r, a):
    return a.astype(r.dt).astype(F)


def kernels_of(run, call, *args):
    """launches of a call by the kernels' names"""
    run.lib.trainlib_profile(1)
    call(run, *args)
    run.lib.trainlib_profile(0)
    return {t[0]: t[1] for t in run.pkg.profile_table(run.lib)}


def conv_outputs(run, x, wt, dy, k, stride=1, bias=False):
    """Y, dX, dW (and dB) of one layer with padding k // 2, and the names of the kernels that ran"""
    n, cin, h, w = x.shape
    cout, Ho, Wo = dy.shape[1:]
    run.lib.trainlib_set_streams(n)
    Y, dX, dW, dB, B, one = run.zeros(*dy.shape), run.zeros(*x.shape), run.zeros(*wt.shape), run.zeros(cout), run.zeros(cout), run.zeros(4)
    a = run.args(run.sname("Conv2D_args"), input=run.blob(run.t(x), dX, C=cin, H=h, W=w), coeff=run.blob(run.t(wt), dW, C=cin, H=k, W=k, dim=wt.size), bias=run.blob(B, dB, dim=cout, W=cout),
                 output=run.blob(Y, run.t(dy), C=cout, H=Ho, W=Wo), Lpad=k // 2, Rpad=k // 2, Upad=k // 2, Dpad=k // 2, stride_h=stride, stride_w=stride,
                 i2c_buffer=one, bt_buffer=one, USE_BIASES=int(bias), USE_IM2COL=0, HWC=0)
    run.lib.trainlib_profile(1)
    for f in ("fw", "bw_param_grads", "bw_input_grads"):
        run.call(run.fname("pulp_conv2d_fp32_%s_cl" % f), a)
    run.lib.trainlib_profile(0)
    return [t.get().astype(F) for t in (Y, dX, dW, dB)[:3 + bias]], [t[0] for t in run.pkg.profile_table(run.lib)]


CONV = [(28, 14, 45, 28, 3, 1, 1), (3, 33, 41, 70, 5, 2, 3), (6, 42, 13, 81, 5, 1, 1), (40, 9, 11, 64, 3, 1, 5), (16, 5, 5, 8, 3, 1, 40), (20, 3, 200, 24, 3, 1, 2),
        (17, 12, 130, 33, 3, 2, 2), (64, 7, 7, 96, 1, 1, 30), (24, 28, 28, 48, 3, 1, 60), (33, 11, 12, 17, 3, 3, 2), (1, 6, 6, 4, 1, 1, 2), (70, 10, 10, 12, 7, 1, 1),
        (12, 8, 9, 16, 1, 2, 3), (64, 12, 12, 64, 5, 1, 4), (16, 7, 8, 8, 3, 1, 150), (8, 10, 16, 16, 3, 1, 63), (16, 32, 32, 16, 3, 1, 9), (8, 12, 32, 8, 3, 1, 30), (64, 16, 17, 64, 1, 1, 70), (36, 13, 15, 100, 1, 1, 100), (64, 40, 40, 72, 1, 1, 10), (72, 12, 12, 64, 1, 1, 110), (33, 9, 8, 130, 1, 1, 230)]


@pytest.mark.parametrize("cin,h,w,cout,k,stride,n", CONV)
def test_conv2d_shapes(run, oracle, cin, h, w, cout, k, stride, n):
    g = geom(cin, h, w, cout, k, stride=stride, pad=k // 2)
    Ho, Wo = out_hw(g)
    rng = seeded(cin + 3 * h + 5 * w + n)
    x, wt, b = rounded(run, rng.uniform(-1, 1, (n, cin, h, w))), rounded(run, rng.uniform(-1, 1, (cout, cin, k, k))), rounded(run, rng.standard_normal(cout))
    dy = rounded(run, rng.standard_normal((n, cout, Ho, Wo)) / 8)
    run.lib.trainlib_set_streams(n)
    X, W_, dY, B = run.t(x), run.t(wt), run.t(dy), run.t(b)
    Y, dX, dW, dB, one = run.zeros(n, cout, Ho, Wo), run.zeros(*x.shape), run.zeros(*wt.shape), run.zeros(cout), run.zeros(4)
    a = run.args(run.sname("Conv2D_args"), input=run.blob(X, dX, C=cin, H=h, W=w), coeff=run.blob(W_, dW, C=cin, H=k, W=k, dim=wt.size), bias=run.blob(B, dB, dim=cout, W=cout),
                 output=run.blob(Y, dY, C=cout, H=Ho, W=Wo), Lpad=k // 2, Rpad=k // 2, Upad=k // 2, Dpad=k // 2, stride_h=stride, stride_w=stride,
                 i2c_buffer=one, bt_buffer=one, USE_BIASES=1, USE_IM2COL=0, HWC=0)
    for f in ("fw", "bw_param_grads", "bw_input_grads"):
        run.call(run.fname("pulp_conv2d_fp32_%s_cl" % f), a)
    tol = FP16_TOL if run.half else FP32_TOL
    y, dx = Y.get().astype(F), dX.get().astype(F)
    for s in range(n):
        assert_close(y[s], oracle.conv2d_fw(x[s], wt, b, g), tol, "fw stream %d" % s)
        assert_close(dx[s], oracle.conv2d_ig(dy[s], wt, g), tol, "ig stream %d" % s)
    want = sum(oracle.conv2d_wg(x[s], dy[s], g)[0].astype(np.float64) for s in range(n)).astype(F)
    assert_close(dW.get().astype(F), want, tol, "wg")
    assert_close(dB.get().astype(F), dy.astype(np.float64).sum(axis=(0, 2, 3)).astype(F), tol, "bias gradient")


# the half-precision kernels on runs of slots (tl_conv_px.cu): loads of one, two and four pixels, planes smaller and larger than a run, runs
# that start inside a row, channel counts at and off multiples of 16, slices of result channels, groups of source channels,
# windows of 1 to 49 taps, strides 2 and 3 with parities that no tap reaches, a bias gradient in a spare channel and on its own.
# The last number: of forward and input gradient, how many run there (the others have too little work, or are products of the GEMM)
SLOTS = [(24, 28, 28, 48, 3, 1, 130, 2), (5, 27, 43, 23, 3, 1, 70, 2), (64, 6, 6, 96, 3, 1, 60, 0), (3, 48, 46, 90, 3, 1, 20, 2), (32, 9, 14, 17, 5, 1, 40, 2), (16, 31, 33, 33, 5, 1, 9, 1), (6, 40, 40, 20, 7, 1, 12, 2), (90, 19, 21, 70, 1, 1, 40, 0),
         (40, 41, 41, 80, 5, 1, 3, 1), (96, 15, 17, 96, 1, 1, 90, 0), (34, 10, 23, 55, 1, 2, 210, 2), (43, 23, 34, 22, 3, 2, 60, 1), (7, 39, 39, 58, 3, 2, 280, 2), (20, 30, 31, 40, 3, 3, 110, 1), (13, 33, 32, 24, 5, 2, 40, 1), (40, 46, 47, 90, 3, 3, 120, 2), (1, 1, 300, 128, 3, 1, 40, 1)]


@pytest.mark.parametrize("cin,h,w,cout,k,stride,n,directions", SLOTS)
def test_conv2d_on_runs_of_slots(run, oracle, cin, h, w, cout, k, stride, n, directions):
    if not run.half:
        pytest.skip("half precision only")
    launches = kernels_of(run, test_conv2d_shapes, oracle, cin, h, w, cout, k, stride, n)
    assert launches.get("conv_px_kernel", 0) == directions and launches.get("conv_px_wg_kernel") == 1, launches


# An infinite or NaN pixel reaches the weight gradients of the taps that pair it with a pixel of the other tensor, and no other one: corners, an
# edge, an even and an odd place of a strided layer, and a pixel inside
@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("cin,h,w,cout,k,stride,n", [(24, 14, 14, 48, 3, 1, 60), (17, 13, 11, 33, 5, 1, 30), (20, 16, 15, 40, 3, 2, 110), (40, 9, 7, 34, 1, 1, 400)])
def test_weight_gradients_on_runs_of_slots_keep_what_is_no_number_apart(run, cin, h, w, cout, k, stride, n, bad):
    if not run.half:
        pytest.skip("half precision only")
    rng = seeded(cin + k)
    Ho, Wo, pad = (h - 1) // stride + 1, (w - 1) // stride + 1, k // 2
    x, wt, dy = (rounded(run, rng.uniform(-1, 1, s)) for s in ((n, cin, h, w), (cout, cin, k, k), (n, cout, Ho, Wo)))
    clean, names = conv_outputs(run, x, wt, dy, k, stride)
    if k > 1:
        assert any("conv_px_wg_kernel" in t for t in names)
    for s, c, r, q in ((0, 0, 0, 0), (n - 1, cin - 1, h - 1, w - 1), (n // 2, 3, 0, w // 2), (3, 2, h // 2, w // 2)):
        v = x.copy(); v[s, c, r, q] = bad
        got = conv_outputs(run, v, wt, dy, k, stride)[0][2]
        touched = np.zeros(got.shape, bool)
        for kh in range(k):
            for kw in range(k):
                i, j = r + pad - kh, q + pad - kw
                touched[:, c, kh, kw] = i % stride == 0 and j % stride == 0 and 0 <= i // stride < Ho and 0 <= j // stride < Wo
        assert not np.isfinite(got[touched]).any()
        assert_close(got[~touched], clean[2][~touched], FP16_TOL, "x %s" % ((s, c, r, q),))
        v = dy.copy(); v[s, min(c, cout - 1), min(r, Ho - 1), min(q, Wo - 1)] = bad
        got = conv_outputs(run, x, wt, v, k, stride)[0][2]
        touched = np.zeros(got.shape, bool)
        for kh in range(k):
            for kw in range(k):
                touched[min(c, cout - 1), :, kh, kw] = 0 <= min(r, Ho - 1) * stride + kh - pad < h and 0 <= min(q, Wo - 1) * stride + kw - pad < w
        assert not np.isfinite(got[touched]).any()
        assert_close(got[~touched], clean[2][~touched], FP16_TOL, "dy %s" % ((s, c, r, q),))


# Long sums of the weight and bias gradient, terms of one sign: the tensor core truncates what it accumulates, up to 2^-23 of the sum at every k-step and half of that in
# the mean.  Over a chain of 32 steps from zero that is 32 / 2 * 2^-24 = 1e-6 of a result, to which the rounding to half precision adds 2^-11 / 1.7
# for one result and 1 / sqrt(results) of it for their mean, 4e-6.  (One chain of all steps of a CTA: 5e-5.)
@pytest.mark.parametrize("cin,h,w,cout,k,stride,n", [(16, 48, 48, 39, 3, 1, 512), (7, 48, 47, 30, 5, 1, 512), (20, 31, 33, 100, 3, 2, 500)])
def test_long_weight_gradients_on_runs_of_slots_do_not_drift(run, cin, h, w, cout, k, stride, n):
    if not run.half:
        pytest.skip("half precision only")
    import torch
    gen = torch.Generator("cuda").manual_seed(cin)
    Ho, Wo = (h - 1) // stride + 1, (w - 1) // stride + 1
    x = torch.rand(n, cin, h, w, device="cuda", generator=gen).half()
    dy = (torch.rand(n, cout, Ho, Wo, device="cuda", generator=gen) / 256).half()
    (_, _, dW, dB), names = conv_outputs(run, x.float().cpu().numpy(), np.ones((cout, cin, k, k), F), dy.float().cpu().numpy(), k, stride, bias=True)
    assert any("conv_px_wg_kernel" in t for t in names)
    d64 = dy.double().permute(1, 0, 2, 3).reshape(cout, -1)
    xp = torch.nn.functional.pad(x.double(), (k // 2,) * 4)
    want = torch.stack([d64 @ xp[:, :, i:i + stride * Ho:stride, j:j + stride * Wo:stride][:, :, :Ho, :Wo].permute(0, 2, 3, 1).reshape(-1, cin) for i in range(k) for j in range(k)], -1)
    rel = lambda got, want: (torch.from_numpy(got.reshape(want.shape)).cuda().double() / want - 1).cpu().numpy()
    e, eb = rel(dW.reshape(cout, cin, k * k), want), rel(dB, d64.sum(1))
    assert abs(e.mean()) <= 1e-5 and np.abs(e).max() <= 2.0 ** -11 * 1.02 and np.abs(eb).max() <= 2.0 ** -11 * 1.02, (e.mean(), np.abs(e).max(), np.abs(eb).max())


# weight gradients of few pixels, one cluster per 16 x 16 channel tile (conv_mma_wg_cluster_kernel): one to sixteen CTAs of a cluster, ranks
# without pixels, a last tile cut short, several streams in a tile, rows longer than a tile, channel remainders, windows of fewer taps
# than the nine warps (which then share the pixels), of more, and of several rounds, strides, odd planes
FEW_PIXELS = [(16, 32, 32, 32, 3, 1, 1), (17, 9, 9, 17, 5, 2, 1), (2, 33, 46, 61, 3, 2, 1), (60, 13, 18, 8, 3, 1, 1), (5, 3, 300, 20, 3, 1, 1), (33, 5, 5, 31, 2, 2, 1), (1, 1, 1, 1, 1, 1, 1), (24, 40, 40, 24, 1, 1, 1),
              (48, 28, 28, 48, 5, 1, 1), (7, 11, 13, 9, 7, 1, 5), (20, 3, 3, 20, 3, 1, 30), (20, 7, 5, 20, 3, 1, 40), (96, 4, 4, 96, 3, 1, 1), (3, 64, 64, 12, 5, 2, 1), (12, 21, 19, 40, 3, 3, 3), (9, 6, 7, 30, 4, 1, 2)]


@pytest.mark.parametrize("cin,h,w,cout,k,stride,n", FEW_PIXELS)
def test_conv2d_of_few_pixels(run, oracle, cin, h, w, cout, k, stride, n):
    run.lib.trainlib_profile(1)
    test_conv2d_shapes(run, oracle, cin, h, w, cout, k, stride, n)
    run.lib.trainlib_profile(0)
    assert any("wg_cluster" in t[0] for t in run.pkg.profile_table(run.lib))


# long sums under few pixels, one cluster per result tile whose CTAs share the source channels: channel counts that divide into unequal
# shares, a last share of few channels, strides whose parities have different taps (some none), more streams in a tile, 1 x 1 windows.
# The last numbers: of forward and input gradient, how many run there in fp32 and in fp16 (the others have shorter sums)
LONG_SUMS = [(96, 9, 13, 96, 3, 2, 1, 2, 1), (60, 13, 18, 8, 3, 1, 1, 1, 0), (130, 7, 9, 100, 3, 1, 1, 2, 2), (400, 4, 4, 390, 1, 1, 1, 2, 2), (50, 5, 5, 52, 5, 1, 3, 2, 2), (75, 3, 3, 66, 3, 3, 7, 1, 0), (200, 5, 7, 17, 2, 1, 1, 1, 1), (48, 28, 28, 40, 5, 1, 1, 2, 2)]


@pytest.mark.parametrize("cin,h,w,cout,k,stride,n,fp32,fp16", LONG_SUMS)
def test_conv2d_of_long_sums(run, oracle, cin, h, w, cout, k, stride, n, fp32, fp16):
    launches = kernels_of(run, test_conv2d_shapes, oracle, cin, h, w, cout, k, stride, n)
    assert launches.get("(conv_mma_kernel<T, MT, WM, WN, WK, BN, true>)", 0) == (fp16 if run.half else fp32), launches


# single-precision pointwise layers over many pixels (tl_conv_pw.cu): CTAs whose last 128 pixels are cut short, planes smaller than that, odd
# ones, one and many pieces of channels, channel counts off multiples of 8 and 16, more than 128 result channels (three products, one
# accumulator), weights that leave room for two, three or four stages, weights that do not fit (another kernel), the GEMM's layers
POINTWISE = [(64, 28, 28, 128, 13), (33, 17, 19, 70, 40), (7, 4, 4, 20, 700), (1, 30, 31, 40, 11), (20, 23, 23, 200, 20), (40, 25, 25, 256, 16), (96, 16, 17, 160, 37), (72, 100, 100, 72, 1), (96, 30, 30, 120, 8), (5, 47, 48, 17, 30),
             (256, 20, 20, 256, 25), (12, 97, 98, 9, 9)]


@pytest.mark.parametrize("cin,h,w,cout,n", POINTWISE)
def test_pointwise_over_many_pixels(run, oracle, cin, h, w, cout, n):
    if run.half:
        pytest.skip("single precision only")
    run.lib.trainlib_profile(1)
    test_conv2d_shapes(run, oracle, cin, h, w, cout, 1, 1, n)
    run.lib.trainlib_profile(0)
    assert any("conv_pw_kernel" in t[0] for t in run.pkg.profile_table(run.lib)) == (cin < 256)


# Terms of one sign show what the tensor core cuts off: half of 2^-23 of the sum in the mean at every step.  Chains of at most twelve steps of eight channels,
# whose sums are added to fp32 registers, leave 12 / 2 * 2^-24 = 3.6e-7 of a result, the three terms of a product and the sum of the chains some
# 1e-7 more (one chain for all channels: 1.4e-6 at 256, 2.3e-6 at 400).  Two sets of accumulators and one, chains of two and of three pieces,
# more than 64 results on small planes, so many channels that the layer runs elsewhere
@pytest.mark.parametrize("cin,h,w,cout,n,here", [(256, 20, 20, 32, 30, 1), (400, 19, 21, 16, 30, 1), (310, 20, 20, 63, 25, 1), (330, 21, 20, 48, 25, 1), (180, 10, 11, 80, 100, 1), (512, 20, 20, 30, 30, 1), (600, 20, 20, 30, 25, 0)])
def test_pointwise_layers_of_many_channels_do_not_drift(run, cin, h, w, cout, n, here):
    if run.half:
        pytest.skip("single precision only")
    rng = seeded(cin)
    x, wt = (rng.uniform(0, 1, s).astype(F) for s in ((n, cin, h, w), (cout, cin, 1, 1)))
    run.lib.trainlib_set_streams(n)
    Y, B, one = run.zeros(n, cout, h, w), run.zeros(cout), run.zeros(4)
    a = run.args("Conv2D_args", input=run.blob(run.t(x), one, C=cin, H=h, W=w), coeff=run.blob(run.t(wt), one, C=cin, H=1, W=1, dim=wt.size), bias=run.blob(B, B, dim=cout, W=cout),
                 output=run.blob(Y, Y, C=cout, H=h, W=w), stride_h=1, stride_w=1, i2c_buffer=one, bt_buffer=one, USE_BIASES=0, USE_IM2COL=0, HWC=0)
    run.lib.trainlib_profile(1)
    run.call("pulp_conv2d_fp32_fw_cl", a)
    run.lib.trainlib_profile(0)
    names = [t[0] for t in run.pkg.profile_table(run.lib)]
    assert any("conv_pw_kernel" in t for t in names) == bool(here), names
    want = np.einsum("oc,nchw->nohw", wt[:, :, 0, 0].astype(np.float64), x[:4].astype(np.float64))
    drift = (Y.get()[:4] / want - 1).mean()
    assert abs(drift) <= 6e-7, drift


# their weight gradient: lanes with hi and lo rows of X (up to 64 source channels) and without, slices of either side's channels, pieces of 16 and
# of 32 pixels, planes that no 16-byte load fits, a last piece cut short
POINTWISE_WG = [(64, 28, 28, 128, 15), (33, 17, 19, 70, 40), (7, 4, 4, 20, 700), (1, 30, 31, 40, 13), (20, 23, 23, 200, 21), (160, 20, 20, 96, 27), (96, 31, 30, 33, 9), (130, 25, 25, 140, 18), (5, 47, 48, 17, 80), (64, 40, 41, 8, 98)]


@pytest.mark.parametrize("cin,h,w,cout,n", POINTWISE_WG)
def test_pointwise_weight_gradient_over_many_pixels(run, oracle, cin, h, w, cout, n):
    if run.half:
        pytest.skip("single precision only")
    run.lib.trainlib_profile(1)
    test_conv2d_shapes(run, oracle, cin, h, w, cout, 1, 1, n)
    run.lib.trainlib_profile(0)
    assert any("conv_pw_wg_kernel" in t[0] for t in run.pkg.profile_table(run.lib))


# NaN and infinity reach every result that they are a factor of, and no other one.  The bits: what operations of the GPU produce and its negative,
# the host's, one whose payload lies below the bits that the tensor core reads, infinity (which the split into two parts turns into NaN)
@pytest.mark.parametrize("bits", [0x7FFFFFFF, 0xFFFFFFFF, 0x7FC00000, 0x7F800001, 0x7F800000])
@pytest.mark.parametrize("cin,cout", [(64, 32), (100, 140)])
def test_pointwise_layers_keep_what_is_no_number(run, cin, cout, bits):
    if run.half:
        pytest.skip("single precision only")
    n, h, w = 26, 28, 28
    rng = seeded(cin)
    bad = np.array([bits], np.uint32).view(F)[0]
    x, wt, dy = (rng.standard_normal(s).astype(F) for s in ((n, cin, h, w), (cout, cin, 1, 1), (n, cout, h, w)))
    clean, names = conv_outputs(run, x, wt, dy, 1)
    assert sum("conv_pw_kernel" in t for t in names) == 1 and any("conv_pw_wg_kernel" in t for t in names)
    with np.errstate(invalid="ignore"):
        for where in ("x", "w", "dy"):
            v = dict(x=x.copy(), w=wt.copy(), dy=dy.copy())
            touched = [np.zeros(t.shape, bool) for t in clean]
            if where == "x":
                v["x"][3, 5, 7, 9] = bad; touched[0][3, :, 7, 9] = True; touched[2][:, 5] = True
            elif where == "w":
                v["w"][6, 2] = bad; touched[0][:, 6] = True; touched[1][:, 2] = True
            else:
                v["dy"][25, 31, 27, 27] = bad; touched[1][25, :, 27, 27] = True; touched[2][31] = True
            got, _ = conv_outputs(run, v["x"], v["w"], v["dy"], 1)
            for g, c, t in zip(got, clean, touched):
                assert not np.isfinite(g[t]).any() and np.array_equal(g[~t], c[~t])


def attention_scale(H):
    """the 1 / sqrt(H) that the layer applies: the guess on the bits and one Newton step, in fp32"""
    y = (np.int32(0x5f3759df) - (F(H).view(np.int32) >> 1)).view(F)
    return y * (F(1.5) - F(H) * F(0.5) * y * y)


# half-precision attention with enough blocks of sixteen queries for the mma.sync kernels: every core product against 64 bits from the
# tensors that the layer leaves behind.  A result is rounded to 2^-11 of itself, and where the stored probabilities or dP stand in
# for the unrounded ones the kernels used, each term by as much again: att and dv two such errors, dq and dk four
@pytest.mark.parametrize("L,E,Fd,heads", [(203, 24, 96, 8), (400, 16, 64, 4), (97, 16, 544, 16), (512, 8, 24, 3), (333, 12, 1280, 5)])
def test_half_precision_attention_core(pkg, gpulib, L, E, Fd, heads):
    gpulib.trainlib_set_streams(1)
    rng = seeded(L + E + Fd)
    half = lambda *s: rng.standard_normal(s).astype(np.float16).astype(F)
    x, dy = half(E, L), half(E, L)
    ws = [(half(E, Fd) / np.sqrt(E)).astype(np.float16).astype(F) for _ in range(3)] + [(half(E, Fd) / np.sqrt(Fd)).astype(np.float16).astype(F)]
    zb = np.zeros(Fd, F)
    r = AbiRunner(pkg, gpulib, device=True, half=True)
    gpulib.trainlib_profile(1)
    got = {k: v.astype(np.float64) for k, v in r.mhsa(x, ws[0], ws[1], ws[2], zb, zb, zb, ws[3], dy, L, E, Fd, heads).items()}
    gpulib.trainlib_profile(0)
    assert sum("mma_attn" in t[0] for t in pkg.profile_table(gpulib)) == 3
    r.close()
    H = Fd // heads
    hd = lambda k: got[k].reshape(heads, H, L)
    P, dP, scale = got["softmax"].reshape(heads, L, L), got["dsoftmax"].reshape(heads, L, L), float(attention_scale(H))
    u = 2.0 ** -11
    def close(a, b, terms, what):
        # the error bound of a sum is that of its terms' absolute values; the largest of them against the largest result
        assert np.abs(a - b).max() <= 1.05 * terms, "%s: %.2e of %.2e" % (what, np.abs(a - b).max(), terms)
    att = np.einsum("hdk,hqk->hdq", hd("v"), P)
    close(hd("att"), att, u * (np.abs(att).max() + np.einsum("hdk,hqk->hdq", np.abs(hd("v")), P).max()), "att")
    want = np.einsum("hdq,hdk->hqk", hd("datt"), hd("v"))
    close(dP, want, u * np.abs(want).max() + 2.0 ** -24, "dP")
    dv = np.einsum("hdq,hqk->hdk", hd("datt"), P)
    close(hd("dv"), dv, u * (np.abs(dv).max() + np.einsum("hdq,hqk->hdk", np.abs(hd("datt")), P).max()) + 2.0 ** -24, "dv")
    # dS = (dP - sum dP P) P from the rounded dP and P, as the kernels form it
    dS = (dP - (dP * P).sum(-1, keepdims=True)) * P
    dq, dk = scale * np.einsum("hdk,hqk->hdq", hd("k"), dS), scale * np.einsum("hdq,hqk->hdk", hd("q"), dS)
    for k, w, m in (("dq", dq, np.einsum("hdk,hqk->hdq", np.abs(hd("k")), np.abs(dS)).max()), ("dk", dk, np.einsum("hdq,hqk->hdk", np.abs(hd("q")), np.abs(dS)).max())):
        close(hd(k), w, u * np.abs(w).max() + 2.0 ** -18 * scale * m + 2.0 ** -24, k)
    # the probabilities sum to one up to their rounding
    assert np.abs(P.sum(-1) - 1).max() <= u * (1 + 1e-3) + L * 2.0 ** -25


# dq and dk of those kernels are as exact as fp32 sums in fused multiply-adds, 32 partial sums a result: what either lets fall on the wrong side of a
# rounding to half precision is counted, some 150 of 262 144 results.  1.2 times as many is two and a half standard deviations (sqrt(150) = 12); a low
# part cut off and chains of four k-steps, in which the tensor core truncates, gave 1.5 times as many
@pytest.mark.parametrize("L,E,Fd,heads", [(512, 128, 256, 4), (256, 256, 512, 8)])
def test_half_precision_attention_core_rounds_like_fp32_sums(pkg, gpulib, L, E, Fd, heads):
    gpulib.trainlib_set_streams(1)
    rng = seeded(L + E + Fd)
    x, dy = (rng.standard_normal((E, L)).astype(np.float16).astype(F) for _ in range(2))
    ws = [(rng.standard_normal((E, Fd)) / np.sqrt(E)).astype(np.float16).astype(F) for _ in range(4)]
    zb = np.zeros(Fd, F)
    r = AbiRunner(pkg, gpulib, device=True, half=True)
    gpulib.trainlib_profile(1)
    got = r.mhsa(x, ws[0], ws[1], ws[2], zb, zb, zb, ws[3], dy, L, E, Fd, heads)
    gpulib.trainlib_profile(0)
    assert sum("mma_attn_bw" in t[0] for t in pkg.profile_table(gpulib)) == 2
    r.close()
    H = Fd // heads
    P, dP = (got[k].astype(F).reshape(heads, L, L) for k in ("softmax", "dsoftmax"))

    def fma_sum(a, b):
        """sum over the last axis of a * b (broadcast): 32 partial sums, then added in pairs, every step rounded to fp32"""
        acc = np.zeros(np.broadcast_shapes(a.shape, b.shape)[:-1] + (32,), F)
        for j in range(0, L, 32):
            acc = (acc.astype(np.float64) + a[..., j:j + 32].astype(np.float64) * b[..., j:j + 32]).astype(F)
        while acc.shape[-1] > 1:
            acc = acc[..., :acc.shape[-1] // 2] + acc[..., acc.shape[-1] // 2:]
        return acc[..., 0]

    scale = attention_scale(H)
    dS = (dP - fma_sum(dP, P)[..., None]) * P
    dS64 = (dP.astype(np.float64) - (dP.astype(np.float64) * P).sum(-1, keepdims=True)) * P
    wrong = wrong_fma = 0
    for name, other, t in (("dq", "k", dS), ("dk", "q", dS.transpose(0, 2, 1))):
        M = got[other].astype(F).reshape(heads, H, L)
        exact = (float(scale) * np.einsum("hdj,hnj->hdn", M.astype(np.float64), dS64 if name == "dq" else dS64.transpose(0, 2, 1))).astype(np.float16)
        fma = np.stack([np.stack([fma_sum(M[h, d], t[h]) for d in range(H)]) for h in range(heads)]) * scale
        wrong += int((got[name].astype(np.float16).reshape(exact.shape) != exact).sum())
        wrong_fma += int((fma.astype(np.float16) != exact).sum())
    assert wrong <= 1.2 * wrong_fma, "%d and %d of %d" % (wrong, wrong_fma, 2 * heads * H * L)


@pytest.mark.parametrize("c,h,w,k,pad,n", [(5, 9, 7, 3, 1, 3), (64, 28, 28, 3, 1, 4), (3, 33, 18, 3, 0, 2), (8, 6, 6, 5, 2, 9), (2, 40, 41, 3, 2, 1), (7, 4, 4, 3, 1, 700), (4, 12, 12, 4, 1, 2)])
def test_depthwise_shapes(run, oracle, c, h, w, k, pad, n, stride=1):
    g = geom(c, h, w, c, k, stride=stride, pad=pad)
    Ho, Wo = out_hw(g)
    rng = seeded(c + h + w + n)
    x, wt, dy = rounded(run, rng.standard_normal((n, c, h, w))), rounded(run, rng.standard_normal((c, k, k)) / k), rounded(run, rng.standard_normal((n, c, Ho, Wo)) / 4)
    run.lib.trainlib_set_streams(n)
    X, W_, dY = run.t(x), run.t(wt), run.t(dy)
    Y, dX, dW = run.zeros(n, c, Ho, Wo), run.zeros(*x.shape), run.zeros(*wt.shape)
    fields = {} if run.half else dict(stride_h=stride, stride_w=stride)
    a = run.args(run.sname("DepthWise_Conv_args"), input=run.blob(X, dX, C=c, H=h, W=w), coeff=run.blob(W_, dW, C=c, H=k, W=k), output=run.blob(Y, dY, C=c, H=Ho, W=Wo),
                 Lpad=pad, Rpad=pad, Upad=pad, Dpad=pad, skip_wg_grad=0, skip_in_grad=0, HWC=0, **fields)
    run.call(run.fname("pulp_conv_dw_fp32_fw_cl"), a); run.call(run.fname("pulp_conv_dw_fp32_bw_cl"), a)
    tol = FP16_TOL if run.half else FP32_TOL
    y, dx = Y.get().astype(F), dX.get().astype(F)
    for s in range(0, n, max(1, n // 5)):
        assert_close(y[s], oracle.dw_fw(x[s], wt, g), tol, "fw stream %d" % s)
        assert_close(dx[s], oracle.dw_ig(dy[s], wt, g), tol, "ig stream %d" % s)
    want = sum(oracle.dw_wg(x[s], dy[s], g).astype(np.float64) for s in range(n)).astype(F)
    assert_close(dW.get().astype(F), want, tol, "wg")


# 3 x 3 with stride 1 in register strips: rows of whole 16-byte groups and not, one row, one column, strips of unequal rows, many planes in a CTA
# (more than there are channels), several rounds of a CTA's threads, padding of two columns beside whole groups, so many channels that the
# weight gradient takes more than one wave of CTAs
@pytest.mark.parametrize("c,h,w,pad,n", [(6, 31, 20, 1, 5), (3, 1, 8, 1, 2), (2, 9, 1, 1, 40), (1, 1, 1, 1, 3), (3, 6, 8, 1, 900), (200, 9, 12, 1, 3), (2, 130, 131, 1, 1), (4, 17, 12, 2, 6), (5, 18, 16, 0, 4), (1, 300, 260, 1, 1), (297, 6, 8, 1, 7), (600, 5, 7, 1, 2)])
def test_depthwise_in_register_strips(run, oracle, c, h, w, pad, n):
    launches = kernels_of(run, test_depthwise_shapes, oracle, c, h, w, 3, pad, n)
    assert sum(v for t, v in launches.items() if "dw3_strip_kernel" in t) == 2 and sum(v for t, v in launches.items() if "dw3_strip_wg_kernel" in t) == 1, launches


# Planes whose staged windows come to just below, exactly and just above the 48 KB that a launch gets without asking: the weight
# gradients keep static arrays beside them.  Floats staged: 3x3 with pad 1 11 880, 12 276, 12 288, 11 446 (past that kernel's own
# limit), with pad 0 and 2 12 288; 5x5 11 881, 12 100, 12 544; stride 2 (fp32 only) 12 285, 12 519.
@pytest.mark.parametrize("c,h,w,k,pad,stride,n", [(2, 97, 108, 3, 1, 1, 2), (2, 97, 112, 3, 1, 1, 2), (3, 94, 116, 3, 1, 1, 3), (2, 95, 116, 3, 1, 1, 1), (2, 96, 118, 3, 0, 1, 2), (2, 92, 114, 3, 2, 1, 2),
                                                  (2, 105, 105, 5, 2, 1, 2), (3, 106, 106, 5, 2, 1, 2), (2, 108, 108, 5, 2, 1, 1), (2, 104, 115, 3, 1, 2, 2), (2, 106, 115, 3, 1, 2, 2)])
def test_depthwise_planes_at_the_shared_memory_limit(run, oracle, c, h, w, k, pad, stride, n):
    if run.half and stride != 1:
        pytest.skip("the fp16 argument struct has no stride")
    test_depthwise_shapes(run, oracle, c, h, w, k, pad, n, stride)


@pytest.mark.parametrize("N,K,M", [(1, 1, 1), (17, 3001, 41), (16, 2048, 300), (33, 64, 31), (130, 7, 130), (64, 129, 65), (500, 40, 333), (1000, 60, 520), (128, 512, 128)])
@pytest.mark.parametrize("trans_B", [0, 1])
def test_products_of_small_groups(run, N, K, M, trans_B):
    rng = seeded(N + K + M)
    A, B = rounded(run, rng.standard_normal((N, K)) / np.sqrt(K)), rounded(run, rng.standard_normal((M, K) if trans_B else (K, M)))
    want = (A.astype(np.float64) @ (B.T if trans_B else B).astype(np.float64)).astype(F)
    assert_close(run.mm(A, B, N, K, M, trans_B=trans_B).astype(F), want, FP16_TOL if run.half else FP32_TOL, "mm")


# the tcgen05 kernel: one CTA per tile, CTA pairs, split contractions; operands in place (multiples of 16 bytes) and packed
@pytest.mark.parametrize("N,K,M", [(257, 512, 1030), (129, 200, 4100), (300, 2048, 912), (1000, 1001, 700), (2504, 1304, 2600), (2600, 1800, 5001), (2560, 1800, 5008)])
@pytest.mark.parametrize("trans_B", [0, 1])
def test_products_of_tiles(run, N, K, M, trans_B):
    test_products_of_small_groups(run, N, K, M, trans_B)


# host arrays: odd byte counts, at and past the size that goes through the page-locked block, and more than the block holds
@pytest.mark.parametrize("N,K,M", [(1, 3, 5), (96, 1024, 7), (97, 1024, 3), (300, 320, 330), (330, 297, 1)])
def test_products_of_host_arrays(pkg, gpulib, N, K, M):
    r = AbiRunner(pkg, gpulib, device=False)
    rng = seeded(N + K + M)
    A, B = (rng.standard_normal(s).astype(F) for s in ((N, K), (K, M)))
    want = (A.astype(np.float64) @ B.astype(np.float64)).astype(F)
    assert_close(r.mm(A, B, N, K, M), want, FP32_TOL, "mm")
    r.close()


# both gradients and the bias gradient of one stream, rows that are no multiple of 16 bytes
@pytest.mark.parametrize("inn,out", [(1, 1), (21, 1398), (1001, 70), (34, 3001), (3, 9000), (2050, 33)])
def test_linear_rows_of_any_length(run, oracle, inn, out):
    rng = seeded(inn + out)
    W, x = rounded(run, rng.standard_normal((out, inn)) / np.sqrt(inn)), rounded(run, rng.standard_normal(inn))
    dy, bias = rounded(run, rng.standard_normal(out)), rounded(run, rng.standard_normal(out))
    want, got = oracle.linear(W, x, dy, bias), run.linear(W, x, dy, bias, one_backward_call=True)
    for k in ("y", "dW", "dx", "db"):
        assert_close(got[k].astype(F).reshape(want[k].shape), want[k], FP16_TOL if run.half else FP32_TOL, k)


def test_products_alternating_between_streams(run):
    """split contractions use scratch and counters of the library: calls of two streams, never synchronised in between"""
    import torch
    N, K, M = 16, 2048, 300
    rng = seeded(5)
    mats = [(rounded(run, rng.standard_normal((N, K)) / np.sqrt(K)), rounded(run, rng.standard_normal((K, M)))) for _ in range(8)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    args, outs = [], []
    for A, B in mats:
        a, b, c = run.t(A), run.t(B), run.zeros(N, M)
        args.append(run.args(run.sname("matMul_args"), A=a, B=b, C=c, N=N, K=K, M=M, trans_B=0, USE_BIASES=0)); outs.append(c)
    torch.cuda.synchronize()
    try:
        for rep in range(5):
            for i, a in enumerate(args):
                run.lib.trainlib_set_stream(streams[i % 2].cuda_stream)
                run.call("mm_fp16" if run.half else "mm", a)
        torch.cuda.synchronize()
    finally:
        run.lib.trainlib_set_stream(None)
    for (A, B), c in zip(mats, outs):
        assert_close(c.get().astype(F), (A.astype(np.float64) @ B.astype(np.float64)).astype(F), FP16_TOL if run.half else FP32_TOL, "mm")


@pytest.mark.parametrize("rows,width", [(1, 1), (7, 33), (200, 128), (700, 250), (300, 512), (5, 1024), (9, 1500)])
def test_layernorm_shapes(run, oracle, rows, width):
    rng = seeded(rows + width)
    x, w, b, dy = (rounded(run, a) for a in (rng.standard_normal((rows, width)), rng.standard_normal(width), rng.standard_normal(width), rng.standard_normal((rows, width)) / 16))
    eps = float(np.asarray(1e-3, run.dt))
    got = run.layernorm_ext(x, w, b, dy, rows, width, eps)
    tol = FP16_TOL if run.half else FP32_TOL
    assert_close(got["y"].astype(F), oracle.layernorm_fw(x, w, b, rows, width, eps), tol, "y")
    dx, dw, db = oracle.layernorm_bw(x, w, dy, rows, width, eps)
    for k, v in (("dx", dx), ("dw", dw), ("db", db)):
        if np.abs(v).max() > 1e-6:                          # (a row of one element has no gradient)
            assert_close(got[k].astype(F), v, tol, k)


# the backward pass of a few rows as one cluster: fewest and most rows and columns, and just past them
@pytest.mark.parametrize("rows,width", [(9, 1), (128, 129), (129, 257), (512, 512), (513, 512), (512, 513), (17, 31), (384, 128), (385, 128), (385, 129), (8, 40)])
def test_layernorm_of_one_cluster(run, oracle, rows, width):
    names = kernels_of(run, test_layernorm_shapes, oracle, rows, width)
    assert any("layernorm_bw_cluster" in t for t in names) == (8 < rows <= (512 if width > 128 else 384) and width <= 512), names


@pytest.mark.parametrize("dim", [1, 5, 1023, 1025, 70001, 400000])
def test_mse_lengths(run, oracle, dim):
    rng = seeded(dim)
    y, t = rounded(run, rng.standard_normal(dim)), rounded(run, rng.standard_normal(dim))
    loss, dy = run.loss("MSELoss", y, t)
    tol = FP16_TOL if run.half else FP32_TOL
    assert_close(np.asarray([loss], F), np.asarray([np.mean((t.astype(np.float64) - y) ** 2)], F), tol, "loss")
    assert_close(dy.astype(F) * dim, (2.0 * (y.astype(np.float64) - t)).astype(F), tol if dim < 5000 or not run.half else 0.1, "dy")


def test_conv2d_planes_of_one_pixel_and_millions_of_channels(pkg, gpulib):
    """128 streams of nine million channels on 1 x 1: the streams that share a tile of the weight gradient lie past 4 GB"""
    import torch
    n, c = 128, 9000000
    r = AbiRunner(pkg, gpulib, device=True)
    gen = torch.Generator("cuda").manual_seed(6)
    x, dw, dy = torch.randn(n, c, device="cuda", generator=gen), torch.empty(c, 9, device="cuda"), torch.randn(n, device="cuda", generator=gen)
    one = r.zeros(4)
    mk = lambda d, g, C, H, W, dim=None: pkg.make_blob(r.keep, d, g, C=C, H=H, W=W, dim=dim)
    a = r.args("Conv2D_args", input=mk(x.data_ptr(), one.arg, c, 1, 1), coeff=mk(one.arg, dw.data_ptr(), c, 3, 3, 9 * c), bias=mk(one.arg, one.arg, 1, 1, 1), output=mk(one.arg, dy.data_ptr(), 1, 1, 1),
               Lpad=1, Rpad=1, Upad=1, Dpad=1, stride_h=1, stride_w=1, i2c_buffer=one, bt_buffer=one, USE_BIASES=0, USE_IM2COL=0, HWC=0)
    torch.cuda.synchronize()
    try:
        gpulib.trainlib_set_streams(n)
        r.call("pulp_conv2d_fp32_bw_param_grads_cl", a)
        gpulib.trainlib_synchronize()
    finally:
        gpulib.trainlib_set_streams(1)
        r.close()
    err = top = 0.0
    for k in range(0, c, 1000000):
        want = (x[:, k:k + 1000000].double() * dy.double()[:, None]).sum(0)
        top = max(top, float(want.abs().max())); err = max(err, float((dw[k:k + 1000000, 4] - want).abs().max()))
    assert err <= FP32_TOL * top, (err, top)
    assert float(dw[:, :4].abs().max()) == 0 and float(dw[:, 5:].abs().max()) == 0
