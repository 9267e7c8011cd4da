"""CPU: the library's host code on a CUDA runtime without a device (fake_cudart.c), where launches can be made to fail."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
HEAD = r'''
import ctypes, sys
sys.path.insert(0, %r)
import numpy as np
from conftest import load_pkg
pkg = load_pkg()
fake = ctypes.CDLL(%r)
lib = pkg.load()
assert lib.trainlib_init(0) == 0
'''


@pytest.fixture(scope="module")
def on_fake_runtime(tmp_path_factory):
    if not os.path.exists(os.path.join(INCLUDE, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.check_call(["gcc", "-O1", "-Wall", "-shared", "-fPIC", "-I" + INCLUDE, os.path.join(HERE, "fake_cudart.c"), "-o", so])

    def run(program):
        r = subprocess.run([sys.executable, "-c", HEAD % (HERE, so) + program], env=dict(os.environ, LD_PRELOAD=so), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


def test_a_failed_upload_stops_its_call(on_fake_runtime):
    """host arrays: without its inputs no kernel of the call runs and no output is written; a failed download writes none either"""
    on_fake_runtime(r'''
rng = np.random.default_rng(0)
A, B = rng.standard_normal((9, 8)).astype(np.float32), rng.standard_normal((8, 7)).astype(np.float32)
def call(fail):
    keep = pkg.Keep()
    C = np.full((9, 7), 3.0, np.float32)
    a = pkg.make_args(keep, "matMul_args", A=A, B=B, C=C, N=9, K=8, M=7, trans_B=0, USE_BIASES=0)
    lib.trainlib_clear_error()
    fake.fake_reset(fail)
    lib.mm(ctypes.byref(a))
    return fake.fake_launches(), lib.trainlib_last_error(), bool((C == 3.0).all())
n, err, same = call(0)
assert n >= 3 and err == pkg.TL_OK and not same, (n, err, same)             # uploads, products, downloads
assert call(1) == (1, 2, True), call(1)
assert call(n)[1:] == (2, True), call(n)
assert call(0) == (n, pkg.TL_OK, False)
''')


def test_depthwise_weight_gradients_occupy_the_chip(on_fake_runtime):
    """3 x 3 layers with 64 streams on 148 SMs that hold four CTAs each: up to 296 channels one wave at most and two thirds of one at least (where there are
    as many planes), beyond a wave and a half and less than a CTA a channel more"""
    on_fake_runtime(r"""
x = lib.trainlib_malloc(1 << 22)
lib.trainlib_set_streams(64)
keep = pkg.Keep()
for c in list(range(1, 800, 7)) + [296, 297, 592, 593]:
    b = lambda ch, h: pkg.make_blob(keep, x, x, C=ch, H=h, W=h)
    a = pkg.make_args(keep, "DepthWise_Conv_args", input=b(c, 8), coeff=b(c, 3), output=b(c, 8), Lpad=1, Rpad=1, Upad=1, Dpad=1, stride_h=1, stride_w=1, HWC=0)
    fake.fake_reset(0)
    lib.pulp_conv_dw_fp32_bw_param_grads_cl(ctypes.byref(a))
    n = fake.fake_max_blocks()
    assert lib.trainlib_last_error() == 0
    if c <= 296: assert min(c * 64, 592 * 2 // 3) <= n <= 592, (c, n)
    else: assert 888 <= n < 888 + c, (c, n)
""")


@pytest.mark.parametrize("limit", [8, 16])
def test_clusters_of_sixteen_only_where_they_can_be_placed(on_fake_runtime, limit):
    """weight gradients of few pixels run as clusters of up to sixteen CTAs, on a device that places eight at most as smaller ones or on another kernel"""
    on_fake_runtime(r"""
fake.fake_cluster_limit(%d)
x = lib.trainlib_malloc(1 << 22)
keep = pkg.Keep()
most = 0
for half in ("", "_fp16"):
    for cin, h, k in ((16, 32, 3), (16, 45, 3), (24, 40, 1), (12, 44, 5), (5, 41, 7), (8, 12, 3)):
        b = lambda ch, hh, dim=None: pkg.make_blob(keep, x, x, C=ch, H=hh, W=hh, dim=dim, half=bool(half))
        a = pkg.make_args(keep, "Conv2D_args" + half, input=b(cin, h), coeff=b(cin, k, 32 * cin * k * k), bias=b(32, 1), output=b(32, h), Lpad=k // 2, Rpad=k // 2, Upad=k // 2, Dpad=k // 2,
                          stride_h=1, stride_w=1, i2c_buffer=x, bt_buffer=x, USE_BIASES=0, USE_IM2COL=0, HWC=0)
        fake.fake_reset(0)
        getattr(lib, "pulp_conv2d_fp%%s_bw_param_grads_cl" %% ("16" if half else "32"))(ctypes.byref(a))
        assert fake.fake_launches() >= 1 and lib.trainlib_last_error() == 0, (half, cin, h, k)
        most = max(most, fake.fake_max_cluster())
assert most == %d, most
""" % (limit, limit))
