"""The kernel families of the bench's roofline: no GPU needed."""
import glob
import os
import re
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench_nets  # noqa: E402

Net = next(c for c in vars(bench_nets).values() if isinstance(c, type) and hasattr(c, "FAMILIES"))
PEAKS = {"bf16_tflops": 1642.0, "bf16_tflops_sustained": 1368.0, "hbm_gbs": 6547.0, "source": "test"}


def test_every_convolution_kernel_has_a_family():
    members = {m for _, names, _, _ in Net.FAMILIES for m in names}
    kernels = set()
    for path in glob.glob(os.path.join(ROOT, "pulp-trainlib_b200", "csrc", "*.cu")):
        kernels |= set(re.findall(r"__global__[^;{]*?\b(conv\w*_kernel)\s*\(", open(path).read()))
    kernels -= {"conv_dilate_dy_kernel"}              # spreads samples, multiplies nothing
    assert len(kernels) >= 12 and kernels <= members, sorted(kernels - members)


def test_launches_go_by_the_name_of_their_kernel():
    """the profile takes the name that a launch is written with: never a local variable's (upper case: a macro's parameter)"""
    for path in glob.glob(os.path.join(ROOT, "pulp-trainlib_b200", "csrc", "*.cu")):
        for name in re.findall(r"TL_LAUNCH(?:_CLUSTER)?\(\(*(\w+)", open(path).read()):
            assert name.endswith("_kernel") or name.isupper(), "%s: %s" % (os.path.basename(path), name)


@pytest.mark.parametrize("name,bound", [("(conv_wgy_kernel<2, 2>)", "tensor"), ("(conv_mma_kernel<T, 1, 1, 8, 1, 128>)", "tensor"), ("some_kernel", "unclassified")])
def test_a_contraction_is_never_reported_as_bandwidth_bound(name, bound):
    table = [(name, 2, 0.5, 4e10), ("(act_bw_kernel<T>)", 3, 0.2, 0.0)]
    top = Net.roofline(object.__new__(Net), table, 512, PEAKS)
    assert top["bound"] == bound and top["algorithmic_flops"] == 4e10 and abs(top["achieved"] - 80.0) < 1e-9
    assert (top["frac"] is None) == (bound == "unclassified")
    assert [f["bound"] for f in top["families"]] == ["hbm"]
