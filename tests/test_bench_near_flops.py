"""The near field's operation count in bench.py is the profiled kernel's."""
import os
import re

from conftest import ROOT


def test_near_flops_are_those_of_the_profile():
    import bench
    text = open(os.path.join(ROOT, "profiles", "near_leaf_sphere5120.md")).read()
    add, mul, fma = (int(re.search(r"FP64 %s[^|]*\| ([\d,]+)" % k, text).group(1).replace(",", ""))
                     for k in ("adds", "multiplies", "FMAs"))
    pairs = int(re.search(r"([\d,]+) \(point, triangle\) near\s+pairs", text).group(1).replace(",", ""))
    assert abs(bench.NEAR_FLOPS_PER_PAIR * pairs / (add + mul + 2 * fma) - 1) < 1e-3
    # the profiled kernel is the one in the tree: its registers fill three CTAs of 128 threads per SM
    regs = int(re.search(r"registers per thread \| (\d+)", text).group(1))
    src = open(os.path.join(ROOT, "elfmmlib3d_b200", "csrc", "nearfield.cu")).read()
    minb = int(re.search(r"constexpr int NL_MINB = (\d+)", src).group(1))
    assert regs <= 65536 // (128 * minb)
