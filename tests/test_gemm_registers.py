"""The GEMM kernels of divided k-loops keep their values in registers: what was spilled cost 0.5 us of a launch and more."""
import os
import re
import subprocess

from spoc_b200.build import CSRC, _nvcc

ARGS = {"split": ", ".join(["const __grid_constant__ CUtensorMap"] * 5), "convert": "const ConvOperands, " + ", ".join(["const __grid_constant__ CUtensorMap"] * 2)}
# BN, CTAS, ROWS, divided within a cluster; MODE, BN, quads, divided within a cluster
INSTANCES = [("split", f"{form}, true") for form in ("64, 1, 64", "128, 1, 64", "64, 1, 128", "128, 1, 128", "64, 2, 128", "128, 2, 128", "192, 2, 128", "256, 2, 128")]
INSTANCES += [("convert", f"{form}, true, true") for form in ("1, 64", "1, 128", "3, 64", "3, 128")]


def test_divided_k_loops_spill_nothing(tmp_path):
    src = ['#include "gemm_convert.cuh"', '#include "gemm_split.cuh"', "using namespace sb200;"]
    src += [f"template __global__ void sb200::gemm_{kind}_kernel<{form}>({ARGS[kind]}, const GemmParams);" for kind, form in INSTANCES]
    path = tmp_path / "divided.cu"
    path.write_text("\n".join(src) + "\n")
    cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-I", CSRC, "-Xptxas", "-v", "-cubin",
           "-o", str(tmp_path / "divided.cubin"), str(path)]
    res = subprocess.run(cmd, capture_output=True, text=True, timeout=900, stdin=subprocess.DEVNULL, cwd=os.path.dirname(str(path)))
    assert res.returncode == 0, res.stderr
    seen = re.findall(r"Function properties for (\S*gemm_(?:split|convert)_kernel\S*)\n.*?(\d+) bytes spill stores, (\d+) bytes spill loads", res.stderr)
    assert len(seen) == len(INSTANCES), res.stderr
    assert all(stores == loads == "0" for _, stores, loads in seen), seen
