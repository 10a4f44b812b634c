"""The hand-over of gemm_pair_kernel's accumulators, on the host: however late a warp of either epilogue group comes to look, it finds the tile
it waits for.  The kernel's own counts of arrivals, with barriers that follow the parity rule."""
import os
import subprocess

from spoc_b200.build import CSRC, _nvcc

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_epilogue_warp_misses_an_accumulator(tmp_path):
    exe = str(tmp_path / "epilogue_groups")
    cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-I", CSRC, "-o", exe, os.path.join(HERE, "epilogue_groups.cu")]
    res = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr
    lines = subprocess.run([exe], capture_output=True, text=True, timeout=300, check=True).stdout.splitlines()
    assert len(lines) == 31
    for line in lines:
        f = dict(x.split("=") for x in line.split()[4:])
        assert f["mistakes"] == "0", line
        # the model sees the fault: with two groups, of which only the first hands accumulators back
        assert (int(f["first"]) > 0) == (f["groups"] == "2"), line
