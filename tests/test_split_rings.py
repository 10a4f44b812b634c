"""The waits of the splitting GEMM's rings, on the host: whatever order its loads land in, no group takes a raw stage for a k-block that has
not landed.  The kernel's own order of waits and its own ring lengths, with barriers that follow the parity rule."""
import os
import subprocess

from spoc_b200.build import CSRC, _nvcc

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_raw_stage_is_read_before_it_has_landed(tmp_path):
    exe = str(tmp_path / "split_rings")
    cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-I", CSRC, "-o", exe, os.path.join(HERE, "split_rings.cu")]
    res = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr
    lines = subprocess.run([exe], capture_output=True, text=True, timeout=300, check=True).stdout.splitlines()
    assert len(lines) == 8
    for line in lines:
        f = dict(x.split("=") for x in line.split()[3:])
        raw, parts, groups = (int(f[x]) for x in ("raw", "parts", "groups"))
        assert f["early"] == "0", line
        # the model sees the fault: with the raw stage waited for first, it shows wherever neither rule about the lengths holds
        assert (int(f["other"]) > 0) == (raw % groups != 0 and raw < groups + parts), line
