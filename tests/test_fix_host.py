"""CPU test of the fixed-point arithmetic behind the FP64 line sums: the same
header the GPU kernels include is compiled for the host with g++ and compared
with long double (conversions, range check, one row of a line sum)."""
import os
import subprocess

from helpers import ROOT


def test_fixed_point_line_sums_on_the_host(tmp_path):
    exe = str(tmp_path / "fix_host_check")
    src = os.path.join(ROOT, "tests", "fix_host_check.cpp")
    inc = os.path.join(ROOT, "scale-dg-kernel-extraction_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{inc}", src, "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
