"""CPU test of the page mapping ahead of downloads: compiled with g++, with a
thread that writes to the same pages."""
import os
import platform
import subprocess

import pytest

from helpers import ROOT


@pytest.mark.skipif(tuple(int(x) for x in platform.release().split(".")[:2]) < (5, 14),
                    reason="the kernel maps no pages ahead")
def test_mapping_pages_loses_no_write(tmp_path):
    exe = str(tmp_path / "pages_host_check")
    src = os.path.join(ROOT, "tests", "pages_host_check.cpp")
    inc = os.path.join(ROOT, "scale-dg-kernel-extraction_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", f"-I{inc}", src, "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
