"""The absorbing layers' targets are formed on the host (solvers) and on the
device (a server's gradual start) and have to agree to the bit: compiled with the
library's own flags for a host that has fused multiply-adds."""
import os
import platform
import subprocess

import pytest

from orrery_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(platform.machine() != "x86_64", reason="names an x86-64 instruction set")
def test_host_targets_are_not_contracted(tmp_path):
    with open("/proc/cpuinfo") as info:
        if " fma " not in info.read():
            pytest.skip("this host has no fused multiply-add")
    exe = str(tmp_path / "inlet_targets_test")
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "-Xcompiler", "-mfma", "-x", "cu",
                    os.path.join(ROOT, "tests", "native", "inlet_targets_test.cu"), "-o", exe, "-cudart", "static"],
                   check=True, capture_output=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split() == ["0", "0"]
