"""The block of a batch or server member's row step (orrery_b200/csrc/ops3d.h): a
member in linear order takes the block that a solver of its size takes, unless
the caller named one."""
import os
import subprocess

from orrery_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

LINE = 5_500_000   # nodes from which the linear-order step takes 256 threads


def test_members_take_a_solvers_block(tmp_path):
    exe = str(tmp_path / "row_block_test")
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "-x", "c++",
                    os.path.join(ROOT, "tests", "native", "row_block_test.cpp"), "-o", exe, "-cudart", "static"],
                   check=True, capture_output=True)
    cases = [(0, 1, LINE - 1, 128), (0, 1, LINE, 256), (0, 1, 2 ** 26, 256), (0, 1, 27, 128),
             (0, 0, LINE, 128),          # row tiles keep the schedule's
             (1, 1, LINE, 128), (1, 0, LINE, 128), (1, 1, LINE - 1, 128)]
    out = subprocess.run([exe], input="\n".join(" ".join(map(str, c[:3])) for c in cases), capture_output=True,
                         text=True, check=True).stdout
    assert [int(line) for line in out.split()] == [c[3] for c in cases]
