"""Division by multiplication (orrery_b200/csrc/fast_div.h), compiled with g++:
exact for every divisor from 2 on, a divisor it has no form for refused."""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


def test_quotients_are_exact(tmp_path):
    exe = str(tmp_path / "fast_div_test")
    subprocess.run(["g++", "-std=c++20", "-O1", "-I", os.path.join(ROOT, "orrery_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "fast_div_test.cpp"), "-o", exe], check=True)
    rng = random.Random(3)
    divisors = sorted(set(list(range(2, 300)) + [2 ** b + k for b in range(9, 31) for k in (-1, 0, 1)] +
                          [2 ** 31 - 1] + [rng.randrange(3, 2 ** 27) for _ in range(200)]))
    out = subprocess.run([exe, "0", "1", *map(str, divisors)], capture_output=True, text=True, check=True).stdout
    assert out.splitlines() == ["0 refused", "1 refused"] + [f"{d} 0" for d in divisors]
