"""Staged host copies of several streams (orrery_b200/csrc/host_copy.cpp) on the
CPU, as test_host_copy.py builds them: a copy behind a busy stream does not hold
the staging ring."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("sanitize", [False, True])
def test_a_busy_stream_leaves_the_ring(tmp_path, sanitize):
    exe = str(tmp_path / "host_copy_ring_test")
    cmd = ["g++", "-std=c++20", "-O1", "-g", "-pthread", *(["-fsanitize=thread"] if sanitize else []),
           "-I", os.path.join(ROOT, "tests", "native", "fake_cuda"), "-I", os.path.join(ROOT, "include"),
           "-I", os.path.join(ROOT, "orrery_b200", "csrc"),
           os.path.join(ROOT, "tests", "native", "host_copy_ring_test.cpp"),
           os.path.join(ROOT, "orrery_b200", "csrc", "host_copy.cpp"), "-o", exe]
    built = subprocess.run(cmd, capture_output=True, text=True)
    if sanitize and built.returncode != 0:
        pytest.skip("no thread sanitizer runtime")
    assert built.returncode == 0, built.stderr
    res = subprocess.run([exe], capture_output=True, text=True, timeout=600,
                         env=dict(os.environ, TSAN_OPTIONS="halt_on_error=1"))
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout + res.stderr
    assert "WARNING: ThreadSanitizer" not in res.stderr
