"""The autotuner's buffer holds every poly its timings transform, for any limb count (tests/tune_sample_check.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_batch_sized_calls_stay_inside_the_buffer(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "tune_sample_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "tune_sample_check.cpp")], check=True,
                   capture_output=True, timeout=120)
    out = subprocess.run([exe], check=False, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
