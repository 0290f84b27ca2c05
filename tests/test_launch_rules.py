"""Host checks of the rules that size launches and their buffers: the autotuner's sample (tune_sample_check.cpp) and
the grid of a transform pass (ntt_grid_check.cpp), over all sizes they are used at."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("check", ["tune_sample_check", "ntt_grid_check"])
def test_rule(tmp_path, check):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / check)
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, check + ".cpp")], check=True,
                   capture_output=True, timeout=120)
    out = subprocess.run([exe], check=False, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
