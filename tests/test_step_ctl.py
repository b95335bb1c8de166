"""The device clock's initial state (compiled for the host)."""

import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


def test_a_fresh_clock_takes_any_step(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "step_ctl_check"
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", str(HERE.parent / "dgcom_gb300" / "csrc"),
                    str(HERE / "step_ctl_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
