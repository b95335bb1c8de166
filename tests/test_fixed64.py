"""The fixed-point arithmetic of the kernels (dgcom_gb300/csrc/fixed64.hpp),
compiled for the host and held to long double."""

import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


CSRC = HERE.parent / "dgcom_gb300" / "csrc"


def run_check(tmp_path, name, *flags):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / name
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", *flags,
                    "-I", str(CSRC), str(HERE / f"{name}.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.startswith("ok ")


@pytest.mark.parametrize("seed_error", ["0.0f", "4.0e-7f", "-4.0e-7f"])
def test_roots_reciprocals_and_powers(tmp_path, seed_error):
    """√x, 1/x and x^(-4/3) within 0.75 ulp, with seeds off by up to 2^-21."""
    run_check(tmp_path, "fixed64_check", f"-DDGSWE_SEED_ERROR={seed_error}")


@pytest.mark.parametrize("seed_error", ["0.0f", "4.0e-7f", "-4.0e-7f"])
def test_face_fluxes_and_wet_element_sums(tmp_path, seed_error):
    """The interior face's flux and the wet element's sums of orders 1 to 4:
    their error no larger than the FP64 formulas', nothing overflows."""
    run_check(tmp_path, "fixed64_flux_check", f"-DDGSWE_SEED_ERROR={seed_error}",
              "-fsanitize=undefined", "-fno-sanitize-recover=undefined", str(CSRC / "setup.cpp"))
