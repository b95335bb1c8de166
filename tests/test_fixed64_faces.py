"""The fixed-point flux between two sides, side by side (compiled for the host
and held to long double)."""

import pytest

from test_fixed64 import CSRC, run_check


@pytest.mark.parametrize("seed_error", ["0.0f", "-4.0e-7f"])
def test_face_fluxes_side_by_side(tmp_path, seed_error):
    """Neither side's flux less exact than FP64's for its own depth and current,
    the largest errors included."""
    run_check(tmp_path, "fixed64_faces_check", f"-DDGSWE_SEED_ERROR={seed_error}",
              "-fsanitize=undefined", "-fno-sanitize-recover=undefined", str(CSRC / "setup.cpp"))
