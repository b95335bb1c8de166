"""The fixed-point sums of the wet elements, node by node (compiled for the
host and held to long double)."""

import pytest

from test_fixed64 import CSRC, run_check


@pytest.mark.parametrize("seed_error", ["0.0f", "4.0e-7f"])
def test_wet_element_sums_node_by_node(tmp_path, seed_error):
    """No node's sums less exact than FP64's, over the elements that are left
    to fixed point; nothing overflows."""
    run_check(tmp_path, "fixed64_nodes_check", f"-DDGSWE_SEED_ERROR={seed_error}",
              "-fsanitize=undefined", "-fno-sanitize-recover=undefined", str(CSRC / "setup.cpp"))
