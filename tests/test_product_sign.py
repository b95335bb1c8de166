"""The sign of a product without the product (compiled for the host), which the
subcells' slopes take: an extremum is where dm·dp <= 0 as it rounds."""

from test_fixed64 import run_check


def test_the_sign_of_a_product(tmp_path):
    run_check(tmp_path, "product_sign_check")
