"""Which kernel the products over a mixture's experts go to: pairs of SMs only where they were measured to be the faster ones."""
import pytest

ONE_CTA, PAIRS = (0, 0), (256, 32)


@pytest.mark.parametrize("rows,experts,shared,where", [
    (12, 8, False, ONE_CTA), (48, 8, False, ONE_CTA), (96, 8, False, ONE_CTA), (16, 64, False, ONE_CTA), (32, 32, False, ONE_CTA), (127, 128, False, ONE_CTA),
    (15, 8, False, PAIRS), (64, 4, False, PAIRS), (128, 8, False, PAIRS), (128, 128, False, PAIRS), (300, 32, False, PAIRS),
    (65, 8, True, PAIRS), (16, 128, True, PAIRS), (30, 64, True, PAIRS)])
def test_the_line_between_pairs_and_one_cta(rows, experts, shared, where):
    from lia_rs_b200.kernels import ops
    assert ops.moe_pair_tile_rows(rows * experts, experts, shared) == where
