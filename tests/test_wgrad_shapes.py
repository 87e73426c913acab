"""The weight-gradient kernel over the layouts its shape rule picks: one to
three 16-block instruction groups, with and without the row of ones, one to four
stages (and more tiles per block than stages), tap rows split over two blocks.
Bounds as test_denoiser_wgrad: the same sums of the same BF16 products in FP32."""
import pytest

import test_denoiser_wgrad as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,cin,cout", [
    (1, 1, 1, 16, 16),        # less than a tile
    (3, 16, 9, 16, 64),       # one group, four stages
    (9, 150, 170, 32, 32),    # several tiles per block: the ring wraps
    (1, 17, 8, 48, 64),       # two groups, three stages
    (2, 31, 33, 64, 64),      # two groups, the largest accumulators of one block
    (5, 130, 140, 80, 32),    # two stages, wrapping
    (1, 20, 50, 96, 48),
    (4, 100, 110, 128, 16),   # three full groups: no row of ones, one stage, wrapping
    (2, 18, 23, 128, 48),
])
def test_wgrad_layouts(n, h, w, cin, cout):
    base.test_wgrad_matches_torch(n, h, w, cin, cout)
