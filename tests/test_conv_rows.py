"""The row form of the denoiser's convolution (widths from 80 pixels on) at the
edges of its 128-pixel strips, its row pairs and runs, its TMEM and row rings:
every channel pair of the U-Net and of its backward pass. Tolerance as
test_denoiser_conv (FP32 sums, BF16 output)."""
import pytest

import test_denoiser_conv as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,cin,cout,relu,ych,yoff", [
    (1, 1, 80, 16, 32, 1, 32, 0),      # one row: no neighbours above or below
    (1, 2, 127, 32, 32, 1, 80, 0),     # a strip's last pixel missing
    (2, 3, 128, 32, 48, 0, 48, 0),     # exactly a strip, an odd height
    (1, 5, 129, 48, 48, 1, 112, 0),    # a strip of one pixel (the tiled kernel)
    (1, 37, 200, 48, 64, 1, 64, 0),
    (3, 64, 256, 64, 64, 1, 112, 48),  # four TMEM slots
    (1, 33, 160, 112, 48, 1, 48, 0),
    (1, 33, 230, 112, 48, 1, 48, 0),   # two row stages
    (2, 90, 333, 80, 32, 1, 32, 0),
    (4, 481, 640, 32, 16, 0, 16, 0),   # long runs over several columns
    (1, 700, 90, 16, 64, 0, 64, 0),
])
def test_conv_rows_matches_torch(n, h, w, cin, cout, relu, ych, yoff):
    base.test_conv3x3_matches_torch(n, h, w, cin, cout, relu, ych, yoff)
