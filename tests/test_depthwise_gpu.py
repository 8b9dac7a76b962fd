"""The tensor-core kernel for depthwise 3 x 3 layers (csrc/kernels/conv_dw.cu): edges of its tiles of 16 x 32 output pixels
(8 x 16 with stride 2), images stacked in one tile, 32 and 64 channels a tile, more tiles than CTAs."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


# (n, c, h, w, stride, pad), each enough images for a tile an SM: whole tiles; one pixel more and less in each direction; odd
# sizes; images of few lines, two and three in a tile, the last tile half empty; no padding; many channel blocks; pairs of
# pixels (32 and 64 channels, even widths) in and out; several tiles a CTA
SHAPES = [(80, 64, 32, 16, 1, 1), (75, 64, 33, 17, 1, 1), (40, 64, 33, 18, 1, 1), (150, 64, 31, 15, 1, 1), (17, 96, 29, 45, 1, 1),
          (151, 128, 14, 14, 1, 1), (99, 192, 10, 16, 1, 1), (148, 192, 8, 16, 1, 1), (60, 64, 12, 70, 1, 0), (20, 1024, 14, 14, 1, 1),
          (75, 64, 30, 31, 1, 1), (41, 32, 56, 56, 1, 1), (301, 128, 14, 14, 1, 1), (60, 32, 57, 63, 1, 1), (3, 32, 256, 254, 1, 1),
          (80, 64, 32, 16, 2, 1), (75, 64, 34, 18, 2, 1), (150, 64, 31, 15, 2, 1), (9, 96, 29, 93, 2, 1), (151, 128, 14, 14, 2, 1),
          (99, 192, 11, 16, 2, 1), (148, 32, 8, 16, 2, 1), (34, 64, 13, 141, 2, 0), (20, 1024, 14, 14, 2, 1), (41, 32, 112, 56, 2, 1),
          (301, 128, 14, 14, 2, 1), (30, 128, 28, 56, 2, 1)]


@pytest.mark.parametrize("n,c,h,w,stride,pad", SHAPES)
@pytest.mark.parametrize("relu,bias", [(True, True), (False, False)])
def test_depthwise(n, c, h, w, stride, pad, relu, bias, gpu_run, oracle, wl):
    js, pb, x = cases.conv_case(c + h + n, n, c, h, w, c, 3, stride, pad, groups=c, bias=bias, relu=relu, shift=wl.GraphBuilder.default_shift(9))
    assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))
