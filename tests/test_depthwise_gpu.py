"""The tensor-core kernel for depthwise 3 x 3 layers (csrc/kernels/conv_dw.cu): edges of its tiles of 16 x 32 output pixels
(8 x 16 with stride 2), images stacked in one tile, 32 and 64 channels a tile, more tiles than CTAs."""
import ctypes as ct

import numpy as np
import pytest

import cases
from kernel_desc import I8, Direct, shape

pytestmark = pytest.mark.gpu


# (n, c, h, w, stride, pad), each enough images for a tile an SM: whole tiles; one pixel more and less in each direction; odd
# sizes; images of few lines, two and three in a tile, the last tile half empty; no padding; many channel blocks; pairs of
# pixels (32 and 64 channels, even widths) in and out; several tiles a CTA
SHAPES = [(80, 64, 32, 16, 1, 1), (75, 64, 33, 17, 1, 1), (40, 64, 33, 18, 1, 1), (150, 64, 31, 15, 1, 1), (17, 96, 29, 45, 1, 1),
          (151, 128, 14, 14, 1, 1), (99, 192, 10, 16, 1, 1), (148, 192, 8, 16, 1, 1), (60, 64, 12, 70, 1, 0), (20, 1024, 14, 14, 1, 1),
          (75, 64, 30, 31, 1, 1), (41, 32, 56, 56, 1, 1), (301, 128, 14, 14, 1, 1), (60, 32, 57, 63, 1, 1), (3, 32, 256, 254, 1, 1),
          (80, 64, 32, 16, 2, 1), (75, 64, 34, 18, 2, 1), (150, 64, 31, 15, 2, 1), (9, 96, 29, 93, 2, 1), (151, 128, 14, 14, 2, 1),
          (99, 192, 11, 16, 2, 1), (148, 32, 8, 16, 2, 1), (34, 64, 13, 141, 2, 0), (20, 1024, 14, 14, 2, 1), (41, 32, 112, 56, 2, 1),
          (301, 128, 14, 14, 2, 1), (30, 128, 28, 56, 2, 1),
          # images cut into bands of lines, several images' bands in a tile: 16, 15, 18 and 38 lines, the last band shorter, the
          # last tile not full; 32 channels; stride 2
          (151, 64, 16, 24, 1, 1), (200, 128, 15, 16, 1, 1), (299, 64, 18, 14, 1, 1), (75, 128, 38, 21, 1, 1), (299, 32, 16, 32, 1, 1),
          (150, 128, 15, 20, 1, 1), (99, 192, 19, 19, 1, 1), (200, 64, 40, 16, 1, 0), (301, 64, 16, 48, 2, 1), (151, 128, 37, 31, 2, 1)]


@pytest.mark.parametrize("n,c,h,w,stride,pad", SHAPES)
@pytest.mark.parametrize("relu,bias", [(True, True), (False, False)])
def test_depthwise(n, c, h, w, stride, pad, relu, bias, gpu_run, oracle, wl):
    js, pb, x = cases.conv_case(c + h + n, n, c, h, w, c, 3, stride, pad, groups=c, bias=bias, relu=relu, shift=wl.GraphBuilder.default_shift(9))
    assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))


# one output pixel, one operand line and one operand row more than whole tiles (33 x 25 rows of 16 x 8 a tile), in planes and in
# pairs of pixels, of 32 and 64 channels; every layer runs on the tensor cores
@pytest.mark.parametrize("n,c,h,w,stride", [(10, 64, 66, 50, 1), (10, 64, 65, 50, 1), (14, 64, 65, 49, 1), (7, 128, 66, 50, 1), (7, 128, 65, 49, 1), (10, 32, 66, 50, 1),
                                            (5, 96, 66, 49, 1), (10, 64, 65, 50, 2), (10, 64, 66, 50, 2), (14, 64, 65, 49, 2), (7, 128, 66, 50, 2), (7, 128, 65, 49, 2),
                                            (10, 32, 65, 50, 2), (5, 96, 66, 49, 2), (50, 64, 33, 32, 1), (37, 128, 33, 31, 1)])
def test_depthwise_edges(n, c, h, w, stride, gpu_run, oracle, wl, rt):
    d = Direct()
    shape(d, n, c, h, w, c, 3, stride, 1)
    d.x_dtype = d.y_dtype = I8
    d.groups, d.depthwise, d.dil_h, d.dil_w = c, 1, 1, 1
    assert rt.lib().cvmk_conv2d_direct_tensor_cores(ct.byref(d)) == 1
    js, pb, x = cases.conv_case(c + h + n, n, c, h, w, c, 3, stride, 1, groups=c, relu=bool(n % 2), shift=wl.GraphBuilder.default_shift(9))
    assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))


# chains that are not just a shift: a clip without one, a shift that leaves more than 16 bits, a tensor operand (whole batches
# and parts of them), a bias that is computed on the way, and a chain that is run step by step with a tensor operand in it;
# a tile an SM and more, and fewer
CHAINS = ["clip", "wide", "residual", "activation_bias", "steps"]


@pytest.mark.parametrize("n,c,h,w,stride", [(80, 64, 33, 17, 1), (40, 128, 28, 28, 1), (75, 64, 34, 18, 2), (151, 96, 14, 14, 1), (41, 32, 56, 56, 1), (2, 128, 28, 28, 1)])
@pytest.mark.parametrize("chain", CHAINS)
def test_depthwise_chain(n, c, h, w, stride, chain, gpu_run, oracle, wl):
    g = wl.GraphBuilder(c + h)
    x = cases.rnd(np.random.RandomState(n), (n, c, h, w), 8)
    d = g.var("data", x.shape, 8)
    if chain == "activation_bias":
        one = g.op("cvm_right_shift", [d], x.shape, {"precision": 4, "shift_bit": 4})
        b = g.op("sum", [one], (c,), {"axis": (0, 2, 3), "keepdims": False, "exclude": False})
        wt = g.var("w", (c, 1, 3, 3), 8, g.weight8((c, 1, 3, 3)))
        oh, ow = (h - 1) // stride + 1, (w - 1) // stride + 1
        y = g.op("conv2d", [d, wt, b], (n, c, oh, ow), {"channels": c, "kernel_size": (3, 3), "strides": (stride, stride), "padding": (1, 1),
                 "dilation": (1, 1), "groups": c, "layout": "NCHW", "kernel_layout": "OIHW", "use_bias": True})
        y = g.op("cvm_right_shift", [y], g.shape_of(y), {"precision": 8, "shift_bit": 7})
    else:
        y = g.conv(d, c, 3, stride, 1, groups=c, relu=chain == "wide", shift={"clip": 0, "wide": 2}.get(chain))
    if chain == "clip":
        y = g.op("cvm_clip", [y], g.shape_of(y), {"precision": 8})
    if chain in ("residual", "steps"):
        z = g.conv(d, c, 1, stride, 0, relu=False)
        y = g.op("elemwise_sub", [y, z] if chain == "residual" else [z, y], g.shape_of(y))
        if chain == "steps":
            y = g.op("abs", [y], g.shape_of(y))
        y = g.op("cvm_clip", [y], g.shape_of(y), {"precision": 8})
    js, pb = g.finish(y)
    assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))
