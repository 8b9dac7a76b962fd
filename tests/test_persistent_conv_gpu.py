"""The persistent convolution kernel (csrc/kernels/conv_tc.cu), whose 256-row tiles belong to two CTAs: last tiles
without a second half, channels that end inside a tile's first or second half, every way operands are loaded."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


# (n, c, h, w, oc, k, stride, groups): an odd number of 128-row tiles (291, 229, 399) over one, two and more N tiles, weights
# resident and in the ring, spatial patches, im2col loads, halo tiles with resident weights of one and two channel
# blocks, 256-column tiles over 160 channels, 128-column ones over 136, depthwise layers (tiles of two images in one pair)
@pytest.mark.parametrize("n,c,h,w,oc,k,stride,groups", [
    (10, 64, 61, 61, 72, 1, 1, 1), (9, 64, 57, 57, 256, 1, 1, 1), (13, 256, 62, 63, 64, 1, 1, 1), (13, 256, 62, 63, 512, 1, 1, 1),
    (10, 64, 61, 61, 160, 3, 1, 1), (21, 96, 111, 77, 136, 3, 2, 1), (15, 64, 72, 72, 64, 3, 1, 1), (15, 128, 72, 72, 96, 3, 1, 1),
    (171, 128, 16, 24, 128, 3, 1, 128), (130, 256, 15, 16, 256, 3, 1, 256), (61, 32, 40, 44, 32, 3, 1, 32)])
def test_convolution(n, c, h, w, oc, k, stride, groups, gpu_run, oracle, wl):
    for shift, relu in ((wl.GraphBuilder.default_shift(c // groups * k * k), True), (None, False)):   # packed and step by step
        if shift is None and c * k * k > 600:
            continue
        js, pb, x = cases.conv_case(c + oc, n, c, h, w, oc, k, stride, k // 2, groups=groups, shift=shift, relu=relu)
        assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))


# residual joins: operand tiles that arrive in one or two staging buffers, the last pair's second half missing
@pytest.mark.parametrize("n,c,h,w,oc", [(9, 64, 57, 57, 256), (10, 256, 61, 61, 512), (10, 128, 61, 61, 96)])
def test_residual_join(n, c, h, w, oc, gpu_run, oracle, wl):
    g = wl.GraphBuilder(c + oc)
    x = cases.rnd(np.random.RandomState(n), (n, c, h, w), 8)
    d = g.var("data", x.shape, 8)
    sc = g.conv(d, oc, 1, 1, 0, relu=False)
    z = g.conv(d, oc, 1, 1, 0, relu=False)
    a = g.op("elemwise_add", [z, sc], g.shape_of(z))
    a = g.op("relu", [a], g.shape_of(a))
    js, pb = g.finish(g.op("cvm_clip", [a], g.shape_of(a), {"precision": 8}))
    assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))
