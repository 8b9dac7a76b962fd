"""The persistent convolution kernel (csrc/kernels/conv_tc.cu), whose 256-row tiles belong to two CTAs: last tiles
without a second half, channels that end inside a tile's first or second half, every way operands are loaded."""
import numpy as np
import pytest

import cases
import kernel_desc

pytestmark = pytest.mark.gpu


# (n, c, h, w, oc, k, stride, groups): layers as the executor cuts them: an odd number of 128-row tiles, one, two and more N
# tiles, spatial patches, im2col loads, halo tiles with resident weights of one and two channel blocks, 256-column tiles over
# 160 channels, 128-column ones over 136.  The first and third (1 x 1 over 72 and 64 channels) and the last join below go to the
# kernel of small launches, the depthwise layers to their own
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


# Straight through the kernel interface, with a look at the plan.  (n, c, h, w, oc, k, stride, block_n, resident): 1 x 1 layers of
# 32, 64, 128 and 256 columns, weights resident and in the ring, output channels that end inside a tile; 3 x 3 of each way
# to load; every one with an odd number of 128-row tiles, so that the last pair lacks its second half
PLANS = [(33, 64, 111, 111, 32, 1, 1, 32, True), (40, 64, 61, 61, 64, 1, 1, 64, True), (21, 256, 62, 63, 64, 1, 1, 64, True),
         (62, 32, 61, 61, 64, 1, 1, 64, True), (40, 64, 61, 61, 72, 1, 1, 128, False), (21, 128, 61, 61, 128, 1, 1, 128, True),
         (32, 64, 61, 61, 96, 1, 1, 128, False), (21, 128, 61, 61, 384, 1, 1, 128, False), (9, 64, 57, 57, 256, 1, 1, 256, False),
         (13, 256, 62, 63, 512, 1, 1, 256, True), (21, 96, 111, 77, 136, 3, 2, 256, False), (10, 64, 61, 61, 160, 3, 1, 256, False),
         (15, 64, 72, 72, 64, 3, 1, 64, False), (15, 128, 72, 72, 96, 3, 1, 128, False)]


@pytest.mark.parametrize("n,c,h,w,oc,k,stride,block_n,resident", PLANS)
@pytest.mark.parametrize("packed", [True, False])
def test_plan(n, c, h, w, oc, k, stride, block_n, resident, packed, rt):
    plan = kernel_desc.run_conv(rt, n, c, h, w, oc, k, stride, packed, seed=n + oc)
    m_tiles = -(-n * plan.d.OH * plan.d.OW // 128) if plan.a_im2col < 2 else \
        -(-plan.d.OW // plan.patch_w) * -(-plan.d.OH // plan.patch_h) * -(-n // plan.patch_n)
    assert plan.small_split == 0 and plan.block_n == block_n and plan.b_resident == int(resident) and m_tiles % 2 == 1


@pytest.mark.parametrize("n,c,h,w,oc,block_n", [(32, 128, 61, 61, 96, 128), (40, 64, 61, 61, 64, 64), (10, 256, 61, 61, 512, 256), (21, 256, 61, 61, 1024, 256)])
@pytest.mark.parametrize("packed", [True, False])
def test_plan_with_join(n, c, h, w, oc, block_n, packed, rt):
    plan = kernel_desc.run_conv(rt, n, c, h, w, oc, 1, 1, packed, join=True, seed=n + oc)
    assert plan.small_split == 0 and plan.block_n == block_n and plan.res_step == 2 and -(-n * h * w // 128) % 2 == 1
