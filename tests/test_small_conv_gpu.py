"""The convolution kernel of launches that do not fill the GPU (csrc/kernels/conv_small.cu), at the edges of
its tiles, rings and clusters."""
import numpy as np
import pytest

import cases
import kernel_desc

pytestmark = pytest.mark.gpu


# (n, c, h, w, oc, k, stride): one unit of 32 channels (a ring smaller than the tile it stages on the way
# out), 64- and 32-column tiles, channels that end inside a tile, ragged last tiles, two to four units behind one
# barrier, rings that turn, reductions whole and cut over four CTAs with rows the cut does not divide,
# strided filters (im2col loads), patches of several images; two and three CTAs an SM whose rings turn, one unit
# behind each of eight barriers
@pytest.mark.parametrize("n,c,h,w,oc,k,stride", [
    (5, 32, 85, 85, 64, 1, 1), (3, 32, 85, 85, 64, 3, 2), (5, 32, 85, 85, 40, 1, 1), (1, 32, 9, 9, 8, 1, 1), (2, 64, 61, 61, 72, 1, 1),
    (1, 128, 57, 57, 128, 1, 1), (1, 256, 29, 31, 64, 1, 1), (1, 512, 14, 14, 32, 1, 1), (1, 1024, 14, 14, 256, 1, 1),
    (1, 512, 7, 7, 512, 3, 1), (3, 256, 7, 7, 128, 3, 1), (1, 512, 13, 13, 512, 3, 2), (1, 2048, 7, 7, 512, 1, 1), (1, 128, 11, 5, 136, 3, 1),
    (11, 512, 29, 29, 192, 1, 1), (13, 512, 41, 43, 128, 1, 1), (5, 256, 27, 27, 264, 3, 1), (10, 1024, 14, 14, 520, 1, 1)])
def test_convolution(n, c, h, w, oc, k, stride, gpu_run, oracle, wl):
    for shift, relu in ((wl.GraphBuilder.default_shift(c * k * k), True), (None, False)):   # packed and step by step
        js, pb, x = cases.conv_case(c + oc, n, c, h, w, oc, k, stride, k // 2, shift=shift, relu=relu)
        assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))


# the weights as the 128-row operand: rows around the widths of the narrow one, channels that end inside a tile
@pytest.mark.parametrize("rows", [1, 31, 33, 64, 65, 128, 129])
@pytest.mark.parametrize("k,units", [(1024, 1000), (4096, 136), (16384, 1024)])   # (the last: rings that turn, cut over eight CTAs)
def test_dense(rows, k, units, gpu_run, oracle, wl):
    g = wl.GraphBuilder(rows)
    y = g.dense(g.var("data", (rows, k), 8), units, shift=0 if rows % 2 else None)
    js, pb = g.finish(y)
    x = np.random.RandomState(rows).randint(-127, 128, size=(rows, k)).astype(np.int8)
    assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))


# The cut that the rule gives for 148 SMs, straight through the kernel interface: reductions over one, two, four and eight CTAs, of
# tiles of 9, 25, 35, 49, 105 (361 in three tiles) and 128 rows, channels that end inside a tile, im2col loads and patches
@pytest.mark.parametrize("n,c,h,w,oc,k,stride,split,block_n", [
    (1, 256, 19, 19, 512, 3, 1, 2, 32), (1, 256, 19, 19, 520, 3, 1, 2, 32), (1, 2048, 19, 19, 512, 1, 1, 2, 32), (2, 256, 19, 19, 264, 3, 1, 2, 32),
    (1, 512, 7, 7, 512, 3, 1, 4, 32), (1, 512, 13, 13, 512, 3, 2, 4, 32), (3, 256, 7, 7, 128, 3, 1, 4, 32), (1, 2048, 7, 7, 512, 1, 1, 4, 32),
    (1, 512, 3, 3, 64, 3, 1, 8, 32), (1, 512, 5, 5, 72, 3, 1, 8, 32), (1, 512, 7, 7, 40, 3, 1, 8, 32), (1, 1024, 5, 7, 72, 3, 1, 8, 32),
    (3, 256, 27, 27, 264, 3, 1, 1, 64), (10, 1024, 14, 14, 520, 1, 1, 1, 64)])
@pytest.mark.parametrize("packed,join", [(True, False), (False, False), (True, True)])
def test_cut(n, c, h, w, oc, k, stride, split, block_n, packed, join, rt):
    import torch
    plan = kernel_desc.run_conv(rt, n, c, h, w, oc, k, stride, packed, join, seed=n + oc)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert (plan.small_split, plan.block_n) == (split, block_n)
