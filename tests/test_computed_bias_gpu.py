"""Biases that the graph computes: a kernel that starts while the one before it drains has to read them after that one has
ended.  The first inference of a handle decides it: the timing at load ran on zeros, so a bias read too early is zero."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


# (n, c, h, w, oc, k, stride, groups, shift): depthwise on the tensor cores, of both strides, with one channel group a tile and
# two, and step by step; depthwise on the CUDA cores, tiled, by rows and of 5 x 5; a grouped layer; the persistent
# kernel and the one for small launches, packed and step by step; an image stem
@pytest.mark.parametrize("n,c,h,w,oc,k,stride,groups,shift", [
    (40, 128, 28, 28, 128, 3, 1, 128, 7), (80, 96, 33, 17, 96, 3, 1, 96, 7), (40, 64, 28, 28, 64, 3, 2, 64, 7), (40, 64, 28, 28, 64, 3, 1, 64, 2),
    (2, 64, 14, 14, 64, 3, 1, 64, 7), (9, 48, 28, 28, 48, 3, 1, 48, 7), (9, 64, 28, 28, 64, 5, 1, 64, 8), (9, 16, 28, 28, 32, 3, 1, 4, 8),
    (40, 64, 56, 56, 128, 1, 1, 1, 9), (40, 64, 56, 56, 64, 3, 1, 1, 11), (40, 64, 56, 56, 72, 1, 1, 1, 0), (4, 64, 28, 28, 64, 3, 1, 1, 11),
    (4, 64, 28, 28, 40, 1, 1, 1, 0), (9, 3, 64, 64, 32, 3, 2, 1, 8)])
def test_computed_bias(n, c, h, w, oc, k, stride, groups, shift, gpu_run, oracle, wl):
    g = wl.GraphBuilder(c + h)
    x = cases.rnd(np.random.RandomState(n), (n, c, h, w), 8)
    d = g.var("data", x.shape, 8)
    small = g.op("cvm_right_shift", [d], x.shape, {"precision": 4, "shift_bit": 4})
    per_channel = g.op("sum", [small], (c,), {"axis": (0, 2, 3), "keepdims": False, "exclude": False})
    bias = per_channel
    if oc != c:   # repeated, or cut, to the output channels
        bias = g.op("repeat", [bias], (c * -(-oc // c),), {"repeats": -(-oc // c), "axis": 0})
        bias = g.op("strided_slice", [bias], (oc,), {"begin": (0,), "end": (oc,), "stride": (1,)})
    shape = (oc, c // groups, k, k)
    wt = g.var("w", shape, 8, g.weight8(shape))
    oh, ow = (h + 2 * (k // 2) - k) // stride + 1, (w + 2 * (k // 2) - k) // stride + 1
    y = g.op("conv2d", [d, wt, bias], (n, oc, oh, ow), {
        "channels": oc, "kernel_size": (k, k), "strides": (stride, stride), "padding": (k // 2, k // 2), "dilation": (1, 1), "groups": groups,
        "layout": "NCHW", "kernel_layout": "OIHW", "use_bias": True})
    if shift:
        y = g.op("cvm_right_shift", [y], g.shape_of(y), {"precision": 8, "shift_bit": shift})
    js, pb = g.finish(y)
    assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))
