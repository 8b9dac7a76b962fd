"""The image stem (csrc/kernels/conv_stem.cu): 1 to 4 channels, both strides, every filter form that has products of its own
and one that has not, blocks of different numbers of rows with a last one that is not full, and inputs of -128."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,h,w,oc,k,stride,pad", [
    (1, 3, 224, 224, 64, 7, 2, 3), (37, 3, 97, 112, 64, 7, 2, 3), (5, 3, 224, 224, 64, 3, 1, 1), (70, 3, 61, 64, 32, 3, 1, 1),
    (60, 3, 112, 96, 32, 3, 2, 1), (3, 1, 64, 80, 128, 8, 2, 0), (9, 2, 50, 48, 32, 5, 1, 2), (4, 4, 33, 32, 64, 4, 1, 0),
    (11, 4, 64, 64, 32, 3, 2, 1), (2, 3, 300, 304, 64, 7, 2, 3), (6, 2, 40, 50, 64, 5, 2, 2)])
def test_stem(n, c, h, w, oc, k, stride, pad, gpu_run, oracle, wl):
    js, pb, x = cases.conv_case(c + k + n, n, c, h, w, oc, k, stride, pad, relu=n % 2 == 0, shift=wl.GraphBuilder.default_shift(c * k * k))
    x = np.array(x)
    x.reshape(-1)[::7] = -128
    assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))
