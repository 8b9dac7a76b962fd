"""Launchers of the kernel C-ABI (include/cvmk_kernels.h) called directly, in ways that the executor does not."""
import ctypes as ct

import numpy as np
import pytest

from kernel_desc import (ADD_C, I8, I32, RSHIFT, Conv, ConvPlan, Direct, Reduce, Stem, chain, conv_sums, int8, right_shift, shape)

pytestmark = pytest.mark.gpu


def shift_clip(desc, shift, bias=None):
    chain(desc, ([(ADD_C, 0, 0, I32, bias)] if bias else []) + [(RSHIFT, shift, 8, 0, None)])


# Weights and a bias that the kernel in front of the launch writes, with bias_static left 0.  That kernel is a sum of many rows
# (all zero but the last) in one block: it is at work long after a kernel that starts early has got to its weights.
@pytest.mark.parametrize("kind", ["depthwise", "stem"])
def test_weights_written_by_the_kernel_before(kind, rt):
    import torch
    lib, rng = rt.lib(), np.random.RandomState(5)
    n, c, h, oc, k, step, groups, shift = (40, 64, 56, 64, 3, 1, 64, 7) if kind == "depthwise" else (8, 3, 224, 64, 7, 2, 1, 9)
    oh = (h + 2 * (k // 2) - k) // step + 1
    x, w = int8(torch, rng, n, c, h, h), int8(torch, rng, oc, c // groups, k, k)
    bias = torch.from_numpy(rng.randint(-5000, 5000, size=oc).astype(np.int32)).cuda()
    y = torch.empty(n, oh, oh, oc, dtype=torch.int8, device="cuda")
    if kind == "depthwise":
        d, xin, wk = Direct(), x.permute(0, 2, 3, 1).contiguous(), w.reshape(oc, 9).t().contiguous().reshape(-1)
        d.x_dtype, d.y_dtype, d.depthwise, d.groups, d.dil_h, d.dil_w = 1, 1, 1, groups, 1, 1
    else:
        d, xin, wk = Stem(), x, None
        d.clamp = 127
    shape(d, n, c, h, h, oc, k, step, k // 2)
    d.acc_bound = (c // groups) * k * k * 128 * 128 + 5000
    if wk is None:
        packed = np.zeros(lib.cvmk_conv2d_stem_weight_bytes(ct.byref(d)), np.int8)
        wide = np.ascontiguousarray(w.cpu().numpy().astype(np.int32))
        assert lib.cvmk_conv2d_stem_pack_weights(ct.byref(d), wide.ctypes.data_as(ct.c_void_p), packed.ctypes.data_as(ct.c_void_p)) == 0
        wk = torch.from_numpy(packed).cuda()
    params = torch.cat([wk.view(torch.int32), bias])
    rows = 100000
    source = torch.zeros(rows, params.numel(), dtype=torch.int32, device="cuda")
    source[-1] = params
    target = torch.zeros_like(params)
    at_b = wk.numel()
    d.x, d.y, d.w = xin.data_ptr(), y.data_ptr(), target.data_ptr()
    shift_clip(d, shift, target.data_ptr() + at_b)
    total = Reduce(n_keep=1, n_red=1, x=source.data_ptr(), x_dtype=4, y=target.data_ptr(), y_dtype=4)
    total.keep_extent[0], total.keep_stride[0], total.red_extent[0], total.red_stride[0] = params.numel(), 1, rows, params.numel()
    plan = None
    if kind == "stem":
        raw = ct.create_string_buffer(4096)
        plan = ct.c_void_p((ct.addressof(raw) + 63) & ~63)
        assert lib.cvmk_conv2d_stem_prepare(ct.byref(d), plan) == 0
    stream = torch.cuda.Stream()   # (kernels of the default stream do not overlap)
    for _ in range(2):             # (the first launch of a kernel loads it and waits)
        target.zero_()
        torch.cuda.synchronize()
        at = ct.c_void_p(stream.cuda_stream)
        assert lib.cvmk_reduce(ct.byref(total), at) == 0
        assert (lib.cvmk_conv2d_stem_launch(plan, at) if plan else lib.cvmk_conv2d_direct(ct.byref(d), at)) == 0
        torch.cuda.synchronize()
    want = conv_sums(torch, x, w, step, k // 2, groups) + bias.long()
    assert torch.equal(y, right_shift(want, shift).to(torch.int8))


# The grouped form of the persistent kernel, which the executor does not launch.  (n, channels, h, w, fold), sizes of the
# real image: one to three N tiles of 4, 2 and 1 groups of 32 channels; folded pixels, 2 of 64 channels and 4 of 32; an odd
# number of 128-row tiles, and patches that end outside the image
@pytest.mark.parametrize("n,c,h,w,fold", [(171, 128, 16, 24, 1), (129, 256, 15, 24, 1), (75, 96, 16, 24, 1), (33, 192, 31, 23, 1), (1, 128, 16, 8, 1),
                                          (171, 64, 16, 48, 2), (75, 64, 30, 46, 2), (171, 32, 16, 96, 4), (75, 32, 30, 92, 4)])
@pytest.mark.parametrize("packed", [True, False])
def test_grouped(n, c, h, w, fold, packed, rt):
    import torch
    lib, rng = rt.lib(), np.random.RandomState(n + c)
    x, wt = int8(torch, rng, n, c, h, w), int8(torch, rng, c, 32, 3, 3)
    bias = torch.from_numpy(rng.randint(-5000, 5000, size=c).astype(np.int32)).cuda()
    d, shift = Conv(), 11
    shape(d, n, c * fold, h, w // fold, c * fold, 3, 1, 1)
    d.dil_h = d.dil_w = 1
    d.groups, d.group_fold = c * fold // 32, fold
    d.acc_bound = 32 * 9 * 127 * 127 + 5000 if packed else 0
    xin, y = x.permute(0, 2, 3, 1).contiguous(), torch.zeros(n, h, w, c, dtype=torch.int8, device="cuda")
    wk, bias_k = wt.permute(0, 2, 3, 1).contiguous().repeat(fold, 1, 1, 1), bias.repeat(fold)   # (once per sub-pixel)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    d.x, d.w, d.y, d.y_dtype, d.status = xin.data_ptr(), wk.data_ptr(), y.data_ptr(), I8, status.data_ptr()
    shift_clip(d, shift, bias_k.data_ptr())
    raw = ct.create_string_buffer(4096)
    plan = ConvPlan.from_buffer(raw, (-ct.addressof(raw)) % 64)
    assert lib.cvmk_conv2d_tc_supported(ct.byref(d)) == 1
    assert lib.cvmk_conv2d_tc_prepare(ct.byref(d), ct.byref(plan)) == 0 and plan.a_im2col == 4
    torch.cuda.synchronize()
    assert lib.cvmk_conv2d_tc_launch(ct.byref(plan), ct.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    want = conv_sums(torch, x, wt, 1, 1, c // 32) + bias.long()
    assert int(status) == 0
    assert torch.equal(y, right_shift(want, shift).to(torch.int8))
