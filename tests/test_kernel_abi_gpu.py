"""Launchers of the kernel C-ABI (include/cvmk_kernels.h) called directly, in ways that the executor does not."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RSHIFT, ADD_C = 2, 8


class Step(ct.Structure):
    _fields_ = [("op", ct.c_int32), ("a", ct.c_int32), ("b", ct.c_int32), ("ptr_dtype", ct.c_int32), ("ptr", ct.c_void_p)]


class Epilogue(ct.Structure):
    _fields_ = [("n", ct.c_int32), ("reserved", ct.c_int32), ("s", Step * 8)]


def ints(names):
    return [(n, ct.c_int32) for n in names.split()]


class Direct(ct.Structure):
    _fields_ = ([("x", ct.c_void_p)] + ints("x_dtype narrow_x") + [("w", ct.c_void_p), ("y", ct.c_void_p)] +
                ints("y_dtype N H W C OC KH KW OH OW groups stride_h stride_w pad_h pad_w dil_h dil_w depthwise bias_static") +
                [("acc_bound", ct.c_int64), ("ep", Epilogue), ("status", ct.c_void_p)])


class Stem(ct.Structure):
    _fields_ = ([("x", ct.c_void_p), ("w", ct.c_void_p), ("y", ct.c_void_p)] +
                ints("N H W C OC KH KW OH OW stride_h stride_w pad_h pad_w clamp") +
                [("status", ct.c_void_p), ("acc_bound", ct.c_int64), ("ep", Epilogue)] + ints("x_pitch bias_static"))


class Reduce(ct.Structure):
    _fields_ = (ints("is_max init_zero n_keep n_red") + [(n, ct.c_int64 * 6) for n in ("keep_extent", "keep_stride", "red_extent", "red_stride")] +
                [("x", ct.c_void_p)] + ints("x_dtype pad0") + [("y", ct.c_void_p)] + ints("y_dtype pad1") + [("ep", Epilogue)])


def shift_clip(desc, shift, bias=None):
    steps = ([(ADD_C, 0, 0, 4, bias)] if bias else []) + [(RSHIFT, shift, 8, 0, None)]
    desc.ep.n = len(steps)
    for i, s in enumerate(steps):
        desc.ep.s[i] = Step(*s)


def conv(torch, x, w, bias, shift, stride, pad, groups):
    """int8 NCHW in, int8 NHWC out: the sums in 64 bits, exact, then cvm_right_shift to 8 bits."""
    s = torch.nn.functional.conv2d(x.double(), w.double(), bias.double() if bias is not None else None, stride, pad, 1, groups).long()
    return (((s >> (shift - 1)) + 1) >> 1).clamp(-127, 127).to(torch.int8).permute(0, 2, 3, 1).contiguous()


def int8(torch, rng, *shape):
    return torch.from_numpy(rng.randint(-127, 128, size=shape).astype(np.int8)).cuda()


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
    for name, value in dict(N=n, H=h, W=h, C=c, OC=oc, KH=k, KW=k, OH=oh, OW=oh, stride_h=step, stride_w=step, pad_h=k // 2, pad_w=k // 2).items():
        setattr(d, name, value)
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
    assert torch.equal(y, conv(torch, x, w, bias, shift, step, k // 2, groups))
