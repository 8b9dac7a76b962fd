"""Descriptors of the kernel C-ABI (include/cvmk_kernels.h) for tests that call its launchers directly, and exact results."""
import ctypes as ct

import numpy as np

I8, I32 = 1, 4
RSHIFT, CLIP, ADD_T, ADD_C = 2, 4, 5, 8


class Step(ct.Structure):
    _fields_ = [("op", ct.c_int32), ("a", ct.c_int32), ("b", ct.c_int32), ("ptr_dtype", ct.c_int32), ("ptr", ct.c_void_p)]


class Epilogue(ct.Structure):
    _fields_ = [("n", ct.c_int32), ("reserved", ct.c_int32), ("s", Step * 8)]


def ints(names):
    return [(n, ct.c_int32) for n in names.split()]


class Conv(ct.Structure):
    _fields_ = ([("x", ct.c_void_p), ("w", ct.c_void_p), ("y", ct.c_void_p)] +
                ints("y_dtype N H W C OC KH KW OH OW stride_h stride_w pad_h pad_w dil_h dil_w") +
                [("status", ct.c_void_p), ("acc_bound", ct.c_int64)] + ints("bias_static groups group_fold reserved1") +
                [("workspace", ct.c_void_p), ("workspace_bytes", ct.c_int64), ("ep", Epilogue)])


class ConvPlan(ct.Structure):
    _fields_ = ([(n, ct.c_uint8 * 128) for n in ("tmap_a", "tmap_b", "tmap_y", "tmap_r")] + [("d", Conv)] +
                ints("block_k block_n a_im2col stages grid smem_bytes tma_out res_step panels panel_bytes io_bufs ring_bytes "
                     "patch_w patch_h patch_n units small_swap b_resident small_split"))


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


def chain(desc, steps):
    desc.ep.n = len(steps)
    for i, s in enumerate(steps):
        desc.ep.s[i] = Step(*s)


def shape(desc, n, c, h, w, oc, k, stride, pad):
    oh, ow = (h + 2 * pad - k) // stride + 1, (w + 2 * pad - k) // stride + 1
    for name, value in dict(N=n, H=h, W=w, C=c, OC=oc, KH=k, KW=k, OH=oh, OW=ow, stride_h=stride, stride_w=stride, pad_h=pad, pad_w=pad).items():
        setattr(desc, name, value)
    return oh, ow


def int8(torch, rng, *shape):
    return torch.from_numpy(rng.randint(-127, 128, size=shape).astype(np.int8)).cuda()


def right_shift(s, shift):
    """cvm_right_shift to 8 bits of whole numbers."""
    return (((s >> (shift - 1)) + 1) >> 1).clamp(-127, 127)


def conv_sums(torch, x, w, stride, pad, groups=1):
    """int8 NCHW in: the sums as whole numbers, NHWC (products and sums in float64 are exact far beyond them)."""
    s = torch.nn.functional.conv2d(x.double(), w.double(), None, stride, pad, 1, groups)
    return s.round().long().permute(0, 2, 3, 1).contiguous()


def run_conv(rt, n, c, h, w, oc, k, stride, packed, join=False, seed=0):
    """One cvmk_conv2d_tc_* layer of random data with bias, shift and clamp, and an int8 tensor added and the result clamped again where
    `join`: its plan.  Asserts that every output byte is right.  `packed`: with the bound that lets the kernel requantise 16 bits at a time."""
    import torch
    lib, rng = rt.lib(), np.random.RandomState(seed)
    x, wt = int8(torch, rng, n, c, h, w), int8(torch, rng, oc, c, k, k)
    bias = torch.from_numpy(rng.randint(-5000, 5000, size=oc).astype(np.int32)).cuda()
    d = Conv()
    oh, ow = shape(d, n, c, h, w, oc, k, stride, k // 2)
    d.dil_h = d.dil_w = d.groups = 1
    xin, wk = x.permute(0, 2, 3, 1).contiguous(), wt.permute(0, 2, 3, 1).contiguous()
    y, r = torch.zeros(n, oh, ow, oc, dtype=torch.int8, device="cuda"), int8(torch, rng, n, oh, ow, oc)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    d.x, d.w, d.y, d.y_dtype, d.status = xin.data_ptr(), wk.data_ptr(), y.data_ptr(), I8, status.data_ptr()
    shift = 7 + int(np.ceil(np.log2(np.sqrt(c) * k)))
    d.acc_bound = c * k * k * 127 * 127 + 5000 if packed else 0
    chain(d, [(ADD_C, 0, 0, I32, bias.data_ptr()), (RSHIFT, shift, 8, 0, None)] +
          ([(ADD_T, 0, 0, I8, r.data_ptr()), (CLIP, -127, 127, 0, None)] if join else []))
    raw = ct.create_string_buffer(4096)
    plan = ConvPlan.from_buffer(raw, (-ct.addressof(raw)) % 64)
    assert lib.cvmk_conv2d_tc_prepare(ct.byref(d), ct.byref(plan)) == 0
    torch.cuda.synchronize()
    assert lib.cvmk_conv2d_tc_launch(ct.byref(plan), ct.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    want = right_shift(conv_sums(torch, x, wt, stride, k // 2) + bias.long(), shift)
    if join:
        want = (want + r.long()).clamp(-127, 127)
    assert int(status) == 0
    assert torch.equal(y, want.to(torch.int8))
    return plan
