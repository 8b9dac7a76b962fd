"""How inputs reach the GPU and results the caller: every path of the executor against the oracle."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def copy_case(wl, n):
    """One operator over n int8 elements: the result is as large as the input."""
    g = wl.GraphBuilder(3)
    d = g.var("data", (1, n), 8)
    y = g.op("clip", [d], (1, n), {"a_min": -100, "a_max": 90})
    js, pb = g.finish(y)
    return js, pb, np.random.RandomState(n).randint(-127, 128, size=(1, n)).astype(np.int8)


# one kernel writes heads of up to 1 MiB, larger ones leave in 1 MiB pieces; inputs above 1 MiB are
# staged by the host threads in 256 KiB pieces
@pytest.mark.parametrize("n", [1, 15, 4099, 300001, 1 << 20, (1 << 20) + 1, (3 << 20) + 77])
@pytest.mark.parametrize("where", ["pageable", "pinned", "device"])
def test_sizes_and_buffers(n, where, rt, wl, oracle):
    import torch
    js, pb, x = copy_case(wl, n)
    want = oracle.run_model(js, pb, x)
    net = rt.CVMAPILoadModel(js, pb, 0)
    try:
        flat = torch.from_numpy(x.reshape(-1).view(np.uint8).copy())
        src = {"pageable": flat, "pinned": flat.pin_memory(), "device": flat.cuda()}[where]
        out = torch.zeros(n, dtype=torch.uint8)
        for dst in (out, torch.zeros(n, dtype=torch.uint8).pin_memory()):
            for _ in range(4):   # (the helpers are awake from the third on)
                dst.zero_()
                rt.check_call(rt.lib().CVMAPIInference(net, ctypes.c_void_p(src.data_ptr()), n, ctypes.c_void_p(dst.data_ptr())))
                assert np.array_equal(dst.numpy(), want.view(np.uint8))
    finally:
        rt.CVMAPIFreeModel(net)


# rows past top_k / max_output_size are not downloaded; the operator's loop ends at an image without
# valid boxes, whose successors keep what their memory held (zeros in a fresh handle)
@pytest.mark.parametrize("empty", [None, 0, 1, 3])
@pytest.mark.parametrize("batch", [4, 9])
@pytest.mark.parametrize("anchors,top_k,mos", [(1001, 100, -1), (1000, 100, 37), (700, 800, 20), (5003, 1, -1)])
def test_nms_head(batch, anchors, top_k, mos, empty, gpu_run, wl, oracle):
    js, pb, x = wl.ssd_tail(batch=batch, anchors=anchors, top_k=top_k, max_output_size=mos)
    if empty is not None:
        x = x.copy()
        x[empty, :, 1] = 3
    got = gpu_run(js, pb, x).view(np.int32).reshape(batch, anchors, 6)
    want = oracle.run_model(js, pb, x).view(np.int32).reshape(batch, anchors, 6)
    last = batch if empty is None else empty + 1
    assert np.array_equal(got[:last], want[:last])


# stems over rows that do not start on 16-byte boundaries (moved apart first), widths beyond one TMA box, and
# batches that are and are not cut into parts while they upload
@pytest.mark.parametrize("width", [17, 31, 48, 100, 191, 224, 250, 301])
@pytest.mark.parametrize("batch", [1, 8, 11])
def test_image_stem(width, batch, rt, wl, oracle):
    import torch
    g = wl.GraphBuilder(width)
    d = g.var("data", (batch, 3, 29, width), 8)
    k = 7 if width % 2 else 3
    y = g.conv(d, 32, k, 2, k // 2)
    y = g.max_pool(y, 3, 2, 1)
    y = g.conv(y, 64, 1, 1, 0)
    y = g.conv(y, 64, 3, 1, 1)
    js, pb = g.finish(y)
    x = np.random.RandomState(width).randint(-128, 128, size=(batch, 3, 29, width)).astype(np.int8)
    want = oracle.run_model(js, pb, x)
    net = rt.CVMAPILoadModel(js, pb, 0)
    try:
        flat = torch.from_numpy(x.reshape(-1).view(np.uint8).copy())
        for src in (flat, flat.pin_memory(), flat.cuda()):
            out = torch.zeros(want.nbytes, dtype=torch.uint8)
            rt.check_call(rt.lib().CVMAPIInference(net, ctypes.c_void_p(src.data_ptr()), flat.numel(), ctypes.c_void_p(out.data_ptr())))
            assert np.array_equal(out.numpy(), want.view(np.uint8))
    finally:
        rt.CVMAPIFreeModel(net)


# graphs that are cut along the batch as a whole: the parts of the head leave while later parts compute;
# widths whose images are and are not whole 16-byte words, a head below and some above the size that leaves in pieces
@pytest.mark.parametrize("batch,channels,size", [(8, 32, 14), (9, 64, 33), (31, 32, 37), (40, 64, 56), (3, 128, 61)])
def test_head_in_parts(batch, channels, size, rt, wl, oracle):
    import torch
    js, pb, x = wl.conv_chain(batch=batch, channels=channels, size=size)
    net = rt.CVMAPILoadModel(js, pb, 0)
    try:
        for turn in range(2):
            x = np.roll(x, 1, axis=0)
            want = oracle.run_model(js, pb, x).view(np.uint8).reshape(-1)
            flat = torch.from_numpy(x.reshape(-1).view(np.uint8).copy())
            for src in (flat, flat.pin_memory(), flat.cuda()):
                for dst in (torch.zeros(want.size, dtype=torch.uint8), torch.zeros(want.size, dtype=torch.uint8).pin_memory()):
                    rt.check_call(rt.lib().CVMAPIInference(net, ctypes.c_void_p(src.data_ptr()), flat.numel(), ctypes.c_void_p(dst.data_ptr())))
                    assert np.array_equal(dst.numpy(), want)
    finally:
        rt.CVMAPIFreeModel(net)


# layers whose parts of the batch would not start on 16 bytes (odd images of 8 or 24 channels) are not cut
@pytest.mark.parametrize("oc", [8, 24, 40])
@pytest.mark.parametrize("batch", [8, 9, 15])
def test_parts_that_do_not_align(oc, batch, gpu_run, wl, oracle):
    g = wl.GraphBuilder(oc)
    d = g.var("data", (batch, 3, 37, 37), 8)
    y = g.conv(d, 32, 3, 2, 1)
    y = g.conv(y, oc, 3, 1, 1)
    y = g.max_pool(y, 3, 2, 1)
    js, pb = g.finish(g.conv(y, oc, 1, 1, 0, relu=False))
    x = np.random.RandomState(batch).randint(-128, 128, size=(batch, 3, 37, 37)).astype(np.int8)
    assert np.array_equal(gpu_run(js, pb, x), oracle.run_model(js, pb, x))
