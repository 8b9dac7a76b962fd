"""The executor's host logic on a device made of host memory (tests/executor_host/fake_device.cc): what
happens to the caller's buffers, to queued transfers and to memory when a call fails on the way.

The host sources of the library are compiled against the fake with the address sanitizer, so that a helper
or a queued copy that touches memory that is gone ends the program.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = os.path.join(HERE, "executor_host")
OUT = os.path.join(SRC, "build")
BIN = os.path.join(OUT, "executor_host")
HOST = os.path.join(ROOT, "cvm-runtime_b200", "csrc", "host")
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    srcs = [os.path.join(HOST, f) for f in ("ops.cc", "graph.cc", "host_pool.cc", "executor.cc", "c_api.cc")]
    srcs += [os.path.join(SRC, f) for f in ("fake_device.cc", "main.cc")]
    inc = os.path.join(ROOT, "include")
    headers = [os.path.join(d, f) for d in (HOST, SRC, inc, os.path.join(inc, "cvm")) for f in os.listdir(d) if f.endswith(".h")]
    newest = max(os.path.getmtime(h) for h in headers)
    os.makedirs(OUT, exist_ok=True)
    objs, procs = [], []
    flags = ["-std=c++17", "-O0", "-g1", "-fsanitize=address", "-pthread", "-I" + CUDA, "-I" + inc, "-I" + HOST]
    for s in srcs:
        o = os.path.join(OUT, os.path.basename(s) + ".o")
        objs.append(o)
        if not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), newest):
            procs.append(subprocess.Popen(["g++"] + flags + ["-c", s, "-o", o]))
    assert all(p.wait() == 0 for p in procs)
    if procs or not os.path.exists(BIN):
        subprocess.check_call(["g++", "-fsanitize=address", "-pthread"] + objs + ["-o", BIN])

    pool = os.path.join(OUT, "pool")
    if procs or not os.path.exists(pool) or os.path.getmtime(pool) < os.path.getmtime(os.path.join(SRC, "pool.cc")):
        subprocess.check_call(["g++"] + flags + [os.path.join(SRC, "pool.cc"), os.path.join(OUT, "host_pool.cc.o"), "-o", pool, "-ldl"])

    def run(work, *args, slow_images=0, binary=BIN):
        env = dict(os.environ, SLOW_IMAGES=str(slow_images), ASAN_OPTIONS="detect_leaks=0:alloc_dealloc_mismatch=0")
        p = subprocess.run([os.path.join(OUT, binary)] + [str(a) for a in args], cwd=work, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True,
                           env=env, timeout=60)
        assert p.returncode == 0, p.stderr[-4000:]
        return dict(tok[1:].split("=", 1) for tok in p.stdout.split() if tok.startswith("@"))
    return run


def put(path, js, pb, x):
    for name, data in (("graph.json", js.encode() if isinstance(js, str) else js), ("params.bin", pb), ("input.bin", x.tobytes())):
        with open(os.path.join(path, name), "wb") as f:
            f.write(data)


def chain(wl, batch):   # on the fake device the result is the input; 2 MiB at batch 8: staged, cut into parts, leaves in pieces
    return wl.conv_chain(batch=batch, channels=64, size=64)


@pytest.mark.parametrize("when", ["late", "early"])
@pytest.mark.parametrize("src,dst", [("pageable", "pageable"), ("pinned", "pinned"), ("pageable", "pinned"), ("pinned", "pageable")])
@pytest.mark.parametrize("batch", [1, 8])
def test_a_failing_call_leaves_no_transfer_behind(when, src, dst, batch, host, wl, tmp_path):
    js, pb, x = chain(wl, batch)
    put(tmp_path, js, pb, x)
    f = host(tmp_path, "fail_run", when, src, dst, slow_images=8)   # (batch 8: runs in parts)
    assert int(f["failed"]) > 0 and f["last_status"] == "0"
    assert f["in_flight"] == "0"      # nothing queued that reads the input or writes the output
    assert f["wrong_after"] == "0"    # the handle answers the next call
    assert np.array_equal(np.fromfile(tmp_path / "output.bin", np.int8), x.reshape(-1))


# The caller's input and output may overlap, as with the reference, which copies the input before it computes:
# nothing is written there before the whole input is on the device.
@pytest.mark.parametrize("when", ["late", "early"])
@pytest.mark.parametrize("src", ["pageable", "pinned"])
@pytest.mark.parametrize("ahead", [0, 300000])
def test_output_over_the_input(when, src, ahead, host, wl, tmp_path):
    js, pb, x = chain(wl, 9)
    put(tmp_path, js, pb, x)
    assert host(tmp_path, "in_place", when, src, ahead, slow_images=9)["status"] == "0"
    assert np.array_equal(np.fromfile(tmp_path / "output.bin", np.int8), x.reshape(-1))
    js, pb, x = wl.ssd_tail(batch=9, anchors=1500, top_k=100)
    put(tmp_path, js, pb, x)
    assert host(tmp_path, "in_place", when, src, ahead)["status"] == "0"
    want = np.full(x.shape, -1, np.int32)
    want[:, :100] = x[:, -100:]   # (what the fake device's operators do)
    assert np.array_equal(np.fromfile(tmp_path / "output.bin", np.int32), want.reshape(-1))


# a copy between the device and memory that is page-locked in part is refused by the driver; such buffers go the way
# of pageable ones
@pytest.mark.parametrize("src,dst", [("half", "pageable"), ("pageable", "half"), ("half", "half")])
def test_buffers_that_are_page_locked_in_part(src, dst, host, wl, tmp_path):
    js, pb, x = chain(wl, 9)
    put(tmp_path, js, pb, x)
    assert host(tmp_path, "half", "early", src, dst, slow_images=9)["status"] == "0"
    assert np.array_equal(np.fromfile(tmp_path / "output.bin", np.int8), x.reshape(-1))


@pytest.mark.parametrize("when", ["late", "early"])
def test_a_failing_load_gives_everything_back(when, host, wl, tmp_path):
    put(tmp_path, *wl.conv_chain(batch=8, channels=64, size=48))   # (1.2 MB: timed from pageable memory too)
    f = host(tmp_path, "fail_load", when, "-", "-")
    assert int(f["failed"]) > 100
    assert f["left"] == "0" and f["odd"] == "0"


def test_the_memory_a_model_holds_is_enough_to_load_it(host, wl, tmp_path):
    put(tmp_path, *wl.mobilenet_v1(batch=16, size=96))
    f = host(tmp_path, "tight", "early", "-", "-")
    assert int(f["sizes"]) > 0 and f["refused"] == "0" and f["left"] == "0"


# plans for the parts of the batch are made for the (at most fourteen) leading steps that run in parts, not for every
# layer of the network: 53 convolutions, and nine parts of no more than thirteen of them
def test_parts_are_prepared_for_the_steps_that_run_in_parts(host, wl, tmp_path):
    put(tmp_path, *wl.resnet50(batch=8, size=64))
    f = host(tmp_path, "plans", "early", "-", "-", slow_images=8)
    assert f["status"] == "0" and 53 <= int(f["plans"]) <= 53 + 13 * 9
    # ... and the handle says what it chose: steps and parts for each place an input can lie in
    steps, parts = map(int, f["pinned"].split(":"))
    assert 0 < steps <= 14 and parts in (2, 4, 5)
    assert f["device"] == "0:1" and f["short"] == "2"


# handles of one GPU share its helpers; one handle starts and ends them each time, several come and go beside one
# that stays
@pytest.mark.parametrize("handles", [1, 2, 5])
def test_handles_share_the_helpers_of_a_device(handles, host, tmp_path):
    f = host(tmp_path, "share", handles, binary="pool")
    assert f["wrong"] == "0" and f["left"] == "0"
    assert 1 <= int(f["helpers"]) <= 5


def test_callers_do_without_helpers(host, tmp_path):
    f = host(tmp_path, "none", binary="pool")
    assert f["wrong"] == "0" and f["threads"] == "1"
