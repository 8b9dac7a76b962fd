"""The calls whose speed matters to a user of this runtime, as cases that can be timed and compared.

A user loads a quantised model once (CVMAPILoadModel) and then calls CVMAPIInference on one batch
after the other.  A case is such a call: a model, its sizes, and where the caller's input lies.  The
models are the benchmark and parity configurations of workloads.py (seeded synthetic weights); the
network input is drawn from the case's seed.

Where the input lies:
  pageable   an ordinary buffer: what the Go and Python callers of the C-ABI pass
  pinned     page-locked host memory: a server that keeps its input buffers
  device     GPU memory: a caller whose pre-processing runs on the same GPU
The output always goes to a buffer of the caller's in host memory, as the C-ABI has it.
"""
import ctypes
import functools
import importlib
import json
import math
import weakref

import numpy as np
import torch

_pkg = importlib.import_module("cvm-runtime_b200")
_rt, _wl = _pkg.runtime, _pkg.workloads


def listed():
    return [
        # One operator chain on one image: the smallest call, all latency and launches.
        {"name": "conv_chain_b1", "model": "conv_chain", "batch": 1, "channels": 64, "size": 56, "input": "pageable"},
        # The same chain on a batch: the plain convolution rate.
        {"name": "conv_chain_b64", "model": "conv_chain", "batch": 64, "channels": 64, "size": 56, "input": "device"},
        # One image through a classifier: what a node that verifies one inference waits for.
        {"name": "resnet50_b1", "model": "resnet50", "batch": 1, "size": 224, "input": "pageable"},
        {"name": "vgg19_b1", "model": "vgg19", "batch": 1, "size": 224, "input": "pageable"},
        # A few images of an odd size: ragged rows, partial tiles, a batch that does not divide.
        {"name": "mobilenet_b5_s191", "model": "mobilenet_v1", "batch": 5, "size": 191, "input": "pageable"},
        # Middling batches of a server that fills them as requests come.
        {"name": "resnet50_b13_s197", "model": "resnet50", "batch": 13, "size": 197, "input": "pinned"},
        {"name": "resnet50_b64", "model": "resnet50", "batch": 64, "size": 224, "input": "device"},
        # Throughput: the largest batches, one GPU's share of them for the largest network.
        {"name": "resnet50_b256", "model": "resnet50", "batch": 256, "size": 224, "input": "pinned"},
        {"name": "mobilenet_b256", "model": "mobilenet_v1", "batch": 256, "size": 224, "input": "pinned"},
        {"name": "vgg19_b32", "model": "vgg19", "batch": 32, "size": 224, "input": "pageable"},
        # Detection: image to boxes in one graph, and the post-processing of a whole batch on its own.
        {"name": "ssd_full_b8_s512", "model": "ssd_full", "batch": 8, "size": 512, "input": "pageable", "top_k": 100},
        {"name": "ssd_tail_b64", "model": "ssd_tail", "batch": 64, "anchors": 24564, "top_k": 400, "force": False, "input": "pageable"},
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, evenly spread over its logarithm."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    model = rng.choice(["conv_chain", "resnet50", "resnet50", "mobilenet_v1", "mobilenet_v1", "vgg19", "ssd_full", "ssd_tail"])
    c = {"model": model, "input": rng.choice(["pageable", "pinned", "device"])}
    if model == "conv_chain":
        c.update(batch=_log(rng, 1, 128), channels=rng.choice([32, 64, 128]), size=rng.randint(14, 64))
        c["batch"] = min(c["batch"], (24 << 20) // (c["channels"] * c["size"] ** 2))
    elif model == "ssd_tail":
        c.update(batch=_log(rng, 1, 64), anchors=_log(rng, 1000, 24564), top_k=rng.choice([100, 200, 400, 800]),
                 force=rng.random() < 0.25)
    else:
        # the largest batch keeps a drawn case within the pixels of the largest listed one
        lo, hi, most, at = {"resnet50": (96, 288, 256, 224), "mobilenet_v1": (96, 288, 256, 224),
                            "vgg19": (64, 224, 32, 224), "ssd_full": (128, 512, 8, 512)}[model]
        c["size"] = 224 if lo <= 224 <= hi and rng.random() < 0.4 else rng.randint(lo, hi)
        c["batch"] = min(_log(rng, 1, most), most * at * at // c["size"] ** 2)
        if model == "ssd_full":
            c["top_k"] = rng.choice([100, 400])
    return c


def _key(case):
    return json.dumps({k: v for k, v in case.items() if k not in ("name", "input")}, sort_keys=True)


@functools.lru_cache(maxsize=2)
def _built(key):
    """(graph JSON, params blob, bytes of the parameters) of a case's model."""
    c = json.loads(key)
    if c["model"] == "conv_chain":
        js, pb, _ = _wl.conv_chain(batch=c["batch"], channels=c["channels"], size=c["size"])
    elif c["model"] == "ssd_tail":
        js, pb, _ = _wl.ssd_tail(batch=c["batch"], anchors=c["anchors"], top_k=c["top_k"], force_suppress=c["force"])
    elif c["model"] == "ssd_full":
        js, pb, _ = _wl.ssd_full(batch=c["batch"], size=c["size"], top_k=c["top_k"])
    else:
        js, pb, _ = getattr(_wl, c["model"])(batch=c["batch"], size=c["size"])
    return js, pb, len(pb)


class _Model:
    """A loaded model, freed with its last user."""

    def __init__(self, key):
        js, pb, _ = _built(key)
        self.net = _rt.CVMAPILoadModel(js, pb, 0)

    def __del__(self):
        if getattr(self, "net", None):
            _rt.CVMAPIFreeModel(self.net)


_loaded = weakref.WeakValueDictionary()  # a program loads a model once, whatever inputs it then runs


def _model(case):
    key = _key(case)
    m = _loaded.get(key)
    if m is None:
        m = _loaded[key] = _Model(key)
    return m


def _input(case, seed):
    rng = np.random.RandomState(seed % (1 << 32))
    b = case["batch"]
    if case["model"] == "ssd_tail":
        return _wl.ssd_boxes(b, case["anchors"], seed % (1 << 32))
    c = case["channels"] if case["model"] == "conv_chain" else 3
    raw = np.frombuffer(rng.bytes(b * c * case["size"] ** 2), np.int8)  # uniform in [-127, 127]
    return np.maximum(raw, np.int8(-127)).reshape(b, c, case["size"], case["size"])


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.model = _model(case)
    s.x = np.ascontiguousarray(_input(case, seed))
    s.nbytes, s.device = s.x.nbytes, None
    if case["input"] != "pageable":
        flat = torch.from_numpy(s.x.reshape(-1).view(np.uint8))
        if case["input"] == "device":
            s.device, s.x = flat.cuda(), None
        else:
            s.pinned = torch.empty(flat.numel(), dtype=torch.uint8, pin_memory=True)
            s.pinned.copy_(flat)
            s.x = s.pinned.numpy()
    s.out = np.zeros(_rt.CVMAPIGetOutputLength(s.model.net), np.uint8)
    s.wide = _rt.CVMAPIGetOutputTypeSize(s.model.net) == 4
    return s


def run(s):
    if s.device is None:
        _rt.inference_bytes(s.model.net, s.x, s.out)
    else:
        _rt.check_call(_rt.lib().CVMAPIInference(s.model.net, ctypes.c_void_p(s.device.data_ptr()), ctypes.c_int(s.nbytes),
                                                 s.out.ctypes.data_as(ctypes.c_char_p)), "CVMAPIInference")
    return s.out.view(np.int32 if s.wide else np.int8)


def work(case):
    """Input, parameters and output once each; two operations for each multiply-add of a convolution."""
    js, _, params = _built(_key(case))
    g = json.loads(js)
    b = case["batch"]
    if case["model"] == "ssd_tail":
        n = b * case["anchors"] * 24
        return {"bytes": 2 * n, "flops": 0}
    out_eid = g["node_row_ptr"][g["heads"][0][0]] + g["heads"][0][1]
    out = int(np.prod(g["attrs"]["shape"][1][out_eid])) * (1 if case["model"] == "conv_chain" else 4)
    c = case["channels"] if case["model"] == "conv_chain" else 3
    return {"bytes": b * c * case["size"] ** 2 + params + out, "flops": b * _wl.conv_ops_per_image(js)}


def tolerance(case):
    return "exact"  # every operator works on whole numbers
