"""Performance cases of the quantized-inference path, as a user's program drives it.

A pass is what an application does per request: Tensor::CopyDataToTensor, Graph::Run, Tensor::CopyDataFromTensor on host
buffers (the only way data goes in and out of this API), with the graph compiled once beforehand.  Two kinds of graphs:

  kind "net"  a whole network built through the tim::vx C++ API (tim-vx_b200/samples): LeNet-5 with uint8 weights,
              MobileNetV2-1.0 uint8 asymmetric, ResNet-50 v1.5 with per-channel int8 weights
  kind "op"   a graph of one operator family through the C ABI and its Python binding (tim-vx_b200/opworkloads.py):
              fcchain:<rows>:<width>:<layers>, conv:<k>:<cin>:<cout>:<hw>:<stride>, convadd:<same>

"pinned" says whether the caller's host buffers are page-locked (a server that cares) or ordinary memory (the sample
programs, a numpy array).  Runs from the repository's root.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.abspath("tim-vx_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import opworkloads  # noqa: E402
import pyb2vx  # noqa: E402

# per image: operations (2 x multiply-accumulate), input bytes, output bytes; once: weight and bias bytes
_NETS = {
    "lenet": (4.586e6, 28 * 28, 10, 432.8e3),
    "mobilenetv2": (0.6015e9, 224 * 224 * 3, 1000, 3.47e6),
    "resnet50": (8.178e9, 224 * 224 * 3, 1000, 25.5e6),
}
_MAX_BATCH = {"lenet": 1024, "mobilenetv2": 1024, "resnet50": 256}


def _net(name, net, batch, pinned):
    return {"name": name, "kind": "net", "net": net, "batch": batch, "pinned": pinned}


def _op(name, spec, batch, pinned):
    return {"name": name, "kind": "op", "spec": spec, "batch": batch, "pinned": pinned}


def listed():
    return [
        # one digit at a time, as the LeNet sample program does: all launch and copy latency
        _net("lenet_b1", "lenet", 1, False),
        # the benchmark configuration's batch of digits
        _net("lenet_b256", "lenet", 256, False),
        # one camera frame: the latency of an interactive classifier
        _net("mobilenetv2_b1", "mobilenetv2", 1, False),
        # a server's batch
        _net("mobilenetv2_b64", "mobilenetv2", 64, True),
        # offline labelling: the largest batch of the benchmark configurations
        _net("mobilenetv2_b1024", "mobilenetv2", 1024, True),
        # one image through the headline network
        _net("resnet50_b1", "resnet50", 1, False),
        # what a dynamic batcher happens to have collected: a batch that divides nothing
        _net("resnet50_b13", "resnet50", 13, True),
        # the headline configuration
        _net("resnet50_b64", "resnet50", 64, True),
        # decode-like fully-connected layers: one row, twelve layers, every weight read once
        _op("fc_1x4096x12", "fcchain:1:4096:12", 1, False),
        # the same for a handful of concurrent requests on wide layers
        _op("fc_16x8192x4", "fcchain:16:8192:4", 1, False),
        # prefill-like: many rows through a deep stack of fully-connected layers
        _op("fc_2048x4096x8", "fcchain:2048:4096:8", 1, True),
        # the convolution sweep's 3x3 layer as a graph of its own, converters included
        _op("conv3x3_b32", "conv:3:64:64:56:1", 32, True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in known:
            return case


def _draw(rng):
    pinned = rng.random() < 0.6
    what = rng.random()
    if what < 0.5:
        net = rng.choice(sorted(_NETS))
        return {"kind": "net", "net": net, "batch": _log(rng, 2, _MAX_BATCH[net]), "pinned": pinned}
    if what < 0.75:
        m, n, layers = _log(rng, 1, 4096), _log(rng, 128, 8192), _log(rng, 1, 12)
        if rng.random() < 0.5:
            n = max(128, n // 64 * 64)
        while layers > 1 and (n * n * layers > 270e6 or m * n * n * layers > 2.7e11):
            layers -= 1
        m = max(1, min(m, int(2.7e11 / (n * n * layers))))
        return {"kind": "op", "spec": "fcchain:%d:%d:%d" % (m, n, layers), "batch": 1, "pinned": pinned}
    form = rng.choice(["conv", "conv", "convadd"])
    k, stride = rng.choice([1, 3, 3, 5]), rng.choice([1, 1, 2])
    cin, cout, hw = _log(rng, 8, 512), _log(rng, 16, 512), _log(rng, 7, 112)
    if rng.random() < 0.5:
        cin, cout = max(16, cin // 16 * 16), max(16, cout // 16 * 16)
    per_image = hw * hw * (cin + 2 * cout)
    batch = max(1, min(_log(rng, 1, 64), int(40e6 / per_image)))
    return {"kind": "op", "spec": "%s:%d:%d:%d:%d:%d" % (form, k, cin, cout, hw, stride), "batch": batch, "pinned": pinned}


class _Net:
    """A sample network and its host buffers."""

    _lib = None

    @classmethod
    def library(cls):
        if cls._lib is None:
            lib = ctypes.CDLL(os.path.join(_PACKAGE, "samples", "libb2vx_samples.so"))
            vp = ctypes.c_void_p
            for name, res, args in (("create", vp, [ctypes.c_char_p, ctypes.c_int32, ctypes.c_uint64, ctypes.c_int32]),
                                    ("destroy", None, [vp]), ("input_bytes", ctypes.c_size_t, [vp]), ("output_bytes", ctypes.c_size_t, [vp]),
                                    ("synthetic_input", None, [vp, ctypes.c_uint64, vp]), ("set_input", ctypes.c_int32, [vp, vp]),
                                    ("run", ctypes.c_int32, [vp]), ("get_output", ctypes.c_int32, [vp, vp])):
                fn = getattr(lib, "b2vx_net_" + name)
                fn.restype, fn.argtypes = res, args
            cls._lib = lib
        return cls._lib

    def __init__(self, net, batch, seed, pinned):
        self.lib, self.net = self.library(), None
        self.net = self.lib.b2vx_net_create(net.encode(), batch, seed, 0)
        if not self.net:
            raise RuntimeError("cannot build %s at batch %d" % (net, batch))
        self.x = torch.empty(self.lib.b2vx_net_input_bytes(self.net), dtype=torch.uint8, pin_memory=pinned)
        self.y = torch.empty(self.lib.b2vx_net_output_bytes(self.net), dtype=torch.uint8, pin_memory=pinned)
        self.px, self.py = self.x.data_ptr(), self.y.data_ptr()
        self.lib.b2vx_net_synthetic_input(self.net, seed, self.px)

    def __del__(self):
        if self.net:
            self.lib.b2vx_net_destroy(self.net)

    def run(self):
        lib, net = self.lib, self.net
        if lib.b2vx_net_set_input(net, self.px) or lib.b2vx_net_run(net) or lib.b2vx_net_get_output(net, self.py):
            raise RuntimeError("the pass failed")
        return self.y


class _Op:
    """A compiled operator graph; host data as numpy arrays, or page-locked buffers handed over by address."""

    def __init__(self, spec, batch, seed, pinned):
        self.g = pyb2vx.Graph(pyb2vx.load(pyb2vx.PRODUCT_LIB), 0)
        work = opworkloads.build(spec, batch, self.g, np.random.default_rng(seed))
        self.g.compile()
        self.inputs, self.outputs, self.pinned = work["inputs"], work["outputs"], pinned
        if pinned:
            self.keep = [torch.from_numpy(a).pin_memory() for _, a in self.inputs]
            self.out = [torch.empty(self.g.shape(t)[::-1], dtype=torch.uint8, pin_memory=True) for t in self.outputs]
            self.px = [(t, b.data_ptr(), b.numel()) for (t, _), b in zip(self.inputs, self.keep)]
            self.py = [(t, b.data_ptr(), b.numel()) for t, b in zip(self.outputs, self.out)]

    def run(self):
        g = self.g
        if self.pinned:
            for t, p, n in self.px:
                g.write_ptr(t, p, n)
            g.run()
            for t, p, n in self.py:
                g.read_ptr(t, p, n)
            return self.out
        for t, a in self.inputs:
            g.write(t, a)
        g.run()
        return [g.read(t) for t in self.outputs]


def prepare(case, seed):
    if case["kind"] == "net":
        return _Net(case["net"], case["batch"], seed, case["pinned"])
    return _Op(case["spec"], case["batch"], seed, case["pinned"])


def run(state):
    return state.run()


def work(case):
    n = case["batch"]
    if case["kind"] == "net":
        ops, x, y, w = _NETS[case["net"]]
        return {"bytes": n * (x + y) + w, "flops": n * ops}
    kind, v = opworkloads.parse(case["spec"])
    if kind == "fcchain":
        m, width, layers = v
        return {"bytes": 2 * m * width + layers * (width * width + 8 * width), "flops": 2.0 * m * width * width * layers}
    k, cin, cout, hw, stride = v
    ho = (hw + stride - 1) // stride
    outs = n * ho * ho * cout
    return {"bytes": n * hw * hw * cin + outs * (2 if kind == "convadd" else 1) + k * k * cin * cout + 8 * cout,
            "flops": 2.0 * outs * cin * k * k}


def tolerance(case):
    # quantized outputs: the rounding of every value is fixed by the reference's float sequence
    return "exact"
