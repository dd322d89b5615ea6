"""The work that a user of this library has it do, as cases that can be timed.

A case is a dict of plain values; `kind` names the entry point.  Everything goes through the C ABI
(include/mdc_gpu_ops.h) with device pointers on a stream of the runtime's own, except for `graph`,
which is a lowered graph module called with host memref descriptors the way multi-device-gpu-runner
calls it.  Matrix shapes are those of the library's benchmark and of the reference's End2End tests,
or generic ones of the same range.
"""
import ctypes
import importlib
import math
import os

import numpy as np
import torch

mdc = importlib.import_module("multi-device-model-compiler_b200")

F16, BF16 = mdc.F16, mdc.BF16
RELU, GELU = mdc.ACT_RELU, mdc.ACT_GELU_ERF
EPS = 1e-5


def listed():
    return [
        # One ONNX Add node on the tensors of the reference's example, a batch of four.
        {"name": "add-images", "kind": "add", "n": 4 * 3 * 640 * 640},
        # LayerNorm over the hidden dimension, fp32 with affine parameters, 32 sequences of 512.
        {"name": "layernorm-32x512x768", "kind": "layernorm", "rows": 32 * 512, "cols": 768},
        # ONNX Gemm / torch.nn.Linear through the reference's fp32 entry point: a batch of tokens ...
        {"name": "linear-2048x4096x4096", "kind": "linear", "m": 2048, "n": 4096, "k": 4096},
        # ... and the classifier at the end of a network, a few rows and an odd width.
        {"name": "linear-16x1000x2048", "kind": "linear", "m": 16, "n": 1000, "k": 2048},
        # First layer of an image network (the layer of test/End2End/GPU/conv.mlir): three channels
        # in, output much larger than input.
        {"name": "conv-image", "kind": "conv", "batch": 16, "ic": 3, "h": 256, "w": 256, "oc": 64, "kernel": 3,
         "stride": 1, "pad": 1, "dilation": 1, "post_add": False, "relu": False},
        # Second convolution of a residual block: residual add and ReLU ride in the call.
        {"name": "conv-residual", "kind": "conv", "batch": 32, "ic": 64, "h": 56, "w": 56, "oc": 64, "kernel": 3,
         "stride": 1, "pad": 1, "dilation": 1, "post_add": True, "relu": True},
        # The pooling layer of test/End2End/GPU/pool.mlir.
        {"name": "pool-image", "kind": "pool", "planes": 128 * 3, "h": 256, "w": 256, "kernel": 4, "stride": 4,
         "pad": 0, "average": False},
        # The reference's own transformer entry point with its own head geometry (8 x 128), pre-LN,
        # causal, ReLU; fp32 weights come with every call.
        {"name": "context-layer-8x256", "kind": "context_layer", "batch": 8, "seq": 256, "heads": 8, "head_dim": 128,
         "ffn": 4096, "norm_first": True, "causal": True, "relu": True},
        # One post-LN encoder layer with padded sequences (valid lengths uniform in half .. full).
        {"name": "encoder-layer-padded", "kind": "stack", "layers": 1, "batch": 32, "seq": 384, "heads": 12,
         "head_dim": 64, "ffn": 3072, "norm_first": False, "causal": False, "gelu": True, "dtype": "f16", "padded": True},
        # The benchmark's workload: throughput of a 12-layer encoder at a large batch.
        {"name": "encoder-12-layers-256x128", "kind": "stack", "layers": 12, "batch": 256, "seq": 128, "heads": 12,
         "head_dim": 64, "ffn": 3072, "norm_first": False, "causal": False, "gelu": True, "dtype": "f16", "padded": False},
        # Prefill of a single prompt of odd length, bf16, pre-LN, causal: latency.
        {"name": "decoder-12-layers-1x99", "kind": "stack", "layers": 12, "batch": 1, "seq": 99, "heads": 12,
         "head_dim": 64, "ffn": 3072, "norm_first": True, "causal": True, "gelu": True, "dtype": "bf16", "padded": False},
        # A compiled model (encoder layer, weights inside the module) called on pageable host
        # tensors: upload, layer, download, result allocated by the callee.
        {"name": "graph-encoder-32x128", "kind": "graph", "batch": 32, "seq": 128},
    ]


# How often draw() gives each kind: the shares of the listed cases.
_KINDS = ["add", "layernorm", "linear", "linear", "conv", "conv", "pool", "context_layer", "stack", "stack", "stack", "graph"]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, step):
    """A size from lo to hi: usually a multiple of `step`, otherwise any."""
    v = _log(rng, lo, hi)
    return min(hi, max(step, v // step * step)) if rng.random() < 0.7 else v


def draw(rng):
    kind = rng.choice(_KINDS)
    if kind == "add":
        return {"kind": kind, "n": _log(rng, 4_000_000, 100_000_000)}
    if kind == "layernorm":
        cols = _size(rng, 128, 4096, 64)
        return {"kind": kind, "rows": max(min(_log(rng, 2048, 131072), 100_000_000 // cols), 5_000_000 // cols), "cols": cols}
    if kind == "linear":
        return {"kind": kind, "m": _size(rng, 1, 4096, 16), "n": _size(rng, 256, 4096, 64), "k": _size(rng, 256, 4096, 64)}
    if kind == "conv":
        while True:
            ic = 3 if rng.random() < 0.3 else _size(rng, 16, 512, 32)
            h = _log(rng, 7, 256)
            w = max(7, min(256, int(h * rng.uniform(0.6, 1.7))))
            c = {"kind": kind, "batch": _log(rng, 1, 64), "ic": ic, "h": h, "w": w,
                 "oc": _size(rng, 16, 512, 32), "kernel": rng.choice([1, 3, 3, 3, 5, 7]), "stride": rng.choice([1, 1, 2]),
                 "dilation": rng.choice([1, 1, 1, 2])}
            c["pad"] = c["dilation"] * (c["kernel"] - 1) // 2
            c["post_add"], c["relu"] = rng.random() < 0.4, rng.random() < 0.6
            if _conv_out(c)[0] >= 1 and work(c)["bytes"] <= 4e8 and work(c)["flops"] <= 4e10:
                return c
    if kind == "pool":
        kernel = rng.choice([2, 3, 4])
        stride = rng.choice([2, kernel])
        h = _log(rng, 56, 256)
        return {"kind": kind, "planes": _log(rng, 256, 4096) * 56 // h + 128, "h": h, "w": int(h * rng.uniform(0.7, 1.4)), "kernel": kernel,
                "stride": stride, "pad": rng.choice([0, kernel // 2]) if kernel == 3 else 0, "average": rng.random() < 0.4}
    if kind == "context_layer":
        head_dim = rng.choice([64, 128])
        d = rng.choice([512, 768, 1024])
        seq = _log(rng, 32, 512)
        return {"kind": kind, "batch": min(_log(rng, 1, 16), max(1, 4096 // seq)), "seq": seq, "heads": d // head_dim,
                "head_dim": head_dim, "ffn": rng.choice([2, 4]) * d, "norm_first": rng.random() < 0.7,
                "causal": rng.random() < 0.7, "relu": rng.random() < 0.7}
    if kind == "stack":
        padded = rng.random() < 0.35
        seq = _log(rng, 16, 512)
        batch = max(1, min(48 if padded else 256, _log(rng, 32, 32768) // seq))
        heads, head_dim = rng.choice([(12, 64), (12, 64), (16, 64), (8, 128)])
        d = heads * head_dim
        return {"kind": kind, "layers": rng.choice([1, 2, 6, 12]) if d == 768 else rng.choice([1, 2, 4]), "batch": batch,
                "seq": seq, "heads": heads, "head_dim": head_dim, "ffn": 4 * d, "norm_first": rng.random() < 0.5,
                "causal": rng.random() < 0.4, "gelu": rng.random() < 0.7, "dtype": rng.choice(["f16", "bf16"]), "padded": padded}
    seq = _log(rng, 32, 384)
    return {"kind": "graph", "batch": max(1, min(32, 9000 // seq, _log(rng, 1, 32))), "seq": seq}


# ------------------------------------------------------------------ state
class _State:
    """Buffers (torch tensors), the stream and the handle of one prepared case."""

    def __init__(self, case):
        mdc.init(0)
        self.case = case
        self.ops = mdc.ops()
        self.stream = _stream()
        self.stack = None
        self.result = None
        self.call = None

    def __del__(self):
        if self.stack:
            self.ops.mgpuEncoderStackDestroy(self.stack)
        if self.result:
            _libc.free(self.result)


_streams = []


def _stream():
    """The one stream that the program works on."""
    if not _streams:
        _streams.append(mdc.runtime().mgpuStreamCreate())
    return _streams[0]


_libc = ctypes.CDLL(None)
_libc.free.argtypes = [ctypes.c_void_p]


def _conv_out(c):
    def out(n):
        return (n + 2 * c["pad"] - c["dilation"] * (c["kernel"] - 1) - 1) // c["stride"] + 1
    return (out(c["h"]), out(c["w"])) if min(out(c["h"]), out(c["w"])) >= 1 else (0, 0)


def _pool_out(c):
    return [(c[n] + 2 * c["pad"] - c["kernel"]) // c["stride"] + 1 for n in ("h", "w")]


def _lengths(case):
    """Valid lengths spread over half .. full; the same for every seed, so that outputs have one shape."""
    rng = np.random.default_rng(case["batch"] * 1000 + case["seq"])
    lens = rng.integers(max(1, case["seq"] // 2), case["seq"] + 1, case["batch"])
    return torch.tensor(lens, device="cuda", dtype=torch.int32)


class MemRef3(ctypes.Structure):
    _fields_ = [("allocated", ctypes.c_void_p), ("aligned", ctypes.c_void_p), ("offset", ctypes.c_ssize_t),
                ("sizes", ctypes.c_ssize_t * 3), ("strides", ctypes.c_ssize_t * 3)]


class MemRef1(ctypes.Structure):
    _fields_ = [("allocated", ctypes.c_void_p), ("aligned", ctypes.c_void_p), ("offset", ctypes.c_ssize_t),
                ("sizes", ctypes.c_ssize_t * 1), ("strides", ctypes.c_ssize_t * 1)]


def _encoder_graph():
    path = os.path.join(mdc.LIB_DIR, "graph_encoder.so")
    fn = ctypes.CDLL(path)._mlir_ciface_main_graph
    fn.argtypes = [ctypes.c_void_p] * 3
    fn.restype = None
    return fn


def prepare(case, seed):
    s = _State(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)

    def normal(*shape, std=1.0, mean=0.0):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32).mul_(std).add_(mean)

    def empty(*shape):
        return torch.zeros(*shape, device="cuda", dtype=torch.float32)

    kind = case["kind"]
    if kind == "add":
        s.a = torch.rand(case["n"], generator=gen, device="cuda").mul_(2).sub_(1)
        s.b = torch.rand(case["n"], generator=gen, device="cuda").mul_(2).sub_(1)
        s.out = empty(case["n"])
        s.args = (s.a.data_ptr(), s.b.data_ptr(), s.out.data_ptr(), case["n"], s.stream)
        s.call = s.ops.mgpuAdd
    elif kind == "layernorm":
        s.x = normal(case["rows"], case["cols"])
        s.gamma, s.beta = normal(case["cols"], std=0.1, mean=1.0), normal(case["cols"], std=0.1)
        s.out = empty(case["rows"], case["cols"])
        s.args = (s.x.data_ptr(), s.gamma.data_ptr(), s.beta.data_ptr(), s.out.data_ptr(), EPS, case["rows"], case["cols"], s.stream)
        s.call = s.ops.mgpuLayerNormF32
    elif kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        s.x, s.w, s.bias = normal(m, k), normal(k, n, std=0.02), normal(n, std=0.02)
        s.out = empty(m, n)
        s.args = (s.x.data_ptr(), s.w.data_ptr(), s.bias.data_ptr(), s.out.data_ptr(), m, n, k, s.stream)
        s.call = s.ops.mgpuMatmul
    elif kind == "conv":
        oh, ow = _conv_out(case)
        k, p = case["kernel"], case["pad"]
        s.x = normal(case["batch"], case["ic"], case["h"], case["w"])
        s.w = normal(case["oc"], case["ic"], k, k, std=math.sqrt(2.0 / (case["ic"] * k * k)))
        s.bias = normal(case["oc"], std=0.1)
        s.out = empty(case["batch"], case["oc"], oh, ow)
        s.add = normal(case["batch"], case["oc"], oh, ow) if case["post_add"] else None
        s.args = (s.x.data_ptr(), s.w.data_ptr(), s.bias.data_ptr(), s.out.data_ptr(), s.add.data_ptr() if case["post_add"] else None,
                  case["batch"], case["ic"], case["h"], case["w"], case["oc"], k, k, oh, ow, p, p, p, p, case["stride"],
                  case["stride"], case["dilation"], case["dilation"], case["post_add"], case["relu"], s.stream)
        s.call = s.ops.mgpuConv2d
    elif kind == "pool":
        oh, ow = _pool_out(case)
        s.x = normal(case["planes"], case["h"], case["w"])
        s.out = empty(case["planes"], oh, ow)
        k, p, st = case["kernel"], case["pad"], case["stride"]
        s.args = (s.x.data_ptr(), s.out.data_ptr(), 1, case["planes"], case["h"], case["w"], oh, ow, k, k, p, p, p, p, st, st,
                  1 if case["average"] else 0, s.stream)
        s.call = s.ops.mgpuPool2d
    elif kind == "context_layer":
        d, ffn = case["heads"] * case["head_dim"], case["ffn"]
        s.x = normal(case["batch"], case["seq"], d)
        s.weights = [normal(d, 3 * d, std=0.02), normal(d, d, std=0.02), normal(d, std=0.02), normal(d, ffn, std=0.02),
                     normal(ffn, std=0.02), normal(ffn, d, std=0.02), normal(d, std=0.02)]
        s.out = empty(case["batch"], case["seq"], d)
        s.args = (s.x.data_ptr(), *[w.data_ptr() for w in s.weights], s.out.data_ptr(), case["batch"], case["seq"], d, ffn,
                  case["heads"], case["norm_first"], case["causal"], case["relu"], s.stream)
        s.call = s.ops.mgpuLLMDecodingContextLayer
    elif kind == "stack":
        d, ffn = case["heads"] * case["head_dim"], case["ffn"]
        s.stack = s.ops.mgpuEncoderStackCreate(case["layers"], d, ffn, case["heads"], case["norm_first"], case["causal"],
                                               GELU if case["gelu"] else RELU, F16 if case["dtype"] == "f16" else BF16, EPS)
        for layer in range(case["layers"]):
            w = [normal(d, 3 * d, std=0.02), normal(3 * d, std=0.02), normal(d, d, std=0.02), normal(d, std=0.02),
                 normal(d, ffn, std=0.02), normal(ffn, std=0.02), normal(ffn, d, std=0.02), normal(d, std=0.02),
                 normal(d, std=0.1, mean=1.0), normal(d, std=0.1), normal(d, std=0.1, mean=1.0), normal(d, std=0.1)]
            torch.cuda.current_stream().synchronize()  # the handle reads the weights on its own stream
            s.ops.mgpuEncoderStackSetLayer(s.stack, layer, *[t.data_ptr() for t in w], s.stream)
            mdc.runtime().mgpuStreamSynchronize(s.stream)
        s.x = normal(case["batch"], case["seq"], d)
        s.y = empty(case["batch"], case["seq"], d)
        s.lens = _lengths(case) if case["padded"] else None
        # rows of padded positions carry no meaning: a user reads each sequence's valid rows
        s.out = [s.y[b, :n] for b, n in enumerate(s.lens.tolist())] if case["padded"] else s.y
        s.args = (s.stack, s.x.data_ptr(), s.lens.data_ptr() if case["padded"] else None, s.y.data_ptr(), case["batch"],
                  case["seq"], s.stream)
        s.call = s.ops.mgpuEncoderStackRun
    else:
        B, S, d = case["batch"], case["seq"], 768
        s.x = normal(B, S, d).cpu().numpy()
        s.lens = np.full(B, S, np.float32)
        s.x_ref = MemRef3(s.x.ctypes.data, s.x.ctypes.data, 0, (B, S, d), (S * d, d, 1))
        s.lens_ref = MemRef1(s.lens.ctypes.data, s.lens.ctypes.data, 0, (B,), (1,))
        s.out_ref = MemRef3()
        s.args = (ctypes.addressof(s.out_ref), ctypes.addressof(s.x_ref), ctypes.addressof(s.lens_ref))
        s.shape, s.floats = (B, S, d), ctypes.c_float * (B * S * d)
        s.call = _encoder_graph()
    torch.cuda.current_stream().synchronize()  # inputs are ready for calls on any stream
    mdc.check("prepare")
    return s


def run(state):
    if state.case["kind"] != "graph":
        state.call(*state.args)
        return state.out
    if state.result:  # the result of a call belongs to the caller, who frees it when done with it
        _libc.free(state.result)
        state.result = None
    state.call(*state.args)
    state.result = state.out_ref.allocated
    return np.frombuffer(state.floats.from_address(state.out_ref.aligned), np.float32).reshape(state.shape)


# ------------------------------------------------------------------ work and tolerance
def _layer_flops(tokens, pairs, d, ffn, causal):
    """One transformer layer: four Gemms over `tokens` rows, and attention over `pairs` (query, key) pairs."""
    return 2.0 * tokens * (4 * d * d + 2 * d * ffn) + 4.0 * pairs * d * (0.5 if causal else 1.0)


def work(case):
    kind = case["kind"]
    if kind == "add":
        return {"bytes": 12.0 * case["n"], "flops": 1.0 * case["n"]}
    if kind == "layernorm":
        return {"bytes": 8.0 * (case["rows"] + 1) * case["cols"], "flops": 8.0 * case["rows"] * case["cols"]}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4.0 * (m * k + k * n + n + m * n), "flops": 2.0 * m * n * k}
    if kind == "conv":
        oh, ow = _conv_out(case)
        out, taps = case["batch"] * case["oc"] * oh * ow, case["ic"] * case["kernel"] ** 2
        return {"bytes": 4.0 * (case["batch"] * case["ic"] * case["h"] * case["w"] + case["oc"] * (taps + 1) + out * (2 if case["post_add"] else 1)),
                "flops": 2.0 * out * taps}
    if kind == "pool":
        oh, ow = _pool_out(case)
        return {"bytes": 4.0 * case["planes"] * (case["h"] * case["w"] + oh * ow), "flops": 1.0 * case["planes"] * oh * ow * case["kernel"] ** 2}
    if kind == "graph":
        tokens, d, ffn = case["batch"] * case["seq"], 768, 3072
        return {"bytes": 8.0 * tokens * d + 2.0 * (4 * d * d + 2 * d * ffn),
                "flops": _layer_flops(tokens, case["batch"] * case["seq"] ** 2, d, ffn, False)}
    d, ffn = case["heads"] * case["head_dim"], case["ffn"]
    tokens, pairs = case["batch"] * case["seq"], case["batch"] * case["seq"] ** 2
    if kind == "context_layer":
        return {"bytes": 8.0 * tokens * d + 4.0 * (4 * d * d + 2 * d * ffn + 2 * d + ffn), "flops": _layer_flops(tokens, pairs, d, ffn, case["causal"])}
    if case["padded"]:  # mean and mean square of a length uniform in half .. full
        tokens, pairs = 0.75 * tokens, 7.0 / 12.0 * pairs
    return {"bytes": 8.0 * tokens * d + case["layers"] * (2.0 * (4 * d * d + 2 * d * ffn) + 4.0 * (9 * d + ffn)),
            "flops": case["layers"] * _layer_flops(tokens, pairs, d, ffn, case["causal"])}


def tolerance(case):
    kind = case["kind"]
    if kind == "add" or (kind == "pool" and not case["average"]):
        return "exact"
    if kind in ("layernorm", "pool"):
        return {"rel": 1e-5, "max": 1e-4}  # fp32 statistics and sums
    if kind in ("linear", "conv"):
        # operands rounded once to fp16 (to nearest), fp32 accumulation: two such results differ by
        # the order of the sum and by nothing else
        return {"rel": 1e-4, "max": 2e-3}
    # Layers keep activations, softmax weights and matrix operands in 16 bits: a few roundings of
    # half an ulp (2^-12 fp16, 2^-9 bf16) per layer, independent from layer to layer.
    bf16 = kind == "stack" and case["dtype"] == "bf16"
    layers = case["layers"] if kind == "stack" else 1
    return {"rel": (6e-3 if bf16 else 8e-4) * math.sqrt(layers)}
