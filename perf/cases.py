"""The work a user of this framework has it do, as measurable cases.

A case names a kind of model or layer and its sizes. `prepare` loads the model (graph -> torq-b200-ops blob ->
Executable, kept while the same case is prepared again, as a program keeps the model it serves) and makes the inputs
of one call from the seed; `run` makes that call through the public entry points: Executable.dispatch on device
buffers, InferenceRunner.infer and Executable.invoke_host_async on host arrays, and the upload / dispatch / download
loop of token-by-token decoding. Sizes are those of the benchmark configurations and of the tests, and the ranges
around them.
"""
import math
import os
import sys

import numpy as np
import torch

for _p in (os.getcwd(), os.path.join(os.getcwd(), "torq-compiler_b200")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from torq_b200.bf16 import to_bf16  # noqa: E402
from torq_b200.oplist import Graph  # noqa: E402
from torq_b200.quant import add_rescale_params, quantize_multiplier, quantize_multipliers  # noqa: E402
from torq_b200.runtime import MEMORY_HOST_PINNED, Device, Executable, InferenceRunner  # noqa: E402
from torq_b200.workloads import gemma3  # noqa: E402
from torq_b200.workloads.mobilenet_v2 import build_mobilenet_v2  # noqa: E402
from torq_b200.workloads.yolov8n import build_yolov8n  # noqa: E402

_TORCH = {"i8": torch.int8, "i16": torch.int16, "i32": torch.int32, "f32": torch.float32, "bf16": torch.bfloat16}


def listed():
    return [
        # the smallest call: one convolution layer on one image (the single-layer configuration), a dispatch of its own
        {"name": "conv3x3 one image", "kind": "conv", "batch": 1, "size": 56, "ic": 64, "oc": 64, "k": 3, "stride": 1},
        # a classifier answering one request: host array in, host array out
        {"name": "classifier one image", "kind": "classifier", "batch": 1, "res": 224, "call": "runner"},
        # a small ragged batch of smaller images, pipelined host calls from pinned memory
        {"name": "classifier 23 at 160", "kind": "classifier", "batch": 23, "res": 160, "call": "pipelined"},
        # the headline workload: a full batch, inputs and results on the device
        {"name": "classifier 256", "kind": "classifier", "batch": 256, "res": 224, "call": "device"},
        # a detector on one camera frame, and on a batch of them
        {"name": "detector one frame", "kind": "detector", "batch": 1, "res": 640, "call": "device"},
        {"name": "detector 64", "kind": "detector", "batch": 64, "res": 640, "call": "device"},
        # FullyConnected: few rows against many weights, and the compute-bound corner of the sweep
        {"name": "fc 64 x 4096", "kind": "fc", "rows": 64, "k": 4096, "n": 4096, "zp": -7},
        {"name": "fc 4096 x 8192", "kind": "fc", "rows": 4096, "k": 8192, "n": 8192, "zp": 0},
        # pooling, table and rescaled add at the size of the pooling configuration
        {"name": "pools and add", "kind": "block", "batch": 64, "size": 112, "c": 64},
        # bf16 tensor ops: one attention head op by op (transpose, matmul, softmax, cast, matmul)
        {"name": "bf16 attention head", "kind": "head", "rows": 512, "d": 64, "dtype": "bf16"},
        # text generation: a greedy token loop behind a 1024-token prompt, for one user and for a batch of them
        {"name": "decode one sequence", "kind": "decode", "batch": 1, "layers": 26, "vocab": 262144, "prompt": 1024, "steps": 8, "feed": "greedy"},
        {"name": "decode 32 sequences", "kind": "decode", "batch": 32, "layers": 26, "vocab": 262144, "prompt": 1024, "steps": 8, "feed": "greedy"},
    ]


def _log(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 0.999)))
    return int(min(hi, max(lo, multiple * max(1, round(v / multiple)) if multiple > 1 else int(v))))


def draw(rng):
    kind = rng.choice(["conv", "classifier", "detector", "fc", "block", "head", "decode"])
    if kind == "conv":
        c = {"kind": kind, "batch": _log(rng, 1, 256), "size": _log(rng, 7, 112), "ic": _log(rng, 8, 256, rng.choice([1, 8, 16, 16, 32])),
             "oc": _log(rng, 8, 256, rng.choice([1, 8, 16, 16, 32])), "k": rng.choice([1, 3, 3, 5]), "stride": rng.choice([1, 1, 2])}
        while c["batch"] > 1 and work(c)["flops"] > 3e10:
            c["batch"] = (c["batch"] + 1) // 2
        return c
    if kind == "classifier":
        return {"kind": kind, "batch": _log(rng, 1, 200), "res": rng.choice([96, 128, 160, 192, 224]),
                "call": rng.choice(["device", "runner", "pipelined"])}
    if kind == "detector":
        res = 32 * _log(rng, 4, 20)
        return {"kind": kind, "batch": _log(rng, 1, 48), "res": res, "call": rng.choice(["device", "device", "runner"])}
    if kind == "fc":
        m = rng.choice([1, 8, 16, 64])
        return {"kind": kind, "rows": _log(rng, 1, 4096), "k": _log(rng, 512, 8192, m), "n": _log(rng, 512, 8192, m), "zp": rng.choice([0, -7])}
    if kind == "block":
        return {"kind": kind, "batch": _log(rng, 1, 64), "size": _log(rng, 14, 112), "c": _log(rng, 16, 256, rng.choice([1, 4, 16, 32]))}
    if kind == "head":
        return {"kind": kind, "rows": _log(rng, 64, 1024), "d": _log(rng, 32, 256, rng.choice([1, 8, 32])), "dtype": rng.choice(["bf16", "f32", "i16"])}
    return {"kind": kind, "batch": _log(rng, 1, 32), "layers": rng.randint(2, 8), "vocab": 4096 * _log(rng, 2, 16),
            "prompt": _log(rng, 16, 1024), "steps": rng.randint(4, 8), "feed": rng.choice(["greedy", "prompt"])}


# ---- models ---------------------------------------------------------------------------------------------------

_device = None
_loaded = (None, None)  # the last model and its case: the one a program is serving


def _dev():
    global _device
    if _device is None:
        _device = Device(0)
    return _device


def _dim(size, k, s, p0, p1):
    return (size + p0 + p1 - k) // s + 1


def _pool_pad(size):
    return (0, 1) if size % 2 == 0 else (1, 1)


def _conv_graph(c):
    # weights, scales and zero points as in the single-convolution configuration: uniform symmetric int8 weights,
    # per-channel scales, int32 bias, SAME padding; the scale keeps the spread of the result inside int8
    rng = np.random.default_rng(1234)
    k, p = c["k"], (c["k"] - 1) // 2
    w = rng.integers(-127, 128, (c["oc"], k, k, c["ic"]), dtype=np.int8)
    m, s = quantize_multipliers(rng.uniform(0.5, 1.5, c["oc"]) * 40.0 / (math.sqrt(k * k * c["ic"]) * 74 * 73))
    g = Graph()
    g.output(g.conv2d(g.input((c["batch"], c["size"], c["size"], c["ic"])), w, np.round(rng.normal(0, 2000, c["oc"])).astype(np.int32), m, s,
                      stride=(c["stride"], c["stride"]), pad=(p, p, p, p), input_zp=-3, out_zp=5))
    return g


def _fc_graph(c):
    rng = np.random.default_rng(1234)
    w = rng.integers(-127, 128, (c["n"], c["k"]), dtype=np.int8)
    m, s = quantize_multipliers(rng.uniform(0.5, 1.5, c["n"]) * 40.0 / (math.sqrt(c["k"]) * 74 * 73))
    g = Graph()
    g.output(g.fully_connected(g.input((c["rows"], c["k"])), w, np.round(rng.normal(0, 1000, c["n"])).astype(np.int32), m, s,
                               input_zp=c["zp"], out_zp=3))
    return g


def _block_graph(c):
    # max pool with a sigmoid table behind it, average pool, and their rescaled sum
    pad = _pool_pad(c["size"]) * 2
    q = np.arange(-128, 128)
    sigmoid = np.clip(np.round(256.0 / (1.0 + np.exp(-0.05 * (q + 4)))) - 128, -128, 127).astype(np.int8)
    m0, m1, mo = add_rescale_params(1.0 / 256, 0.07, 0.06)
    g = Graph()
    x = g.input((c["batch"], c["size"], c["size"], c["c"]))
    mx = g.table(g.maxpool2d(x, (3, 3), (2, 2), pad=pad), sigmoid)
    av = g.avg_pool2d(x, (3, 3), (2, 2), pad=pad, input_zp=-3, output_zp=2)
    g.output(g.add(mx, av, a_zp=-128, a_ms=m0, b_zp=2, b_ms=m1, out_ms=mo, out_zp=1))
    return g


def _head_graph(c):
    g = Graph()
    s, d, dt = c["rows"], c["d"], c["dtype"]
    q, k, v = (g.input((s, d), dt) for _ in range(3))
    kt = g.transpose(k, (1, 0))
    if dt == "i16":
        # integer form: int16 products, the scores rescaled to int16, an interpolated exp table, int16 weights
        scores = g.matmul_i32(q, kt)
        m, sh = quantize_multiplier(6000.0 / (math.sqrt(d) * 1000.0 * 1000.0))
        p16 = g.rescale(scores, m, sh, out_dtype="i16")
        e = g.table16(p16, np.round(4000.0 * np.exp((np.arange(513) - 512) / 96.0)).astype(np.int16))
        m, sh = quantize_multiplier(1.0 / 128.0)
        g.output(g.matmul_i32(g.rescale(e, m, sh, out_dtype="i16"), v))
        return g
    scores = g.matmul_f(q, kt, "f32")
    scale = np.full((1, 1), 1.0 / math.sqrt(d), np.float32)
    p = g.softmax(g.ew("mul", scores, g.const(scale)))
    if dt == "bf16":
        p = g.ew("cast", p, out_dtype="bf16")
    g.output(g.matmul_f(p, v, dt))
    return g


def _gemma_config(c):
    return gemma3.GemmaConfig(layers=c["layers"], vocab=c["vocab"], max_seq=c["prompt"] + 128)


def _gemma_weights(cfg):
    """gemma3.random_weights with its distributions (embedding gain 6.0: peaked logits, as trained weights have),
    drawn on the GPU: a gigabyte of them."""
    gen = torch.Generator("cuda").manual_seed(1234)
    rng = np.random.default_rng(1234)
    H, D = cfg.hidden, cfg.head_dim

    def weight(n, k, gain=1.0):
        w = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=gen).cpu().numpy()
        scale = gain / (127.0 / math.sqrt(3.0) * math.sqrt(k)) * rng.uniform(0.8, 1.25, n)
        return w, to_bf16(scale.astype(np.float32))

    def norm(n, mean=0.0):
        return to_bf16(rng.normal(mean, 0.1 if mean == 0.0 else 0.03, n).astype(np.float32))

    params = {"embed": weight(cfg.vocab, H, 6.0), "final_norm": norm(H), "layers": []}
    for _ in range(cfg.layers):
        params["layers"].append({
            "in_norm": norm(H), "post_attn_norm": norm(H, -0.75), "pre_ffn_norm": norm(H), "post_ffn_norm": norm(H, -0.75),
            "q_norm": norm(D), "k_norm": norm(D), "qkv": weight((cfg.n_q + 2 * cfg.n_kv) * D, H), "o": weight(H, cfg.n_q * D),
            "gate_up": weight(2 * cfg.intermediate, H, 1.5), "down": weight(H, cfg.intermediate)})
    return params


class _Model:
    """What a program keeps between calls: the loaded executable or runner."""

    def __init__(self, c):
        self.runner = None
        if c["kind"] == "decode":
            self._load_decoder(c)
            return
        graph = {"conv": _conv_graph, "fc": _fc_graph, "block": _block_graph, "head": _head_graph,
                 "classifier": lambda c: build_mobilenet_v2(c["batch"], resolution=c["res"])[0],
                 "detector": lambda c: build_yolov8n(c["batch"], c["res"])[0]}[c["kind"]](c)
        blob = graph.serialize()
        if c.get("call") == "runner":
            self.runner = InferenceRunner(blob, device=_dev())
            self.ex = self.runner.executable
        else:
            self.ex = Executable(_dev(), blob)

    def _load_decoder(self, c):
        cfg = _gemma_config(c)
        graph = gemma3.build_decode_step(cfg, c["batch"], _gemma_weights(cfg), with_logits=True)
        self.ex = Executable(_dev(), graph.serialize())
        # the prompt that every request shares, already in the caches
        self.tok, self.pos, self.next = _dev().alloc(4 * c["batch"]), _dev().alloc(4), _dev().alloc(4 * c["batch"])
        logits = _dev().alloc(4 * c["batch"] * c["vocab"])
        prompt = np.random.default_rng(1234).integers(0, c["vocab"], (c["prompt"], c["batch"])).astype(np.int32)
        for i in range(c["prompt"]):
            self.tok.upload(prompt[i])
            self.pos.upload(np.array([i], np.int32))
            self.ex.dispatch([self.tok, self.pos], [self.next, logits])
        _dev().wait()
        logits.free()

    def __del__(self):
        if self.runner is not None:
            self.runner.close()
        elif hasattr(self, "ex"):
            self.ex.destroy()
        for b in (getattr(self, n, None) for n in ("tok", "pos", "next")):
            if b is not None:
                b.free()


def _model(c):
    global _loaded
    key = tuple(sorted((k, v) for k, v in c.items() if k != "name"))
    if _loaded[0] != key:
        _loaded = (None, None)  # the old one goes before the new one comes
        _loaded = (key, _Model(c))
    return _loaded[1]


# ---- one call -------------------------------------------------------------------------------------------------

class _State:
    """One call's inputs and the places its results go to."""

    def __init__(self, model):
        self.model, self.buffers = model, []

    def bind(self, tensor):
        b = _dev().import_pointer(tensor.data_ptr(), tensor.numel() * tensor.element_size())
        self.buffers.append(b)
        return b

    def __del__(self):
        for b in self.buffers:
            b.free()


def _random(info, gen):
    """Activations as the path meets them: int8 over its whole range, int16 of a moderate range, unit-variance floats."""
    if info.dtype == "i8":
        return torch.randint(-128, 128, info.shape, dtype=torch.int8, device="cuda", generator=gen)
    if info.dtype == "i16":
        return torch.randint(-1730, 1731, info.shape, dtype=torch.int16, device="cuda", generator=gen)
    return torch.randn(info.shape, device="cuda", generator=gen).to(_TORCH[info.dtype])


def prepare(case, seed):
    model = _model(case)
    s = _State(model)
    s.kind, s.call = case["kind"], case.get("call", "device")
    gen = torch.Generator("cuda").manual_seed(seed)
    if s.kind == "decode":
        s.prompt, s.steps, s.feed, s.batch = case["prompt"], case["steps"], case["feed"], case["batch"]
        s.tokens = torch.randint(0, case["vocab"], (s.steps, s.batch), dtype=torch.int32, device="cuda", generator=gen).cpu().numpy()
        s.logits = torch.empty((s.batch, case["vocab"]), dtype=torch.float32, device="cuda")
        s.logits_buffer = s.bind(s.logits)
        s.positions = [np.array([s.prompt + i], np.int32) for i in range(s.steps)]
        torch.cuda.synchronize()
        return s
    ins = [_random(i, gen) for i in model.ex.inputs_info]
    if s.call == "runner":
        s.host_in = [t.cpu().numpy() for t in ins]
    elif s.call == "pipelined":
        pairs = [(i, _dev().alloc(i.nbytes, MEMORY_HOST_PINNED)) for i in model.ex.inputs_info + model.ex.outputs_info]
        s.buffers += [b for _, b in pairs]
        arrays = [b.as_numpy(i.shape, i.np_dtype) for i, b in pairs]
        s.host_in, s.host_out = arrays[:len(ins)], arrays[len(ins):]
        for a, t in zip(s.host_in, ins):
            a[...] = t.cpu().numpy()
    else:
        s.tensors = ins
        s.outs = [torch.empty(o.shape, dtype=_TORCH[o.dtype], device="cuda") for o in model.ex.outputs_info]
        s.ins_bound = [s.bind(t) for t in ins]
        s.outs_bound = [s.bind(t) for t in s.outs]
    torch.cuda.synchronize()
    return s


def run(state):
    s, m = state, state.model
    if s.kind == "decode":
        ids = []
        tokens = s.tokens[0]
        for i in range(s.steps):
            m.tok.upload(tokens)
            m.pos.upload(s.positions[i])
            m.ex.dispatch([m.tok, m.pos], [m.next, s.logits_buffer])
            if s.feed == "greedy":  # the program reads each token (to stream it) and feeds it back
                tokens = m.next.download((s.batch,), np.int32)
                ids.append(tokens)
            elif i + 1 < s.steps:   # the program feeds a prompt and reads what comes after its end
                tokens = s.tokens[i + 1]
        if s.feed == "prompt":
            ids.append(m.next.download((s.batch,), np.int32))
        return {"ids": np.stack(ids), "logits": s.logits}
    if s.call == "runner":
        return m.runner.infer(s.host_in)
    if s.call == "pipelined":
        m.ex.invoke_host_async(s.host_in, s.host_out)
        return s.host_out
    m.ex.dispatch(s.ins_bound, s.outs_bound)
    return s.outs


# ---- what a pass cannot do without ------------------------------------------------------------------------------

_macs = {}


def _network(c):
    """(multiply-adds, weight and bias bytes, input bytes, output bytes) of one image of a network."""
    key = (c["kind"], c["res"])
    if key not in _macs:
        if c["kind"] == "classifier":
            g, layers = build_mobilenet_v2(1, resolution=c["res"])
            macs = sum(layer["macs"] for layer in layers)
        else:
            g, macs = build_yolov8n(1, c["res"])
        const = sum(t.nbytes for t in g.tensors if t.data is not None)
        _macs[key] = (macs, const, sum(t.nbytes for t in g.inputs), sum(t.nbytes for t in g.outputs))
    return _macs[key]


def work(case):
    c, kind = case, case["kind"]
    if kind in ("classifier", "detector"):
        macs, const, n_in, n_out = _network(c)
        return {"bytes": const + c["batch"] * (n_in + n_out), "flops": 2 * macs * c["batch"]}
    if kind == "conv":
        p = (c["k"] - 1) // 2
        o = _dim(c["size"], c["k"], c["stride"], p, p)
        pixels = c["batch"] * o * o
        return {"bytes": c["batch"] * c["size"] ** 2 * c["ic"] + pixels * c["oc"] + c["oc"] * (c["k"] ** 2 * c["ic"] + 9),
                "flops": 2 * pixels * c["oc"] * c["k"] ** 2 * c["ic"]}
    if kind == "fc":
        return {"bytes": c["rows"] * (c["k"] + c["n"]) + c["n"] * (c["k"] + 9), "flops": 2 * c["rows"] * c["k"] * c["n"]}
    if kind == "block":
        o = _dim(c["size"], 3, 2, *_pool_pad(c["size"]))
        out = c["batch"] * o * o * c["c"]
        return {"bytes": c["batch"] * c["size"] ** 2 * c["c"] + out + 256, "flops": 20 * out}
    if kind == "head":
        size = {"bf16": 2, "f32": 4, "i16": 2}[c["dtype"]]
        out = 4 if c["dtype"] == "i16" else size
        return {"bytes": c["rows"] * c["d"] * (3 * size + out), "flops": 4 * c["rows"] ** 2 * c["d"]}
    cfg = _gemma_config(c)
    weights = gemma3.weight_bytes_per_token(cfg)
    nbytes = flops = 0
    for i in range(c["steps"]):
        t = c["prompt"] + i + 1
        seen = sum(t if cfg.is_global(layer) else min(t, cfg.window) for layer in range(cfg.layers))
        nbytes += weights + c["batch"] * (2 * seen * cfg.head_dim * 2 + 4 * cfg.vocab)
        flops += 2 * c["batch"] * (weights + 2 * seen * cfg.n_q * cfg.head_dim)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "decode":
        return {"rel": 1e-2}  # bf16 activations; the ids have to be the same
    if case["kind"] == "head" and case["dtype"] != "i16":
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 1e-5}
    return "exact"
