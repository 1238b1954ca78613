"""Performance cases of the library: what a program that uses it has it do, call by call.

Three ways of use, each through the public entry points (aspen_b200.api makes the same calls a C program makes):

* ``call``   -- a program written against the ASPEN header: rpool_add_nasm_raw_input (or token ids), dse_group_run,
                dse_wait_for_nasm_completion, dse_group_stop, dse_get_nasm_result.  Input and result are host memory.
* ``serve``  -- a serving loop in service mode: dse_group_run once, several graphs of one network in rotation, an upload,
                a completed pass and a download per request, dse_group_stop at the end of the burst.
* ``matmul`` -- aspen_b200_matmul_noalloc on device buffers: one layer for a caller that must not allocate.

Networks are the ones of aspen_b200.cfgs with seeded random weights.  ``tiling`` is how the program asked for its tile
graph: "reference" is the geometry every unchanged program gets, "b200" is the tensor-core geometry
(aspen_b200_set_tile_profile(1), or the quanta given).  ``precision``: 0 TF32 operands, 1 fp32.
"""
import math
import os
import tempfile

import numpy as np
import torch

from aspen_b200 import api, cfgs, weights

# network -> (weight scheme, weight seed, order of the result's dimensions)
_NETS = {
    "custom": ("he", 5, (api.BATCH, api.OUT_C)),
    "resnet50": ("he", 1, (api.BATCH, api.OUT_H, api.OUT_W, api.OUT_C)),
    "vgg16": ("he", 2, (api.BATCH, api.OUT_C)),
    "bert_base": ("n002", 3, (api.BATCH, api.MAT_N, api.MAT_M)),
    "gpt2_124M": ("n002", 4, (api.BATCH, api.MAT_N, api.MAT_M)),
}
_IMAGE = {"custom": (32, 10), "resnet50": (224, 1000), "vgg16": (224, 1000)}      # input side, classes
_VOCAB = {"bert_base": 30522, "gpt2_124M": 50257}
_LAYERS, _D, _HEADS, _FFN = 12, 768, 12, 3072                                     # both transformers


def listed():
    return [
        # one token through one projection layer of a plug-in: nothing but latency
        {"name": "matmul_1x768x768", "mode": "matmul", "n": 1, "k": 768, "m": 768, "act": 8},
        # a classifier head over a ragged batch; k is not a multiple of four
        {"name": "matmul_333x770x1000", "mode": "matmul", "n": 333, "k": 770, "m": 1000, "act": 0},
        # an FFN-up layer over 32 sequences of 128 tokens
        {"name": "matmul_4096x768x3072", "mode": "matmul", "n": 4096, "k": 768, "m": 3072, "act": 8},
        # the CIFAR-10 example program, one image at a time
        {"name": "custom_b1_call", "mode": "call", "net": "custom", "batch": 1, "seq": 0, "tiling": "reference", "precision": 0},
        # the ResNet-50 example program as it is, one image, in the fp32 mode a validation run uses
        {"name": "resnet50_b1_fp32_call", "mode": "call", "net": "resnet50", "batch": 1, "seq": 0, "tiling": "reference", "precision": 1},
        # the same program with a batch
        {"name": "resnet50_b32_call", "mode": "call", "net": "resnet50", "batch": 32, "seq": 0, "tiling": "reference", "precision": 0},
        # two networks in one pool (co-inference)
        {"name": "resnet50_vgg16_b16_call", "mode": "call", "net": "resnet50+vgg16", "batch": 16, "seq": 0, "tiling": "b200", "precision": 0},
        # one short sentence of odd length through an unchanged program
        {"name": "bert_b1_s37_call", "mode": "call", "net": "bert_base", "batch": 1, "seq": 37, "tiling": "reference", "precision": 0},
        # prefill of 8 prompts of 512 tokens, causal attention
        {"name": "gpt2_b8_s512_call", "mode": "call", "net": "gpt2_124M", "batch": 8, "seq": 512, "tiling": "b200", "precision": 0},
        # image serving: full batches, and the small batches of a latency-bound or sharded service
        {"name": "resnet50_b32_serve", "mode": "serve", "net": "resnet50", "batch": 32, "seq": 0, "graphs": 3, "requests": 12, "tiling": "128x128/100", "precision": 0},
        {"name": "resnet50_b4_serve", "mode": "serve", "net": "resnet50", "batch": 4, "seq": 0, "graphs": 8, "requests": 32, "tiling": "128x128/100", "precision": 0},
        # text serving from token ids
        {"name": "bert_b16_s128_serve", "mode": "serve", "net": "bert_base", "batch": 16, "seq": 128, "graphs": 4, "requests": 16, "tiling": "256x128/148", "precision": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed() if c["mode"] != "matmul")
    while True:
        kind = rng.choice(["matmul", "custom", "resnet50", "fp32", "pair", "bert_base", "gpt2_124M", "serve_image", "serve_text"])
        if kind == "matmul":
            return {"mode": "matmul", "n": _log(rng, 1, 4096), "k": _log(rng, 64, 3072), "m": _log(rng, 64, 3072), "act": rng.choice([0, 4, 8])}
        c = {"mode": "call", "net": kind, "batch": 1, "seq": 0, "tiling": rng.choice(["reference", "b200"]), "precision": 0}
        if kind == "custom":
            c.update(batch=_log(rng, 1, 256), precision=rng.choice([0, 0, 1]))
        elif kind == "resnet50":
            c.update(batch=_log(rng, 1, 32))
        elif kind == "fp32":
            c.update(net="resnet50", batch=_log(rng, 1, 4), precision=1)
        elif kind == "pair":
            c.update(net="resnet50+vgg16", batch=_log(rng, 1, 16))
        elif kind == "bert_base":
            c.update(batch=_log(rng, 1, 32), seq=_log(rng, 8, 384))
        elif kind == "gpt2_124M":
            c.update(batch=_log(rng, 1, 8), seq=_log(rng, 16, 512))
        else:
            batch = _log(rng, 1, 32)
            graphs = 3 if batch > 16 else rng.choice([3, 4, 8]) if batch <= 4 else rng.choice([3, 4])
            c.update(mode="serve", net="resnet50", batch=batch, graphs=graphs, requests=graphs * rng.choice([2, 3]), tiling="128x128/100")
            if kind == "serve_text":
                c.update(net="bert_base", batch=max(1, batch // 2), seq=_log(rng, 16, 256), tiling="256x128/148")
        if work(c)["flops"] <= most:
            return c


_models = {}


def _model(net):
    """The network with its weights, read once by a program and shared by its graphs."""
    if net not in _models:
        scheme, seed, _ = _NETS[net]
        with tempfile.TemporaryDirectory(prefix="aspen_perf_") as d:
            cfg, wfile = os.path.join(d, net + ".cfg"), os.path.join(d, net + ".bin")
            weights.write_aspen_data(wfile, weights.make_weights(cfgs.write_cfg(net, cfg), seed, scheme))
            dnn = api.Dnn(cfg, wfile)
        if net in _VOCAB:
            rng = np.random.default_rng(seed + 100)
            dnn.set_embedding(np.float32(0.02) * rng.standard_normal((_VOCAB[net], _D), dtype=np.float32),
                              np.float32(0.02) * rng.standard_normal((512, _D), dtype=np.float32))
        _models[net] = dnn
    return _models[net]


def _graph(net, case):
    L, tiling, count = api.lib(), case["tiling"], 100
    if "/" in tiling:
        quanta, count = tiling.split("/")
        L.aspen_b200_set_tile_quanta(*(int(v) for v in quanta.split("x")), 100000000)
    else:
        L.aspen_b200_set_tile_profile(1 if tiling == "b200" else 0)
    nasm = api.Nasm(_model(net), case["batch"], case["seq"], int(count))
    L.aspen_b200_set_tile_profile(0)
    return nasm


class _Program:
    """A pool, its scheduling engines and the tile graphs in it: what a program builds once and keeps."""

    def __init__(self, case, inputs):
        self.serve = case["mode"] == "serve"
        nets = case["net"].split("+")
        self.order = [_NETS[n][2] for n in nets]
        self.rpool, self.group = api.Rpool(), api.DseGroup(0, case["precision"])
        self.group.set_rpool(self.rpool)
        self.graphs = [_graph(n, case) for n in nets * case.get("graphs", 1)]
        if self.serve:
            # the serving loop returns the last layer only, so the outputs a fused residual add swallows need not be kept
            api.lib().aspen_b200_set_hidden_states(0)
            self.group.set_service(True)
        for g, x in zip(self.graphs, inputs):
            self.add(g, x)
        self.group.run()
        for g in self.graphs:
            self.group.wait(g)
        self.group.stop()
        api.lib().aspen_b200_set_hidden_states(1)

    def add(self, graph, x):
        if x.dtype == np.int32:
            self.rpool.add_tokens(graph, x)
        else:
            self.rpool.add(graph, x)

    def call(self, inputs):
        for g, x in zip(self.graphs, inputs):
            self.add(g, x)
        self.group.run()
        for g in self.graphs:
            self.group.wait(g)
        self.group.stop()
        return [g.result(o) for g, o in zip(self.graphs, self.order)]

    def burst(self, inputs):
        out, n, order = [], len(self.graphs), self.order[0]
        self.group.run()
        for i, x in enumerate(inputs):
            g = self.graphs[i % n]
            if i >= n:
                self.group.wait(g)
                out.append(g.result(order))
            self.add(g, x)
        for i in range(len(inputs), len(inputs) + n):
            g = self.graphs[i % n]
            self.group.wait(g)
            out.append(g.result(order))
        self.group.stop()
        return out

    def close(self):
        self.group.close()
        for g in self.graphs:
            g.close()
        self.rpool.close()


_programs = {}      # by case; building a tile graph takes seconds, so a program does it once and feeds it ever new inputs


def _program(case, inputs):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _programs:
        while len(_programs) >= 16:
            _programs.pop(next(iter(_programs))).close()
        _programs[key] = _Program(case, inputs)
    return _programs[key]


def _input(rng, case, net):
    """Images are N(0, 1); text is token ids in a serving loop and for GPT-2, hidden states in a reference-style call.
    A serving loop keeps its input buffers in pinned memory, a plain program does not."""
    batch, seq, serve = case["batch"], case["seq"], case["mode"] == "serve"
    if net in _IMAGE:
        side = _IMAGE[net][0]
        x = rng.standard_normal((batch * side * side, 3), dtype=np.float32)
    elif serve or net == "gpt2_124M":
        x = rng.integers(0, _VOCAB[net], (batch, seq), dtype=np.int32)
    else:
        x = rng.standard_normal((batch * seq, _D), dtype=np.float32)
    return torch.from_numpy(x).pin_memory().numpy() if serve else x


def prepare(case, seed):
    if case["mode"] != "matmul":
        rng = np.random.default_rng(seed)
        inputs = [_input(rng, case, net) for net in case["net"].split("+") * case.get("requests", 1)]
        return _program(case, inputs), inputs
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, k, m = case["n"], case["k"], case["m"]
    return {"x": torch.randn(n, k, generator=g, device="cuda"), "w": torch.randn(m, k, generator=g, device="cuda") * (2.0 / k) ** 0.5,
            "bias": torch.randn(m, generator=g, device="cuda") * 0.01, "out": torch.empty(n, m, device="cuda"), "act": case["act"]}


def run(state):
    if isinstance(state, tuple):
        program, inputs = state
        return program.burst(inputs) if program.serve else program.call(inputs)
    x, w, out = state["x"], state["w"], state["out"]
    rc = api.lib().aspen_b200_matmul_noalloc(x.data_ptr(), w.data_ptr(), state["bias"].data_ptr(), out.data_ptr(), x.shape[0], x.shape[1],
                                             w.shape[0], state["act"], torch.cuda.current_stream().cuda_stream)
    if rc != 0:
        raise RuntimeError("aspen_b200_matmul_noalloc: " + api.last_error())
    return out


def _conv_flops(net):
    """Multiply-adds of one image times two: [(output side, rows x K of the weight)] of every weighted layer."""
    if net == "custom":
        shape = [(32, 32 * 75), (16, 64 * 288), (1, 256 * 4096), (1, 128 * 256), (1, 10 * 128)]
    elif net == "vgg16":
        shape, cin = [], 3
        for side, n, c in ((224, 2, 64), (112, 2, 128), (56, 3, 256), (28, 3, 512), (14, 3, 512)):
            for _ in range(n):
                shape.append((side, c * cin * 9))
                cin = c
        shape += [(1, 4096 * 25088), (1, 4096 * 4096), (1, 1000 * 4096)]
    else:
        shape, cin = [(112, 64 * 147)], 64
        for side, n, c in ((56, 3, 64), (28, 4, 128), (14, 6, 256), (7, 3, 512)):
            for b in range(n):
                before = side * 2 if b == 0 and c > 64 else side
                shape += [(before, c * cin), (side, c * c * 9), (side, 4 * c * c)]
                if b == 0:
                    shape.append((side, 4 * c * cin))
                cin = 4 * c
        shape.append((1, 1000 * 2048))
    return sum(2.0 * s * s * wk for s, wk in shape), sum(wk for _, wk in shape)


def work(case):
    if case["mode"] == "matmul":
        n, k, m = case["n"], case["k"], case["m"]
        return {"bytes": 4.0 * (n * k + m * k + m + n * m), "flops": 2.0 * n * k * m}
    nbytes = flops = 0.0
    for net in case["net"].split("+"):
        b, s, r = case["batch"], case["seq"], case.get("requests", 1)
        if net in _IMAGE:
            side, classes = _IMAGE[net]
            f, params = _conv_flops(net)
            nbytes += 4.0 * (params + r * b * (3 * side * side + classes))
            flops += r * b * f
        else:
            params = _LAYERS * (4 * _D * _D + 2 * _D * _FFN)
            keys = (s + 1) / 2 if net == "gpt2_124M" else s               # keys a query sees on average (causal or all)
            per_token = 4 if case["mode"] == "serve" or net == "gpt2_124M" else 4 * _D
            nbytes += 4.0 * params + r * b * s * (per_token + 4.0 * _D)
            flops += r * b * s * (2.0 * params + _LAYERS * 4.0 * _D * keys)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # fp32 sums in another order; with TF32 operands (2**-11 per rounding) what the rounding of a chain of layers adds up to
    return {"rel": 1e-5, "max": 1e-3} if case["mode"] == "matmul" or case["precision"] == 1 else {"rel": 3e-3, "max": 5e-2}
