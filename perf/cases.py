"""What the decoder token loop is measured on: calls of the public entry points as a program that serves a model makes them, over the
range of batches, contexts and designs that the library takes.

A case names its `path`; `listed()` has one or more fixed cases of every path, `draw()` others of the same ranges:

  decode     steps of a grouped-query decoder with the host in the loop (`Generation.step_host`): the next token of every sequence comes from the
             program (forced tokens, as speculative, constrained or scored decoding has them), the chosen tokens go back to it; in the
             end the logits of the last step.  The cache is cut back to the prompt before the pass, so every pass does the same work.
  prefill    prompts of equal or unequal length through `Generation.prefill` into an empty cache, logits of every prompt's last token.
  attention  the decode attention alone, as a program binds it over the kernel-level C ABI, on sequences of very unequal length.
  hybrid     state-space and latent-attention decoder: prompts, then forced steps, as a chat turn.
  parallel   chunked-attention decoder with a looped range: one packed pass of unequal prompts through `LanguageModel.run`.
  experts    router and gated experts of a mixture on the rows of a pass, over the kernel-level C ABI.

Weights are seeded random numbers of the benchmark configurations' sizes (`ctorch_b200.workloads`): a loaded model is kept between the
inputs, as a serving program keeps it.  Tokens, keys, queries and rows come from the case's seed."""
from __future__ import annotations

import copy
import ctypes as C
import math

import numpy as np
import torch

import ctorch_b200 as B
from ctorch_b200 import workloads as W

# ---- models --------------------------------------------------------------------------------------------------------------------------------------

DECODERS = {
    "byte": dict(W.CONFIGS["c1"], context=512),                          # f32, the byte-level decoder that also runs on a CPU
    "small": dict(W.CONFIGS["c2"], context=1536),                        # bf16, 12 layers of width 768
    "1b": dict(W.CONFIGS["c4"], context=1536),                           # bf16, 16 layers of width 2048
    "8b": dict(W.CONFIGS["c5"], layers=2, context=4608),                 # two layers of the 8B shape, rank-16 adapters, its vocabulary
}
_DENSE = {"kind": "dense", "ff": 4096}


def _hybrid():
    return W.hybrid_config(**W.HYBRID_SIZES["1k"][0])


def _parallel():
    """The parallel decoder of width 1024 with dense feed-forwards (the experts are a path of their own, with routes that do not hang on rounding)."""
    config = W.parallel_config(width=1024, layers=12, ff=4096, heads=16, kv_heads=4, experts=16, chunk=512, loop=(4, 8, 2))
    config["layers"] = [dict(layer, mlp=_DENSE) for layer in config["layers"]]
    return config


_kept: dict = {}


def _keep(key, make):
    """A loaded model, kept while the next inputs are for it."""
    if key not in _kept:
        while len(_kept) >= 2:
            _kept.pop(next(iter(_kept)))
        _kept[key] = make()
    return _kept[key]


def _normal(index, shape, scale, dtype, around=0.0):
    g = torch.Generator(device="cuda").manual_seed(1_000_003 + index)
    return (around + scale * torch.randn(shape, generator=g, device="cuda")).to(dtype)


def _host(tensor):
    return (tensor.view(torch.int16).cpu().numpy().view(np.uint16) if tensor.dtype == torch.bfloat16 else tensor.cpu().numpy())


def _decoder_weight(spec, index):
    """Tensor `index` of the canonical list, on the GPU in the model's dtype."""
    name, shape = W.tensor_shapes(spec)[index]
    dtype = torch.bfloat16 if spec["dtype"] == "bf16" else torch.float32
    return _normal(index, shape, 0.1, dtype, 1.0) if len(shape) == 1 else _normal(index, shape, 0.02, dtype)


def _adapter_weight(spec, layer, j):
    """q down, q up, v down, v up of one layer."""
    d, r, kv = spec["d_model"], spec["lora_rank"], spec["kv_heads"] * spec["d_model"] // spec["heads"]
    return _normal(50_000 + 4 * layer + j, [(r, d), (d, r), (r, d), (kv, r)][j], 0.05, torch.bfloat16)


def _decoder(name):
    spec = DECODERS[name]

    def make():
        tensors = [_host(_decoder_weight(spec, i)) for i in range(len(W.tensor_shapes(spec)))]
        lora = [_host(_adapter_weight(spec, i, j)) for i in range(spec["layers"]) for j in range(4)] if spec.get("lora_rank") else None
        return B.DecoderModel(spec, tensors, lora=lora)
    return _keep(name, make)


def _shapes(config):
    return {n: t.shape for n, t in B.LanguageModel(config, None, device=None).module.state().items() if "rotary." not in n}


def _named_weight(index, name, shape):
    if len(shape) == 2:
        return _normal(index, shape, shape[1] ** -0.5, torch.bfloat16)
    if name.endswith((".b", "A_log", "dt_bias")):
        return _normal(index, shape, 0.2, torch.bfloat16)
    return _normal(index, shape, 0.05, torch.bfloat16, 1.0)


def _language_model(name, config):
    def make():
        return B.LanguageModel(config, {n: _host(_named_weight(i, n, s)) for i, (n, s) in enumerate(_shapes(config).items())})
    return _keep(name, make)


# ---- cases ---------------------------------------------------------------------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: one sequence of the f32 byte decoder, bound by latency and launches
        {"name": "byte_decode", "path": "decode", "model": "byte", "batch": 1, "context": 64, "steps": 16},
        # a small model that answers several users at once
        {"name": "small_decode_16", "path": "decode", "model": "small", "batch": 16, "context": 549, "steps": 8},
        # one user of the 1B shape, near the end of the context
        {"name": "1b_decode_1", "path": "decode", "model": "1b", "batch": 1, "context": 1501, "steps": 8},
        # the headline: a full decode batch of the 1B shape
        {"name": "1b_decode_256", "path": "decode", "model": "1b", "batch": 256, "context": 1024, "steps": 2},
        # adapters on the 8B shape's layers, long contexts, the 128k vocabulary
        {"name": "8b_adapters_decode_32", "path": "decode", "model": "8b", "batch": 32, "context": 4096, "steps": 4},
        # prompts of the 1B shape, a full pass of rows
        {"name": "1b_prefill_8x1024", "path": "prefill", "model": "1b", "batch": 8, "longest": 1024, "ragged": False},
        # decode attention of a large cache, contexts from 1k to 32k
        {"name": "attention_64x32k", "path": "attention", "batch": 64, "heads": 32, "kv_heads": 8, "dim": 128, "shortest": 1024, "longest": 32768},
        # the hybrid decoder on long prompts, and on short ones with a longer answer
        {"name": "hybrid_prompts", "path": "hybrid", "batch": 8, "longest": 1024, "ragged": False, "steps": 1},
        {"name": "hybrid_answers", "path": "hybrid", "batch": 64, "longest": 24, "ragged": True, "steps": 16},
        # arrivals of a serving queue in one packed pass
        {"name": "parallel_packed", "path": "parallel", "batch": 24, "longest": 700},
        # a mixture's rows in a decode batch and in a prompt
        {"name": "experts_256", "path": "experts", "rows": 256, "width": 2048, "ff": 4096, "experts": 16, "top": 2},
        {"name": "experts_8192", "path": "experts", "rows": 8192, "width": 2048, "ff": 4096, "experts": 16, "top": 2},
    ]


def _spread(rng, low, high):
    """A whole number from low to high, evenly over the logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.5))))))


def draw(rng):
    path = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "attention", "hybrid", "parallel", "experts", "experts"])
    if path == "decode":
        model = rng.choice(["byte", "small", "1b", "1b", "8b"])
        most_batch, most_context = {"byte": (4, 400), "small": (256, 1400), "1b": (256, 1400), "8b": (32, 4096)}[model]
        batch = _spread(rng, 1, most_batch)
        context = _spread(rng, 9, most_context if batch <= 128 else 1000)
        return {"path": path, "model": model, "batch": batch, "context": context, "steps": 2 if batch > 128 else 4 if batch > 24 else 8}
    if path == "prefill":
        model = rng.choice(["small", "1b"])
        longest = _spread(rng, 16, 1400)
        return {"path": path, "model": model, "batch": _spread(rng, 1, min(64, max(1, 8192 // longest))), "longest": longest, "ragged": rng.random() < 0.5}
    if path == "attention":
        dim, kv_heads = rng.choice([64, 128]), rng.choice([2, 4, 8])
        longest = _spread(rng, 300, 32768)
        return {"path": path, "batch": _spread(rng, 1, 64), "heads": kv_heads * rng.choice([1, 3, 4, 8]), "kv_heads": kv_heads, "dim": dim,
                "shortest": max(1, longest // 32), "longest": longest}
    if path == "hybrid":
        longest = _spread(rng, 4, 1024)
        return {"path": path, "batch": _spread(rng, 1, min(128, max(1, 8192 // longest))), "longest": longest, "ragged": rng.random() < 0.5, "steps": rng.randint(1, 16)}
    if path == "parallel":
        longest = _spread(rng, 8, 1400)
        return {"path": path, "batch": _spread(rng, 1, min(64, max(1, 12000 // longest))), "longest": longest}
    return {"path": path, "rows": _spread(rng, 9, 8192), "width": rng.choice([1024, 1536, 2048]), "ff": rng.choice([2048, 2752, 4096]),
            "experts": rng.choice([8, 16]), "top": rng.choice([1, 2, 4])}


# ---- inputs --------------------------------------------------------------------------------------------------------------------------------------

DISTINCT = 8      # different prompts of a decode batch: the sequences of a batch continue these (several samples of one prompt)


def _tokens(case, seed, vocab):
    """Prompts, their lengths, and forced tokens [steps, batch]."""
    rng = np.random.default_rng([seed, 17])
    batch, steps = case["batch"], case.get("steps", 0)
    if case["path"] == "decode":
        prompts = rng.integers(0, vocab, (min(batch, 2 if case["model"] == "8b" else DISTINCT), case["context"]))
        lengths = np.full(batch, case["context"])
    else:
        longest = case["longest"]
        prompts = rng.integers(0, vocab, (batch, longest))
        unequal = case.get("ragged", True)
        lengths = rng.integers(max(1, longest // 8), longest + 1, batch) if unequal else np.full(batch, longest)
        lengths[0] = longest
    return prompts, lengths, rng.integers(0, vocab, (steps, batch))


def _budget(batch):
    """Steps that a generation object may make: its history stays below 70 MB."""
    return 1 << 23 if batch == 1 else (1 << 23) // batch


def _attention_inputs(case, seed):
    """Lengths and queries, and the chunks of keys and values (on the bf16 grid, as f32)."""
    n, longest = case["batch"], case["longest"]
    lengths = np.random.default_rng([seed, 11]).integers(case["shortest"], longest + 1, n).astype(np.int32)
    lengths[0] = longest
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn((n, case["heads"], case["dim"]), device="cuda", generator=g)

    def chunks():
        for first in range(0, longest, 1024):
            count = min(1024, longest - first)
            yield tuple(torch.randn((n, case["kv_heads"], count, case["dim"]), device="cuda", generator=g).bfloat16().float() for _ in range(2))
    return lengths, q, chunks()


def _expert_inputs(case, seed):
    def normal(index, shape, scale, dtype):   # weights, the same for every seed
        return _normal(90_000 + index, shape, scale, dtype)
    e, width, ff = case["experts"], case["width"], case["ff"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    return {"up": normal(0, (e, 2 * ff, width), width ** -0.5, torch.bfloat16), "down": normal(1, (e, width, ff), ff ** -0.5, torch.bfloat16),
            "x": torch.randn((case["rows"], width), device="cuda", generator=g), "residual": torch.randn((case["rows"], width), device="cuda", generator=g),
            "logits": torch.randn((case["rows"], e), device="cuda", generator=g)}


# ---- a program's objects ---------------------------------------------------------------------------------------------------------------------------

class DeviceMatrix:
    """A device result of the library, for torch to look at where it lies."""

    def __init__(self, tensor):
        self.tensor = tensor
        self.__cuda_array_interface__ = {"shape": tensor.shape, "typestr": "<f4", "data": (tensor.data_ptr, False), "version": 3}


def _logits(generation):
    """Logits of the last step, on the device."""
    out = C.c_void_p()
    B.check(B.lib().dl_generation_logits(generation.h, C.byref(out)))
    return torch.as_tensor(DeviceMatrix(B.Tensor(out)), device="cuda")


class AttentionState:
    def __init__(self, case, seed):
        l = B.lib()
        self.case = case
        n, longest = case["batch"], case["longest"]
        self.cache = C.c_void_p()
        B.kcheck(l.b200_kv_cache_create(0, B.BF16, n, case["kv_heads"], case["dim"], longest, 64, C.byref(self.cache)))
        lengths, self.q, chunks = _attention_inputs(case, seed)
        stream = torch.cuda.current_stream().cuda_stream
        for k, v in chunks:
            B.kcheck(l.b200_kv_cache_append(self.cache, k.data_ptr(), v.data_ptr(), k.shape[2], stream))
            B.kcheck(l.b200_kv_cache_advance((C.c_void_p * 1)(self.cache), 1, k.shape[2], stream))
        B.kcheck(l.b200_kv_cache_set_lengths(self.cache, (lengths - 1).ctypes.data_as(C.POINTER(C.c_int32)), stream))   # the step's own token counts
        self.need = l.b200_attention_scratch_bytes(n, case["heads"], case["kv_heads"], case["dim"], longest, 64)
        self.scratch = torch.empty((self.need,), dtype=torch.uint8, device="cuda")
        self.out = torch.empty((n, case["heads"], case["dim"]), device="cuda")
        torch.cuda.synchronize()

    def run(self):
        c = self.case
        B.kcheck(B.lib().b200_attention_decode(self.q.data_ptr(), c["batch"], 1, c["heads"], self.cache, c["longest"], 1, self.scratch.data_ptr(), self.need,
                                               self.out.data_ptr(), torch.cuda.current_stream().cuda_stream))
        return {"attended": self.out}

    def __del__(self):
        B.lib().b200_kv_cache_release(self.cache)


class ExpertState:
    def __init__(self, case, seed):
        self.t = t = _expert_inputs(case, seed)
        rows, top, experts, width, ff = case["rows"], case["top"], case["experts"], case["width"], case["ff"]
        self.rows, self.experts = rows, experts
        hi = t["x"].bfloat16()
        lo = (t["x"] - hi.float()).bfloat16()
        integers = lambda *shape: torch.zeros(shape, dtype=torch.int32, device="cuda")
        self.chosen, self.rank, self.counts, self.weight = integers(rows, top), integers(rows, top), integers(experts), torch.zeros((rows, top), device="cuda")
        self.y = torch.empty((rows, width), device="cuda")
        self.route = B.Route(experts=experts, top=top, column=0, chosen=self.chosen.data_ptr(), weight=self.weight.data_ptr(), rank=self.rank.data_ptr(),
                             counts=self.counts.data_ptr(), chosen_softmax=1)
        self.args = B.Experts(experts=experts, top=top, rows=rows, inner=width, ff=ff, weight_dtype=B.BF16, up=t["up"].data_ptr(), down=t["down"].data_ptr(),
                              chosen=self.chosen.data_ptr(), weight=self.weight.data_ptr(), residual=t["residual"].data_ptr(), y=self.y.data_ptr(), gated=1,
                              weigh_results=1, eps=1e-5)
        self.args.x_hi, self.args.x_lo = hi.data_ptr(), lo.data_ptr()
        self.planes = hi, lo
        self.grouped = bool(B.lib().b200_experts_takes_grouped(C.byref(self.args)))
        self.need = B.lib().b200_experts_grouped_bytes(C.byref(self.args)) if self.grouped else 4 * rows * top * ff
        self.scratch = torch.empty((self.need,), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def run(self):
        l, stream = B.lib(), torch.cuda.current_stream().cuda_stream
        self.counts.zero_()
        B.kcheck(l.b200_route_rows(self.t["logits"].data_ptr(), self.rows, self.experts, C.byref(self.route), stream))
        if self.grouped:
            B.kcheck(l.b200_experts_grouped(C.byref(self.args), self.rank.data_ptr(), self.counts.data_ptr(), self.scratch.data_ptr(), self.need, stream))
        else:
            B.kcheck(l.b200_experts_streamed(C.byref(self.args), self.scratch.data_ptr(), stream))
        return {"chosen": self.chosen, "weight": self.weight, "y": self.y}


class DecodeState:
    """A batch of sequences whose prompts are in the cache."""

    def __init__(self, case, seed):
        shared = _decoder(case["model"])
        self.model = copy.copy(shared)          # the loaded model with a cache of this batch's own
        self.model.cache = None
        self.model.new_cache()
        prompts, _, self.forced = _tokens(case, seed, shared.spec["vocab"])
        self.forced = np.ascontiguousarray(self.forced, dtype=np.int64)
        batch = case["batch"]
        self.context = case["context"]
        self.generation = B.Generation(self.model, batch, _budget(batch))
        self.generation.prefill(prompts[np.arange(batch) % len(prompts)])
        self.chosen = np.empty(self.forced.shape, dtype=np.int64)

    def run(self):
        self.model.truncate(self.context)
        for ids, chosen in zip(self.forced, self.chosen):
            self.generation.step_host(ids, chosen)
        return {"chosen": self.chosen, "logits": _logits(self.generation)}


class PrefillState:
    def __init__(self, case, seed):
        shared = _decoder(case["model"])
        self.model = copy.copy(shared)
        self.model.cache = None
        self.model.new_cache()
        self.prompts, self.lengths, _ = _tokens(case, seed, shared.spec["vocab"])
        if not case["ragged"]:
            self.lengths = None
        self.generation = B.Generation(self.model, case["batch"], _budget(case["batch"]))

    def run(self):
        self.model.clear()
        self.generation.prefill(self.prompts, lengths=self.lengths)
        return {"logits": _logits(self.generation)}


class HybridState:
    def __init__(self, case, seed):
        self.model = copy.copy(_language_model("hybrid", _hybrid()))
        self.prompts, self.lengths, forced = _tokens(case, seed, self.model.vocab)
        self.forced = np.ascontiguousarray(forced, dtype=np.int64)
        self.model.new_cache(case["batch"], case["longest"] + case["steps"])
        self.generation = B.Generation(self.model, case["batch"], _budget(case["batch"]))
        self.chosen = np.empty(self.forced.shape, dtype=np.int64)

    def run(self):
        self.model.cache.clear()
        self.generation.prefill(self.prompts, lengths=self.lengths)
        for ids, chosen in zip(self.forced, self.chosen):
            self.generation.step_host(ids, chosen)
        return {"logits": _logits(self.generation)}


class ParallelState:
    def __init__(self, case, seed):
        self.model = _language_model("parallel", _parallel())
        prompts, lengths, _ = _tokens(case, seed, self.model.vocab)
        self.entries = [(slot, prompt[:n], [int(n) - 1]) for slot, (prompt, n) in enumerate(zip(prompts, lengths))]
        self.cache = B.SlotCache(self.model, case["batch"], case["longest"])

    def run(self):
        self.cache.clear()
        return {"logits": self.model.run(self.entries, self.cache)}


_STATES = {"decode": DecodeState, "prefill": PrefillState, "attention": AttentionState, "hybrid": HybridState, "parallel": ParallelState, "experts": ExpertState}


def prepare(case, seed):
    return _STATES[case["path"]](case, seed)


def run(state):
    return state.run()


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------------------------------

def _matrix_elements(path_model):
    """Weights that a pass of every layer reads, head included, counted once per layer run."""
    if path_model in DECODERS:
        spec = DECODERS[path_model]
        d, f, kv = spec["d_model"], spec["hidden"], spec["kv_heads"] * spec["d_model"] // spec["heads"]
        layer = 2 * d * d + 2 * d * kv + 3 * d * f
        if spec.get("lora_rank"):
            layer += spec["lora_rank"] * (3 * d + kv)
        return spec["layers"] * layer, spec["vocab"] * d
    config = _hybrid() if path_model == "hybrid" else _parallel()
    d, total = config["width"], 0
    loop = config.get("loop") or {"start": 0, "stop": 0, "times": 1}
    for i, layer in enumerate(config["layers"]):
        m = layer["mixer"]
        if layer["type"] == "mamba2":
            inner = m["heads"] * m["vdim"]
            own = d * (2 * inner + 2 * m["groups"] * m["state"] + m["heads"]) + inner * d
        elif layer["type"] == "latent_attention":
            own = d * (m["q_rank"] + m["kv_rank"] + m["rot_dim"] + m["heads"] * m["vdim"]) + m["q_rank"] * m["heads"] * (m["dim"] + m["rot_dim"]) \
                + m["kv_rank"] * m["heads"] * (m["dim"] + m["vdim"]) + m["heads"] * m["vdim"] * d
        else:
            own = d * (m["heads"] * (m["dim"] + 1) + m["kv_heads"] * (m["dim"] + m["vdim"])) + m["heads"] * m["vdim"] * d
        own += 3 * d * layer["mlp"]["ff"]
        total += own * (loop["times"] if loop["start"] <= i < loop["stop"] else 1)
    if config.get("loop"):
        total += (loop["times"] + 1) * d * d
    return total, config["vocab"] * d


def work(case):
    path = case["path"]
    if path == "attention":
        mean = (case["shortest"] + case["longest"]) / 2
        keys = case["batch"] * mean * case["kv_heads"] * case["dim"]
        rows = case["batch"] * case["heads"] * case["dim"]
        return {"bytes": 4 * keys + 8 * rows, "flops": 4 * case["batch"] * mean * case["heads"] * case["dim"]}
    if path == "experts":
        rows, top, width, ff = case["rows"], case["top"], case["width"], case["ff"]
        used = min(case["experts"], rows * top)
        return {"bytes": used * 3 * width * ff * 2 + rows * width * 12, "flops": 6 * rows * top * width * ff}
    if path == "decode":
        spec = DECODERS[case["model"]]
        size, (layers, head) = 2 if spec["dtype"] == "bf16" else 4, _matrix_elements(case["model"])
        batch, context = case["batch"], case["context"]
        hd = spec["d_model"] // spec["heads"]
        cached = spec["layers"] * batch * context * spec["kv_heads"] * hd * 2
        step = {"bytes": size * (layers + head + cached) + 4 * batch * spec["vocab"] / case["steps"],
                "flops": 2 * batch * (layers + head) + 4 * spec["layers"] * batch * context * spec["d_model"]}
        return {k: case["steps"] * v for k, v in step.items()}
    mean = (max(1, case["longest"] // 8) + case["longest"]) / 2 if case.get("ragged", True) else case["longest"]
    tokens, batch = case["batch"] * mean, case["batch"]
    if path == "prefill":
        spec = DECODERS[case["model"]]
        layers, head = _matrix_elements(case["model"])
        flops = 2 * tokens * layers + 2 * batch * head + 2 * spec["layers"] * tokens * mean * spec["d_model"]
        written = spec["layers"] * tokens * spec["kv_heads"] * (spec["d_model"] // spec["heads"]) * 2
        return {"bytes": 2 * (layers + head + written) + 4 * batch * spec["vocab"], "flops": flops}
    layers, head = _matrix_elements(path)
    vocab = _hybrid()["vocab"]
    passes = 1 + case.get("steps", 0)
    rows = tokens + batch * case.get("steps", 0)
    data = {"bytes": passes * 2 * (layers + head) + 4 * batch * vocab, "flops": 2 * rows * layers + 2 * batch * passes * head}
    if path == "hybrid":    # states of the recurrence, read and written by every step
        m = _hybrid()["layers"][0]["mixer"]
        state = m["heads"] * m["state"] * m["vdim"]
        data["bytes"] += 6 * batch * state * 4 * (1 + 2 * case["steps"])
        data["flops"] += 6 * rows * state * 6
    return data


def tolerance(case):
    """About four times the distance from 64 bits that was measured: 2.2e-7 in the byte decoder (f32 throughout), 7.4e-6 in the experts (planes of 16 bits),
    2.1e-3 in the attention (bf16 queries and softmax weights).  Whole models reach 1e-3 to 1e-2 (bf16 keys, values, queries and weights in up to 16 layers); of
    that only the part that hangs on the order of sums may change.  Chosen tokens may differ where two logits are closer than that."""
    path = case["path"]
    if path == "experts":
        return {"rel": 3e-5, "max": 1e-3}
    if path == "attention":
        return {"rel": 8e-3, "max": 8e-2}
    if path == "decode" and case["model"] == "byte":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    return {"rel": 1e-2, "max": 1e-1, "differ": 0.01}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------------------------------------

F = torch.float64


def _silu(z):
    return z * torch.sigmoid(z)


def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _turned(x, positions, dims, base, pairs):
    """x [..., T, d] with its first `dims` entries turned by their positions: entry 2i with 2i + 1 (pairs), or i with i + dims / 2."""
    half = dims // 2
    angle = positions.to(F)[:, None] * float(base) ** (-2.0 * torch.arange(half, dtype=F, device=x.device) / dims)
    c, s = angle.cos(), angle.sin()
    out = x.clone()
    u, v = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, half), slice(half, dims))
    out[..., u] = x[..., u] * c - x[..., v] * s
    out[..., v] = x[..., v] * c + x[..., u] * s
    return out


def _causal(q, k, v, scale, past=0, chunk=None):
    """q [..., H, T, d], k and v [..., G, S, d]: position past + i sees the keys up to itself (of its own chunk)."""
    group = q.shape[-3] // k.shape[-3]
    k, v = k.repeat_interleave(group, -3), v.repeat_interleave(group, -3)
    score = q @ k.transpose(-1, -2) * scale
    i, j = torch.arange(q.shape[-2], device=q.device)[:, None] + past, torch.arange(k.shape[-2], device=q.device)[None]
    hidden = j > i
    if chunk:
        hidden = hidden | (i // chunk != j // chunk)
    return score.masked_fill_(hidden, -math.inf).softmax(-1) @ v


def _exact_decoder(case, seed):
    spec = DECODERS[case["model"]]
    D, H, G, eps = spec["d_model"], spec["heads"], spec["kv_heads"], spec["eps"]
    hd = D // H
    prompts, lengths, forced = _tokens(case, seed, spec["vocab"])
    batch, steps = case["batch"], len(forced)
    which = torch.arange(batch, device="cuda") % len(prompts)
    embedding = _decoder_weight(spec, 0).to(F)
    ids = torch.from_numpy(prompts).cuda()
    x = embedding[ids]
    y = embedding[torch.from_numpy(np.ascontiguousarray(forced.T)).cuda()]      # [batch, steps, D], after the prompts
    P = ids.shape[1]
    places = torch.arange(P, device="cuda"), torch.arange(steps, device="cuda") + P
    last = torch.from_numpy(lengths).cuda() - 1
    for i in range(spec["layers"]):
        wq, wk, wv, wo, gate, up, down, n1, n2 = (_decoder_weight(spec, 1 + 9 * i + j).to(F) for j in range(9))
        if spec.get("lora_rank"):
            qd, qu, vd, vu = (_adapter_weight(spec, i, j).to(F) for j in range(4))
            factor = spec["lora_alpha"] / spec["lora_rank"]
            wq, wv = wq + factor * qu @ qd, wv + factor * vu @ vd

        def heads(h, w, n, place):
            r = (h @ w.T).unflatten(-1, (n, hd)).transpose(-2, -3)
            return r if place is None else _turned(r, place, hd, spec["rope_base"], True)

        def finish(z, o):
            z = z + o.transpose(-2, -3).flatten(-2) @ wo.T
            h = _rms(z, eps) * n2
            return z + (_silu(h @ gate.T) * (h @ up.T)) @ down.T
        h = _rms(x, eps) * n1
        k, v = heads(h, wk, G, places[0]), heads(h, wv, G, None)
        attended = []
        for first in range(0, P, 512):      # in blocks of queries: a whole score matrix is large in 64 bits
            part = slice(first, min(P, first + 512))
            q = heads(h[:, part], wq, H, places[0][part])
            attended.append(torch.stack([_causal(a, b[:, :part.stop], c[:, :part.stop], hd ** -0.5, first) for a, b, c in zip(q, k, v)]))
        x = finish(x, torch.cat(attended, -2))
        if steps:
            h = _rms(y, eps) * n1
            q, ky, vy = heads(h, wq, H, places[1]), heads(h, wk, G, places[1]), heads(h, wv, G, None)
            o = [_causal(q[b], torch.cat([k[which[b]], ky[b]], -2), torch.cat([v[which[b]], vy[b]], -2), hd ** -0.5, P) for b in range(batch)]
            y = finish(y, torch.stack(o))
    end = y[:, -1] if steps else x[torch.arange(batch, device="cuda"), last]
    logits = (_rms(end, eps) * _decoder_weight(spec, 9 * spec["layers"] + 1).to(F)) @ embedding.T
    return {"chosen": None, "logits": logits} if case["path"] == "decode" else {"logits": logits}


def _whole_sequences(case, seed, vocab):
    """Prompt and forced tokens of every sequence side by side, padded behind, and the place of its last token."""
    prompts, lengths, forced = _tokens(case, seed, vocab)
    ids = np.zeros((len(prompts), prompts.shape[1] + len(forced)), dtype=np.int64)
    for row, prompt, n, more in zip(ids, prompts, lengths, forced.T):
        row[:n], row[n:n + len(more)] = prompt[:n], more
    return torch.from_numpy(ids).cuda(), torch.from_numpy(lengths).cuda() + len(forced) - 1


def _exact_mamba(h, w, p, m, eps):
    heads, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    inner, batch, T = heads * P, h.shape[0], h.shape[1]
    rows = h @ w(p + "in").T
    z, xbc, dt = rows[..., :inner], rows[..., inner:2 * inner + 2 * G * N], rows[..., 2 * inner + 2 * G * N:]
    taps = w(p + "conv")
    padded = torch.nn.functional.pad(xbc, (0, 0, taps.shape[1] - 1, 0))
    xbc = _silu(sum(taps[:, j] * padded[:, j:j + T] for j in range(taps.shape[1])) + w(p + "conv.b"))
    x = xbc[..., :inner].unflatten(-1, (heads, P))
    b, c = (v.unflatten(-1, (G, N)).repeat_interleave(heads // G, -2) for v in (xbc[..., inner:inner + G * N], xbc[..., inner + G * N:]))
    dt = torch.nn.functional.softplus(dt + w(p + "dt_bias"), threshold=60.0)
    decay = torch.exp(-torch.exp(w(p + "A_log")) * dt)
    x_dt = x * dt[..., None]
    state, y = torch.zeros((batch, heads, N, P), dtype=F, device=h.device), torch.empty_like(x)
    for t in range(T):
        state.mul_(decay[:, t, :, None, None]).add_(b[:, t, :, :, None] * x_dt[:, t, :, None, :])
        torch.matmul(c[:, t, :, None, :], state, out=y[:, t, :, None, :])
    y = (y + w(p + "D")[:, None] * x).flatten(-2) * _silu(z)
    return (_rms(y.unflatten(-1, (m["norm_groups"], -1)), eps).flatten(-2) * w(p + "norm")) @ w(p + "o").T


def _exact_latent(h, w, p, m, eps):
    H, d, r, e, K = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    place = torch.arange(h.shape[1], device=h.device)
    turned = lambda v: _turned(v, place, m["rot"]["dims"], m["rot"]["base"], True)
    q = (_rms(h @ w(p + "dq").T, eps) * w(p + "dq.norm") @ w(p + "uq").T).unflatten(-1, (H, d + r)).transpose(1, 2)
    low = h @ w(p + "dkv").T
    c = _rms(low[..., :K], eps) * w(p + "dkv.norm")
    k, v = ((c @ w(p + n).T).unflatten(-1, (H, -1)).transpose(1, 2) for n in ("uk", "uv"))
    q = torch.cat([q[..., :d], turned(q[..., d:])], -1)
    k = torch.cat([k, turned(low[..., K:])[:, None].expand(-1, H, -1, -1)], -1)
    o = torch.stack([_causal(*x, m["scale"]) for x in zip(q, k, v)]).transpose(1, 2).flatten(-2)
    return (o * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T


def _exact_chunked(h, w, p, m, eps):
    H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    place = torch.arange(h.shape[1], device=h.device)
    turned = lambda n, heads: _turned((_rms(h @ w(p + n).T, eps) * w(p + n + ".norm")).unflatten(-1, (heads, d)).transpose(1, 2), place, m["rot"]["dims"],
                                      m["rot"]["base"], False)
    q, k = turned("q", H), turned("k", G)
    v = (h @ w(p + "v").T).unflatten(-1, (G, e)).transpose(1, 2)
    o = torch.stack([_causal(*x, m["scale"], chunk=m["mask"]["size"]) for x in zip(q, k, v)]).transpose(1, 2)
    return (o * torch.sigmoid(h @ w(p + "g").T)[..., None]).flatten(-2) @ w(p + "o").T


def _exact_model(case, seed):
    hybrid = case["path"] == "hybrid"
    config = _hybrid() if hybrid else _parallel()
    order = {n: (i, s) for i, (n, s) in enumerate(_shapes(config).items())}
    w = lambda name: _named_weight(order[name][0], name, order[name][1]).to(F)
    norm = (lambda n, x: torch.tanh(w(n + ".alpha") * x) * w(n) + w(n + ".b")) if hybrid else (lambda n, x: _rms(x, eps) * w(n))
    eps = config["norm"]["eps"]
    ids, last = _whole_sequences(case, seed, config["vocab"])
    x = first = w("embed")[ids]
    loop = config.get("loop") or {"start": 0, "stop": 0, "times": 0}
    runs = [(i, False) for i in range(loop["start"])]
    for _ in range(loop["times"]):
        runs += [(i, i == loop["start"]) for i in range(loop["start"], loop["stop"])]
    for i, enters in runs + [(i, False) for i in range(loop["stop"], len(config["layers"]))]:
        layer = config["layers"][i]
        if enters:
            x = torch.cat([x, first], -1) @ w("loop.in").T
        dense = lambda h: (_silu(h @ w(f"l{i}.mlp.gate").T) * (h @ w(f"l{i}.mlp.up").T)) @ w(f"l{i}.mlp.down").T
        mix = {"mamba2": _exact_mamba, "latent_attention": _exact_latent, "attention": _exact_chunked}[layer["type"]]
        h = norm(f"l{i}.norm1", x)
        if hybrid:
            x = x + mix(h, w, f"l{i}.mix.", layer["mixer"], eps)
            x = x + dense(norm(f"l{i}.norm2", x))
        else:
            x = x + mix(h, w, f"l{i}.mix.", layer["mixer"], eps) + dense(h)
    end = norm("final.norm", x[torch.arange(len(ids), device="cuda"), last])
    return {"logits": end @ w("head").T * config.get("logit_scale", 1.0)}


def _exact_attention(case, seed):
    lengths, q, chunks = _attention_inputs(case, seed)
    n, G, d = case["batch"], case["kv_heads"], case["dim"]
    q = q.to(F).view(n, G, -1, d) * d ** -0.5
    ends = torch.from_numpy(lengths).cuda()[:, None, None, None]
    top, total, sums = q.new_full((n, G, q.shape[2], 1), -math.inf), 0.0, 0.0
    for i, (k, v) in enumerate(chunks):
        score = q @ k.to(F).transpose(-1, -2)
        score.masked_fill_(torch.arange(score.shape[-1], device="cuda") + 1024 * i >= ends, -math.inf)
        above = torch.maximum(top, score.amax(-1, keepdim=True))
        p, old = torch.exp(score - above), torch.exp(top - above)
        top, total, sums = above, total * old + p.sum(-1, keepdim=True), sums * old + p @ v.to(F)
    return {"attended": (sums / total).flatten(1, 2)}


def _exact_experts(case, seed):
    t = _expert_inputs(case, seed)
    logits, chosen = t["logits"].to(F).sort(dim=-1, descending=True, stable=True)
    weight, chosen = logits[:, :case["top"]].softmax(-1), chosen[:, :case["top"]]
    x, y = t["x"].to(F), t["residual"].to(F)
    for e in range(case["experts"]):
        row, place = (chosen == e).nonzero(as_tuple=True)
        up, down = t["up"][e].to(F), t["down"][e].to(F)
        h = x[row]
        y[row] += weight[row, place, None] * ((_silu(h @ up[0::2].T) * (h @ up[1::2].T)) @ down.T)
    return {"chosen": None, "weight": weight, "y": y}


def exact(case, seed):
    return {"decode": _exact_decoder, "prefill": _exact_decoder, "hybrid": _exact_model, "parallel": _exact_model, "attention": _exact_attention,
            "experts": _exact_experts}[case["path"]](case, seed)
