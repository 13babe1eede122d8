"""Workloads by which the speed of this package is judged on one GPU.

Each case is one call (or one serving step) a program makes through the public entry points: an
all-reduce of a symmetric tensor, a decode GEMV, a projection GEMM, the prefill of a decoder layer and
a decode step through a stack of layers.  With one process the collectives are a world of one: what is
left is the rank's own part, which every rank of a larger world runs as well.  The layers are one rank's
share of the Llama-3-70B layer under tensor parallelism (`LlamaTPConfig.llama3_70b`, divided by 8 or 4).
`listed()` are the fixed cases, `draw(rng)` gives others of the same ranges.
"""
import functools
import math

import torch

import symm_mem_recipes_b200 as smr
from symm_mem_recipes_b200.models.llama_tp_layer import DecodeGraph, LlamaTPConfig, LlamaTPDecoderLayer, new_kv_caches
from symm_mem_recipes_b200.ops import interleave_gate_up
from symm_mem_recipes_b200.parallel import symm_mem


def listed():
    return [
        # one-shot all-reduce of 8192 elements, the size of the upstream correctness test: pure call latency
        {"name": "all_reduce_16KiB", "kind": "all_reduce", "numel": 8192},
        # the message size at which bus bandwidth is quoted
        {"name": "all_reduce_64MiB", "kind": "all_reduce", "numel": 1 << 25},
        # decode, one sequence: column-parallel QKV projection of a rank at TP8 (weight stored [N, K])
        {"name": "gemv_qkv_b1", "kind": "gemv", "batch": 1, "n": 1280, "k": 8192, "nk": True},
        # decode, full batch: row-parallel down projection of a rank at TP8 (weight stored [K, N])
        {"name": "gemv_down_b16", "kind": "gemv", "batch": 16, "n": 8192, "k": 3584, "nk": False},
        # a short, ragged prompt: o-projection of a rank at TP8
        {"name": "project_o_m129", "kind": "project", "m": 129, "n": 8192, "k": 1024, "dtype": "bf16", "swiglu": False},
        # a chunk of a prompt through the gate / up projection with the activation in the epilogue
        {"name": "project_swiglu_m2048", "kind": "project", "m": 2048, "n": 7168, "k": 8192, "dtype": "bf16",
         "swiglu": True},
        # the fp8 form (A, B and C in e4m3) of the up projection
        {"name": "project_fp8_m4096", "kind": "project", "m": 4096, "n": 3584, "k": 8192, "dtype": "fp8",
         "swiglu": False},
        # the headline shape: up projection at TP8 over all 16384 tokens
        {"name": "project_up_m16384", "kind": "project", "m": 16384, "n": 3584, "k": 8192, "dtype": "bf16",
         "swiglu": False},
        # a single ragged prompt through one layer into its KV cache
        {"name": "prefill_1x509", "kind": "prefill", "tp": 8, "batch": 1, "seq": 509},
        # the prefill the layer benchmark times: batch 16 x 2048 tokens
        {"name": "prefill_16x2048", "kind": "prefill", "tp": 8, "batch": 16, "seq": 2048},
        # serving: one token for one sequence, two layers replayed from one CUDA graph
        {"name": "decode_b1", "kind": "decode", "tp": 8, "batch": 1, "max_seq": 4096, "pos": 3000, "graph": True},
        # serving: one token for a full batch with long contexts
        {"name": "decode_b16", "kind": "decode", "tp": 8, "batch": 16, "max_seq": 8192, "pos": 6500, "graph": True},
    ]


def _log_int(rng, lo, hi, step=1):
    """An integer in [lo, hi], uniform in its logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(step, min(hi // step, round(v / step)) * step)


def draw(rng):
    kind = rng.choice(("all_reduce", "gemv", "gemv", "project", "project", "prefill", "prefill", "decode", "decode"))
    if kind == "all_reduce":
        # 4 KiB to 64 MiB; 16-byte vectors are the only granularity asked of a caller
        return {"kind": kind, "numel": _log_int(rng, 2048, 1 << 25, 8)}
    if kind == "gemv":
        return {"kind": kind, "batch": rng.randint(1, 16), "n": _log_int(rng, 512, 16384, 8),
                "k": _log_int(rng, 512, 8192, 8), "nk": rng.random() < 0.5}
    if kind == "project":
        dtype = "fp8" if rng.random() < 0.25 else "bf16"
        swiglu = dtype == "bf16" and rng.random() < 0.3
        return {"kind": kind, "m": _log_int(rng, 17, 16384), "n": _log_int(rng, 512, 8192, 256 if swiglu else 16),
                "k": _log_int(rng, 512, 8192, 16), "dtype": dtype, "swiglu": swiglu}
    tp = rng.choice((8, 4))
    if kind == "prefill":
        batch = _log_int(rng, 1, 16)
        return {"kind": kind, "tp": tp, "batch": batch, "seq": _log_int(rng, 33, min(2048, 2048 * tp // batch))}
    max_seq = _log_int(rng, 256, 8192)
    return {"kind": kind, "tp": tp, "batch": rng.randint(1, 16), "max_seq": max_seq,
            "pos": rng.randint(max_seq // 2, max_seq - 1), "graph": rng.random() < 0.75}


_DECODE_LAYERS = 2


def _share(tp):
    """One rank's share of the 70B layer, as a layer of its own."""
    full = LlamaTPConfig.llama3_70b()
    return LlamaTPConfig(hidden=full.hidden, n_heads=full.n_heads // tp, n_kv_heads=full.n_kv_heads // tp,
                         head_dim=full.head_dim, ffn=full.ffn // tp)


@functools.lru_cache(maxsize=None)
def _layer(tp, index):
    """A program loads its weights once and serves every request with them."""
    return LlamaTPDecoderLayer(_share(tp), torch.device("cuda", torch.cuda.current_device()), seed=1 + 1000 * index)


def _normal(gen, *shape, std=1.0):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.bfloat16).mul_(std)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "all_reduce":
        t = symm_mem.empty(case["numel"], dtype=torch.bfloat16, device="cuda")
        t.copy_(_normal(gen, case["numel"]))
        symm_mem.rendezvous(t)
        return kind, t
    if kind == "gemv":
        n, k = case["n"], case["k"]
        w = _normal(gen, *((n, k) if case["nk"] else (k, n)), std=0.02)
        return kind, _normal(gen, case["batch"], k), w, case["nk"]
    if kind == "project":
        a, b = _normal(gen, case["m"], case["k"]), _normal(gen, case["n"], case["k"], std=0.02)
        if case["swiglu"]:
            return kind, a, interleave_gate_up(b[: case["n"] // 2], b[case["n"] // 2:]), "swiglu"
        if case["dtype"] == "fp8":
            # e4m3 has no scale factors here: weights are kept in the range of its normal numbers
            return kind, a.to(torch.float8_e4m3fn), (b * 4).to(torch.float8_e4m3fn), None
        return kind, a, b, None
    if kind == "prefill":
        layer, batch, seq = _layer(case["tp"], 0), case["batch"], case["seq"]
        x = _normal(gen, batch * seq, layer.cfg.hidden, std=0.5)
        return kind, layer, x, batch, seq, new_kv_caches([layer], batch, seq + 64)[0]
    layers = [_layer(case["tp"], i) for i in range(_DECODE_LAYERS)]
    x = _normal(gen, case["batch"], layers[0].cfg.hidden, std=0.5)
    if case["graph"]:
        graph = DecodeGraph(layers, case["batch"], case["max_seq"])
        caches = graph.caches
    else:
        graph, caches = None, new_kv_caches(layers, case["batch"], case["max_seq"])
    for kc, vc in caches:           # the context: keys and values of the positions before `pos`
        for t in (kc, vc):
            t[:, : case["pos"]] = _normal(gen, case["batch"], case["pos"], *t.shape[2:])
    return kind, layers, graph, x, case["pos"], caches


def run(state):
    kind = state[0]
    if kind == "all_reduce":
        return smr.one_shot_all_reduce(state[1])
    if kind == "gemv":
        _, x, w, nk = state
        # row-parallel weights ([K, N]) end in the all-reduce, column-parallel ones ([N, K]) are rank-local
        return smr.gemv(x, w, weights_nk=True) if nk else smr.gemv_all_reduce(x, w)
    if kind == "project":
        _, a, b, epilogue = state
        return smr.all_gather_matmul(a, b, epilogue=epilogue)
    if kind == "prefill":
        _, layer, x, batch, seq, cache = state
        return layer.forward(x, batch, seq, kv_cache=cache), cache
    _, layers, graph, x, pos, caches = state
    if graph is not None:
        return graph.step(x, pos), caches
    h = x
    for layer, (kc, vc) in zip(layers, caches):
        h = layer.decode(h, kc, vc, pos)
    return h, caches


def _layer_elements(cfg):
    """Weights of a layer, in elements."""
    d, h = cfg.head_dim, cfg.hidden
    return h * ((cfg.n_heads + 2 * cfg.n_kv_heads) * d + cfg.n_heads * d + 3 * cfg.ffn)


def work(case):
    kind = case["kind"]
    if kind == "all_reduce":
        return {"bytes": 4 * case["numel"], "flops": 0}
    if kind == "gemv":
        b, n, k = case["batch"], case["n"], case["k"]
        return {"bytes": 2 * (n * k + b * k + b * n), "flops": 2 * b * n * k}
    if kind == "project":
        m, n, k = case["m"], case["n"], case["k"]
        size = 1 if case["dtype"] == "fp8" else 2
        return {"bytes": size * (m * k + n * k + m * (n // 2 if case["swiglu"] else n)), "flops": 2 * m * n * k}
    cfg, b = _share(case["tp"]), case["batch"]
    weights, kv_row = _layer_elements(cfg), 2 * cfg.n_kv_heads * cfg.head_dim
    if kind == "prefill":
        s = case["seq"]
        attention = 2 * b * s * (s + 1) * cfg.n_heads * cfg.head_dim          # causal: half of the square, QK and PV
        return {"bytes": 2 * (weights + 2 * b * s * cfg.hidden + b * s * kv_row), "flops": 2 * b * s * weights + attention}
    seen = case["pos"] + 1
    return {"bytes": 2 * (_DECODE_LAYERS * (weights + b * seen * kv_row) + 2 * b * cfg.hidden),
            "flops": _DECODE_LAYERS * (2 * b * weights + 4 * b * seen * cfg.n_heads * cfg.head_dim)}


def tolerance(case):
    kind = case["kind"]
    if kind == "all_reduce":
        return "exact"                       # a sum over one rank in a fixed order
    if kind in ("gemv", "project"):
        # fp32 sums in another order, then one rounding to bf16 (or e4m3, where a flipped rounding is 2^-3)
        return {"rel": 1e-2 if case.get("dtype") == "fp8" else 4e-3, "max": 0.15 if case.get("dtype") == "fp8" else 0.04}
    return {"rel": 1e-2}                     # a chain of bf16 tensors between the kernels
