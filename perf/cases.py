"""The work that programs built on this library have it do, as measurable cases.

A case is either a whole encoder forward through the replay program (every kernel of the path
in the order a lowered BERT calls them) or one entry point of the runner-utils ABI at the sizes
the benchmark configurations name.  `listed()` names twelve of them, `draw()` makes more over
the same ranges, `prepare()` builds what a program holds before the call (weights, inputs,
descriptors), `run()` is the call.

Encoder cases cover both model sizes, one sequence to the largest batch, short, odd and the
longest sequences, full and ragged lengths, both weight layouts, and the three ways a program
is driven: CUDA-graph replay, plain calls (what a compiled model library does) and host buffers
in, host buffers out.
"""
from __future__ import annotations

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = "hands_on_mlir_b200"  # the directory's name has a hyphen: loaded by path


def _package():
    if _PACKAGE not in sys.modules:
        root = Path.cwd() / "hands-on-mlir_b200"
        spec = importlib.util.spec_from_file_location(_PACKAGE, root / "__init__.py",
                                                      submodule_search_locations=[str(root)])
        module = importlib.util.module_from_spec(spec)
        sys.modules[_PACKAGE] = module
        spec.loader.exec_module(module)
    return sys.modules[_PACKAGE]


def _program_module():
    _package()
    return importlib.import_module(_PACKAGE + ".bert_program")


_MODELS = {
    "base": dict(layers=12, hidden=768, heads=12, ffn=3072),
    "large": dict(layers=24, hidden=1024, heads=16, ffn=4096),
}
_VOCAB = 30522
_EPS = 1e-12


def _encoder(name, model, batch, seq, shortest, nk, mode):
    """Valid lengths are uniform in [shortest, seq]."""
    return dict(name=name, kind="encoder", model=model, batch=batch, seq=seq, shortest=shortest, nk=nk, mode=mode)


def listed():
    return [
        # one short query, latency: the smallest row of the benchmark grid, replayed as a graph
        _encoder("base_1x64_graph", "base", 1, 64, 64, False, "graph"),
        # one sentence padded to the sequence length, driven call by call like a compiled model
        _encoder("base_1x128_eager", "base", 1, 128, 12, False, "eager"),
        # a handful of odd-sized requests, weights stored [N, K]
        _encoder("base_5x77_ragged_nk", "base", 5, 77, 20, True, "graph"),
        # a small serving batch end to end: host token ids in, host hidden states out
        _encoder("base_8x128_host", "base", 8, 128, 128, False, "host"),
        # the configuration the throughput metric is quoted on
        _encoder("base_32x128_graph", "base", 32, 128, 128, False, "graph"),
        # a few paragraphs through the large model: several key tiles per query, small batch
        _encoder("large_6x384_ragged", "large", 6, 384, 150, False, "graph"),
        # the largest configuration: BERT-large, padded batch of 256 x 512
        _encoder("large_256x512_ragged", "large", 256, 512, 256, False, "graph"),
        # one fused GEMM + bias + GELU on batch 4 x seq 128 rows: a single call
        dict(name="gemm_bias_gelu_512", kind="gemm_gelu", m=512, n=3072, k=768),
        # residual add + affine LayerNorm on batch 32 x seq 128 rows
        dict(name="residual_layernorm_4096", kind="layernorm", rows=4096, hidden=768),
        # packed-QKV attention with padding, batch 32 x seq 128
        dict(name="attention_32x128", kind="attention", batch=32, seq=128, shortest=64, heads=12),
        # GEMM that also emits row statistics, then the GEMM that applies them to its input
        dict(name="gemm_stats_ln_gemm_4096", kind="ln_pair", m=4096, k=768, n=768, n2=3072),
        # vocabulary projection of the masked positions (20 in each of 32 sequences): N = 30522
        dict(name="vocab_projection_640", kind="vocab", m=640, n=_VOCAB, k=768),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["encoder"] * 5 + ["gemm_gelu", "layernorm", "attention", "ln_pair", "vocab"])
    if kind == "encoder":
        model = rng.choice(["base", "large"])
        seq = _log_int(rng, 16, 512)
        mode = rng.choice(["graph", "graph", "eager", "host"])
        # up to the largest listed case's tokens; a host step also moves its outputs
        most = {"graph": 256 * 512, "eager": 256 * 128, "host": 64 * 128}[mode]
        batch = _log_int(rng, 1, min(256, max(1, most // seq)))
        shortest = seq if rng.random() < 0.4 else max(1, int(seq * rng.uniform(0.1, 0.9)))
        case = _encoder("", model, batch, seq, shortest, rng.random() < 0.3, mode)
        del case["name"]
        return case
    model = _MODELS[rng.choice(["base", "large"])]
    rows = _log_int(rng, 16, 32768)
    if kind == "gemm_gelu":
        return dict(kind=kind, m=rows, n=model["ffn"], k=model["hidden"])
    if kind == "layernorm":
        return dict(kind=kind, rows=_log_int(rng, 16, 131072), hidden=model["hidden"])
    if kind == "attention":
        seq = _log_int(rng, 16, 512)
        batch = _log_int(rng, 1, max(1, min(256, 32768 // seq)))
        return dict(kind=kind, batch=batch, seq=seq, shortest=max(1, int(seq * rng.uniform(0.3, 1.0))),
                    heads=model["heads"])
    if kind == "ln_pair":
        return dict(kind=kind, m=rows, k=model["hidden"], n=model["hidden"], n2=rng.choice([3 * model["hidden"], model["ffn"]]))
    return dict(kind="vocab", m=_log_int(rng, 16, 2048), n=_VOCAB, k=model["hidden"])


class _DeviceResult:
    """A zero-copy tensor view of the program-owned fp16 result buffer (keeps the program alive)."""

    def __init__(self, program, memref):
        self.program = program
        self.__cuda_array_interface__ = {"shape": tuple(memref.shape), "typestr": "<f2", "version": 2,
                                         "data": (memref.data_ptr, False)}


class _Weight:
    """A GEMM weight declared constant for as long as this object lives."""

    def __init__(self, hom, tensor):
        self.hom, self.tensor = hom, tensor
        hom.declare_weights(tensor)

    def __del__(self):
        try:
            self.hom.forget_weights(self.tensor)
        except Exception:
            pass


_stream = None


def prepare(case, seed):
    global _stream
    hom = _package().runner()
    if _stream is None:
        _stream = torch.cuda.Stream()  # a program's own stream: the default one cannot be captured
    hom.set_stream(_stream.cuda_stream)
    gen, rng = _sources(seed)
    state = {"case": case, "hom": hom, "call": getattr(sys.modules[__name__], "_run_" + case["kind"])}
    getattr(sys.modules[__name__], "_prepare_" + case["kind"])(case, state, gen, rng)
    _stream.wait_stream(torch.cuda.current_stream())
    return state


def exact(case, seed):
    """What `run` returns for these inputs, in 64 bits with plain torch (no rounding in between)."""
    with torch.no_grad():
        return getattr(sys.modules[__name__], "_exact_" + case["kind"])(case, *_sources(seed))


def _sources(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen, np.random.default_rng(seed)


def run(state):
    return state["call"](state["hom"], state)


def _normal(gen, shape, std=1.0, mean=0.0):
    return torch.empty(shape, dtype=torch.float16, device="cuda").normal_(mean, std, generator=gen)


def _uniform(gen, shape):
    return torch.empty(shape, dtype=torch.float16, device="cuda").uniform_(-1, 1, generator=gen)


def _memref(tensor):
    """The descriptor a compiled program keeps for a buffer it calls with."""
    return _package().MemRef.of(tensor)


# ------------------------------------------------------------------------------- encoder

def _encoder_inputs(case, gen, rng):
    """Weights in call order, then token ids and mask on the host."""
    m = _MODELS[case["model"]]
    batch, seq, h, f = case["batch"], case["seq"], m["hidden"], m["ffn"]
    shapes = {"word_emb": (1, _VOCAB, h), "pos_emb": (1, seq, h), "type_emb": (1, 2, h)}
    for i in range(m["layers"]):
        for name, (k, n) in {"wqkv": (h, 3 * h), "wo": (h, h), "w1": (h, f), "w2": (f, h)}.items():
            shapes[f"{name}_{i}"] = (1, n, k) if case["nk"] else (1, k, n)
    weights = {name: _normal(gen, shape, 0.02) for name, shape in shapes.items()}
    ids = rng.integers(1000, _VOCAB, (batch, seq)).astype(np.int64)
    lengths = rng.integers(case["shortest"], seq + 1, batch)
    mask = (np.arange(seq)[None, :] < lengths[:, None]).astype(np.int64)
    return weights, ids, mask


def _prepare_encoder(case, state, gen, rng):
    mod = _program_module()
    cfg = mod.BertConfig(vocab=_VOCAB, type_vocab=2, eps=_EPS, **_MODELS[case["model"]])
    batch, seq = case["batch"], case["seq"]
    weights, ids, mask = _encoder_inputs(case, gen, rng)
    program = mod.BertProgram(cfg, batch, seq, weights_nk=case["nk"])
    program.set_weights(weights)
    inputs = [torch.from_numpy(x) for x in (ids, mask, np.zeros_like(ids))]
    if case["mode"] == "host":
        state["inputs"] = [x.pin_memory() for x in inputs]
        state["out"] = torch.empty((batch, seq, cfg.hidden), dtype=torch.float16).pin_memory()
    else:
        state["inputs"] = [x.cuda() for x in inputs]
    state["program"] = program


def _run_encoder(hom, state):
    program, mode = state["program"], state["case"]["mode"]
    if mode == "host":
        program.forward_host(*state["inputs"], state["out"], use_graph=True)
        return state["out"]
    memref = program.forward(*state["inputs"], use_graph=mode == "graph")
    return torch.as_tensor(_DeviceResult(program, memref), device="cuda")


def _exact_encoder(case, gen, rng):
    weights, ids, mask = _encoder_inputs(case, gen, rng)
    m = _MODELS[case["model"]]

    def matrix(name):
        w = weights[name][0].double()
        return w.t() if case["nk"] else w

    valid = torch.from_numpy(mask.astype(bool)).cuda()
    ids = torch.from_numpy(ids).cuda()
    x = weights["word_emb"][0][ids].double() + weights["type_emb"][0][0].double() + weights["pos_emb"][0].double()
    x = _layernorm64(x, _EPS)
    for i in range(m["layers"]):
        qkv = x @ matrix(f"wqkv_{i}")
        x = _layernorm64(_attention64(qkv, valid, m["heads"]) @ matrix(f"wo_{i}") + x, _EPS)
        del qkv
        hidden = x @ matrix(f"w1_{i}")
        x = _layernorm64(torch.nn.functional.gelu(hidden) @ matrix(f"w2_{i}") + x, _EPS)
    return x


def _layernorm64(x, eps):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], eps=eps)


def _attention64(qkv, valid, heads):
    """Keys of padding are left out, query rows of padding are zero; a few sequences at a time."""
    batch, seq, _ = qkv.shape
    out = torch.zeros((batch, seq, heads * 64), dtype=torch.float64, device=qkv.device)
    step = max(1, (1 << 28) // (heads * seq * seq))
    for lo in range(0, batch, step):
        part = qkv[lo:lo + step].reshape(-1, seq, 3, heads, 64)
        q, k, v = (part[:, :, i].transpose(1, 2) for i in range(3))
        here = valid[lo:lo + step]
        scores = (q @ k.transpose(-1, -2) * 0.125).masked_fill(~here[:, None, None, :], float("-inf"))
        rows = (torch.softmax(scores, -1) @ v).transpose(1, 2).reshape(-1, seq, heads * 64)
        out[lo:lo + step] = rows * here[:, :, None]
    return out


# ---------------------------------------------------------------------- single entry points

def _gemm_gelu_inputs(case, gen, rng):
    m, n, k = case["m"], case["n"], case["k"]
    return _normal(gen, (1, k, n), 0.02), _uniform(gen, (1, m, k)), _uniform(gen, (1, 1, n))


def _prepare_gemm_gelu(case, state, gen, rng):
    weight, x, bias = _gemm_gelu_inputs(case, gen, rng)
    state["weight"] = _Weight(state["hom"], weight)
    state["out"] = torch.empty((1, case["m"], case["n"]), dtype=torch.float16, device="cuda")
    state["args"] = [_memref(t) for t in (x, weight, bias, state["out"])]


def _run_gemm_gelu(hom, state):
    hom.cutlassGemmF16(*state["args"], activation=1, alpha=1.0, beta=1.0)
    return state["out"]


def _exact_gemm_gelu(case, gen, rng):
    weight, x, bias = (t.double() for t in _gemm_gelu_inputs(case, gen, rng))
    return torch.nn.functional.gelu(x @ weight + bias)


def _layernorm_inputs(case, gen, rng):
    rows, hidden = case["rows"], case["hidden"]
    return (_normal(gen, (1, rows, hidden)), _normal(gen, (1, rows, hidden)), _normal(gen, (hidden,), 0.1, 1.0),
            _normal(gen, (hidden,), 0.1))


def _prepare_layernorm(case, state, gen, rng):
    inputs = _layernorm_inputs(case, gen, rng)
    state["out"] = torch.empty_like(inputs[0])
    state["args"] = [_memref(t) for t in (*inputs, state["out"])]


def _run_layernorm(hom, state):
    hom.homResidualLayernormF16(*state["args"], eps=_EPS)
    return state["out"]


def _exact_layernorm(case, gen, rng):
    x, residual, gamma, beta = (t.double() for t in _layernorm_inputs(case, gen, rng))
    return torch.nn.functional.layer_norm(x + residual, x.shape[-1:], gamma, beta, eps=_EPS)


def _attention_inputs(case, gen, rng):
    batch, seq, heads = case["batch"], case["seq"], case["heads"]
    lengths = rng.integers(case["shortest"], seq + 1, batch)
    return lengths, _normal(gen, (batch, seq, 3 * heads * 64))


def _prepare_attention(case, state, gen, rng):
    lengths, qkv = _attention_inputs(case, gen, rng)
    batch, seq, heads = case["batch"], case["seq"], case["heads"]
    cu = torch.from_numpy(np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)).cuda()
    state["out"] = torch.empty((batch, seq, heads * 64), dtype=torch.float16, device="cuda")
    state["args"] = [_memref(t) for t in (qkv, cu, state["out"])]
    state["heads"] = heads


def _run_attention(hom, state):
    hom.nvteBertAttentionF16(*state["args"], 0.125, state["heads"])
    return state["out"]


def _exact_attention(case, gen, rng):
    lengths, qkv = _attention_inputs(case, gen, rng)
    valid = torch.from_numpy(np.arange(case["seq"])[None, :] < lengths[:, None]).cuda()
    return _attention64(qkv.double(), valid, case["heads"])


def _ln_pair_inputs(case, gen, rng):
    m, k, n, n2 = case["m"], case["k"], case["n"], case["n2"]
    return (_normal(gen, (1, k, n), 0.02), _normal(gen, (1, n, n2), 0.02), _normal(gen, (1, m, n)),
            _normal(gen, (1, 1, n2), 0.1), _normal(gen, (1, m, k)))


def _prepare_ln_pair(case, state, gen, rng):
    m, n, n2 = case["m"], case["n"], case["n2"]
    half = dict(dtype=torch.float16, device="cuda")
    first, second, residual, bias, x = _ln_pair_inputs(case, gen, rng)
    state["weights"] = [_Weight(state["hom"], first), _Weight(state["hom"], second)]
    state["outs"] = [torch.empty((1, m, n), **half), torch.empty((m,), **half), torch.empty((m,), **half),
                     torch.empty((1, m, n2), **half)]
    hidden, var, mean, out = (_memref(t) for t in state["outs"])
    state["first"] = [_memref(x), _memref(first), _memref(residual), hidden, var, mean]
    state["second"] = [hidden, _memref(second), _memref(bias), out, var, mean]


def _run_ln_pair(hom, state):
    hom.cutlassGemmWithVarMeanF16(*state["first"], alpha=1.0, beta=1.0, eps=1e-5)
    hom.cutlassLayernormGemmF16(*state["second"], alpha=1.0, beta=1.0)
    return state["outs"]


def _exact_ln_pair(case, gen, rng):
    """The statistics travel as 1/std and -mean/std."""
    first, second, residual, bias, x = (t.double() for t in _ln_pair_inputs(case, gen, rng))
    hidden = x @ first + residual
    mean = hidden.mean(-1, keepdim=True)
    rstd = ((hidden - mean).square().mean(-1, keepdim=True) + 1e-5).rsqrt()
    return [hidden, rstd.reshape(-1), (-mean * rstd).reshape(-1), (hidden - mean) * rstd @ second + bias]


def _vocab_inputs(case, gen, rng):
    m, n, k = case["m"], case["n"], case["k"]
    return _normal(gen, (1, k, n), 0.02), _normal(gen, (1, m, k)), _normal(gen, (1, 1, n), 0.02)


def _prepare_vocab(case, state, gen, rng):
    weight, x, bias = _vocab_inputs(case, gen, rng)
    state["weight"] = _Weight(state["hom"], weight)
    state["out"] = torch.empty((1, case["m"], case["n"]), dtype=torch.float16, device="cuda")
    state["args"] = [_memref(t) for t in (x, weight, bias, state["out"])]


def _run_vocab(hom, state):
    hom.cutlassGemmF16(*state["args"], activation=0, alpha=1.0, beta=1.0)
    return state["out"]


def _exact_vocab(case, gen, rng):
    weight, x, bias = (t.double() for t in _vocab_inputs(case, gen, rng))
    return x @ weight + bias


# ------------------------------------------------------------------------ work and tolerance

def _gemm_flops(m, n, k):
    return 2.0 * m * n * k


def _mean_pairs(shortest, seq):
    """Expected query x key pairs of one sequence whose length is uniform in [shortest, seq]."""
    lengths = np.arange(shortest, seq + 1, dtype=np.float64)
    return float((lengths ** 2).mean())


def work(case):
    """Bytes: every input and weight read once, every output written once.  Operations: the
    contractions, attention over valid query x key pairs only."""
    kind = case["kind"]
    if kind == "encoder":
        m = _MODELS[case["model"]]
        h, f, layers = m["hidden"], m["ffn"], m["layers"]
        tokens = case["batch"] * case["seq"]
        flops = layers * _gemm_flops(tokens, 4 * h + 2 * f, h)
        flops += layers * 4.0 * h * case["batch"] * _mean_pairs(case["shortest"], case["seq"])
        weights = 2.0 * (layers * (4 * h * h + 2 * h * f) + case["seq"] * h + 2 * h)
        words = 2.0 * h * min(tokens, _VOCAB)
        return {"bytes": weights + words + 24.0 * tokens + 2.0 * tokens * h, "flops": flops}
    if kind == "layernorm":
        return {"bytes": 2.0 * (3 * case["rows"] * case["hidden"] + 2 * case["hidden"]), "flops": 0.0}
    if kind == "attention":
        h = 64 * case["heads"]
        return {"bytes": 2.0 * 4 * case["batch"] * case["seq"] * h + 4.0 * (case["batch"] + 1),
                "flops": 4.0 * h * case["batch"] * _mean_pairs(case["shortest"], case["seq"])}
    m, n, k = case["m"], case["n"], case["k"]
    if kind == "ln_pair":
        n2 = case["n2"]
        return {"bytes": 2.0 * (m * k + k * n + 2 * m * n + n * n2 + n2 + m * n2 + 2 * m),
                "flops": _gemm_flops(m, n, k) + _gemm_flops(m, n2, n)}
    return {"bytes": 2.0 * (m * k + k * n + n + m * n), "flops": _gemm_flops(m, n, k)}


def tolerance(case):
    """Four times what the path differs from a 64-bit evaluation of the same inputs: encoders
    1.4e-3 (largest element 9e-3, roundings of 12 or 24 layers), single calls 2e-4 to 3.3e-4
    (largest element 1.5e-3)."""
    return {"rel": 6e-3, "max": 4e-2} if case["kind"] == "encoder" else {"rel": 1.5e-3, "max": 6e-3}
