"""What a program that embeds this backend has it do, as timed cases: prompts, generated text, sampled text, the verify
step of speculative decoding and the scoring of a text, over the weight formats and layer families that are in use.

A case names a model shape, the format of its weights, an operation, the position it starts at (`context`) and its number
of tokens `n`. Each state has a session of its own, as a conversation has, already holding the conversation so far.
"""
import math
from dataclasses import replace

import numpy as np

from brisk_llm_b200 import formats as F
from brisk_llm_b200 import synth
from brisk_llm_b200.engine import CudaSession

SHAPES = {"qwen3-0.6b": synth.QWEN3_0_6B, "llama-3.2-1b": synth.LLAMA_3_2_1B, "bitnet-2b4t": synth.BITNET_2B,
          "mistral-7b": synth.MISTRAL_7B, "gemma3-1b": synth.GEMMA3_1B}
# The usual "medium" mixes of files keep the V and down projections and the embedding in Q6_K.
MEDIUM = {"v": F.Q6_K, "down": F.Q6_K, "embd": F.Q6_K}
WEIGHTS = {"Q4_0": (F.Q4_0, {}), "Q8_0": (F.Q8_0, {}), "Q4_K_M": (F.Q4_K, MEDIUM), "Q5_K_M": (F.Q5_K, MEDIUM), "TQ2_0": (F.TQ2_0, {"embd": F.F16})}
# Formats in which each shape is distributed (rows of 1152 values do not hold whole K-quant super-blocks).
IN_USE = {"qwen3-0.6b": ("Q4_0", "Q8_0", "Q4_K_M"), "llama-3.2-1b": ("Q4_K_M", "Q5_K_M", "Q8_0"), "bitnet-2b4t": ("TQ2_0",),
          "mistral-7b": ("Q4_0", "Q4_K_M"), "gemma3-1b": ("Q4_0", "Q8_0")}
TOP_K = 40  # candidates a sampler keeps


def listed():
    def case(name, model, weights, op, context, n):
        return {"name": name, "model": model, "weights": weights, "op": op, "context": context, "n": n}

    return [
        # The smallest calls: a greeting as the whole prompt, and one token of a chat whose host picks from the logits itself.
        case("short-prompt", "qwen3-0.6b", "Q4_0", "prompt", 0, 23),
        case("chat-token", "qwen3-0.6b", "Q4_0", "chat", 181, 1),
        # The headline workload in its two halves: a 512-token prompt, then greedy text after it.
        case("prompt", "qwen3-0.6b", "Q4_0", "prompt", 0, 512),
        case("generate", "qwen3-0.6b", "Q4_0", "greedy", 512, 32),
        # Perplexity of a text: log-likelihood, rows of logits for every token.
        case("score", "qwen3-0.6b", "Q8_0", "score", 0, 333),
        # A K-quant mix: a page of text as the prompt (ragged: the last batch is odd), then text after it.
        case("prompt-k-quant", "llama-3.2-1b", "Q4_K_M", "prompt", 0, 1023),
        case("generate-k-quant", "llama-3.2-1b", "Q4_K_M", "greedy", 1024, 32),
        # Ternary weights with an F16 head, sampled on the host from the device's best candidates.
        case("sample-ternary", "bitnet-2b4t", "TQ2_0", "sample", 517, 16),
        # Sliding-window layers, post-norms, GELU, heads of 256 values: text past the window.
        case("generate-sliding", "gemma3-1b", "Q4_0", "greedy", 700, 16),
        # The 7B class: a long document as the prompt, text at the end of a full context, and one speculative verify step
        # (the carried token and eight drafted ones).
        case("prompt-7b", "mistral-7b", "Q4_0", "prompt", 0, 4096),
        case("generate-7b", "mistral-7b", "Q4_0", "greedy", 8192, 16),
        case("verify-7b", "mistral-7b", "Q4_0", "verify", 2064, 9),
    ]


def _between(rng, low, high):
    """A whole number of [low, high], spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    model = rng.choice(sorted(SHAPES))
    op = rng.choice(["prompt", "chat", "greedy", "greedy", "sample", "verify", "score"])
    most = min(SHAPES[model].context, 4096 if op == "prompt" else 8192)
    n = {"prompt": lambda: _between(rng, 2, most - 1), "chat": lambda: _between(rng, 1, 8), "greedy": lambda: _between(rng, 8, 64),
         "sample": lambda: _between(rng, 4, 32), "verify": lambda: _between(rng, 2, 17), "score": lambda: _between(rng, 65, 512)}[op]()
    context = 0 if op in ("prompt", "score") else _between(rng, 24, most - 1 - n)
    return {"model": model, "weights": rng.choice(IN_USE[model]), "op": op, "context": context, "n": n}


# ---- models and sessions ----------------------------------------------------------------------------------------------

_models = {}  # (shape, weights) -> HostModel
_idle = {}    # (shape, weights) -> sessions whose state is gone: the next conversation takes one of them


def _spec(case):
    fmt, overrides = WEIGHTS[case["weights"]]
    return replace(SHAPES[case["model"]], name=case["model"] + "-" + case["weights"].lower(), fmt=fmt, fmt_overrides=overrides)


def _matrices(s):
    """role -> (tensor name, rows, cols) of one layer."""
    return {"q": ("attn_q", s.q_dim, s.hidden), "k": ("attn_k", s.kv_dim, s.hidden), "v": ("attn_v", s.kv_dim, s.hidden),
            "o": ("attn_output", s.hidden, s.q_dim), "gate": ("ffn_gate", s.ffn, s.hidden), "up": ("ffn_up", s.ffn, s.hidden),
            "down": ("ffn_down", s.hidden, s.ffn)}


def _host_model(spec):
    """Random weights of the shape: f32 ~N(0, 0.02) (ternary: uniform thirds) quantised by the package's encoders. Blocks are
    drawn from an encoded pool and the layers share their host tensors, which keeps building a 7B shape to a second; on the
    device every layer has weights of its own."""
    rng = np.random.default_rng(7)
    pools, t = {}, {}

    def matrix(fmt, rows, cols):
        unit = max(F.BLOCK_ELEMS[fmt], 32)
        if fmt not in pools:
            if fmt == F.TQ2_0:
                x = rng.integers(-1, 2, size=(1 << 20)).astype(np.float32) * np.float32(spec.std)
                x[::256] = np.float32(spec.std)  # every block holds a weight of full size: one scale for the tensor
            else:
                x = rng.standard_normal(1 << 20, dtype=np.float32) * np.float32(spec.std)
            pools[fmt] = np.ascontiguousarray(F.quantize(fmt, x)).view(np.uint8).reshape((1 << 20) // unit, -1)
        pool = pools[fmt]
        return fmt, (rows, cols), np.take(pool, rng.integers(0, len(pool), rows * (cols // unit)), axis=0).reshape(-1)

    def norm(n):
        return F.F32, (1, n), (1.0 + 0.05 * rng.standard_normal(n)).astype(np.float32)

    t["token_embd.weight"] = matrix(spec.fmt_of("embd"), spec.vocab, spec.hidden)
    if not spec.tied:
        t["output.weight"] = matrix(spec.fmt_of("output"), spec.vocab, spec.hidden)
    t["output_norm.weight"] = norm(spec.hidden)
    layer = {name + ".weight": matrix(spec.fmt_of(role), rows, cols) for role, (name, rows, cols) in _matrices(spec).items()}
    layer["attn_norm.weight"], layer["ffn_norm.weight"] = norm(spec.hidden), norm(spec.hidden)
    if spec.arch in ("qwen3", "gemma3"):
        layer["attn_q_norm.weight"], layer["attn_k_norm.weight"] = norm(spec.head_dim), norm(spec.head_dim)
    if spec.arch == "gemma3":
        layer["post_attention_norm.weight"], layer["post_ffw_norm.weight"] = norm(spec.hidden), norm(spec.hidden)
    if spec.arch == "bitnet":
        layer["attn_sub_norm.weight"], layer["ffn_sub_norm.weight"] = norm(spec.q_dim), norm(spec.ffn)
    for i in range(spec.layers):
        t.update({"blk.%d.%s" % (i, name): v for name, v in layer.items()})
    factors = None
    if spec.llama3_rope is not None:
        factors = synth.llama3_rope_factors(spec.head_dim, spec.rope_base, *spec.llama3_rope)
    return synth.HostModel(spec, t, factors)


class _State:
    """One conversation: a session and the tokens of its next call. The session serves another conversation afterwards."""

    def __init__(self, case, seed):
        self.case, self.key = case, (case["model"], case["weights"])
        for key in [k for k in _idle if k != self.key]:  # a program serves one model at a time
            for session in _idle.pop(key):
                session.close()
        waiting = _idle.get(self.key)
        if waiting:
            self.session = waiting.pop()
        else:
            if self.key not in _models:
                _models[self.key] = _host_model(_spec(case))
            self.session = CudaSession(_models[self.key])
        rng = np.random.default_rng([seed, 2])
        vocab = SHAPES[case["model"]].vocab
        self.tokens = rng.integers(0, vocab, case["n"] if case["op"] in ("prompt", "verify", "score") else 1, dtype=np.int32)
        self.uniform = rng.random(case["n"])  # the draws of a sampler
        self.session.rollback(0)
        if case["context"]:
            self.session.eval(rng.integers(0, vocab, case["context"], dtype=np.int32), copy=False)

    def __del__(self):
        if getattr(self, "session", None) is not None:
            _idle.setdefault(self.key, []).append(self.session)


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    s, case = state.session, state.case
    s.rollback(case["context"])  # where the call starts: back over what an earlier pass appended
    if case["op"] == "prompt":
        return s.eval(state.tokens)
    if case["op"] == "verify":
        return s.eval_all(state.tokens)
    if case["op"] == "score":
        return s.log_likelihood(state.tokens)
    if case["op"] == "greedy":
        return s.generate_greedy(int(state.tokens[0]), case["n"])
    token, out = int(state.tokens[0]), []
    if case["op"] == "chat":
        for _ in range(case["n"]):
            logits = s.eval([token])
            token = int(np.argmax(logits))
            out.append(logits)
        return out
    picked, values = [], []
    for u in state.uniform:  # sample: softmax over the best candidates, then one draw
        ids, best = s.eval_topk([token], TOP_K)
        share = np.exp(best.astype(np.float64) - float(best[0]))
        token = int(ids[min(int(np.searchsorted(np.cumsum(share), u * share.sum())), TOP_K - 1)])
        picked.append(ids)
        values.append(best)
    return {"ids": np.stack(picked), "values": np.stack(values)}


def work(case):
    """Weights once for each pass over them that depends on the one before (a generated token), cached keys and values read
    and written once, the logits that leave; two operations for each weight and token and for each cached value a query meets."""
    s, n, context = _spec(case), case["n"], case["context"]

    def sizes(role, rows, cols):
        return rows * F.row_bytes(s.fmt_of(role), cols), rows * cols

    per_layer = [sizes(role, rows, cols) for role, (_, rows, cols) in _matrices(s).items()]
    layer_bytes, layer_weights = s.layers * sum(b for b, _ in per_layer), s.layers * sum(w for _, w in per_layer)
    head_bytes, head_weights = sizes("embd" if s.tied else "output", s.vocab, s.hidden)
    serial = case["op"] in ("greedy", "chat", "sample")
    passes = n if serial else 1
    heads = {"prompt": 1}.get(case["op"], n)  # rows that meet the output head
    out_values = {"prompt": s.vocab, "chat": n * s.vocab, "verify": n * s.vocab, "sample": 2 * n * TOP_K}.get(case["op"], n)
    seen = written = read = 0  # (token, visible position) pairs; K/V rows written; K/V rows read
    for layer in range(s.layers):
        window = s.sliding_window if s.layer_slides(layer) else 1 << 30
        visible = [min(window, context + i + 1) for i in range(n)]
        seen += sum(visible)
        written += n
        read += sum(visible) if serial else min(context, window)
    kv_row = 2 * s.kv_dim * 2  # one position of keys and values, f16
    return {"bytes": passes * (layer_bytes + head_bytes) + (read + written) * kv_row + out_values * 4,
            "flops": 2 * (n * layer_weights + heads * head_weights) + 4 * seen * s.q_dim}


def tolerance(case):
    # The engine repeats the arithmetic of the CPU engine in its order: ids are equal, logits equal to 32-bit rounding.
    return {"rel": 1e-5}
