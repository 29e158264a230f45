"""The work that users of this library have it do, as cases that can be timed and compared.

Each case is a dict of plain values. ``prepare`` builds what a user's program holds before the call (a context, registered
weights, a model, inputs on the device), ``run`` makes the calls, ``work`` counts the bytes and operations that the path
cannot do without, ``tolerance`` says how far two correct implementations may differ.

Kinds of cases:

``linear``    one GPTQ int4 projection through ``QwenGpt.gemm``: any K, N, group size and number of rows.
``layer``     the seven projections of one transformer layer (q, k, v, o, gate, up, down) of a 0.5B- or 7B-shaped model, called
              one by one or recorded once as a command batch and submitted.
``dequant``   ``dequantize_gptq_int4``: packed host tensors in, the dense host matrix out.
``prefill``   a prompt through the whole 24-layer 0.5B-shaped model, logits of its last row or of all rows.
``score``     a prompt, then given tokens one at a time with every logits row read back (scoring a continuation, constrained
              decoding, a host program's own sampler).
``greedy``    ``generate_qwen`` at temperature 0: the decode loop stays on the device.
``sampled``   ``generate_qwen`` with temperature, top-k and top-p.
``forward``   ``QwenGpt.forward``: B sequences of T tokens without a cache, all logits (evaluation).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from webllm_b200 import GptqInt4Params, Gpu, QwenGpt, SamplerOptions, dequantize_gptq_int4, generate_qwen
from webllm_b200.synthetic import QWEN05B_SHAPES, QWEN25_05B, QWEN7B_SHAPES, GptqTensors

LAYERS = {"0.5b": QWEN05B_SHAPES, "7b": QWEN7B_SHAPES}
MB = 1 << 20


def listed():
    return [
        # one up projection at decode: the smallest call there is, where host time and launch latency count
        {"name": "up_05b_m1", "kind": "linear", "K": 896, "N": 4864, "M": 1, "group": 128, "act": "f32", "bias": False, "exact": False},
        # a ragged matrix in the fp32-activation mode, as a parity check of a small model runs it
        {"name": "ragged_exact_m145", "kind": "linear", "K": 1000, "N": 1236, "M": 145, "group": 128, "act": "f32", "bias": True,
         "exact": True},
        # four sequences decoded together, the layer recorded once and replayed
        {"name": "layer_05b_m4_recorded", "kind": "layer", "model": "0.5b", "M": 4, "act": "f16", "recorded": True},
        # decode of a larger model: bound by the weights
        {"name": "layer_7b_m1", "kind": "layer", "model": "7b", "M": 1, "act": "f16", "recorded": False},
        # a served batch of a larger model
        {"name": "layer_7b_m24", "kind": "layer", "model": "7b", "M": 24, "act": "f32", "recorded": False},
        # a long prefill of a larger model: bound by the tensor cores
        {"name": "layer_7b_m4096", "kind": "layer", "model": "7b", "M": 4096, "act": "f16", "recorded": False},
        # a dense copy of one projection for inspection or for another engine
        {"name": "dequant_up_05b", "kind": "dequant", "K": 896, "N": 4864, "group": 128, "dtype": "f32"},
        # a long document before the first token
        {"name": "prefill_2048", "kind": "prefill", "n": 2048, "last_only": True, "kv": "f16"},
        # a few-shot prompt and the continuation that is scored against it
        {"name": "score_512_16", "kind": "score", "n": 512, "steps": 16, "kv": "f16"},
        # a short question and a greedy answer
        {"name": "greedy_8_128", "kind": "greedy", "n": 8, "new": 128, "kv": "f16"},
        # the same with a chat program's sampler
        {"name": "sampled_6_8", "kind": "sampled", "n": 6, "new": 8, "temperature": 0.8, "top_k": 40, "top_p": 0.95, "kv": "f32"},
        # a batch of evaluation sequences
        {"name": "forward_4x101", "kind": "forward", "B": 4, "T": 101, "kv": "f32"},
    ]


def _log_int(rng: random.Random, lo: int, hi: int, step: int = 1) -> int:
    """A multiple of ``step`` between lo and hi, spread evenly over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // step * step, max(-(-lo // step) * step, round(v / step) * step))


def draw(rng: random.Random):
    kind = rng.choice(["linear", "linear", "linear", "layer", "layer", "dequant", "prefill", "score", "greedy", "sampled", "forward"])
    kv = rng.choice(["f16", "f32"])
    if kind == "linear":
        exact = rng.random() < 0.2
        K = _log_int(rng, 256, 8192, 8 if rng.random() < 0.3 else 128)
        N = _log_int(rng, 128, 19456, 8)
        group = rng.choice([64, 128, 128])
        # the fp32-activation mode and K that is no multiple of 64 are for small matrices and few rows
        most = 2 ** 28 if exact or K % 64 else 2 ** 36
        M = _log_int(rng, 1, max(1, min(4096, most // (K * N))))
        return {"kind": kind, "K": K, "N": N, "M": M, "group": group, "act": "f32" if exact else rng.choice(["f16", "f32"]),
                "bias": rng.random() < 0.4, "exact": exact}
    if kind == "layer":
        model = rng.choice(["0.5b", "7b"])
        return {"kind": kind, "model": model, "M": _log_int(rng, 1, 4096), "act": rng.choice(["f16", "f32"]),
                "recorded": rng.random() < 0.3}
    if kind == "dequant":
        return {"kind": kind, "K": _log_int(rng, 256, 4864, 8), "N": _log_int(rng, 128, 4864, 8), "group": rng.choice([32, 64, 128]),
                "dtype": rng.choice(["f32", "f16"])}
    if kind == "prefill":
        last_only = rng.random() < 0.7
        return {"kind": kind, "n": _log_int(rng, 3, 2048 if last_only else 384), "last_only": last_only, "kv": kv}
    if kind == "score":
        return {"kind": kind, "n": _log_int(rng, 16, 1500), "steps": rng.randint(4, 24), "kv": kv}
    if kind == "greedy":
        return {"kind": kind, "n": rng.randint(2, 8), "new": _log_int(rng, 16, 160), "kv": kv}
    if kind == "sampled":
        return {"kind": kind, "n": rng.randint(2, 8), "new": rng.randint(3, 8), "temperature": round(rng.uniform(0.6, 1.2), 2),
                "top_k": _log_int(rng, 10, 60), "top_p": rng.choice([1.0, 0.95, 0.9]), "kv": kv}
    B = rng.randint(1, 6)
    return {"kind": "forward", "B": B, "T": _log_int(rng, 12, 400 // B), "kv": kv}


# ---------------------------------------------------------------------------------------------------- inputs
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _gptq(K: int, N: int, group: int, g: torch.Generator, std: float = 0.02) -> GptqTensors:
    """One projection in checkpoint layout: nibbles distributed as those of a round-to-nearest quantised normal weight,
    stored zero points 7 and 8, scales that make the weight's standard deviation ``std``. Made on the GPU, held on the host."""
    rows, groups, cols = -(-K // 8), -(-K // group), -(-N // 8)
    q = torch.randn(rows, 8, N, device="cuda", generator=g).mul_(2.8).add_(8).round_().clamp_(0, 15).to(torch.int32)
    words = torch.zeros(rows, N, dtype=torch.int32, device="cuda")
    for j in range(8):
        words |= q[:, j] << (4 * j)
    z = torch.randint(7, 9, (groups, cols, 8), device="cuda", generator=g, dtype=torch.int32)
    zeros = torch.zeros(groups, cols, dtype=torch.int32, device="cuda")
    for j in range(8):
        zeros |= z[:, :, j] << (4 * j)
    scales = (torch.randn(groups, N, device="cuda", generator=g) * 0.1 + 1).abs_().mul_(std / 2.8).half()
    return GptqTensors(words.cpu().numpy(), zeros.cpu().numpy(), scales.cpu().numpy(), K, N, group)


class _State:
    """What one program holds: the context over an activation slab that is a torch tensor, the model object, the inputs."""

    def __init__(self, weight_bytes: int, act_bytes: int):
        self.slab = torch.empty(act_bytes, dtype=torch.uint8, device="cuda")
        self.gpu = Gpu(0, weight_bytes=weight_bytes, act_slab=(self.slab.data_ptr(), act_bytes))
        self.model = self.batch = None

    def view(self, t):
        """The device tensor behind a handle of the library."""
        flat = self.slab[t.offset:t.offset + t.nbytes].view(torch.float32 if t.dtype == "f32" else torch.float16)
        return flat.view(t.shape)

    def __del__(self):
        if self.batch is not None:
            self.batch.destroy()
        if self.model is not None:
            self.model.close()
        self.gpu.close()


def _shapes(case):
    return LAYERS[case["model"]] if case["kind"] == "layer" else {"w": (case["K"], case["N"])}


def _prepare_linear(case, seed):
    g, shapes, M, act = _gen(seed), _shapes(case), case["M"], case["act"]
    group, size = case.get("group", 128), 4 if act == "f32" else 2
    wbytes = sum(K * N for K, N in shapes.values())
    rows = sum({K: K for K, _ in shapes.values()}.values()) + sum(N for _, N in shapes.values())
    s = _State(wbytes + 4 * MB, M * rows * size + 4 * MB)
    s.model = QwenGpt(s.gpu, QWEN25_05B)
    s.calls, x = [], {}
    for name, (K, N) in shapes.items():
        s.model.upload_gptq(name, _gptq(K, N, group, g))
        bias = None
        if case.get("bias"):
            bias = name + ".bias"
            s.model.upload_f32(bias, torch.randn(N, device="cuda", generator=g).mul_(0.1).cpu().numpy())
        if K not in x:  # q, k, v and gate, up read the same input
            x[K] = s.gpu.arena.alloc(M * K, [M, K], act)
            s.view(x[K]).copy_(torch.randn(M, K, device="cuda", generator=g))
        s.calls.append((x[K], name, s.gpu.arena.alloc(M * N, [M, N], act), bias, M, N, K))
    s.exact = case.get("exact", False)
    s.out = [s.view(c[2]) for c in s.calls]
    torch.cuda.synchronize()
    if case.get("recorded"):
        with s.gpu.batch() as s.batch:
            for c in s.calls:
                s.model.gemm(*c)
    return s


def _prepare_model(case, seed):
    """The 24-layer model: int4 projections, fp16 tied embedding whose rows differ in length as those of trained models do,
    a final norm that spreads the logits over a few units."""
    g, cfg = _gen(seed), QWEN25_05B
    kind = case["kind"]
    C, KV, I, V = cfg.n_embd, cfg.kv_dim, cfg.intermediate, cfg.vocab_size
    rows = case["B"] * case["T"] if kind == "forward" else case["n"]
    max_t = case["T"] if kind == "forward" else case["n"] + case.get("new", case.get("steps", 0)) + 1
    logit_rows = rows if kind == "forward" or not case.get("last_only", True) else 1
    # (the library's own guide to sizes: everything one pass holds in f32, some 20 rows of the hidden size and 4 of the MLP's)
    s = _State(800 * MB + 200 * 1024 * max_t, rows * (24 * C + 4 * I) * 4 + logit_rows * V * 4 + 64 * MB)
    s.model = QwenGpt(s.gpu, cfg, max_t=max_t, kv_dtype=case["kv"])

    def normal(n, std, mean=0.0):
        return torch.randn(n, device="cuda", generator=g).mul_(std).add_(mean).cpu().numpy()

    embed = torch.randn(V, C, device="cuda", generator=g).mul_(0.02)
    embed *= torch.randn(V, 1, device="cuda", generator=g).mul_(0.25).exp_()
    s.model.upload_f16_bits("embed", embed.half().cpu().numpy(), V)
    s.model.upload_f32("finalNorm", normal(C, 0.08, 4.0))
    for i in range(cfg.n_layer):
        layer = {name: _gptq(K, N, 128, g) for name, (K, N) in QWEN05B_SHAPES.items()}
        layer.update(q_bias=normal(C, 0.02), k_bias=normal(KV, 0.02), v_bias=normal(KV, 0.02), input_norm=normal(C, 0.02, 1.0),
                     post_norm=normal(C, 0.02, 1.0))
        s.model.upload_gptq_layer(i, layer)
    s.tokens = torch.randint(0, V, (rows,), device="cuda", generator=g).cpu().numpy().astype(np.uint32)
    s.seed, s.case = seed, case
    if kind == "score":
        s.given = torch.randint(0, V, (case["steps"],), device="cuda", generator=g).tolist()
    return s


def _prepare_dequant(case, seed):
    t = _gptq(case["K"], case["N"], case["group"], _gen(seed))
    s = _State(case["K"] * case["N"] + 4 * MB, case["K"] * case["N"] * 4 + 4 * MB)
    s.params = GptqInt4Params(t.qweight, t.scales, t.in_features, t.out_features, t.qzeros, t.group_size)
    s.dtype = case["dtype"]
    return s


def prepare(case, seed):
    if case["kind"] in ("linear", "layer"):
        s = _prepare_linear(case, seed)
    elif case["kind"] == "dequant":
        s = _prepare_dequant(case, seed)
    else:
        s = _prepare_model(case, seed)
    s.kind = case["kind"]
    return s


# ---------------------------------------------------------------------------------------------------- one pass
def run(s):
    if s.kind in ("linear", "layer"):
        if s.batch is not None:
            s.batch.submit()
        else:
            for c in s.calls:
                s.model.gemm(*c, exact=s.exact)
        return s.out
    if s.kind == "dequant":
        return dequantize_gptq_int4(s.gpu, s.params, s.dtype)
    m, case, vocab = s.model, s.case, s.model.config.vocab_size
    if s.kind == "forward":
        return s.view(m.forward(s.tokens, case["B"], case["T"]))
    if s.kind == "prefill":
        m.reset_cache()
        return s.view(m.prefill(s.tokens, last_only=case["last_only"]))
    if s.kind == "score":
        m.reset_cache()
        rows = [m.read_tensor_slice(m.prefill(s.tokens, last_only=True), 0, vocab)]
        rows += [m.read_tensor_slice(m.decode_step(t), 0, vocab) for t in s.given]
        return rows
    if s.kind == "greedy":
        r = generate_qwen(m, m.config, s.tokens.tolist(), case["new"], SamplerOptions(temperature=0))
        return np.array(r.ids), m.last_logits()
    r = generate_qwen(m, m.config, s.tokens.tolist(), case["new"],
                      SamplerOptions(case["temperature"], case["top_k"], case["top_p"], random.Random(s.seed).random))
    return np.array(r.ids)


# ---------------------------------------------------------------------------------------------------- what a pass needs
def _packed_bytes(K, N, group):
    return K * N / 2 + -(-K // group) * N * 2.5


def work(case):
    kind = case["kind"]
    if kind in ("linear", "layer"):
        shapes, M, size = _shapes(case), case["M"], 4 if case["act"] == "f32" else 2
        inputs = sum({K for K, _ in shapes.values()})
        return {"bytes": sum(_packed_bytes(K, N, case.get("group", 128)) + M * N * size for K, N in shapes.values()) + M * inputs * size,
                "flops": sum(2.0 * M * N * K for K, N in shapes.values())}
    if kind == "dequant":
        K, N = case["K"], case["N"]
        return {"bytes": _packed_bytes(K, N, case["group"]) + K * N * (4 if case["dtype"] == "f32" else 2), "flops": 1.0 * K * N}
    cfg = QWEN25_05B
    layers, C, V, kvd, D = cfg.n_layer, cfg.n_embd, cfg.vocab_size, cfg.kv_dim, cfg.n_embd // cfg.n_head
    per_row = layers * sum(2.0 * K * N for K, N in QWEN05B_SHAPES.values())  # operations of the projections
    packed = layers * sum(_packed_bytes(K, N, 128) for K, N in QWEN05B_SHAPES.values())
    head_bytes, head_ops = V * C * 2.0, 2.0 * V * C
    kv_row = layers * 2 * kvd * (2 if case["kv"] == "f16" else 4)  # one position of the cache

    def attend(keys):
        return layers * 4.0 * cfg.n_head * D * keys

    if kind == "forward":
        B, T = case["B"], case["T"]
        return {"bytes": packed + head_bytes + 4.0 * B * T * V,
                "flops": B * T * (per_row + head_ops) + B * attend(T * (T + 1) / 2)}
    n = case["n"]
    rows = n if kind == "prefill" and not case["last_only"] else 1
    total = {"bytes": packed + head_bytes + n * kv_row + 4.0 * rows * V, "flops": n * per_row + rows * head_ops + attend(n * (n + 1) / 2)}
    steps = case["steps"] if kind == "score" else case.get("new", 1) - 1
    for i in range(steps):
        total["bytes"] += packed + head_bytes + (n + i + 1) * kv_row + 4.0 * V
        total["flops"] += per_row + head_ops + attend(n + i + 1)
    return total


def tolerance(case):
    kind = case["kind"]
    if kind == "dequant":
        return "exact"  # one rounding per weight: every bit is given
    if kind in ("linear", "layer"):
        # up to 8 rows, and the fp32-activation mode, keep f32 activations; elsewhere operands are fp16
        if case["act"] == "f32" and (case["M"] <= 8 or case.get("exact")):
            # (a group of 64 takes its weights as fp16)
            return {"rel": 1e-5} if case.get("exact") or case.get("group", 128) % 128 == 0 else {"rel": 1e-3}
        return {"rel": 1e-3}
    if kind in ("greedy", "sampled"):
        # short prompts and single steps keep f32 activations; the cache may be fp16
        return {"rel": 2e-3, "differ": 0.0}
    return {"rel": 1e-2}  # fp16 operands through 24 layers
