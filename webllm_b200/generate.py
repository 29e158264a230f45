"""``generateQwen`` and ``sampleToken`` (src/infer/qwen-generate.ts:29-84, src/infer/sampler.ts:18-79)."""
from __future__ import annotations

import math
import random
import time
from dataclasses import dataclass, field, replace

import numpy as np

from .qwen import QwenGpt


@dataclass
class SamplerOptions:
    """``SamplerOptions`` (src/infer/sampler.ts:3-12) plus ``stop_tokens`` of ``QwenGenerateOptions``."""
    temperature: float = 1.0
    top_k: int = 0
    top_p: float = 1.0
    rng: object = None
    stop_tokens: list = field(default_factory=list)


def sample_token(logits: np.ndarray, offset: int, vocab_size: int, options: SamplerOptions | None = None) -> int:
    """``sampleToken``: greedy (first strict maximum) when temperature <= 0, else temperature / top-k /
    top-p sampling with the reference's order of operations."""
    options = options or SamplerOptions()
    if vocab_size <= 0:
        raise ValueError("sampleToken: vocabSize 必须为正")
    if offset < 0 or offset + vocab_size > logits.size:
        raise ValueError(f"sampleToken: logits 越界 offset={offset} vocab={vocab_size}")
    row = np.asarray(logits, np.float32).ravel()[offset:offset + vocab_size]
    if not (options.temperature > 0):
        best = 0
        # np.argmax returns the first maximum; NaNs never win in the reference's strict comparison
        clean = np.where(np.isnan(row), -np.inf, row)
        best = int(np.argmax(clean)) if not np.isnan(row[0]) else 0
        return best
    scaled = (row / np.float32(options.temperature)).astype(np.float32)
    weights = np.exp((scaled - scaled.max()).astype(np.float64)).astype(np.float32)
    limit = min(vocab_size, max(1, int(math.floor(options.top_k)))) if options.top_k > 0 else vocab_size
    if np.isnan(weights).any():
        return _walk(sorted(range(vocab_size), key=lambda i: -float(weights[i]))[:limit], weights, options)
    if limit <= 4096:
        return _walk(_largest(weights, limit).tolist(), weights, options)
    # the whole vocabulary (or nearly): its largest weights usually decide; a prefix of the order that is long enough gives the
    # same answer as all of it
    w64 = weights.astype(np.float64)
    total, keeps_all = float(w64.sum()), not options.top_p < 1
    u = (options.rng or random.random)()
    size = 4096
    while True:
        size = min(size, limit)
        order = _largest(weights, size)
        w = w64[order]
        if keeps_all:
            cut = limit if size == limit else 0
            kept_sum = math.fsum(w64) if limit == vocab_size else math.fsum(w64[_largest(weights, limit)])
        else:
            over = np.flatnonzero(np.cumsum(w / total) >= options.top_p)
            cut = int(over[0]) + 1 if over.size else (limit if size == limit else 0)
            kept_sum = math.fsum(w[:cut])
        if cut or keeps_all:
            reach = np.flatnonzero(np.cumsum(w[:cut or size]) >= u * kept_sum)
            if reach.size:
                return int(order[reach[0]])
            if cut:
                return int(order[min(cut, size) - 1])
        size *= 8


def _largest(weights: np.ndarray, k: int) -> np.ndarray:
    """Indices of the k largest weights, by descending weight and then ascending index (the first k of a stable sort)."""
    if k < weights.size:
        least = np.partition(weights, weights.size - k)[weights.size - k]
        above = np.flatnonzero(weights > least)
        idx = np.sort(np.concatenate([above, np.flatnonzero(weights == least)[:k - above.size]]))
    else:
        idx = np.arange(weights.size)
    return idx[np.argsort(-weights[idx], kind="stable")]


def _walk(kept: list, weights: np.ndarray, options: SamplerOptions) -> int:
    """The reference's loops over the sorted candidates: the top-p cut, then the draw."""
    if options.top_p < 1:
        total = float(weights.astype(np.float64).sum())
        cum = 0.0
        for i, idx in enumerate(kept):
            cum += float(weights[idx]) / total
            if cum >= options.top_p:
                kept = kept[:i + 1]
                break
    kept_sum = sum(float(weights[i]) for i in kept)
    r = (options.rng or random.random)() * kept_sum
    acc = 0.0
    for idx in kept:
        acc += float(weights[idx])
        if acc >= r:
            return idx
    return kept[-1]


@dataclass
class QwenGenerateResult:
    ids: list
    prompt_length: int
    generated: int
    tokens_per_second: float
    prefill_ms: float


def generate_qwen(model: QwenGpt, config, prompt: list, max_new_tokens: int, options: SamplerOptions | None = None,
                  on_device: bool | None = None) -> QwenGenerateResult:
    """``generateQwen``: one prefill, then one decode step per token.

    Greedy decoding without stop tokens runs entirely on the device (``decode_greedy``: argmax and token feedback inside
    one persistent kernel, or a replayed CUDA graph for models that it does not take) unless ``on_device=False``; every
    other option takes the reference's loop with the draw on the device (a top-k of up to 1024) or, from the row read
    back, on the host."""
    options = options or SamplerOptions()
    if len(prompt) == 0:
        raise ValueError("generateQwen: prompt 不能为空")
    if max_new_tokens <= 0:
        raise ValueError("generateQwen: maxNewTokens 必须为正")
    if len(prompt) > model.max_t:
        raise ValueError(f"generateQwen: prompt 长度 {len(prompt)} 超过 blockSize={model.max_t}")
    stop = set(options.stop_tokens or [])
    context = list(prompt)
    vocab = config.vocab_size
    model.reset_cache()

    t0 = time.perf_counter()
    greedy = not (options.temperature > 0)
    k = math.floor(options.top_k) if not greedy and options.top_k > 0 else 0

    on_device_draw = 1 <= k <= 1024  # a short list of candidates is drawn from on the device: the row stays where it is

    def sample(logits, row=None) -> int:
        if on_device_draw:
            u = (options.rng or random.random)()
            token = model.sample(logits, options.temperature, k, options.top_p, u)
            if token is not None:
                return token
            return sample_token(model.read_tensor_slice(logits, 0, vocab), 0, vocab, replace(options, rng=lambda: u))
        return sample_token(model.read_tensor_slice(logits, 0, vocab) if row is None else row, 0, vocab, options)

    # prefill_ms ends with the prompt's logits; the first draw is part of the decoding, as in the reference
    logits, row = model.prefill(np.asarray(prompt, np.uint32), last_only=True), None
    if on_device_draw:
        model.gpu.synchronize()
    else:
        row = model.read_tensor_slice(logits, 0, vocab)
    prefill_ms = (time.perf_counter() - t0) * 1e3

    t1 = time.perf_counter()
    generated = 0
    nxt = sample(logits, row)
    if on_device is None:
        on_device = greedy and not stop
    if on_device and greedy and not stop and max_new_tokens > 1 and nxt not in stop:
        # token 1 is `nxt`; tokens 2..max_new come from max_new-1 device steps
        rest = model.decode_greedy(nxt, max_new_tokens - 1)
        context.append(nxt)
        context.extend(int(t) for t in rest)
        generated = max_new_tokens
    else:
        while generated < max_new_tokens and nxt not in stop:
            context.append(nxt)
            generated += 1
            if generated >= max_new_tokens:
                break
            nxt = sample(model.decode_step(nxt))
    seconds = max(1e-6, time.perf_counter() - t1)
    return QwenGenerateResult(context, len(prompt), generated, generated / seconds, prefill_ms)
