"""The work that users of this package have it do, as cases that can be timed: whole decoding calls, prefills and streams.

Three kinds of call, all through StreamDecoder and DecodeScheduler as a service calls them:

  decode   the encoder frames of `rows` clips are on the device: fill_cross, admit, set_active, then one step per token
           until every row has its `new` tokens (prompt tokens are fed by the steps).
  prefill  fill_cross alone: the cross-attention keys and values of newly admitted clips.
  stream   DecodeScheduler.run over a seeded request stream in pinned host memory: admission and eviction between steps.

Sizes are those of the repository's configurations and tests: 1 to 128 rows, 50 to 375 encoder frames (4 to 30 s of
audio), 10-token prompts and up to 448 new tokens, 8 layers x 1024, 8 heads x 128 with ReLU (the published checkpoint's
decoder) or 16 x 64 with GELU (the benchmark's), every weight mode and both cache formats.

The model is random-init with one exception: the vocabulary projection is tied to a permutation of the token embedding,
so that the best token is clearly the best, as it is for a trained model. With independent random rows a greedy
sequence would hang on near ties that the last bit of a sum decides, and never recover from one. What the layers
compute is held by the keys and values that the decoding appends to the caches, which a pass returns with its tokens.
"""

from __future__ import annotations

import functools
import gc
import math
import random

import numpy as np
import torch

from cohere_inference_b200 import DecodeScheduler, DecoderConfig, StreamDecoder, synthetic_requests
from cohere_inference_b200.synth import SyntheticCohereAsr

LAYERS, WIDTH, FFN, VOCAB = 8, 1024, 4096, 16384
PROMPT, MAX_NEW = 10, 448
BUCKETS = StreamDecoder.BUCKETS
WEIGHTS = {"int8": dict(int8=True), "int8_24": dict(int8=True, ffn_sparse=True), "fp16": dict(fp16_weights=True),
           "bf16": dict()}


def _decode(name, rows, slots, heads, weights, kv, frames_lo, frames_hi, new, frames_dtype):
    return dict(name=name, kind="decode", rows=rows, slots=slots, heads=heads, weights=weights, kv=kv,
                frames_lo=frames_lo, frames_hi=frames_hi, new=new, frames_dtype=frames_dtype)


def _prefill(name, rows, slots, heads, kv, frames_lo, frames_hi, frames_dtype):
    return dict(name=name, kind="prefill", rows=rows, slots=slots, heads=heads, weights="int8", kv=kv,
                frames_lo=frames_lo, frames_hi=frames_hi, frames_dtype=frames_dtype)


def _stream(name, requests, heads, weights, kv, target_hi, fill):
    return dict(name=name, kind="stream", requests=requests, slots=128, heads=heads, weights=weights, kv=kv,
                frames_lo=50, frames_hi=375, target_hi=target_hi, fill=fill)


def listed() -> list[dict]:
    return [
        # a service with 128 slots and one listener: one 14 s clip, 96 steps, int8 weights and caches; latency per token
        _decode("one-clip-int8", 1, 128, 8, "int8", "int8", 175, 175, 87, "bf16"),
        # a handful of clips of different lengths, fewer than the bucket holds
        _decode("six-clips-int8", 6, 8, 16, "int8", "bf16", 50, 375, 96, "fp32"),
        # full-length transcripts of eight 30 s clips with the constructor's default weights
        _decode("batch8-bf16", 8, 8, 16, "bf16", "bf16", 375, 375, 448, "fp32"),
        # 32 clips in one call, 136 steps, int8 weights and caches
        _decode("batch32-int8-kv8", 32, 32, 8, "int8", "int8", 100, 250, 127, "bf16"),
        # the benchmark's configuration: 64 ragged clips, 448 new tokens each
        _decode("batch64-int8", 64, 64, 16, "int8", "bf16", 50, 375, 448, "fp32"),
        # the 16-bit weight mode at the same batch, transcripts of ordinary length
        _decode("batch64-fp16", 64, 64, 8, "fp16", "bf16", 50, 375, 128, "bf16"),
        # an odd batch between two buckets
        _decode("batch100-int8-kv8", 100, 128, 8, "int8", "int8", 50, 375, 96, "bf16"),
        # every slot busy, 2:4 feed-forward weights, short transcripts
        _decode("batch128-24", 128, 128, 16, "int8_24", "bf16", 50, 375, 64, "fp32"),
        # the prefill of one admitted clip
        _prefill("prefill-1", 1, 128, 8, "bf16", 175, 175, "bf16"),
        # the prefill of a whole batch of 64
        _prefill("prefill-64", 64, 64, 16, "bf16", 50, 375, "fp32"),
        # a service with few listeners: a tenth of the slots busy
        _stream("stream-light", 24, 8, "int8", "int8", 128, 0.1),
        # a service at its limit: more requests than slots, 2:4 feed-forward weights
        _stream("stream-full-24", 320, 16, "int8_24", "bf16", 160, 1.05),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))


def draw(rng: random.Random) -> dict:
    most = max(work(c)["bytes"] for c in listed())
    kind = rng.choices(("decode", "prefill", "stream"), (6, 2, 2))[0]
    heads, kv = rng.choice((8, 16)), rng.choice(("bf16", "int8"))
    weights = rng.choice(("int8", "int8", "int8", "int8_24", "fp16", "bf16"))
    if kind == "stream":
        c = _stream("", rng.randint(16, 320), heads, weights, kv, rng.randint(32, 160),
                    round(math.exp(rng.uniform(math.log(0.05), math.log(1.05))), 3))
    else:
        rows = _log_int(rng, 1, 128)
        slots = rng.choice((128, next(b for b in BUCKETS if b >= rows)))
        lo = rng.randint(50, 375)
        hi = rng.randint(lo, 375)
        dtype = rng.choice(("bf16", "fp32"))
        if kind == "prefill":
            c = _prefill("", rows, slots, heads, kv, lo, hi, dtype)
        else:
            c = _decode("", rows, slots, heads, weights, kv, lo, hi, _log_int(rng, 16, MAX_NEW), dtype)
            while work(c)["bytes"] > most:
                c["new"] = c["new"] * 3 // 4
    del c["name"]
    return c


# ---- inputs -------------------------------------------------------------------------------------------------------------


def _lengths(case: dict) -> list[int]:
    """Encoder frames of the rows: the range evenly covered, in a fixed shuffled order (the sizes are the case's, only
    the values come from the seed)."""
    n, lo, hi = case["rows"], case["frames_lo"], case["frames_hi"]
    lens = np.rint(np.linspace(lo, hi, n)).astype(int) if n > 1 else np.array([(lo + hi) // 2])
    return np.random.default_rng(n).permutation(lens).tolist()


def _requests(case: dict) -> list:
    return synthetic_requests(case["requests"], seed=0, vocab=VOCAB, prompt_len=PROMPT,
                              frames=(case["frames_lo"], case["frames_hi"]), targets=(16, case["target_hi"]),
                              slots=case["slots"], fill=case["fill"])


@functools.lru_cache(maxsize=2)
def _model(heads: int):
    """The weights a service has loaded: N(0, 0.02) matrices and embeddings, small biases, LayerNorms around one."""
    cfg = DecoderConfig(num_attention_heads=heads, num_key_value_heads=heads, head_dim=WIDTH // heads,
                        hidden_act="relu" if heads == 8 else "gelu")
    with torch.device("cuda"):
        model = SyntheticCohereAsr(cfg)
    g = torch.Generator(device="cuda").manual_seed(7)
    with torch.no_grad():
        for name, p in model.named_parameters():
            if p.dim() == 2:
                p.normal_(0.0, WIDTH ** -0.5 if name.endswith("decoder.proj.weight") else 0.02, generator=g)
            else:
                p.normal_(1.0 if name.endswith("norm.weight") else 0.0, 0.02, generator=g)
        e = model.model.decoder.embed_tokens.weight
        order = torch.randperm(VOCAB, device="cuda", generator=g)
        model.proj_out.weight.copy_(e[order])
        model.proj_out.bias.zero_()
    return model.eval()


_DECODER: dict[tuple, StreamDecoder] = {}


def _decoder(case: dict) -> StreamDecoder:
    """The one decoder that a program keeps for its GPU; every state of a case works through it, on its stream."""
    key = tuple(sorted((k, str(v)) for k, v in case.items()))
    if key not in _DECODER:
        _DECODER.clear()  # the previous case's, with its caches
        gc.collect()
        torch.cuda.empty_cache()
        _DECODER[key] = StreamDecoder(_model(case["heads"]), slots=case["slots"], max_new_tokens=MAX_NEW, max_prompt=16,
                                      kv_int8=case["kv"] == "int8", eos=-1, **WEIGHTS[case["weights"]])
    return _DECODER[key]


def prepare(case: dict, seed: int) -> dict:
    dec = _decoder(case)
    rng = np.random.default_rng(seed)
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 31)))
    state = dict(case=case, dec=dec)
    if case["kind"] == "stream":
        # encoder frames wait in pinned host memory; a request takes the first of one of sixteen blocks
        pool = torch.randn(16, case["frames_hi"], WIDTH, device="cuda", generator=g).cpu().pin_memory()
        reqs = _requests(case)
        for r in reqs:
            r.prompt = rng.integers(0, VOCAB, PROMPT).astype(np.int64)
        state["requests"] = reqs
        state["sched"] = DecodeScheduler(dec, lambda r: pool[r.mem_seed % 16, : r.frames])
        return state
    lens = _lengths(case)
    memory = torch.randn(sum(lens), WIDTH, device="cuda", generator=g)
    state["memory"] = memory.to(torch.bfloat16) if case["frames_dtype"] == "bf16" else memory
    state["lens"], state["slots"] = lens, list(range(case["rows"]))
    state["prompts"] = [torch.from_numpy(rng.integers(0, VOCAB, PROMPT).astype(np.int64)) for _ in lens]
    torch.cuda.synchronize()
    return state


# ---- one pass -----------------------------------------------------------------------------------------------------------


def run(state: dict):
    case, dec = state["case"], state["dec"]
    if case["kind"] == "stream":
        tokens = state["sched"].run(state["requests"])
        return {"tokens": np.concatenate(tokens), "lengths": np.array([len(t) for t in tokens])}
    with torch.cuda.stream(dec.stream):
        dec.fill_cross(state["memory"], state["lens"], state["slots"])
    if case["kind"] == "prefill":
        got = {"cross_k": dec.cross_k, "cross_v": dec.cross_v}
        if case["kv"] == "int8":
            got.update(cross_ks=dec.cross_ks, cross_vs=dec.cross_vs)
        return got
    dec.admit(state["slots"], state["prompts"], state["lens"], [case["new"]] * case["rows"])
    bucket = dec.set_active(state["slots"])
    for _ in range(PROMPT - 1 + case["new"]):
        dec.step(bucket)
    got = {"tokens": dec.out, "pos": dec.pos}
    # what the steps appended: bf16 keys and values, or the scales of the int8 ones (a code may move by one step when
    # the last bit of the value before rounding does)
    names = ("self_ks", "self_vs") if case["kv"] == "int8" else ("self_k", "self_v")
    got.update({n: getattr(dec, n) for n in names})
    return got


# ---- what a pass cannot do without --------------------------------------------------------------------------------------


def _weight_bytes(weights: str) -> float:
    """One step's projections: 12 x 1024 x 1024 per layer (8 of them feed-forward) and the vocabulary projection."""
    attn, ffn = LAYERS * 4 * WIDTH * WIDTH + LAYERS * 2 * WIDTH * WIDTH, LAYERS * 2 * WIDTH * FFN
    each = {"int8": 1, "int8_24": 1, "fp16": 2, "bf16": 2}[weights]
    return (attn + VOCAB * WIDTH) * each + ffn * (0.625 if weights == "int8_24" else each)


def _rows_work(rows_by_step, kv: str, heads: int, weights: str) -> tuple[float, float]:
    """(bytes, flops) of decoding steps given, per step, the (rows, sum of cached positions, sum of frames)."""
    b_kv = 2.0 if kv == "bf16" else 1 + 4 * heads / WIDTH
    macs = LAYERS * (6 * WIDTH * WIDTH + 2 * WIDTH * FFN) + VOCAB * WIDTH
    w = _weight_bytes(weights)
    total_b = total_f = 0.0
    for rows, positions, frames in rows_by_step:
        keys = positions + rows + frames
        total_b += w + LAYERS * 2 * WIDTH * b_kv * (keys + rows) + rows * 2 * WIDTH * 2
        total_f += 2.0 * rows * macs + 4.0 * LAYERS * WIDTH * keys
    return total_b, total_f


def _prefill_work(frames: int, kv: str, heads: int, frame_bytes: int) -> tuple[float, float]:
    n = LAYERS * 2 * WIDTH
    b_kv = 2.0 if kv == "bf16" else 1 + 4 * heads / WIDTH
    return (WIDTH * WIDTH + n * WIDTH) * 2 + frames * (WIDTH * frame_bytes + n * b_kv), 2.0 * frames * WIDTH * (WIDTH + n)


def work(case: dict) -> dict:
    kv, heads = case["kv"], case["heads"]
    if case["kind"] == "stream":
        reqs = _requests(case)
        b, f = _prefill_work(sum(r.frames for r in reqs), kv, heads, 4)
        b -= (WIDTH * WIDTH + LAYERS * 2 * WIDTH * WIDTH) * 2  # the prefill's weights are counted once per call below
        # every request's own steps; the projections' weights once per step, with all slots busy or as few as arrive
        steps = [PROMPT - 1 + r.target for r in reqs]
        span = max(sum(steps) / case["slots"], max(int(r.arrival) + s for r, s in zip(reqs, steps)))
        rb, rf = _rows_work([(s, s * (s - 1) / 2, s * r.frames) for r, s in zip(reqs, steps)], kv, heads, case["weights"])
        rb += _weight_bytes(case["weights"]) * (span - len(reqs))
        return {"bytes": b + rb, "flops": f + rf}
    lens = _lengths(case)
    b, f = _prefill_work(sum(lens), kv, heads, 2 if case["frames_dtype"] == "bf16" else 4)
    if case["kind"] == "decode":
        n = case["rows"]
        rb, rf = _rows_work([(n, n * t, sum(lens)) for t in range(PROMPT - 1 + case["new"])], kv, heads, case["weights"])
        b, f = b + rb, f + rf
    return {"bytes": b, "flops": f}


def tolerance(case: dict):
    """Tokens, positions and lengths are the same. Keys and values are bf16 (or scales of bf16-rounded vectors) of rows
    that went through 16-bit operands; the prefill's int8 codes may differ where its last bit decides a rounding."""
    if case["kind"] == "stream":
        return "exact"
    return {"rel": 1e-2, "differ": 5e-3 if case["kind"] == "prefill" and case["kv"] == "int8" else 0.0}
