"""What the token sampler is timed on: calls of its public entry points over the range that a
language-model runtime meets, from one token of one conversation to thousands of rows at once.

A case is a dict of plain values:

  entry        'sample'   Sampler.sample: one row, the sampler's own RNG, the token read back
               'rows'     Sampler.sample_rows: a batch resident on the GPU, ids left there
               'rows_ex'  Sampler.sample_rows_ex: every row with its own temperature, top-p and
                          top-k, and a list of banned tokens
               'host'     Sampler.sample_rows_host: logits in pinned host memory
  mode         'topp', 'topk', 'multinomial' or 'greedy' ('mixed' for rows_ex)
  dtype        logits: 'bf16', 'fp16' or 'fp32'
  rows, vocab  batch and vocabulary size; rows are dense, so an odd vocabulary also means rows
               that start on odd addresses
  dist         'zipf'     -slope * log(rank + 1) + sigma * N(0, 1), ranks permuted: the profile of
                          a trained model's logits
               'normal'   sigma * N(0, 1)
               'stress'   half of the rows N(0, 1) with five hot tokens, half almost flat: nuclei of
                          tens of thousands of tokens, as very hot or confused decoding has them
  temperature, topp, topk, slope, sigma

Tokens and RNG states are whole numbers that any correct implementation returns alike.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from executorch_b200 import Sampler, seeds_to_states

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
_GENERATE_ELEMS = 1 << 25  # logits generated at a time: bounds the scratch memory of prepare()


def _case(name, entry, mode, dtype, rows, vocab, dist, temperature, topp=0.9, topk=0, slope=1.1, sigma=0.5):
    c = {"entry": entry, "mode": mode, "dtype": dtype, "rows": rows, "vocab": vocab, "dist": dist,
         "temperature": temperature, "topp": topp, "topk": topk, "slope": slope, "sigma": sigma}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one conversation on a Llama-3 vocabulary: the sampling step between two decode steps,
        # token read back; latency and launches are all there is
        _case("decode1_bf16", "sample", "topp", "bf16", 1, 128_256, "zipf", 0.7),
        # the same on a Llama-2 vocabulary with fp32 logits: the smallest call
        _case("decode1_fp32", "sample", "topp", "fp32", 1, 32_000, "normal", 0.8, sigma=3.0),
        # a handful of conversations served together, Qwen vocabulary
        _case("serve8_bf16", "rows", "topp", "bf16", 8, 151_936, "zipf", 0.7),
        # a mid-size batch on the GPT-2 vocabulary with top-k: an odd vocabulary, so only one row in
        # eight starts on a 16-byte boundary
        _case("serve64_topk_fp16_odd", "rows", "topk", "fp16", 64, 50_257, "normal", 1.0, topk=40, sigma=2.5),
        # a serving batch whose requests bring their own settings and banned tokens
        _case("serve96_own_settings", "rows_ex", "mixed", "bf16", 96, 152_064, "zipf", 0.8),
        # the batch that the sampler's headline figure is quoted on, in its three modes
        _case("batch256_topp_bf16", "rows", "topp", "bf16", 256, 128_256, "zipf", 0.7, topp=0.95),
        _case("batch256_greedy_bf16", "rows", "greedy", "bf16", 256, 128_256, "zipf", 0.0),
        _case("batch256_multinomial_bf16", "rows", "multinomial", "bf16", 256, 128_256, "zipf", 0.7, topp=1.0),
        # logits that a CPU-side model or an external engine leaves in host memory
        _case("host64_topp_bf16", "host", "topp", "bf16", 64, 128_256, "zipf", 0.7),
        # long nuclei: very peaked and almost flat rows
        _case("batch512_stress_fp16", "rows", "topp", "fp16", 512, 151_936, "stress", 1.0),
        # rollout generation: thousands of rows, fp32 logits on a small vocabulary ...
        _case("rollout2048_fp32", "rows", "topp", "fp32", 2048, 32_000, "normal", 0.8, sigma=3.0),
        # ... and bf16 logits on the largest vocabulary in use: the largest call
        _case("rollout2048_bf16_v256000", "rows", "topp", "bf16", 2048, 256_000, "zipf", 0.8, slope=1.0, sigma=0.7),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["sample", "rows", "rows", "rows", "rows", "rows_ex", "host"])
    dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    # half of the vocabularies are multiples of 64, as padded embedding tables have them, half are not
    vocab = _log_int(rng, 16_000, 262_144)
    if rng.random() < 0.5:
        vocab = vocab // 64 * 64
    mode = {"sample": rng.choice(["topp", "topp", "greedy"]), "rows_ex": "mixed", "host": "topp"}.get(
        entry, rng.choice(["topp", "topp", "topp", "topk", "multinomial", "greedy"]))
    dist = rng.choice(["zipf", "zipf", "normal"])
    if mode == "topp" and dtype != "fp32" and entry == "rows" and rng.random() < 0.2:
        dist = "stress"
    # no more logits than the largest listed call of the kind has
    most = {"sample": 1, "rows": 2048, "rows_ex": 128, "host": 64}[entry]
    logits = 64_000_000 if dist == "stress" else {"bf16": 400_000_000, "fp16": 200_000_000, "fp32": 96_000_000}[dtype]
    rows = 1 if most == 1 else _log_int(rng, 2, max(2, min(most, logits // vocab)))
    sigma = {"zipf": rng.uniform(0.4, 0.8), "normal": rng.uniform(2.0, 3.5), "stress": 1.0}[dist]
    temperature = 0.0 if mode == "greedy" else round(rng.uniform(0.6, 1.0), 2)
    topp = 1.0 if mode == "multinomial" else round(rng.uniform(0.8, 0.97), 2)
    topk = rng.randint(10, 100) if mode == "topk" else 0
    return _case(None, entry, mode, dtype, rows, vocab, dist, temperature, topp, topk,
                 round(rng.uniform(1.0, 1.2), 3), round(sigma, 3))


def _logits(case, gen, device):
    """[rows, vocab] logits of the case's distribution, made on the device a few rows at a time."""
    rows, vocab, dist = case["rows"], case["vocab"], case["dist"]
    out = torch.empty((rows, vocab), dtype=_DTYPES[case["dtype"]], device=device)
    chunk = max(1, _GENERATE_ELEMS // vocab)
    for c0 in range(0, rows, chunk):
        n = min(chunk, rows - c0)
        v = torch.randn((n, vocab), generator=gen, device=device)
        if dist == "zipf":
            rank = torch.rand((n, vocab), generator=gen, device=device).argsort(dim=1)
            v = case["sigma"] * v - case["slope"] * torch.log(rank.to(torch.float32) + 1.0)
        elif dist == "normal":
            v *= case["sigma"]
        else:
            flat = torch.arange(c0, c0 + n, device=device) >= rows // 2
            v[flat] *= 0.05
            hot = torch.rand((n, vocab), generator=gen, device=device).topk(5, dim=1).indices
            peak = torch.tensor([12.0, 8.0, 8.0, 8.0, 8.0], device=device).expand(n, 5)
            v[~flat] = v[~flat].scatter(1, hot[~flat], peak[~flat])
        out[c0:c0 + n] = v.to(out.dtype)
    return out


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    rows, vocab = case["rows"], case["vocab"]
    logits = _logits(case, gen, device)
    row_seeds = np.random.default_rng(seed).integers(1, 2**63, size=rows, dtype=np.uint64)
    sampler = Sampler(vocab, case["temperature"], case["topp"], int(row_seeds[0]), device=device)
    if case["mode"] == "topk":
        sampler.set_topk(case["topk"])
    state = {"entry": case["entry"], "sampler": sampler, "logits": logits}
    if case["entry"] == "sample":
        state["logits"] = logits[0]
    elif case["entry"] == "host":
        host = torch.empty(logits.shape, dtype=logits.dtype, pin_memory=True)
        host.copy_(logits)
        state["logits"] = host
        state["states"] = row_seeds
    else:
        state["states"] = seeds_to_states(row_seeds, device)
    if case["entry"] == "rows_ex":
        # requests differ: a third asks for top-k, a sixth samples without a crop, a sixth is greedy
        # and the rest use top-p
        kind = torch.arange(rows, device=device) % 6
        t = case["temperature"] * (0.75 + 0.5 * torch.rand(rows, generator=gen, device=device))
        state["temperature"] = torch.where(kind == 5, torch.zeros_like(t), t)
        p = case["topp"] - 0.1 * torch.rand(rows, generator=gen, device=device)
        state["row_topp"] = torch.where(kind == 4, torch.ones_like(p), p)
        k = torch.randint(10, 100, (rows,), generator=gen, device=device, dtype=torch.int32)
        state["row_topk"] = torch.where(kind < 2, k, torch.zeros_like(k))
        # tokens that no request may produce (banning one twice changes nothing)
        state["ban_ids"] = torch.randint(0, vocab, (32,), generator=gen, device=device, dtype=torch.int32)
        state["ban_bias"] = torch.full((32,), -math.inf, device=device)
    return state


def run(state):
    s, logits = state["sampler"], state["logits"]
    if state["entry"] == "sample":
        return s.sample(logits)
    if state["entry"] == "rows":
        return s.sample_rows(logits, state["states"])
    if state["entry"] == "rows_ex":
        return s.sample_rows_ex(logits, state["states"], temperature=state["temperature"], topp=state["row_topp"],
                                topk=state["row_topk"], edit_ids=state["ban_ids"], edit_bias=state["ban_bias"])
    return s.sample_rows_host(logits, state["states"])


def work(case):
    """Every logit read once; per row an id written and an RNG state read and written. Per logit a
    comparison for the maximum and, unless greedy, a scaled and shifted exponential and its sum."""
    logits = case["rows"] * case["vocab"]
    return {"bytes": logits * _BYTES[case["dtype"]] + case["rows"] * 24,
            "flops": logits * (1 if case["mode"] == "greedy" else 5)}


def tolerance(case):
    return "exact"
