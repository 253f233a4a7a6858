"""The work that users of ring_swa have it do on one GPU, as measurable cases.

Each case is one call of a public entry point the way a program makes it: a training step of an attention
layer (forward and backward), a forward pass alone (prefill of a prompt, evaluation, or the recomputed
forward of activation checkpointing), or the merge of two partial attention results.  Sizes are those of
the benchmark's workloads, of the tests and of the reference's test matrix, or generic; nothing is chosen
for how it happens to fit the kernels' tiles.

The fields of a case:
  fn      swa | swa_varlen | slm | slm_varlen (the four public functions) or merge (ring_swa.ops.merge_attn_out)
  train   forward and backward (true) or forward only
  batch, seq      batch rows and tokens per row; packed functions: lens, the sequences' lengths
  hq, hkv, d      query heads, key/value heads, head dimension
  window, sink    window size, sink tokens
  dtype           bf16 | fp16
  fused           q, k and v are slices of one projection's output instead of tensors of their own
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "ring-sliding-window-attention_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ring_swa  # noqa: E402
from ring_swa.ops import merge_attn_out  # noqa: E402

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _attn(name, fn, train, shape, heads, d, window, sink=0, dtype="bf16", fused=False):
    """shape: (batch, seq), or the packed sequences' lengths as text."""
    c = {"name": name, "fn": fn, "train": train}
    if isinstance(shape, str):
        c["lens"] = shape
    else:
        c["batch"], c["seq"] = shape
    c.update(hq=heads[0], hkv=heads[1], d=d, window=window, sink=sink, dtype=dtype, fused=fused)
    return c


def listed():
    return [
        # the smallest configuration of the benchmark set in a 16-bit type: a step of a small model or a unit
        # test, where launches and host work are all there is
        _attn("train_1k_d64", "swa", True, (1, 1024), (4, 4), 64, 128),
        # the first tokens of a chat: a short prompt of odd length through one layer, forward only
        _attn("prefill_777", "swa", False, (1, 777), (32, 8), 128, 256, fused=True),
        # the shortest shape of the reference's test matrix: 32 query heads on 4 key/value heads
        _attn("train_4k_gqa", "swa", True, (1, 4096), (32, 4), 128, 1000),
        # its packed batch, with the sink token: four documents of very different lengths
        _attn("train_packed_22k_sink", "slm_varlen", True, "512,2000,4000,16000", (32, 4), 128, 1000, sink=1),
        # half precision, two rows of odd length, few key/value heads, a window that is no multiple of anything
        _attn("train_fp16_ragged", "slm", True, (2, 3001), (16, 2), 128, 500, sink=1, dtype="fp16"),
        # a model with 64-wide heads: four rows of 4096 tokens
        _attn("train_d64_batch", "swa", True, (4, 4096), (16, 16), 64, 512),
        # prefill of a long prompt, grouped heads
        _attn("prefill_16k", "swa", False, (1, 16384), (32, 8), 128, 4096, fused=True),
        # the benchmark's default workload
        _attn("train_32k", "swa", True, (2, 32768), (32, 32), 128, 1000),
        # the benchmark's packed workload: seven documents, window 4096
        _attn("train_packed_64k", "swa_varlen", True, "7204,3978,14070,10318,13142,12634,4190", (32, 8), 128, 4096),
        # the benchmark's sink workload: 131072 tokens, 4 sink tokens and a window of 8192
        _attn("train_128k_sink", "slm", True, (1, 131072), (32, 8), 128, 8192, sink=4),
        # a quarter of the benchmark's long-window workload: the window is half of the sequence
        _attn("train_64k_wide", "swa", True, (1, 65536), (64, 8), 128, 32768),
        # folding one hop's partial result into the running float32 accumulators of a ring loop
        {"name": "merge_16k", "fn": "merge", "batch": 1, "seq": 16384, "hq": 32, "d": 128, "dtype": "bf16"},
    ]


_HEADS = [(4, 4), (8, 2), (16, 16), (16, 2), (32, 32), (32, 8), (32, 4), (64, 8)]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the ranges above: 256 to 131072 tokens in all, windows of 64 to 32768, every head layout."""
    most = max(_cost(c) for c in listed())
    if rng.random() < 0.08:
        return {"fn": "merge", "batch": rng.choice((1, 1, 2)), "seq": _log_int(rng, 512, 32768), "hq": rng.choice((8, 16, 32)),
                "d": rng.choice((64, 128, 128)), "dtype": rng.choice(("bf16", "bf16", "fp16"))}
    while True:
        fn = rng.choice(("swa", "swa", "swa", "swa_varlen", "slm", "slm_varlen"))
        tokens = _log_int(rng, 256, 131072)
        if fn.endswith("varlen"):
            n = rng.randint(1, 12)
            cuts = sorted(rng.sample(range(1, tokens), n - 1))
            lens = [b - a for a, b in zip([0] + cuts, cuts + [tokens])]
            shape = ",".join(map(str, lens))
        else:
            batch = rng.choice((1, 1, 1, 2, 4))
            shape = (batch, max(64, tokens // batch))
        c = _attn("", fn, rng.random() < 0.7, shape, rng.choice(_HEADS), rng.choice((64, 128, 128, 128, 128)),
                  _log_int(rng, 64, 32768), sink=rng.choice((1, 1, 4)) if fn.startswith("slm") else 0,
                  dtype=rng.choice(("bf16", "bf16", "bf16", "fp16")), fused=rng.random() < 0.3)
        del c["name"]
        # (the 128-wide equivalent of the arithmetic, and a bound on the bytes)
        if _cost(c) <= most and work(c)["bytes"] <= 6e9:
            return c


def _lens(case):
    if "lens" in case:
        return [int(x) for x in case["lens"].split(",")]
    return [case["seq"]] * case["batch"]


def _pairs(length, window, sink):
    """Visible (query, key) pairs of one sequence: a query sees itself, the `window` tokens before it and
    the first `sink` tokens."""
    full = min(length, window + 1)
    n = full * (full + 1) // 2 + (length - full) * (window + 1)
    for s in range(sink):
        n += max(0, length - (window + 1 + s))
    return n


def _cost(case):
    if case["fn"] == "merge":
        return 0
    pairs = sum(_pairs(n, case["window"], case["sink"]) for n in _lens(case))
    return pairs * case["hq"] * (14 if case["train"] else 4) * 128


def work(case):
    if case["fn"] == "merge":
        rows = case["batch"] * case["seq"] * case["hq"]
        # accumulator read and written (float32), the 16-bit partial result read, one lse read, one updated
        return {"bytes": rows * (case["d"] * (4 + 4 + 2) + 4 + 4 + 4), "flops": rows * case["d"] * 3}
    tokens = sum(_lens(case))
    q, kv = tokens * case["hq"] * case["d"] * 2, tokens * case["hkv"] * case["d"] * 2
    pairs = sum(_pairs(n, case["window"], case["sink"]) for n in _lens(case))
    # forward: q, k, v -> out (two products).  Training: q, k, v, dout -> out, dq, dk, dv (two products
    # and five).
    bytes_ = 2 * q + 2 * kv if not case["train"] else 4 * q + 4 * kv
    return {"bytes": bytes_, "flops": pairs * case["hq"] * case["d"] * (14 if case["train"] else 4)}


def tolerance(case):
    if case["fn"] == "merge":
        return {"rel": 1e-5}  # float32 accumulators
    # 16-bit inputs, probabilities and results around float32 accumulation
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[case["dtype"]]

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32).to(dt)

    if case["fn"] == "merge":
        b, s, h, d = case["batch"], case["seq"], case["hq"], case["d"]
        # log-sum-exp of a few hundred to a few thousand scores each
        return {"case": case, "out": normal(b, s, h, d).float() * 0.05, "new": normal(b, s, h, d) * 0.05,
                "lse": torch.randn(b, h, s, generator=g, device="cuda") + 7.0,
                "new_lse": torch.randn(b, h, s, generator=g, device="cuda") + 6.0}
    lead = (sum(_lens(case)),) if "lens" in case else (case["batch"], case["seq"])
    hq, hkv, d = case["hq"], case["hkv"], case["d"]
    if case["fused"]:
        qkv = normal(*lead, hq + 2 * hkv, d)
        q, k, v = qkv[..., :hq, :], qkv[..., hq:hq + hkv, :], qkv[..., hq + hkv:, :]
    else:
        q, k, v = normal(*lead, hq, d), normal(*lead, hkv, d), normal(*lead, hkv, d)
    st = {"case": case, "q": q, "k": k, "v": v, "kw": {}}
    if case["train"]:
        st["q"], st["k"], st["v"] = (x.detach().requires_grad_(True) for x in (q, k, v))
        st["dout"] = normal(*lead, hq, d)
    if "lens" in case:
        cu = [0]
        for n in _lens(case):
            cu.append(cu[-1] + n)
        st["kw"].update(cu_seqlens=torch.tensor(cu, dtype=torch.int32, device="cuda"), cp_size=1)
    if case["sink"] > 1:
        st["kw"]["num_sink_tokens"] = case["sink"]
    st["call"] = {"swa": ring_swa.ring_sliding_window_attn, "swa_varlen": ring_swa.ring_sliding_window_attn_varlen,
                  "slm": ring_swa.ring_streaming_llm_attn, "slm_varlen": ring_swa.ring_streaming_llm_attn_varlen}[case["fn"]]
    return st


def run(state):
    case = state["case"]
    if case["fn"] == "merge":
        merge_attn_out(state["out"], state["lse"], state["new"], state["new_lse"])
        return state["out"], state["lse"]
    q, k, v = state["q"], state["k"], state["v"]
    if not case["train"]:
        with torch.no_grad():
            return state["call"](q, k, v, case["window"], **state["kw"])
    out = state["call"](q, k, v, case["window"], **state["kw"])
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["dout"])
    return out, dq, dk, dv
