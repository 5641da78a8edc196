"""Performance cases of the attention path: what they are, how their inputs are made, one pass of each, and the
work and the accuracy that a pass implies.

A case is a dict of plain values:

  entry      "dense", "padded" or "varlen": `sigmoid_attention`, `sigmoid_attention_padded`, `sigmoid_attention_varlen`
  backward   forward and gradients of q, k, v (training), or the forward alone without gradients (inference)
  dtype      "fp16", "bf16" or "fp32"
  batch, q_len, k_len, heads, head_dim     extents (packed sequences: q_len = k_len = the longest one)
  causal     causal mask
  shortest   0: every sequence is full; otherwise lengths are spread evenly over [shortest, longest]
  fused      q, k, v are views of one [B, T, 3, H, D] projection output (dense only), the usual form in a model
  bias       sigmoid_bias, None = the default -log(number of keys)
  score_mod  with an additive per-key term
"""

import math

import torch

import triton_sigmoid_b200 as sa

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}


def _case(name, entry, backward, dtype, batch, q_len, heads, head_dim, causal=False, k_len=0, shortest=0, fused=False,
          bias=None, score_mod=False):
    c = {"entry": entry, "backward": backward, "dtype": dtype, "batch": batch, "q_len": q_len,
         "k_len": k_len or q_len, "heads": heads, "head_dim": head_dim, "causal": causal, "shortest": shortest,
         "fused": fused, "bias": bias, "score_mod": score_mod}
    return dict(c, name=name) if name else c


def listed():
    return [
        # One small inference call: the time is the call itself, not the arithmetic.
        _case("fwd_small", "dense", False, "fp16", 2, 256, 4, 64),
        # Training step of a small model with narrow heads and an odd sequence length.
        _case("train_small_d32", "dense", True, "bf16", 8, 300, 8, 32, causal=True),
        # float32 on the smallest benchmark configuration: debugging, gradient checks, small scientific models.
        _case("train_small_fp32", "dense", True, "fp32", 2, 256, 4, 64),
        # float32 at an ordinary training size.
        _case("train_fp32", "dense", True, "fp32", 4, 2048, 8, 64),
        # Many short sequences, the first point of the benchmark's sequence-length sweep (2^18 tokens).
        _case("train_short", "dense", True, "bf16", 512, 512, 16, 64),
        # The benchmark's default workload.
        _case("train_dense", "dense", True, "fp16", 4, 4096, 16, 64),
        # The published chart's setting: 16384 tokens, hidden size 2048, bias 0, forward.
        _case("fwd_bias0", "dense", False, "bf16", 4, 4096, 32, 64, bias=0.0),
        # Causal training on views of a fused projection, a length that is no multiple of a tile.
        _case("train_fused_causal", "dense", True, "bf16", 8, 1000, 16, 64, causal=True, fused=True),
        # Padded batch with very different lengths (the benchmark's padded configuration).
        _case("train_padded", "padded", True, "bf16", 16, 2048, 8, 64, shortest=256),
        # Packed sequences of mixed lengths, causal, wide heads.
        _case("train_packed", "varlen", True, "bf16", 24, 1500, 8, 128, causal=True, shortest=100),
        # Inference with few queries on a long padded context with a per-key term (cross-attention, chunked decoding).
        _case("fwd_cross", "padded", False, "fp16", 8, 64, 8, 64, k_len=4096, shortest=1024, score_mod=True),
        # The largest training configuration: long causal sequences, wide heads.
        _case("train_large", "dense", True, "bf16", 8, 8192, 32, 128, causal=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c):
    """Work in 16-bit tensor-core operations (a float32 one takes tens of times as long)."""
    return work(c)["flops"] * (60.0 if c["dtype"] == "fp32" else 1.0)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        entry = rng.choice(["dense", "dense", "dense", "padded", "padded", "varlen"])
        dtype = rng.choice(["fp16", "bf16", "bf16", "fp32"])
        backward = rng.random() < 0.65
        heads = rng.choice([1, 2, 4, 6, 8, 12, 16, 20, 32])
        head_dim = rng.choice([32, 64, 64, 64, 96, 128, 128])
        k_len = _log_int(rng, 64, 32768)
        if rng.random() < 0.4:
            k_len = max(64, k_len // 128 * 128)
        q_len = k_len
        causal = rng.random() < 0.45
        if entry == "padded" and not causal and rng.random() < 0.4:
            q_len = _log_int(rng, 1, k_len)
        batch = max(1, min(_log_int(rng, 1, 512), (1 << 18) // k_len))
        shortest = 0
        if entry != "dense":
            shortest = max(1, int(k_len * rng.uniform(0.05, 0.8)))
        c = _case(None, entry, backward, dtype, batch, q_len, heads, head_dim, causal=causal, k_len=k_len,
                  shortest=shortest, fused=entry == "dense" and rng.random() < 0.3,
                  bias=rng.choice([None, None, None, 0.0]), score_mod=rng.random() < 0.15)
        if _cost(c) <= most:
            return c


def _lengths(c):
    """Valid lengths of the batch's query and key sequences (in a fixed order; `prepare` shuffles the batch)."""
    B, lo = c["batch"], c["shortest"]

    def spread(hi):
        first = min(lo, hi)
        return [hi - (hi - first) * i // max(1, B - 1) for i in range(B)]

    k = spread(c["k_len"]) if lo else [c["k_len"]] * B
    q = list(k) if c["q_len"] == c["k_len"] else [c["q_len"]] * B
    return q, k


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype, H, D = _DTYPES[c["dtype"]], c["heads"], c["head_dim"]
    std = 0.5 if D > 64 else 1.0

    def normal(*shape):
        return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=gen)

    lens_q, lens_k = _lengths(c)
    order = torch.randperm(c["batch"], generator=torch.Generator().manual_seed(seed)).tolist()
    lens_q, lens_k = [lens_q[i] for i in order], [lens_k[i] for i in order]
    kw = {"is_causal": c["causal"], "sigmoid_bias": c["bias"]}
    state = {"case": c, "kw": kw, "args": ()}
    if c["entry"] == "varlen":
        total = sum(lens_k)
        q_shape, k_shape, mod_shape = (total, H, D), (total, H, D), (total,)
        cu = torch.tensor([0] + lens_k, dtype=torch.int32).cumsum(0).to(device="cuda", dtype=torch.int32)
        state["args"] = (cu, cu, max(lens_k), max(lens_k))
    else:
        q_shape, k_shape = (c["batch"], c["q_len"], H, D), (c["batch"], c["k_len"], H, D)
        mod_shape = (c["batch"], c["k_len"])
        if c["entry"] == "padded":
            state["args"] = (torch.tensor(lens_k, dtype=torch.int32, device="cuda"),
                             torch.tensor(lens_q, dtype=torch.int32, device="cuda"))
    if c["fused"]:
        state["qkv"] = normal(c["batch"], c["q_len"], 3, H, D).requires_grad_(c["backward"])
    else:
        state["qkv"] = tuple(normal(*s).requires_grad_(c["backward"]) for s in (q_shape, k_shape, k_shape))
    if c["backward"]:
        state["dout"] = normal(*q_shape)
    if c["score_mod"]:
        kw["score_mod"] = 0.5 * torch.randn(mod_shape, device="cuda", generator=gen)
    return state


_ENTRY = {"dense": sa.sigmoid_attention, "padded": sa.sigmoid_attention_padded, "varlen": sa.sigmoid_attention_varlen}


def run(state):
    c, leaf = state["case"], state["qkv"]
    q, k, v = leaf.unbind(2) if c["fused"] else leaf
    out = _ENTRY[c["entry"]](q, k, v, *state["args"], **state["kw"])
    if not c["backward"]:
        return out
    return (out.detach(),) + torch.autograd.grad(out, leaf, state["dout"])


def work(case):
    c = case
    size = 4 if c["dtype"] == "fp32" else 2
    lens_q, lens_k = _lengths(c)
    pairs = 0
    for lq, lk in zip(lens_q, lens_k):
        if c["causal"]:  # query i sees keys 0 .. i
            m = min(lq, lk)
            pairs += m * (m + 1) // 2 + (lq - m) * lk
        else:
            pairs += lq * lk
    flops = 4.0 * pairs * c["heads"] * c["head_dim"] * (3.5 if c["backward"] else 1.0)
    # inputs: valid rows; outputs: whole tensors (padded rows are written as zeros)
    if c["entry"] == "varlen":
        rows_q, rows_k = sum(lens_q), sum(lens_k)
    else:
        rows_q, rows_k = c["batch"] * c["q_len"], c["batch"] * c["k_len"]
    rows = sum(lens_q) + 2 * sum(lens_k) + rows_q             # q, k, v, out
    if c["backward"]:
        rows += sum(lens_q) + rows_q + 2 * rows_k             # dout, dq, dk, dv
    return {"bytes": float(rows * c["heads"] * c["head_dim"] * size), "flops": flops}


def tolerance(case):
    # Relative error of results whose products are rounded to the 16-bit type between two contractions (and whose
    # probabilities are below the normal range of fp16 in part), or of sums of 32-bit products.
    return {"rel": {"fp16": 3e-3, "bf16": 1e-2, "fp32": 1e-5}[case["dtype"]]}
