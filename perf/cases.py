"""The work a user of this library has it do, as cases that can be timed and whose outputs can be compared.

A case is a dict of plain values: what is called (``op``), the distribution of the sequence lengths, heads, head
dimension, activation and options.  ``prepare`` makes the inputs of a case on the GPU from a seed (the lengths of a
case are fixed by its ``len_seed``; the seed deals them out to the sequences and draws the values), ``run`` is one
call through the public entry points of ``ads_model_kernel_library_b200.gdpa``; ``exact`` is the same in fp64.
"""
import math

import numpy as np
import torch

import ads_model_kernel_library_b200.gdpa as gdpa

# ------------------------------------------------------------------------------------------------------ the cases

# Field values a case starts from.  `q` / `kv`: length distribution "uniform" (lo .. hi), "lognormal" (median,
# clipped to lo .. hi), "zipf" (multiples of 32 up to hi) or "fixed" (hi); kv = "same" is self-attention.
_BASE = {
    "op": "attention", "train": True, "batch": 1, "heads": 4, "kv_heads": 4, "head_dim": 128, "activation": "gelu_approx",
    "q": "uniform", "q_lo": 1, "q_hi": 256, "q_median": 0, "kv": "same", "kv_lo": 1, "kv_hi": 256, "kv_median": 0,
    "window": -1, "packed": "no", "std": 0.5, "scale": "inverse_max", "len_seed": 0,
}


def _case(**fields):
    c = dict(_BASE)
    c.update(fields)
    if "kv_heads" not in fields:
        c["kv_heads"] = c["heads"]
    return c


def listed():
    return [
        # The smallest training step: eight short sequences, two heads (a unit test's size, a ranking model's user
        # tower on a small batch).  Host time, launches and latency are all of it.
        _case(name="train_tiny", batch=8, heads=2, head_dim=64, q_lo=16, q_hi=256, kv="uniform", kv_lo=16, kv_hi=256, std=1.0),
        # Online inference: a few requests, each with a history of its own that its 64 candidates (short Q sequences)
        # attend to; nothing is trained, the answer is waited for.
        _case(name="serve_shared_kv", op="shared_kv", train=False, batch=4, heads=4, activation="silu", q_lo=1, q_hi=32,
              kv="uniform", kv_lo=200, kv_hi=1500, std=1.0),
        # Cross-attention inference over a large batch: log-normal query and history lengths that do not match.
        _case(name="forward_lognormal", train=False, batch=1024, heads=4, activation="silu", q="lognormal", q_lo=16, q_hi=2048,
              q_median=256, kv="lognormal", kv_lo=16, kv_hi=4096, kv_median=1024, std=1.0),
        # The default training workload: self-attention over histories of 512 to 4096 tokens, eight heads.
        _case(name="train_uniform", batch=512, heads=8, q_lo=512, q_hi=4096),
        # Training on many short histories, lengths anywhere up to 256: every tile is ragged, a work item is a tile or two.
        _case(name="train_short_ragged", batch=1152, heads=4, activation="fast_gelu", q_lo=1, q_hi=256, std=1.0, scale="one"),
        # Cross-attention training against a short fixed-size context (256 keys), queries of 1024 tokens.
        _case(name="train_short_kv", batch=1152, heads=4, activation="fast_gelu", q="fixed", q_hi=1024, kv="fixed", kv_hi=256,
              std=1.0, scale="one"),
        # Heavily skewed lengths: most sequences are one short tile, a few are 8192 tokens long.
        _case(name="train_zipf", batch=128, heads=4, q="zipf", q_hi=8192),
        # The softmax variant, trained: row statistics, log-sum-exp and its backward.
        _case(name="train_softmax", batch=128, heads=4, activation="softmax", q_lo=128, q_hi=2048, std=1.0, scale="inverse_sqrt"),
        # Low-precision inference from bf16 activations: quantise Q, K, V to block-scaled FP8, then the FP8 forward.
        _case(name="forward_fp8", op="fp8", train=False, batch=1024, heads=4, activation="softmax", q_lo=128, q_hi=2048, std=1.0,
              scale="inverse_sqrt"),
        # Low-precision inference from stored MXFP8 tensors (elements and e8m0 scales).
        _case(name="forward_mxfp8", op="mxfp8", train=False, batch=1024, heads=4, activation="softmax", q_lo=128, q_hi=2048,
              std=1.0, scale="inverse_sqrt"),
        # A whole block in training: layer norm of Q, attention, Q residual, RMS norm, residual, and its backward.
        _case(name="train_norms", op="norms", batch=64, heads=8, activation="fast_gelu", q_lo=512, q_hi=4096, std=1.0),
        # Grouped-query heads of 64, K and V packed in one tensor, attention limited to a band of 256 positions.
        _case(name="train_gqa_band", batch=128, heads=8, kv_heads=2, head_dim=64, activation="silu", q_lo=256, q_hi=2048, window=256,
              packed="kv"),
    ]


_MOST_FLOPS = 4.0e13  # of one pass; the largest listed case has 5.0e13
_MOST_VALUES = 1.0e9  # of Q; the largest listed case has 1.2e9


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: a family at random, sizes spread over its range."""
    family = rng.choice(["train", "train", "forward", "shared_kv", "softmax", "fp8", "mxfp8", "norms", "gqa_band", "zipf", "short_kv"])
    seed = rng.randrange(1 << 20)
    acts = ["gelu_approx", "fast_gelu", "silu", "relu"]
    if family in ("train", "forward"):
        hi = _log_int(rng, 32, 4096)
        kv_hi = _log_int(rng, 32, 4096)
        kv = rng.choice(["same", "uniform"]) if family == "train" else "uniform"
        c = _case(train=family == "train", batch=_log_int(rng, 4, 1200), heads=rng.choice([2, 4, 8]), head_dim=rng.choice([64, 128, 128]),
                  activation=rng.choice(acts), q_lo=rng.randint(1, hi), q_hi=hi, kv=kv, kv_lo=rng.randint(1, kv_hi), kv_hi=kv_hi)
    elif family == "shared_kv":
        kv_hi = _log_int(rng, 200, 4000)
        c = _case(op="shared_kv", train=False, batch=_log_int(rng, 1, 64), activation=rng.choice(acts), q_lo=1, q_hi=_log_int(rng, 2, 256),
                  kv="uniform", kv_lo=kv_hi // 4, kv_hi=kv_hi, std=1.0)
    elif family in ("softmax", "fp8", "mxfp8"):
        hi = _log_int(rng, 128, 4096)
        c = _case(op="attention" if family == "softmax" else family, train=family == "softmax", batch=_log_int(rng, 8, 1024),
                  heads=rng.choice([2, 4, 8]), activation="softmax", q_lo=rng.randint(1, hi), q_hi=hi, std=1.0, scale="inverse_sqrt")
    elif family == "norms":
        hi = _log_int(rng, 128, 4096)
        c = _case(op="norms", batch=_log_int(rng, 4, 128), heads=rng.choice([2, 4, 8]), activation=rng.choice(acts),
                  q_lo=rng.randint(1, hi), q_hi=hi, std=1.0)
    elif family == "gqa_band":
        hi = _log_int(rng, 128, 4096)
        kv_heads = rng.choice([1, 2, 4])
        c = _case(batch=_log_int(rng, 4, 256), heads=8, kv_heads=kv_heads, head_dim=rng.choice([64, 128]), activation=rng.choice(acts),
                  q_lo=rng.randint(1, hi), q_hi=hi, window=rng.choice([-1, 64, 256, 300]), packed=rng.choice(["no", "kv"]))
    elif family == "zipf":
        c = _case(batch=_log_int(rng, 8, 256), heads=4, q="zipf", q_hi=8192)
    else:
        c = _case(batch=_log_int(rng, 32, 1152), activation=rng.choice(acts), q="uniform", q_lo=64, q_hi=_log_int(rng, 128, 2048),
                  kv="uniform", kv_lo=32, kv_hi=_log_int(rng, 64, 256), std=1.0)
    c["len_seed"] = seed
    while c["batch"] > 1 and (work(c)["flops"] > _MOST_FLOPS or int(_lengths(c)[0].sum()) * c["heads"] * c["head_dim"] > _MOST_VALUES):
        c["batch"] = c["batch"] * 2 // 3
    return c


# ------------------------------------------------------------------------------------------------------- lengths

_PER_REQUEST = 64  # "shared_kv": candidates of one request


def _draw_lengths(rng, kind, lo, hi, median, n):
    if kind == "fixed":
        return np.full(n, hi, dtype=np.int64)
    if kind == "uniform":
        return rng.integers(lo, hi + 1, n)
    if kind == "lognormal":
        return np.clip(np.rint(np.exp(rng.normal(np.log(median), 0.75, n))), lo, hi).astype(np.int64)
    if kind == "zipf":
        return 32 * np.minimum(rng.zipf(1.2, n), hi // 32).astype(np.int64)
    raise ValueError(kind)


def _lengths(case):
    """(query lengths, KV lengths); for "shared_kv" the query lengths of all candidates and the KV lengths of the requests."""
    rng = np.random.default_rng(case["len_seed"])
    n_kv = case["batch"]
    n_q = n_kv * _PER_REQUEST if case["op"] == "shared_kv" else n_kv
    lq = _draw_lengths(rng, case["q"], case["q_lo"], case["q_hi"], case["q_median"], n_q)
    if case["kv"] == "same":
        return lq, lq.copy()
    return lq, _draw_lengths(rng, case["kv"], case["kv_lo"], case["kv_hi"], case["kv_median"], n_kv)


def _pairs(case):
    """Pairs (query, key) that take part."""
    lq, lk = _lengths(case)
    if case["op"] == "shared_kv":
        return int((lq.reshape(-1, _PER_REQUEST).sum(1) * lk).sum())
    if case["window"] < 0:
        return int((lq * lk).sum())
    w, total = case["window"], 0
    for a, b in zip(lq.tolist(), lk.tolist()):
        i = np.arange(a, dtype=np.int64)
        total += int(np.maximum(0, np.minimum(b, i + w + 1) - np.maximum(0, i - w)).sum())
    return total


# ----------------------------------------------------------------------------------------------- inputs and a pass


def _offsets(lens):
    return torch.from_numpy(np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)).cuda()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    lq, lk = _lengths(case)
    order = np.random.default_rng(seed).permutation(len(lk))  # which sequence has which length
    if case["op"] == "shared_kv":
        lq = lq.reshape(-1, _PER_REQUEST)[order].reshape(-1)
    else:
        lq = lq[order]
    lk = lk[order]
    H, Hk, D = case["heads"], case["kv_heads"], case["head_dim"]
    tq, tk = int(lq.sum()), int(lk.sum())

    def values(*shape, std=case["std"]):
        return (torch.randn(shape, generator=gen, device="cuda") * std).to(torch.bfloat16)

    max_q, max_kv = int(lq.max()), int(lk.max())
    s = {
        "op": case["op"], "train": case["train"], "max_q": max_q, "max_kv": max_kv, "activation": case["activation"],
        "scale": {"one": 1.0, "inverse_max": 1.0 / max_kv, "inverse_sqrt": 1.0 / math.sqrt(D)}[case["scale"]],
        "window": case["window"] if case["window"] >= 0 else None, "qo": _offsets(lq), "ko": _offsets(lk), "q": values(tq, H, D),
    }
    if case["packed"] == "kv":
        s["k"], s["v"] = values(tk, Hk, 2 * D), None
    else:
        s["k"], s["v"] = values(tk, Hk, D), values(tk, Hk, D)
    if case["op"] == "shared_kv":
        s["request_of"] = torch.arange(len(lk), device="cuda").repeat_interleave(_PER_REQUEST)
    if case["op"] == "mxfp8":
        for n, off, axis in (("q", "qo", 0), ("k", "ko", 0), ("v", "ko", 1)):
            s[n], s["sf" + n], _ = gdpa.quantize_varlen_mxfp8_sf_only(s[n], s[off], scale_axis=axis)
    if case["op"] == "norms":
        n = H * D
        for name, base in (("ln_w", 1.0), ("ln_b", 0.0), ("rms_w", 1.0)):
            s[name] = base + 0.1 * torch.randn(n, generator=gen, device="cuda")
        s["residual"] = values(tq, H, D)
    if case["train"]:
        s["dout"] = values(tq, H, D)
        for name in ("q", "k", "v", "ln_w", "ln_b", "rms_w"):
            if s.get(name) is not None:
                s[name].requires_grad_(True)
    return s


def _gradients(out, s, names):
    names = [n for n in names if s[n] is not None]
    return [out, *torch.autograd.grad(out, [s[n] for n in names], s["dout"])]


def run(state):
    s = state
    if s["op"] == "norms":
        out = gdpa.gdpa_megakernel(
            s["q"], s["k"], s["v"], s["qo"], s["ko"], s["max_q"], s["max_kv"], qk_scale=s["scale"], activation=s["activation"],
            fused_rms_norm=True, rms_norm_weight=s["rms_w"], fused_residual_add=True, residual=s["residual"], fused_q_residual_add=True,
            fused_layernorm=True, layernorm_weight=s["ln_w"], layernorm_bias=s["ln_b"])
        return _gradients(out, s, ("q", "k", "v", "ln_w", "ln_b", "rms_w"))
    if s["op"] == "fp8":
        q8, sq, q_blocks = gdpa.quantize_fp8_blockwise(s["q"], s["qo"])
        k8, sk, kv_blocks = gdpa.quantize_fp8_blockwise(s["k"], s["ko"])
        v8, sv, _ = gdpa.quantize_fp8_blockwise(s["v"], s["ko"])
        return gdpa.generalized_dot_product_attention_fp8(
            q8, k8, v8, sq, sk, sv, q_blocks, kv_blocks, s["qo"], s["ko"], s["max_q"], s["max_kv"], qk_scale=s["scale"],
            activation=s["activation"])
    if s["op"] == "mxfp8":
        return gdpa.generalized_dot_product_attention_mxfp8(
            s["q"], s["k"], s["v"], s["sfq"], s["sfk"], s["sfv"], s["qo"], s["ko"], s["max_q"], s["max_kv"], qk_scale=s["scale"],
            activation=s["activation"])
    if s["op"] == "shared_kv":
        with torch.no_grad():
            return gdpa.generalized_dot_product_attention(
                s["q"], s["k"], s["v"], s["qo"], s["ko"], s["max_q"], s["max_kv"], ad_to_request_offset=s["request_of"],
                qk_scale=s["scale"], activation=s["activation"])
    out = gdpa.generalized_dot_product_attention(
        s["q"], s["k"], s["v"], s["qo"], s["ko"], s["max_q"], s["max_kv"], qk_scale=s["scale"], window_size=s["window"],
        activation=s["activation"])
    return _gradients(out, s, ("q", "k", "v")) if s["train"] else out


# ---------------------------------------------------------------------------------------- what a pass cannot do without


def work(case):
    lq, lk = _lengths(case)
    H, Hk, D = case["heads"], case["kv_heads"], case["head_dim"]
    nq, nk = int(lq.sum()) * H * D, int(lk.sum()) * Hk * D
    fwd = 4 * H * D * _pairs(case)
    if case["op"] == "mxfp8":
        n_bytes = (nq + 2 * nk) * 33 // 32 + 2 * nq  # e4m3 elements and their scales in, bf16 out
    else:
        n_bytes = 2 * (2 * nq + 2 * nk)  # Q, K, V in, O out
    if case["train"]:
        n_bytes += 2 * (2 * nq + 2 * nk)  # dO in, dQ, dK, dV out
    if case["op"] == "norms":
        n_bytes += 2 * nq  # the residual
    return {"bytes": n_bytes, "flops": fwd * 7 // 2 if case["train"] else fwd}


def tolerance(case):
    # Four times what the path differs by from the same computation in fp64 on the same inputs (ten sequences of every
    # listed case), largest over the outputs: bf16 P and outputs give rel 2.4e-3 throughout, max 1.3e-2 with an
    # element-wise activation and 2.4e-2 with the softmax; the norm pipeline, whose gradients pass three more bf16
    # tensors, 5.5e-3 and 4.0e-2; FP8, whose P has three mantissa bits, 2.4e-2 and 0.22 (rel held to 0.03).
    if case["op"] == "fp8":
        return {"rel": 0.03, "max": 0.88}
    if case["op"] == "norms":
        return {"rel": 0.02, "max": 0.16}
    return {"rel": 0.01, "max": 0.1 if case["activation"] == "softmax" else 0.06}


# ------------------------------------------------------------------------------------- the same pass in 64 bits


def _mx_values(x, axis):
    """What a block-scaled FP8 tensor of the values `x` ([rows, H, D], one sequence) stands for, in fp64: e4m3 elements, one
    power of two per 32 of them along `axis`, the smallest with amax / scale <= 448."""
    n = x.shape[axis]
    pad = (-n) % 32
    x = x.movedim(axis, -1).float()
    g = torch.nn.functional.pad(x, (0, pad)).unflatten(-1, (-1, 32))
    mantissa, exponent = torch.frexp(g.abs().amax(-1, keepdim=True) * (1.0 / 448.0))
    scale = torch.exp2((exponent - (mantissa == 0.5).int()).double())
    y = (g.double() / scale).float().to(torch.float8_e4m3fn).double() * scale
    return y.flatten(-2)[..., :n].movedim(-1, axis)


def _attention64(q, k, v, s):
    """One sequence: [rows, H, D] tensors in fp64, K and V with a head for each query head."""
    q, k, v = (t.transpose(0, 1) for t in (q, k, v))
    x = q @ k.transpose(1, 2)
    band = None
    if s["window"] is not None:
        i, j = torch.arange(x.shape[1], device=x.device).view(-1, 1), torch.arange(x.shape[2], device=x.device)
        band = (i - j).abs() <= s["window"]
    F = torch.nn.functional
    if s["activation"] == "softmax":
        p = torch.softmax(x * s["scale"], -1)
    else:
        if band is not None:
            x = x * band
        act = {"gelu_approx": lambda t: F.gelu(t, approximate="tanh"), "fast_gelu": lambda t: F.gelu(t, approximate="tanh"),
               "silu": F.silu, "relu": F.relu}[s["activation"]]
        p = act(x) * s["scale"]
        if band is not None:
            p = p * band
    return (p @ v).transpose(0, 1)


def exact(case, seed):
    op, train = case["op"], case["train"]
    s = prepare(dict(case, op="fp8") if op == "mxfp8" else case, seed)  # the inputs before they are quantised
    H, Hk, D = case["heads"], case["kv_heads"], case["head_dim"]
    qo, ko = s["qo"].tolist(), s["ko"].tolist()
    lq, _ = _lengths(case)
    owner = s["request_of"].tolist() if op == "shared_kv" else list(range(len(lq)))
    out = torch.zeros(s["q"].shape, dtype=torch.float64, device="cuda")
    names = [n for n in ("q", "k", "v") if s[n] is not None]
    rows = {n: torch.zeros(s[n].shape, dtype=torch.float64, device="cuda") for n in names} if train else {}
    vectors = {n: s[n].detach().double().requires_grad_(True) for n in ("ln_w", "ln_b", "rms_w")} if op == "norms" else {}
    sums = {n: torch.zeros_like(t.detach()) for n, t in vectors.items()}
    for b, kb in enumerate(owner):
        at = {"q": slice(qo[b], qo[b + 1]), "k": slice(ko[kb], ko[kb + 1]), "v": slice(ko[kb], ko[kb + 1])}
        if at["q"].start == at["q"].stop:
            continue
        x = {n: s[n].detach()[at[n]].double().requires_grad_(train) for n in names}
        q, k = x["q"], x["k"]
        k, v = (k, x["v"]) if "v" in x else k.split(D, -1)
        if Hk != H:
            k, v = (t.repeat_interleave(H // Hk, 1) for t in (k, v))
        if op == "mxfp8":
            q, k, v = _mx_values(s["q"][at["q"]], 2), _mx_values(s["k"][at["k"]], 2), _mx_values(s["v"][at["v"]], 0)
        with torch.set_grad_enabled(train):
            if op == "norms":
                n = H * D
                ln = torch.nn.functional.layer_norm(q.reshape(-1, n), (n,), vectors["ln_w"], vectors["ln_b"], 1e-5)
                y = _attention64(ln.view(q.shape), k, v, s).reshape(-1, n) + ln
                y = y * torch.rsqrt(y.square().mean(1, keepdim=True) + 1e-5) * vectors["rms_w"]
                y = y.view(q.shape) + s["residual"][at["q"]].double()
            else:
                y = _attention64(q, k, v, s)
        out[at["q"]] = y.detach()
        if train:
            wanted = [x[n] for n in names] + list(vectors.values())
            got = torch.autograd.grad(y, wanted, s["dout"][at["q"]].double())
            for n, g in zip(names + list(vectors), got):
                if n in vectors:
                    sums[n] += g
                else:
                    rows[n][at[n]] = g
    return [out, *rows.values(), *sums.values()] if train else out
