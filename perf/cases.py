"""The attention calls whose speed this repository cares about, over the sizes its users call it with.

Every case is one call of `flash_b200.attention`, forward alone or forward and backward through autograd, as a
program that trains, encodes or serves with it makes them. `listed()` names one call per kind of use and `draw()`
gives other sizes of the same kinds. The package is taken from the working folder.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("triton-flash-attention-with-flexible-masks_b200"))
import flash_b200  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(use, B, H, Hk, M, N, D, dtype, causal, backward, docs="none", doc_seed=0, ndoc=0, always=0.0, std=1.0, layout="bhld"):
    """`docs`: how the ids of a mode-1 call are made (see `_lengths`), "none" for a call without ids. `doc_seed` fixes
    the documents' lengths, hence the unmasked entries; their order in the sequence comes from the inputs' seed.
    `layout`: "bhld" contiguous, "blhd" the views that a projection's output [B, L, H, D] is transposed to."""
    return dict(use=use, B=B, H=H, Hk=Hk, M=M, N=N, D=D, dtype=dtype, causal=causal, backward=backward, docs=docs,
                doc_seed=doc_seed, ndoc=ndoc, always=always, std=std, layout=layout)


def listed():
    cases = {
        # The smallest call in use: one short prompt of a small model. Launches and host time are all there is.
        "short_prompt": _case("prompt", 1, 8, 8, 200, 200, 64, "bf16", True, False),
        # Configuration 0 of the benchmark: fp32 training step of a check-sized model, documents and 5 % of
        # positions that attend everywhere.
        "fp32_step": _case("fp32", 2, 4, 4, 512, 512, 64, "fp32", True, True, "uniform", 0, 4, 0.05),
        # One token for each of 16 sequences against a cache of ragged length, grouped-query heads.
        "decode": _case("decode", 16, 32, 8, 1, 4500, 128, "bf16", True, False),
        # A block of new tokens against a long cache (chunked prefill, M < N).
        "prefill_chunk": _case("chunk", 1, 32, 8, 512, 8192, 128, "fp16", True, False),
        # An ordinary training step of a small model on packed documents of a ragged length, heads of 64, q / k / v
        # as the projection leaves them.
        "small_packed_step": _case("small", 4, 12, 12, 1000, 1000, 64, "bf16", True, True, "dirichlet", 5, 8, layout="blhd"),
        # Encoder step without causal mask or ids, narrow heads, odd length (patches and one class token).
        "encoder_step": _case("encoder", 16, 8, 8, 577, 577, 32, "fp16", False, True),
        # Training step with grouped-query heads, plain causal mask, ragged length, projection layout.
        "gqa_step": _case("gqa", 2, 32, 8, 3001, 3001, 128, "bf16", True, True, layout="blhd"),
        # Configuration 2: cross-attention in fp16, keys in 8 documents, queries assigned to them at random.
        "cross_step": _case("cross", 8, 8, 8, 1024, 8192, 64, "fp16", False, True, "random", 2, 8, std=0.5),
        # Configuration 1: packed pretraining step, 4096 tokens, 1 to 16 documents a sequence.
        "packed_step": _case("packed", 4, 16, 16, 4096, 4096, 128, "bf16", True, True, "dirichlet", 1, 16),
        # Configuration 3, the benchmark's headline: long-context packed pretraining step, 64 documents.
        "long_packed_step": _case("long", 1, 32, 32, 32768, 32768, 128, "bf16", True, True, "lognormal", 3, 64),
        # Configuration 4: dense causal prefill in fp16, the largest call.
        "dense_prefill": _case("dense", 16, 32, 32, 8192, 8192, 128, "fp16", True, False),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log_int(rng, lo, hi):
    """An integer from [lo, hi], even over the logarithm."""
    return min(hi, int(lo * (hi / lo) ** rng.random() + 0.5))


def _draw_one(rng):
    use = rng.choice(("prompt", "fp32", "decode", "chunk", "small", "encoder", "gqa", "cross", "packed", "long", "dense"))
    seed = rng.randrange(1 << 20)
    half = rng.choice(("bf16", "fp16"))
    gqa = rng.choice(((32, 8), (16, 4), (64, 8), (16, 16)))
    if use == "prompt":
        h, m = rng.choice((4, 8, 12, 16)), _log_int(rng, 16, 1024)
        return _case(use, rng.choice((1, 1, 2)), h, h, m, m, rng.choice((64, 128)), half, True, False)
    if use == "fp32":
        h, m = rng.choice((2, 4, 8)), _log_int(rng, 100, 1024)
        return _case(use, rng.choice((1, 2, 4)), h, h, m, m, rng.choice((32, 64, 128)), "fp32", True, True, "uniform", seed, 4, 0.05)
    if use == "decode":
        b = _log_int(rng, 1, 64)
        n = _log_int(rng, 512, max(1024, min(32768, (1 << 18) // b)))
        return _case(use, b, gqa[0], gqa[1], 1, n, rng.choice((64, 128)), half, True, False)
    if use == "chunk":
        m = _log_int(rng, 32, 2048)
        return _case(use, rng.choice((1, 1, 2)), gqa[0], gqa[1], m, m + _log_int(rng, 500, 16384), 128, half, True, False)
    if use == "small":
        h, m = rng.choice((8, 12, 16)), _log_int(rng, 256, 2048)
        return _case(use, rng.choice((2, 4, 8)), h, h, m, m, 64, half, True, True, "dirichlet", seed, rng.choice((4, 8)), layout="blhd")
    if use == "encoder":
        h, m = rng.choice((6, 8, 16)), _log_int(rng, 196, 1600)
        return _case(use, rng.choice((8, 16, 32)), h, h, m, m, rng.choice((16, 32, 64)), half, False, True)
    if use == "gqa":
        m = _log_int(rng, 1024, 6000)
        return _case(use, rng.choice((1, 2, 4)), gqa[0], gqa[1], m, m, rng.choice((64, 128)), half, True, True, layout="blhd")
    if use == "cross":
        h = rng.choice((8, 16))
        return _case(use, rng.choice((4, 8)), h, h, _log_int(rng, 300, 2048), _log_int(rng, 2048, 8192), 64, half, False, True, "random",
                     seed, rng.choice((4, 8, 16)), std=0.5)
    if use == "packed":
        h, m = rng.choice((16, 32)), _log_int(rng, 2000, 8192)
        return _case(use, rng.choice((1, 2, 4)), h, h, m, m, 128, half, True, True, "dirichlet", seed, 16)
    if use == "long":
        h, m = rng.choice((4, 8, 16, 32)), _log_int(rng, 12000, 32768)
        return _case(use, 1, h, h, m, m, 128, "bf16", True, True, "lognormal", seed, rng.choice((32, 64)))
    h, m = rng.choice((16, 32)), _log_int(rng, 1500, 8192)
    return _case(use, rng.choice((2, 4, 8, 16)), h, h, m, m, 128, half, True, False)


_LARGEST_FLOPS = 8.8e12  # dense_prefill


def draw(rng):
    while True:
        c = _draw_one(rng)
        if work(c)["flops"] <= _LARGEST_FLOPS:
            return c


def _lengths(c):
    """Document lengths of each sequence, a list of B integer arrays that sum to N each: "uniform" ndoc documents of
    uniform weights, "dirichlet" 1 to ndoc documents of Dirichlet(1) weights, "lognormal" ndoc documents of
    lognormal(6, 1) lengths, "random" ndoc equal ones."""
    rng = np.random.default_rng(c["doc_seed"])
    out = []
    for _ in range(c["B"]):
        if c["docs"] == "uniform":
            w = 0.2 + rng.random(c["ndoc"])
        elif c["docs"] == "dirichlet":
            w = rng.dirichlet(np.ones(int(rng.integers(1, c["ndoc"] + 1))))
        elif c["docs"] == "lognormal":
            w = rng.lognormal(6.0, 1.0, size=c["ndoc"])
        else:
            w = np.ones(c["ndoc"])
        ends = np.round(np.cumsum(w) / w.sum() * c["N"]).astype(np.int64)
        out.append(np.diff(np.concatenate([[0], ends])))
    return out


def _ids(c, rng):
    """(eq, ek), int64 [B, M] and [B, N]: negative document ids, and id 1 where a position attends everywhere."""
    rows = []
    for lengths in _lengths(c):
        order = rng.permutation(len(lengths))
        row = np.repeat(-(np.arange(len(lengths), dtype=np.int64) + 1), lengths[order])
        if c["always"]:
            row[rng.random(c["N"]) < c["always"]] = 1
        rows.append(row)
    ek = np.stack(rows)
    if c["docs"] == "random":  # every query belongs to a document of its own choice
        return -(rng.integers(0, c["ndoc"], size=(c["B"], c["M"])) + 1), ek
    return ek, ek


def _unmasked(c):
    """Unmasked entries of the score matrix, over all batches and heads (expected ones where positions are random)."""
    M, N = c["M"], c["N"]
    full = M * N - (M * (M - 1) // 2 if c["causal"] else 0)
    if c["docs"] == "none":
        return c["B"] * c["H"] * full
    total = 0.0
    for lengths in _lengths(c):
        x = lengths.astype(np.float64)
        if c["docs"] == "random":
            seen = M * float(N) / c["ndoc"]
        else:  # self-attention: inside its document, up to itself
            seen = float((x * (x + 1) / 2 if c["causal"] else x * x).sum())
        total += c["always"] * full + (1 - c["always"]) ** 2 * seen
    return c["H"] * total


def work(case):
    """Flops of the unmasked entries alone (2 products forward, 5 backward); each input read and each output written once."""
    c = case
    size = 4 if c["dtype"] == "fp32" else 2
    q, kv = c["B"] * c["H"] * c["M"] * c["D"] * size, c["B"] * c["Hk"] * c["N"] * c["D"] * size
    tensors = (2 * q + 2 * kv) + (2 * q + 2 * kv if c["backward"] else 0)  # q, k, v, o and dO, dq, dk, dv
    ids = 0 if c["docs"] == "none" else 8 * c["B"] * (c["N"] + (c["M"] if c["docs"] == "random" else 0))
    return {"bytes": tensors + ids, "flops": (14 if c["backward"] else 4) * c["D"] * _unmasked(c)}


def tolerance(case):
    # P and dS are rounded to the inputs' type once on the way, results once more; fp32 sums stay in fp32
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[case["dtype"]]}


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[c["dtype"]]

    def values(heads, length):
        shape = (c["B"], heads, length, c["D"]) if c["layout"] == "bhld" else (c["B"], length, heads, c["D"])
        x = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).mul_(c["std"]).to(dtype)
        return x if c["layout"] == "bhld" else x.transpose(1, 2)

    s = {"causal": c["causal"], "backward": c["backward"], "mode": flash_b200.SCORE_FUNC_MODE0_NOPE, "eq": None, "ek": None,
         "q": values(c["H"], c["M"]), "k": values(c["Hk"], c["N"]), "v": values(c["Hk"], c["N"]), "do": None}
    if c["backward"]:
        s["do"] = values(c["H"], c["M"])
        for n in ("q", "k", "v"):
            s[n].requires_grad_()
    if c["docs"] != "none":
        eq, ek = _ids(c, np.random.default_rng(seed))
        d_ek = torch.from_numpy(ek).cuda()
        d_eq = d_ek if eq is ek else torch.from_numpy(eq).cuda()
        s["mode"] = flash_b200.SCORE_FUNC_MODE1_DOC
        s["eq"] = d_eq[:, None, :].expand(c["B"], c["H"], c["M"])
        s["ek"] = d_ek[:, None, :].expand(c["B"], c["H"], c["N"])
    return s


def run(state):
    s = state
    o = flash_b200.attention(s["q"], s["k"], s["v"], s["causal"], None, s["eq"], s["ek"], s["mode"])
    if not s["backward"]:
        return o
    return (o.detach(), *torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["do"]))


def exact(case, seed):
    """What `run` returns for these inputs, in 64 bits: whole rows of the score matrix, as many at a time as fit in 1 GB."""
    c, s = case, prepare(case, seed)
    B, H, M, N, D = c["B"], c["H"], c["M"], c["N"], c["D"]
    group, gap, scale = H // c["Hk"], max(0, N - M), 1.0 / D ** 0.5
    new = {"device": "cuda", "dtype": torch.float64}
    o = torch.zeros(B, H, M, D, **new)
    dq, dk, dv = (torch.zeros(B, h, n, D, **new) if c["backward"] else None for h, n in ((H, M), (c["Hk"], N), (c["Hk"], N)))
    keys = torch.arange(N, device="cuda")
    step = max(1, min(M, (1 << 27) // N))
    with torch.no_grad():
        for b in range(B):
            for h in range(H):
                hk = h // group
                k, v = s["k"][b, hk].double(), s["v"][b, hk].double()
                for i in range(0, M, step):
                    rows = slice(i, min(i + step, M))
                    last = min(N, rows.stop + gap) if c["causal"] else N  # no row of these sees a later key
                    q = s["q"][b, h, rows].double()
                    p = (q @ k[:last].T).mul_(scale)
                    if c["causal"]:
                        p.masked_fill_(keys[None, :last] > torch.arange(rows.start, rows.stop, device="cuda")[:, None] + gap, -torch.inf)
                    if s["eq"] is not None:
                        eq, ek = s["eq"][b, h, rows, None], s["ek"][b, h, None, :last]
                        p.masked_fill_((eq < 0) & (eq != ek), -torch.inf)
                    p.sub_(p.amax(1, keepdim=True).clamp_(min=-1e300)).exp_()
                    p.div_(p.sum(1, keepdim=True).clamp_(min=1e-300))  # a row without keys gives zeros
                    o[b, h, rows] = p @ v[:last]
                    if c["backward"]:
                        do = s["do"][b, h, rows].double()
                        dv[b, hk, :last] += p.T @ do
                        ds = (do @ v[:last].T).sub_((do * o[b, h, rows]).sum(1, keepdim=True)).mul_(p)
                        dq[b, h, rows] = (ds @ k[:last]).mul_(scale)
                        dk[b, hk, :last] += (ds.T @ q).mul_(scale)
    return (o, dq, dk, dv) if c["backward"] else o
