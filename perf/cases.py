"""The attention calls whose speed this package answers for.

Each case is one call of a public entry point (`sageattn`, `sageattn_qk_int8_pv_fp8` or
`sageattn_varlen`) as a program makes it: inputs already on the GPU, output left there.  The listed
cases are the sizes of the benchmark (H=48; N=288 .. 47520), of the tests and of the documented
options; `draw` takes further ones from the same ranges:

  self    queries and keys of one sequence, 64 .. 47520 tokens, both masks, both types, contiguous
          (HND, NHD) or views of one fused QKV projection, grouped heads, head_dim 64 .. 128
  cross   many image or video tokens against a short text (non-causal, 64 .. 1024 keys)
  few     a few new queries against many keys (non-causal, 1 .. 128 queries)
  packed  a ragged batch of sequences with its cumulative lengths on the GPU

Values are N(0,1) with what the path's options exist for: a K bias per channel (smooth_k), heads of
different magnitude, a few dominant key tokens (0.1 % scaled x50), a V offset (smooth_v).
"""
import math
import os
import random
import sys

import torch

_PKG = os.path.join(os.getcwd(), "sageattention-rdna4_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import sageattention  # noqa: E402

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
_BASE = dict(kind="self", b=1, hq=48, hkv=48, nq=0, nk=0, d=128, dtype="fp16", layout="HND", causal=False,
             lse=False, smooth_v=False, e4m3=False, k_bias=0.5, head_scale=False, dominant=0.0, lengths_seed=0)
#: (query, key) pairs of the largest listed call; nothing drawn has more than 0.6 times as many.
_MOST_PAIRS = 48 * 47520 * 47520


def _case(name, n=None, **kw):
    c = dict(_BASE, name=name, **kw)
    if n is not None:
        c["nq"] = c["nk"] = n
    if c["hkv"] > c["hq"]:
        c["hkv"] = c["hq"]
    return c


def listed():
    return [
        # A small image or a preview step: a handful of launches and the host path are the whole cost.
        _case("self_288", 288),
        # A short sequence of ragged length out of a fused QKV projection, two batch entries.
        _case("self_1000_fused_bf16", 1000, b=2, hq=24, dtype="bf16", layout="fused"),
        # An ordinary square call of the short-call sweep.
        _case("self_4096", 4096),
        # Image-size call, non-causal, K bias and heads of different magnitude (int8 Q.K).
        _case("image_8771", 8771, k_bias=1.0, head_scale=True),
        # Image-size call, causal, bf16 (e4m3 Q.K).
        _case("image_8771_causal_bf16", 8771, dtype="bf16", causal=True, k_bias=1.0),
        # Video-length call with dominant key tokens: the headline benchmark.
        _case("video_47520_dominant", 47520, k_bias=0.0, dominant=0.001),
        # Video-length call without dominant keys, bf16, views of one fused QKV projection.
        _case("video_27280_fused_bf16", 27280, hq=24, dtype="bf16", layout="fused"),
        # Cross attention of a video step: many tokens against a text of a few hundred.
        _case("cross_16384x512", kind="cross", hq=40, nq=16384, nk=512, layout="NHD", dtype="bf16"),
        # A few new queries against a long context, grouped heads.
        _case("few_4x16384_gqa", kind="few", b=2, hq=32, hkv=8, nq=4, nk=16384),
        # Causal prefill with grouped heads and the log-sum-exp a caller merges partial results with.
        _case("prefill_4096_gqa_lse", 4096, b=2, hq=32, hkv=8, causal=True, lse=True, dtype="bf16", layout="NHD"),
        # A packed batch of eleven sequences of very different length.
        _case("packed_11_ragged", kind="packed", b=11, hq=48, nq=8192, nk=8192, lengths_seed=11),
        # Narrow heads, e4m3 Q.K codes for fp16 inputs and smooth_v, batch of four.
        _case("self_2048_d64_smooth_v", 2048, b=4, hq=16, d=64, e4m3=True, smooth_v=True, layout="NHD"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["self", "self", "self", "cross", "few", "packed"])
    hkv = rng.choice([4, 8, 12, 16, 24, 40, 48])
    c = dict(_BASE, kind=kind, dtype=rng.choice(["fp16", "bf16"]), d=rng.choice([128, 128, 128, 96, 64]),
             hkv=hkv, hq=hkv * (rng.choice([1, 1, 2, 4]) if hkv <= 12 else 1),
             layout=rng.choice(["HND", "NHD"]), k_bias=rng.choice([0.0, 0.5, 1.0]))
    if kind == "self":
        c["b"] = rng.choice([1, 1, 2, 4])
        c["causal"] = rng.random() < 0.4
        c["lse"] = rng.random() < 0.25
        c["smooth_v"] = rng.random() < 0.2
        c["e4m3"] = c["dtype"] == "fp16" and rng.random() < 0.25
        c["head_scale"] = rng.random() < 0.25
        if c["hq"] == c["hkv"] and rng.random() < 0.4:
            c["layout"] = "fused"
        most = min(47520, int(math.sqrt(0.6 * _MOST_PAIRS / (c["b"] * c["hq"]))))
        c["nq"] = c["nk"] = _log_int(rng, 64, most)
        if c["nq"] >= 4096 and rng.random() < 0.3:
            c["dominant"] = 0.001
    elif kind == "cross":
        c["b"] = rng.choice([1, 2])
        c["nq"], c["nk"] = _log_int(rng, 256, 32768), _log_int(rng, 64, 1024)
    elif kind == "few":
        c["b"] = rng.choice([1, 2, 4])
        c["nq"], c["nk"] = _log_int(rng, 1, 128), _log_int(rng, 512, 32768)
    else:
        c["b"] = rng.randint(2, 16)
        c["causal"] = rng.random() < 0.5
        c["nq"] = c["nk"] = _log_int(rng, 256, 8192)
        c["lengths_seed"] = rng.randrange(1 << 30)
    return c


def _lengths(case):
    """Sequence lengths of a packed batch: the longest allowed once, the others spread below it."""
    rng = random.Random(case["lengths_seed"])
    lens = [_log_int(rng, max(1, case["nq"] // 16), case["nq"]) for _ in range(case["b"] - 1)]
    lens.insert(rng.randint(0, len(lens)), case["nq"])
    return lens


def _randn(gen, shape, dtype, dev):
    """N(0,1) in fp32, cast; made slice by slice so that the fp32 values of a large input never exist at once."""
    out = torch.empty(shape, dtype=dtype, device=dev)
    for i in range(shape[0]):
        for j in range(0, shape[1], 8192):
            part = out[i, j:j + 8192]
            part.copy_(torch.randn(part.shape, generator=gen, device=dev))
    return out


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(1_000_003 * (seed + 1))
    dt, b, hq, hkv, d = _DTYPES[case["dtype"]], case["b"], case["hq"], case["hkv"], case["d"]
    state = {"case": dict(case)}
    if case["kind"] == "packed":
        lens = _lengths(case)
        b, nq, nk = 1, sum(lens), sum(lens)
        state["cu"] = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=dev)
        state["longest"] = max(lens)
    else:
        nq, nk = case["nq"], case["nk"]
    # everything is made as (B, N, H, D) and laid out below
    if case["layout"] == "fused":
        qkv = _randn(gen, (b, nq, 3, hq, d), dt, dev)
        q, k, v = qkv.unbind(2)
    else:
        q, k, v = (_randn(gen, (b, n, h, d), dt, dev) for n, h in ((nq, hq), (nk, hkv), (nk, hkv)))
    if case["k_bias"] > 0:
        k += (case["k_bias"] * torch.randn((1, 1, hkv, d), generator=gen, device=dev)).to(dt)
    if case["head_scale"]:
        group = hq // hkv
        mult = lambda h: 0.5 + 1.5 * torch.rand((1, 1, h, 1), generator=gen, device=dev)
        q *= mult(hkv).repeat_interleave(group, 2).to(dt)
        k *= mult(hkv).to(dt)
    if case["dominant"] > 0:
        rows = torch.randperm(nk, generator=gen, device=dev)[:max(1, round(case["dominant"] * nk))]
        k[:, rows] = k[:, rows] * 50
    if case["smooth_v"]:
        v += (2.0 * torch.randn((1, 1, hkv, d), generator=gen, device=dev)).to(dt)
    if case["kind"] == "packed":
        q, k, v = q[0], k[0], v[0]
    elif case["layout"] == "HND":
        q, k, v = (t.transpose(1, 2).contiguous() for t in (q, k, v))
    state.update(q=q, k=k, v=v)
    return state


def run(state):
    c, q, k, v = state["case"], state["q"], state["k"], state["v"]
    if c["kind"] == "packed":
        return sageattention.sageattn_varlen(q, k, v, state["cu"], state["cu"], state["longest"], state["longest"],
                                             is_causal=c["causal"])
    layout = "HND" if c["layout"] == "HND" else "NHD"
    if c["smooth_v"] and not c["e4m3"]:
        return sageattention.sageattn_qk_int8_pv_fp8(q, k, v, tensor_layout=layout, is_causal=c["causal"],
                                                     pv_accum_dtype="fp32", smooth_v=True, return_lse=c["lse"])
    return sageattention.sageattn(q, k, v, tensor_layout=layout, is_causal=c["causal"], return_lse=c["lse"],
                                  sk1_int8=False if c["e4m3"] else None, smooth_v=c["smooth_v"])


def work(case):
    """Each input read once, each output written once; the two products, halved when causal."""
    hq, hkv, d = case["hq"], case["hkv"], case["d"]
    if case["kind"] == "packed":
        lens = _lengths(case)
        rows_q = rows_k = sum(lens)
        pairs = sum(n * n for n in lens)
    else:
        rows_q, rows_k = case["b"] * case["nq"], case["b"] * case["nk"]
        pairs = case["b"] * case["nq"] * case["nk"]
    nbytes = 2 * d * (2 * rows_q * hq + 2 * rows_k * hkv)
    if case["lse"]:
        nbytes += 4 * rows_q * hq
    return {"bytes": nbytes, "flops": 4 * pairs * hq * d // (2 if case["causal"] else 1)}


def tolerance(case):
    """P is rounded to e4m3 against the running row maximum, so the order in which keys are visited
    moves the roundings.  Measured with the oracle (tiles of 64 and 256 keys against 128): relative
    2-norm 0.006 .. 0.015 for 288 .. 8771 tokens, largest difference 0.04 .. 0.12 of the result's
    root mean square, 0.23 in the first rows of a causal call."""
    return {"rel": 0.03, "max": 0.5}


def _attend64(q, k, v, causal):
    """(softmax(q k^T / sqrt(d)) v, log-sum-exp) of one head in 64 bits, a block of queries at a time."""
    n, m = q.shape[0], k.shape[0]
    out = torch.empty((n, v.shape[1]), dtype=torch.float64, device=q.device)
    lse = torch.empty((n,), dtype=torch.float64, device=q.device)
    k, v = k.double(), v.double()
    keys = torch.arange(m, device=q.device)
    for i in range(0, n, 4096):
        s = (q[i:i + 4096].double() @ k.T) * q.shape[1] ** -0.5
        if causal:
            s.masked_fill_(keys[None, :] > torch.arange(i, i + s.shape[0], device=q.device)[:, None], -math.inf)
        lse[i:i + 4096] = torch.logsumexp(s, 1)
        out[i:i + 4096] = torch.exp_(s.sub_(lse[i:i + 4096, None])) @ v
    return out, lse


def exact(case, seed):
    """Plain attention in 64 bits.  None where e4m3 score codes meet keys scaled x50: the format alone
    puts such outputs 0.2 off, so the distance says nothing about an implementation."""
    if case["dominant"] > 0 and (case["e4m3"] or case["dtype"] == "bf16"):
        return None
    state = prepare(case, seed)
    q, k, v = state["q"], state["k"], state["v"]
    group = case["hq"] // case["hkv"]
    if case["kind"] == "packed":
        out = torch.zeros(q.shape, dtype=torch.float64, device=q.device)
        cu = state["cu"].tolist()
        for a, z in zip(cu, cu[1:]):
            for h in range(case["hq"]):
                out[a:z, h] = _attend64(q[a:z, h], k[a:z, h // group], v[a:z, h // group], case["causal"])[0]
        return out
    out = torch.empty(q.shape, dtype=torch.float64, device=q.device)
    heads = (lambda t: t) if case["layout"] == "HND" else (lambda t: t.transpose(1, 2))
    lse = torch.empty((case["b"], case["hq"], case["nq"]), dtype=torch.float64, device=q.device)
    for b in range(case["b"]):
        for h in range(case["hq"]):
            o, lse[b, h] = _attend64(heads(q)[b, h], heads(k)[b, h // group], heads(v)[b, h // group], case["causal"])
            heads(out)[b, h] = o
    return (out, lse) if case["lse"] else out
