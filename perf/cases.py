"""The workloads this framework is measured on, through its public entry points.

Sizes are those of the benchmark configurations (bench.py), of the test grid (tests/) and generic ones in
between.  Kinds of case:

  train   flex_block_attn_func forward + backward with a bool block mask that changes from step to step
          (compaction, work orders, forward, backward in every pass)
  sta     the same with prebuilt sliding-tile lists (a static mask: a program builds them once)
  ssta    list building from q and k (window + top-k of pooled scores), forward, backward
  infer   forward alone, no gradients
  layout  inference on raster-order activations [B, S, H, 128]: to_tile_major of q, k, v, forward over
          sliding-tile lists, from_tile_major of the output
  fp8     inference forward over an e4m3 key / value cache
  cache   the cache writer: quantize_kv of one layer's keys and values
"""
import math

import torch

import flex_block_attn_b200 as fba
from flex_block_attn_b200 import masks

D = 128


def _case(kind, name=None, **kw):
    c = {"kind": kind, "B": 1, "Hq": 24, "Hkv": 24, "Sq": 0, "Skv": 0, "qb": 384, "kb": 384, "mask": "random4",
         "keep": 0.4, "std": 1.0, "softmax_scale": 0.0}
    c.update(kw)
    if c["kind"] in ("sta", "ssta", "layout"):
        c["Sq"] = c["Skv"] = c["gt"] * c["gh"] * c["gw"] * c["kb"]
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # Training on a long video latent (18x48x80 tokens) with a fresh random mask per step: the headline workload.
        _case("train", "train_random_s69120", Sq=69120, Skv=69120),
        # The short end of the same sweep: the attention kernels are milliseconds, lists and orders start to count.
        _case("train", "train_random_s11520", Sq=11520, Skv=11520),
        # Dense layers mixed into a sparse model: all-ones mask shared by all heads.
        _case("train", "train_full_s30720", Sq=30720, Skv=30720, mask="full2", std=0.5),
        # Window + top-k selection recomputed from q and k at every step, asymmetric 128 / 384 blocks, batch 2.
        _case("ssta", "train_ssta_s69120_b2", B=2, qb=128, kb=384, gt=3, gh=6, gw=10, topk=8),
        # Fine blocks (64 x 64, below one tile): sub-tile masks inside the kernels, a few heads, a banded mask.
        _case("train", "train_fine_s3072", Hq=4, Hkv=4, Sq=3072, Skv=3072, qb=64, kb=64, mask="band4"),
        # The smallest training call: two heads, a 4 x 4 block grid, latency and launches.
        _case("train", "train_small_s1536", Hq=2, Hkv=2, Sq=1536, Skv=1536, mask="random2", keep=0.5),
        # Cross attention with grouped-query heads, block sizes and lengths that are no multiples of a tile.
        _case("train", "train_gqa_ragged", B=2, Hq=8, Hkv=2, Sq=3696, Skv=4800, qb=48, kb=192),
        # Sampling / prefill: forward only over a medium sequence.
        _case("infer", "infer_random_s30720", Sq=30720, Skv=30720),
        # The smallest inference call: one short prompt, four heads.
        _case("infer", "infer_small_s768", Hq=4, Hkv=4, Sq=768, Skv=768, qb=64, kb=128, mask="band4"),
        # Sampling step of a video model that keeps its activations in raster order: layout change in and out.
        _case("layout", "infer_sta_raster_s69120", gt=3, gh=6, gw=10, tt=6, th=8, tw=8),
        # Inference that reads its keys and values from an 8-bit cache.
        _case("fp8", "infer_fp8_s30720", Sq=30720, Skv=30720),
        # Writing that cache: one layer's keys and values.
        _case("cache", "cache_write_s30720", Sq=30720, Skv=30720),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw(rng):
    kind = rng.choice(["train", "train", "train", "train", "sta", "ssta", "infer", "infer", "layout", "fp8", "cache"])
    keep = round(rng.uniform(0.1, 0.7), 3)
    if kind in ("sta", "ssta", "layout"):
        tile = rng.choice([(6, 8, 8), (4, 8, 8), (4, 4, 8), (2, 8, 8)])
        kb = tile[0] * tile[1] * tile[2]
        g = {"gt": rng.randint(1, 5), "gh": rng.randint(2, 8), "gw": rng.randint(2, 12)}
        B, H = rng.choice([(1, 24), (1, 12), (2, 12), (1, 3), (2, 24)])
        if kind == "ssta":
            qb = rng.choice([q for q in (128, 384) if kb % q == 0])
            return _case(kind, B=B, Hq=H, Hkv=H, qb=qb, kb=kb, topk=rng.randint(2, 12), **g)
        if kind == "layout":
            return _case(kind, B=B, Hq=H, Hkv=H, qb=kb, kb=kb, tt=tile[0], th=tile[1], tw=tile[2], **g)
        return _case(kind, B=B, Hq=H, Hkv=H, qb=kb, kb=kb, **g)
    if kind == "cache":
        kb = 128 * rng.randint(1, 6)
        return _case(kind, B=rng.choice([1, 2]), Hq=24, Hkv=rng.choice([2, 8, 24]), kb=kb,
                     Sq=kb, Skv=kb * _log_int(rng, 3, max(4, 60000 // kb)), qb=kb)
    if kind == "fp8":
        qb, kb = rng.choice([(384, 384), (128, 384), (128, 128), (256, 256)])
        n = _log_int(rng, 2, 40000 // max(qb, kb))
        return _case(kind, B=1, Hq=24, Hkv=rng.choice([24, 8]), Sq=n * max(qb, kb), Skv=n * max(qb, kb), qb=qb, kb=kb,
                     keep=keep)
    B, Hq, Hkv = rng.choice([(1, 24, 24), (1, 24, 24), (1, 3, 3), (2, 8, 2), (1, 2, 2), (2, 12, 12)])
    qb, kb = rng.choice([(384, 384), (384, 384), (128, 384), (128, 128), (64, 64), (48, 192), (16, 128), (192, 64), (256, 256)])
    if kb >= 128 and qb >= 128:
        m = max(qb, kb)
        n = _log_int(rng, 2, 69120 // m)
        Sq = n * m
        Skv = Sq if rng.random() < 0.8 else m * _log_int(rng, 2, 69120 // m)
    else:
        Sq = qb * _log_int(rng, max(2, 400 // qb), 12000 // qb)
        Skv = kb * _log_int(rng, max(2, 400 // kb), 12000 // kb)
    mask = rng.choice(["random4", "random4", "random2", "band4", "full2"])
    return _case(kind, B=B, Hq=Hq, Hkv=Hkv, Sq=Sq, Skv=Skv, qb=qb, kb=kb, mask=mask, keep=keep,
                 std=rng.choice([1.0, 1.0, 0.5]), softmax_scale=rng.choice([0.0, 0.0, 0.0, 0.07]))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        c = _draw(rng)
        w = work(c)
        if w["flops"] <= most and w["bytes"] <= 8e9:
            return c


def _mask(c, g):
    nQ, nK = c["Sq"] // c["qb"], c["Skv"] // c["kb"]
    if c["mask"] == "full2":
        return torch.ones((nQ, nK), dtype=torch.bool, device="cuda")
    shape = (c["B"], c["Hq"], nQ, nK) if c["mask"].endswith("4") else (nQ, nK)
    i, j = torch.arange(nQ, device="cuda"), torch.arange(nK, device="cuda")
    if c["mask"] == "band4":   # |i - j| < 2 in key blocks, plus one column everybody attends to
        m = ((i[:, None] * nK // nQ - j[None, :]).abs() < 2) | (j[None, :] == min(4, nK - 1))
        return m.expand(shape).contiguous()
    m = torch.rand(shape, generator=g, device="cuda") < c["keep"]
    m[..., i, (i * nK) // nQ] = True
    return m


def prepare(case, seed):
    c = dict(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    grads = c["kind"] in ("train", "sta", "ssta")

    def tensor(heads, rows):
        shape = (c["B"], rows, heads, D) if c["kind"] == "layout" else (c["B"], heads, rows, D)
        return torch.randn(shape, generator=g, device="cuda", dtype=torch.bfloat16).mul_(c["std"])

    s = {"case": c, "q": tensor(c["Hq"], c["Sq"]), "k": tensor(c["Hkv"], c["Skv"]), "v": tensor(c["Hkv"], c["Skv"])}
    s["softmax_scale"] = c["softmax_scale"] or None
    if grads:
        s["do"] = tensor(c["Hq"], c["Sq"])
        for x in ("q", "k", "v"):
            s[x].requires_grad_()
    if c["kind"] in ("sta", "layout"):
        s["mask"] = fba.sta_lists((c["gt"], c["gh"], c["gw"]), (1, 1, 1), c["kb"])
    elif c["kind"] in ("train", "infer", "fp8"):
        s["mask"] = _mask(c, g)
    if c["kind"] == "fp8":
        s["cache"] = fba.quantize_kv(s.pop("k"), s.pop("v"), c["kb"])
    if c["kind"] == "layout":
        s["tile"] = (c["tt"], c["th"], c["tw"])
        s["grid"] = (c["gt"] * c["tt"], c["gh"] * c["th"], c["gw"] * c["tw"])
    return s


def run(s):
    c = s["case"]
    kind, qb, kb = c["kind"], c["qb"], c["kb"]
    if kind == "cache":
        r = fba.quantize_kv(s["k"], s["v"], kb)
        return {"k8": r.k8, "v8t": r.v8t, "k_scale": r.k_scale, "v_scale": r.v_scale}
    q = s["q"]
    if kind == "fp8":
        return fba.flex_block_attn_fp8kv(q, s["cache"], qb, kb, s["mask"], s["softmax_scale"])
    k, v = s["k"], s["v"]
    if kind == "infer":
        with torch.no_grad():
            return fba.flex_block_attn_func(q, k, v, qb, kb, s["mask"], s["softmax_scale"])
    if kind == "layout":
        with torch.no_grad():
            q, k, v = (masks.to_tile_major(x, s["grid"], s["tile"]) for x in (q, k, v))
            o = fba.flex_block_attn_func(q, k, v, qb, kb, s["mask"], s["softmax_scale"])
            return masks.from_tile_major(o, s["grid"], s["tile"])
    lists = s.get("mask")
    if kind == "ssta":
        with torch.no_grad():
            lists, _ = fba.ssta_lists(q, k, (c["gt"], c["gh"], c["gw"]), qb, kb, topk=c["topk"])
    o = fba.flex_block_attn_func(q, k, v, qb, kb, lists, s["softmax_scale"])
    dq, dk, dv = torch.autograd.grad(o, (q, k, v), s["do"])
    return {"o": o, "dq": dq, "dk": dk, "dv": dv}


def _active_pairs(c):
    """Active (query block, key block) pairs of one (batch, head); the expected number for random masks."""
    nQ, nK = c["Sq"] // c["qb"], c["Skv"] // c["kb"]
    if c["kind"] in ("sta", "ssta", "layout"):
        near = lambda n: 3 * n - 2          # ordered neighbour pairs |a - b| <= 1 of n positions
        window = near(c["gt"]) * near(c["gh"]) * near(c["gw"]) / nK    # mean tiles per query tile
        if c["kind"] == "ssta":
            window += min(c["topk"], nK) * (1 - window / nK)
        return nQ * window
    if c["mask"] == "full2":
        return nQ * nK
    if c["mask"] == "band4":
        last = min(4, nK - 1)
        n = 0
        for i in range(nQ):
            b = i * nK // nQ
            lo, hi = max(b - 1, 0), min(b + 1, nK - 1)
            n += hi - lo + 1 + (0 if lo <= last <= hi else 1)
        return n
    return nQ * (1 + (nK - 1) * c["keep"])


def work(case):
    c = case
    q_bytes = 2 * D * c["B"] * c["Hq"] * c["Sq"]
    kv_bytes = 2 * D * c["B"] * c["Hkv"] * c["Skv"]
    if c["kind"] == "cache":    # bf16 in, 8-bit out, keys and values
        return {"bytes": 2 * kv_bytes + kv_bytes, "flops": 0}
    pairs = c["B"] * c["Hq"] * _active_pairs(c)
    per_pair = c["qb"] * c["kb"] * D
    if c["kind"] in ("train", "sta", "ssta"):    # q, dO in, O, dQ out; k, v in, dK, dV out
        return {"bytes": 4 * q_bytes + 4 * kv_bytes, "flops": 14 * pairs * per_pair}
    if c["kind"] == "fp8":
        return {"bytes": 2 * q_bytes + kv_bytes, "flops": 4 * pairs * per_pair}
    return {"bytes": 2 * q_bytes + 2 * kv_bytes, "flops": 4 * pairs * per_pair}


def tolerance(case):
    """How far two correct implementations at the same precision may be apart: about four times the distance of
    this one from the same mathematics in 64 bits (measured on four of the cases: 2-norm 2.4e-3, largest 2.8e-2)."""
    if case["kind"] == "cache":
        return "exact"
    if case["kind"] == "fp8":    # three mantissa bits in q and P (measured: 3.7e-2 from the dequantised cache)
        return {"rel": 0.03}
    return {"rel": 1e-2, "max": 0.12}    # P and dS rounded to bf16 before their products, bf16 outputs
