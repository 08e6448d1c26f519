"""The work that programs have this framework do, as cases that can be timed.

A serving program fills a compressed KV cache (prompts in one piece, in chunks, or token by token), attends over it once
per layer and generated token, and runs the dense attention of prompts and encoders beside it. The cases take that work
through the public entry points over the range from one short sequence, where launches and host time count, to caches of
several GB. Sizes are those of the benchmark's workloads where one exists, and generic ones otherwise.

Kinds of a case (`kind`):
  step    TurboKvCache.append of the new token(s) + TurboKvCache.attention: a decode step of one layer
  packed  PackedAttention.run: a prepared decode call over packed rows, one length per sequence in device memory
  blocks  PackedBlocksAttention.run: the same over the blocks of a paged cache
  chunk   TurboKvCache.append + TurboKvCache.attention of a long chunk: prompt pieces over an already compressed cache
  append  prefill_append: causal attention of a whole prompt and its rows written to the cache, one call
  varlen  flash_attn_varlen: prompts of different lengths, packed one behind the other
  dense   flash_attn_with_config: attention over uncompressed keys and values, decode (lq 1) to long encoders
  codec   TurboQuantizer.quantize + dequantize: rows into and out of a format
"""
import numpy as np
import torch

import __graft_entry__

P = __graft_entry__.load_package()
F = P.flash_attn
DEV = "cuda:0"
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
ROW_WORDS = {"mxfp4": lambda d: d // 8 + (d // 32 + 3) // 4 + 2, "nvfp4": lambda d: d // 8 + (d // 16 + 3) // 4 + 2,
             "mxfp8": lambda d: d // 4 + (d // 32 + 3) // 4 + 2, "fp8": lambda d: d // 4 + 2, "turbo4": lambda d: d // 8 + 2}


def listed():
    return [
        # one user's decode step over a short FP8 cache: the smallest call, launches and host time
        dict(name="step_fp8_b1_2k", kind="step", fmt="fp8", rot="none", dt="f16", b=1, hq=32, hkv=8, d=128, lk=2047, lq=1),
        # a small batch over the formats that this device's profile chooses (NVFP4, rotated), at an odd length
        dict(name="step_nvfp4_b8_5k", kind="step", fmt="nvfp4", rot="auto", dt="bf16", b=8, hq=32, hkv=8, d=128, lk=5002, lq=1),
        # continuous batching: 64 sequences of 512 to 8192 keys, outlier channels
        dict(name="ragged_mxfp4_b64", kind="packed", fmt="mxfp4", rot="none", dt="bf16", b=64, hq=32, hkv=8, d=128, lmin=512, lk=8192, lq=1),
        # long contexts in codebook rows, one kv head of a layer whose heads are spread over GPUs
        dict(name="long_turbo4_b32_32k", kind="packed", fmt="turbo4", rot="auto", dt="bf16", b=32, hq=8, hkv=1, d=128, lmin=32768, lk=32768, lq=1),
        # the largest cache: one layer of a full serving batch, 4.7 GB
        dict(name="large_mxfp8_b128_16k", kind="packed", fmt="mxfp8", rot="none", dt="f16", b=128, hq=32, hkv=8, d=128, lmin=16384, lk=16384, lq=1),
        # speculative decoding over a paged cache: four query tokens, sequences of their own lengths, a part-filled last block
        dict(name="paged_mxfp4_b16_4k", kind="blocks", fmt="mxfp4", rot="none", dt="bf16", b=16, hq=32, hkv=8, d=128, page=512, lmin=1000, lk=4000, lq=4),
        # a 1024-token piece of a long prompt over 7168 tokens that are already in the cache
        dict(name="chunk_mxfp8_1k_of_8k", kind="chunk", fmt="mxfp8", rot="auto", dt="bf16", b=1, hq=32, hkv=8, d=128, lk=7168, lq=1024),
        # whole prompts into an NVFP4 cache
        dict(name="prefill_nvfp4_b4_4k", kind="append", fmt="nvfp4", rot="none", dt="bf16", b=4, hq=32, hkv=8, d=128, lk=4096, lq=4096),
        # prompts of a request queue, packed, lengths as they come
        dict(name="varlen_prompts_b12", kind="varlen", dt="bf16", b=12, hq=32, hkv=8, d=128, lmin=100, lk=3000, causal=True),
        # decode over uncompressed keys and values
        dict(name="dense_decode_b64_4k", kind="dense", dt="bf16", b=64, hq=32, hkv=8, d=128, lq=1, lk=4096, causal=True),
        # an encoder: no mask, head dim 64, a length that is no multiple of any tile
        dict(name="encoder_d64_b8_1000", kind="dense", dt="f16", b=8, hq=16, hkv=16, d=64, lq=1000, lk=1000, causal=False),
        # rows of a prompt into codebook rows and back (offload, inspection, moving between formats)
        dict(name="codec_turbo4_64k_rows", kind="codec", fmt="turbo4", rot="auto", dt="bf16", b=1, hkv=8, d=128, lk=8191),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm, odd ones among them."""
    return int(min(hi, max(lo, round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    while True:  # none costs more than the largest listed ones: 4.7 GB, 0.55 TFLOP
        c = _drawn(rng)
        w = work(c)
        if w["bytes"] <= 4.5e9 and w["flops"] <= 5.4e11:
            return c


def _drawn(rng):
    kind = rng.choice(["step", "step", "packed", "packed", "blocks", "chunk", "append", "varlen", "dense", "dense", "codec"])
    fmt = rng.choice(["fp8", "mxfp8", "mxfp4", "nvfp4", "turbo4"])
    hq, hkv = rng.choice([(32, 8), (64, 8), (16, 4), (8, 1), (16, 16)])
    c = dict(kind=kind, dt=rng.choice(["f16", "bf16"]), hq=hq, hkv=hkv, d=128)
    if kind in ("step", "packed", "blocks", "chunk", "append", "codec"):
        c.update(fmt=fmt, rot=rng.choice(["none", "auto"]))
    if kind == "step":
        c.update(b=_log(rng, 1, 32), d=rng.choice([64, 128, 128]), lk=_log(rng, 100, 16000), lq=rng.choice([1, 1, 1, 3]))
    elif kind == "packed":
        b = _log(rng, 4, 128)
        lk = _log(rng, 500, min(32768, 128 * 16384 * 8 // (b * hkv)))
        c.update(b=b, lk=lk, lmin=max(1, lk // rng.choice([1, 4, 16])), lq=rng.choice([1, 1, 2]))
    elif kind == "blocks":
        c.update(b=_log(rng, 1, 32), page=rng.choice([64, 256, 512]), lk=_log(rng, 200, 8000), lq=rng.choice([1, 1, 4]))
        c["lmin"] = max(c["lq"], c["lk"] // 4)
    elif kind == "chunk":
        c.update(b=rng.choice([1, 1, 2]), lq=_log(rng, 256, 2048), lk=_log(rng, 1, 12000))
    elif kind == "append":
        lq = _log(rng, 200, 8192)
        c.update(b=_log(rng, 1, 8), lq=lq, lk=lq)
    elif kind == "varlen":
        c.update(b=_log(rng, 2, 16), lk=_log(rng, 200, 4000), causal=rng.random() < 0.8)
        c["lmin"] = max(1, c["lk"] // 20)
    elif kind == "dense":
        c.update(dt=rng.choice(["f16", "bf16", "bf16", "f32"]), d=rng.choice([64, 64, 96, 128, 256]), causal=rng.random() < 0.6)
        if rng.random() < 0.4:  # decode
            c.update(lq=rng.choice([1, 1, 2]), lk=_log(rng, 200, 8000), b=_log(rng, 1, 64))
        else:
            lq = _log(rng, 60, 4096)
            c.update(lq=lq, lk=lq + rng.choice([0, 0, 0, 333]), b=_log(rng, 1, 16))
    else:
        c.update(b=_log(rng, 1, 8), d=rng.choice([64, 128, 128, 256]), lk=_log(rng, 100, 16000))
        c.pop("hq")
    return c


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, dt, *shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=DTYPES[dt])


def _lens(c, seed):
    """One length per sequence: spread over [lmin, lk] with a random offset each, the same ones for a case, in the seed's order."""
    n, lo, hi = c["b"], c["lmin"], c["lk"]
    lens = lo + ((np.arange(n) + np.random.RandomState(n + hi).random_sample(n)) / n * (hi - lo + 1)).astype(np.int64)
    lens = np.minimum(lens, hi)
    lens[-1] = hi
    np.random.RandomState(seed % (1 << 32)).shuffle(lens)
    return lens


def _rows(c, q, g, *lead):
    """Packed rows (b, hkv, capacity, words) of normal values with 1 % of the channels scaled by eight, as caches have them,
    made a slab of tokens at a time."""
    b, cap = lead
    out = torch.zeros((b, c["hkv"], cap, q.row_words()), dtype=torch.int32, device=DEV)
    scale = torch.ones(c["d"], device=DEV, dtype=DTYPES[c["dt"]])
    scale[torch.randperm(c["d"], generator=g, device=DEV)[: max(1, c["d"] // 100)]] = 8.0
    slab = max(1, (1 << 29) // (b * c["hkv"] * c["d"]))
    for at in range(0, cap, slab):
        t = min(slab, cap - at)
        x = _normal(g, c["dt"], b, c["hkv"], t, c["d"]) * scale
        out[:, :, at:at + t] = q.quantize_rows(x.view(-1, c["d"])).view(b, c["hkv"], t, -1)
    return out


def _quantizers(c):
    f = P.QuantFormat.parse(c["fmt"])
    return P.TurboQuantizer(f, c["d"], c["rot"], 42, DEV), P.TurboQuantizer(f, c["d"], c["rot"], 44, DEV)


def _cfg(c, causal=True):
    cfg = P.FlashAttnConfig(c["d"] ** -0.5)
    return cfg.causal() if causal else cfg


def prepare(case, seed):
    c, g = case, _gen(seed)
    s = dict(c, cfg=_cfg(c, c.get("causal", True)))
    b, d, dt = c["b"], c["d"], c["dt"]
    if c["kind"] in ("step", "chunk"):
        f = P.QuantFormat.parse(c["fmt"])
        s["cache"] = cache = P.TurboKvCache(f, f, d, c["rot"], 42, c["lk"] + c["lq"], DEV)
        cache.append(_normal(g, dt, b, c["hkv"], c["lk"], d), _normal(g, dt, b, c["hkv"], c["lk"], d))
        s["k"], s["v"] = _normal(g, dt, b, c["hkv"], c["lq"], d), _normal(g, dt, b, c["hkv"], c["lq"], d)
        s["q"] = _normal(g, dt, b, c["hq"], c["lq"], d)
    elif c["kind"] == "packed":
        kq, vq = _quantizers(c)
        lens = torch.from_numpy(_lens(c, seed).astype(np.int32)).to(DEV)
        q = _normal(g, dt, b, c["hq"], c["lq"], d)
        s.update(q=q, k=_rows(c, kq, g, b, c["lk"] + 4), v=_rows(c, vq, g, b, c["lk"] + 4), kq=kq, vq=vq)
        s["call"] = P.PackedAttention(q, s["k"], s["v"], lens, kq, vq, s["cfg"])
    elif c["kind"] == "blocks":
        kq, vq = _quantizers(c)
        left, blocks = c["lk"], []
        while left > 0:
            blocks.append(P.KvBlockRef(_rows(c, kq, g, b, c["page"]), _rows(c, vq, g, b, c["page"]), min(left, c["page"])))
            left -= c["page"]
        lens = torch.from_numpy(_lens(c, seed).astype(np.int32)).to(DEV)
        s.update(q=_normal(g, dt, b, c["hq"], c["lq"], d), blocks=blocks, kq=kq, vq=vq)
        s["call"] = P.PackedBlocksAttention(s["q"], blocks, kq, vq, s["cfg"], kv_len=lens)
    elif c["kind"] == "append":
        s["kq"], s["vq"] = _quantizers(c)
        s["q"] = _normal(g, dt, b, c["lq"], c["hq"], d)
        s["k"], s["v"] = _normal(g, dt, b, c["lk"], c["hkv"], d), _normal(g, dt, b, c["lk"], c["hkv"], d)
        for n, q in (("kc", s["kq"]), ("vc", s["vq"])):
            s[n] = torch.zeros((b, c["hkv"], c["lk"] + 64, q.row_words()), dtype=torch.int32, device=DEV)
    elif c["kind"] == "varlen":
        lens = _lens(c, seed)
        s["cu"] = torch.from_numpy(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)).to(DEV)
        s["longest"], n = int(lens.max()), int(lens.sum())
        s["q"], s["k"], s["v"] = (_normal(g, dt, n, h, d) for h in (c["hq"], c["hkv"], c["hkv"]))
    elif c["kind"] == "dense":
        s["q"] = _normal(g, dt, b, c["lq"], c["hq"], d)
        s["k"], s["v"] = (_normal(g, dt, b, c["lk"], c["hkv"], d) for _ in range(2))
    else:
        s["quantizer"] = _quantizers(c)[0]
        s["x"] = _normal(g, dt, b, c["hkv"], c["lk"], d)
    return s


def run(state):
    s = state
    kind = s["kind"]
    if kind in ("step", "chunk"):
        cache = s["cache"]
        cache.len = s["lk"]  # back to the context: the tokens of the pass before were rejected
        cache.append(s["k"], s["v"])
        return cache.attention(s["q"], s["cfg"]), cache.k, cache.v
    if kind in ("packed", "blocks"):
        return s["call"].run()
    if kind == "append":
        return F.prefill_append(s["q"], s["k"], s["v"], s["cfg"], s["kc"], s["vc"], s["kq"], s["vq"], 0), s["kc"], s["vc"]
    if kind == "varlen":
        return F.flash_attn_varlen(s["q"], s["k"], s["v"], s["cu"], s["cu"], s["longest"], s["longest"], s["cfg"].softmax_scale, s["causal"])
    if kind == "dense":
        return F.flash_attn_with_config(s["q"], s["k"], s["v"], s["cfg"])
    packed = s["quantizer"].quantize(s["x"])
    return packed.data, s["quantizer"].dequantize(packed)


def _seen(lq, lk, causal):
    """Pairs of (query, key) that the mask leaves."""
    return lq * lk - (lq * (lq - 1) // 2 if causal else 0)


def work(case):
    """Each input read once, each output written once; packed rows count as stored. Two products of two operations per query
    element and key that the mask leaves."""
    c = case
    e = 4 if c["dt"] == "f32" else 2
    d, b, hkv = c["d"], c["b"], c["hkv"]
    row = 4 * ROW_WORDS[c["fmt"]](d) if "fmt" in c else 0
    if c["kind"] == "codec":
        return {"bytes": b * hkv * c["lk"] * (2 * d * e + 2 * row), "flops": 0}
    hq = c["hq"]
    lens = _lens(c, 1) if "lmin" in c else np.full(b, c["lk"], np.int64)
    if c["kind"] in ("step", "chunk"):
        keys, n = c["lk"] + c["lq"], c["lq"]
        return {"bytes": b * (hkv * keys * 2 * row + hkv * n * 2 * (d * e + row) + 2 * hq * n * d * e),
                "flops": 4 * d * hq * b * _seen(n, keys, True)}
    if c["kind"] in ("packed", "blocks"):
        n = c["lq"]
        return {"bytes": int(lens.sum()) * hkv * 2 * row + 2 * b * hq * n * d * e, "flops": 4 * d * hq * sum(_seen(n, int(l), True) for l in lens)}
    if c["kind"] == "varlen":
        t = int(lens.sum())
        return {"bytes": t * (2 * hq + 2 * hkv) * d * e, "flops": 4 * d * hq * sum(_seen(int(l), int(l), c["causal"]) for l in lens)}
    total = b * (c["lq"] * 2 * hq + c["lk"] * 2 * hkv) * d * e
    if c["kind"] == "append":
        return {"bytes": total + b * hkv * c["lk"] * 2 * row, "flops": 4 * d * hq * b * _seen(c["lq"], c["lk"], True)}
    return {"bytes": total, "flops": 4 * d * hq * b * _seen(c["lq"], c["lk"], c["causal"])}


def tolerance(case):
    """Packed rows are exact. Attention outputs and rows read back: four times the largest relative error against the same sums
    in 64 bits, measured over the ranges of `draw`. bf16: 1.4e-3 to 2.1e-3 (the rounding of the output, and of the softmax weights
    where K and V are bf16), 3.3e-3 for chunks (their keys and values are rounded to bf16 once more). f16 and f32: up to 4.2e-4
    over dense keys (weights and f32 inputs are rounded to f16), 9.3e-4 over packed rows (f16 weights over 27 000 keys)."""
    if case["dt"] == "bf16":
        rel = 1.3e-2 if case["kind"] == "chunk" else 8.5e-3
    else:
        rel = 3.7e-3 if case["kind"] in ("step", "packed", "blocks") else 1.7e-3
    return {"rel": rel, "differ": 0.0}


E2M1 = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0], dtype=torch.float64)


def _decoded(rows, fmt, quantizer):
    """Packed rows (..., words) as 64-bit values, rotated back."""
    d = quantizer.dim
    by = rows.contiguous().view(torch.uint8)
    width = d if fmt in ("fp8", "mxfp8") else d // 2
    scale = by[..., 4 * (rows.shape[-1] - 2):4 * (rows.shape[-1] - 1)].contiguous().view(torch.float32).double()
    e4m3 = lambda x: x.contiguous().view(torch.float8_e4m3fn).to(torch.float64)
    codes = by[..., :width]
    if fmt in ("fp8", "mxfp8"):
        x = e4m3(codes)
    else:
        table = quantizer.tab[:16].double() if fmt == "turbo4" else E2M1.to(DEV)
        x = table[torch.stack([codes & 15, codes >> 4], -1).long()].flatten(-2)
    if fmt in ("mxfp4", "mxfp8"):
        x = x * torch.exp2(by[..., width:width + d // 32].double() - 127).repeat_interleave(32, -1)
    elif fmt == "nvfp4":
        x = x * e4m3(by[..., width:width + d // 16]).repeat_interleave(16, -1)
    x = x * scale
    if quantizer.signs is not None:  # y = H (signs x) / sqrt(d), and H / sqrt(d) is its own inverse
        h = torch.ones(1, 1, dtype=torch.float64, device=DEV)
        while h.shape[0] < d:
            h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
        x = (x @ h) * (d ** -0.5) * quantizer.signs.double()
    return x


def _attend(q, k, v, causal):
    """q (hq, lq, d) over k, v (hkv, lk, d) in 64 bits, masks aligned at the bottom right, a kv head and some rows at a time."""
    hq, lq, d = q.shape
    hkv, lk, _ = k.shape
    out = torch.empty(q.shape, dtype=torch.float64, device=DEV)
    step = max(1, (1 << 27) // (lk * (hq // hkv)))
    for h in range(hkv):
        heads = slice(h * (hq // hkv), (h + 1) * (hq // hkv))
        for at in range(0, lq, step):
            s = (q[heads, at:at + step].double() @ k[h].double().T) * d ** -0.5
            if causal:
                n = torch.arange(at, at + s.shape[1], device=DEV)[:, None] + lk - lq
                s.masked_fill_(torch.arange(lk, device=DEV)[None] > n, -torch.inf)
            out[heads, at:at + step] = torch.softmax(s, -1) @ v[h].double()
    return out


def exact(case, seed):
    """What `run` returns in 64 bits; packed rows have no such value (they are compared as whole numbers)."""
    c, s = case, prepare(case, seed)
    if c["kind"] == "codec":
        return None, _decoded(s["quantizer"].quantize(s["x"]).data, c["fmt"], s["quantizer"]).view(s["x"].shape)
    if c["kind"] == "varlen":
        cu = s["cu"].tolist()
        parts = [[t[i:j].transpose(0, 1) for t in (s["q"], s["k"], s["v"])] for i, j in zip(cu, cu[1:])]
        return torch.cat([_attend(*p, c["causal"]).transpose(0, 1) for p in parts])
    if c["kind"] in ("dense", "append"):
        rows = zip(*(t.transpose(1, 2) for t in (s["q"], s["k"], s["v"])))
        out = torch.stack([_attend(*r, c.get("causal", True)).transpose(0, 1) for r in rows])
        return (out, None, None) if c["kind"] == "append" else out
    if c["kind"] in ("step", "chunk"):
        _, k, v = run(s)
        lens, kq, vq, q = [s["cache"].len] * c["b"], s["cache"].kq, s["cache"].vq, s["q"]
    else:
        q, kq, vq = s["q"], s["kq"], s["vq"]
        if c["kind"] == "blocks":
            k, v = (torch.cat([getattr(x, n)[:, :, :x.rows] for x in s["blocks"]], 2) for n in ("k", "v"))
        else:
            k, v = s["k"], s["v"]
        lens = torch.from_numpy(_lens(c, seed)).tolist()
    out = torch.stack([_attend(q[i], _decoded(k[i, :, :n], c["fmt"], kq), _decoded(v[i, :, :n], c["fmt"], vq), True) for i, n in enumerate(lens)])
    return (out, None, None) if c["kind"] in ("step", "chunk") else out
