"""The work a user of kvcomp_b200 has it do, as measurable cases.

    listed()         named cases over the range of use
    draw(rng)        one more case of the same ranges
    prepare(c, s)    what the caller's program holds before the call, on the GPU
    run(state)       one pass through the public entry points
    work(c)          bytes and operations the pass cannot do without
    tolerance(c)     how far two correct implementations may differ
    exact(c, s)      what run returns for these inputs, in 64 bits, where it is a computed number

Kinds of work (the key "kind"):
  attend     one layer's share of a decode step: KVCompCache.attend over a compressed cache plus its recent window
  generate   a short generation through KVCompCache: prompt in, then per token and layer one append and either one
             attend (the fused path) or the values update() returns (the drop-in contract of the model files)
  prefill    a prompt's keys and values into a fresh KVCompCache: rotate, quantise, build the books, encode; the
             streams go to a pool of the caller's
  readback   KVCompCtx.get() of K and V: decode and dequantise the whole cache (an eager-attention host)
  matvec     KVCompCtx.mat_vec_mul of K and of V: the two unfused halves of decode attention
  operators  the operator module kvcomp_cuda: entropy encode, decode and decode-and-mat-vec of K and V codes

Values follow the distributions of kvcomp_b200.synth: keys with a mean and a spread per channel and a few outlier
channels, values with a log-normal spread per token.  Queries have unit variance here, so that attention weights
are as uneven as trained models make them.
"""
import math

import torch

from kvcomp_b200 import kvcomp_cuda, ops
from kvcomp_b200.cache.kvcomp_cache import KVCompCache
from kvcomp_b200.cache.kvcomp_encode import KVCompCtx
from kvcomp_b200.synth import make_kv
from kvcomp_b200.utils.compute import QuantMode
from kvcomp_b200.utils.config import KVCompCacheConfig, KVCompCacheConfigStatic

D = 128                               # head_dim of every configuration this library takes


def _case(kind, B, Hkv, G, T, kmode="ChannelQuant", vmode="TokenQuant", krel=0.05, vrel=0.1, block=64, recent=0, **more):
    """B sequences of T tokens, Hkv KV heads with G query heads each; K units per block and channel (or per block),
    V units per token (or per token and head); relative error bounds; tokens per K block; recent window."""
    return dict(kind=kind, B=B, Hkv=Hkv, G=G, T=T, kmode=kmode, vmode=vmode, krel=krel, vrel=vrel, block=block,
                recent=recent, **more)


def listed():
    return [
        # one sequence, one short context: the single-layer check configuration; latency and launches count
        dict(_case("attend", 1, 32, 1, 1024, vrel=0.05), name="attend_1x1k"),
        # a served batch in the middle of generating: the headline shape, newest tokens in the recent window
        dict(_case("attend", 8, 32, 1, 4096 + 128, recent=128), name="attend_8x4k"),
        # grouped queries and long contexts: 32 query heads on 8 KV heads
        dict(_case("attend", 16, 8, 4, 32768), name="attend_gqa_16x32k"),
        # grouped queries, a wide batch and the mixed error bounds: 40 query heads on 10 KV heads, blocks of 128
        dict(_case("attend", 32, 10, 4, 16384, krel=0.02, vrel=0.15, block=128), name="attend_gqa_32x16k"),
        # ragged: an odd batch, a length that is no multiple of anything, six query heads per KV head, a window that
        # is no multiple of the block, units of K per block and of V per head
        dict(_case("attend", 3, 4, 6, 2981, kmode="BlockQuant", vmode="VectorQuant", recent=100), name="attend_ragged"),
        # an interactive prompt of a few hundred tokens
        dict(_case("prefill", 1, 8, 4, 333, recent=64), name="prefill_1x333"),
        # the compression sweep's chunk: 1 GiB of keys and 1 GiB of values
        dict(_case("prefill", 32, 32, 1, 4096), name="prefill_32x4k"),
        # an interactive session on the fused path: four layers, 48 tokens generated behind a prompt
        dict(_case("generate", 2, 8, 4, 1000, recent=128, layers=4, steps=48, api="attend"), name="generate_attend"),
        # a model file that takes update()'s values at every step
        dict(_case("generate", 1, 32, 1, 512, recent=128, layers=2, steps=12, api="update"), name="generate_update"),
        # the whole cache read back for eager attention
        dict(_case("readback", 8, 32, 1, 4096), name="readback_8x4k"),
        # the longest context of the mat-vec timings this library is compared by, units as its operator path has them
        dict(_case("matvec", 1, 32, 1, 16384, kmode="BlockQuant"), name="matvec_1x16k"),
        # a program written against the operator module
        dict(_case("operators", 1, 32, 1, 4096, kmode="BlockQuant"), name="operators_1x4k"),
    ]


#: largest number of values of one tensor (tokens x sequences x KV heads x 128) that a drawn case may have
_MOST = {"attend": 32 * 10 * 16384 * D, "prefill": 32 * 32 * 4096 * D, "readback": 16 * 32 * 4096 * D,
         "matvec": 8 * 32 * 16384 * D, "operators": 32 * 16384 * D, "generate": 8 * 8 * 2048 * D}


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attend", "attend", "attend", "prefill", "prefill", "generate", "readback", "matvec", "operators"])
    Hkv, G = rng.choice([(32, 1), (40, 1), (8, 4), (10, 4), (4, 6), (2, 8), (8, 2), (5, 3), (1, 8), (16, 5)])
    block = rng.choice([64, 64, 128])
    krel, vrel = round(math.exp(rng.uniform(math.log(0.01), math.log(0.2))), 4), round(math.exp(rng.uniform(math.log(0.02), math.log(0.2))), 4)
    kmode = rng.choice(["ChannelQuant", "ChannelQuant", "BlockQuant"])
    vmode = rng.choice(["TokenQuant", "TokenQuant", "VectorQuant"])
    B, recent = _spread(rng, 1, 32), rng.choice([0, 32, 100, 128, 256])
    T = _spread(rng, 200, 32768)
    if kind in ("matvec", "operators"):                  # whole blocks of both tensors, units as the operator path has them
        kmode, vmode, block, recent, G = "BlockQuant", "TokenQuant", 64, 0, 1
        T, B = max(128, T // 128 * 128), min(B, 8)
    if kind == "operators":                              # 8-bit child indices bound the operator module's books
        krel, vrel, B = max(krel, 0.03), max(vrel, 0.03), 1
    if kind == "readback":
        B = min(B, 16)
    if kind == "generate":
        B, T = min(B, 8), min(T, 4096)
    most = _MOST[kind] // (Hkv * D)
    B = max(1, min(B, most // 200))
    T = min(T, most // B)
    if kind in ("matvec", "operators"):
        T = T // 128 * 128
    c = _case(kind, B, Hkv, G, T, kmode, vmode, krel, vrel, block, recent)
    if kind == "generate":
        c.update(layers=rng.choice([1, 2, 3]), steps=rng.randint(8, 48), api=rng.choice(["attend", "attend", "update"]))
        if c["api"] == "update":
            c["steps"] = min(c["steps"], 8)
    return c


# ---- inputs -----------------------------------------------------------------------------------------
def _config(c):
    return KVCompCacheConfig("", QuantMode(c["kmode"]), QuantMode(c["vmode"]), c["block"],
                             128 if c["kind"] in ("matvec", "operators") else c["block"], c["recent"], c["recent"],
                             c["krel"], c["vrel"])


def _rotation(first, n, device="cuda"):
    """cos and sin of n positions, fp16 [1, n, D], as a rotary embedding hands them over."""
    inv = 1.0 / (10000.0 ** (torch.arange(0, D, 2, dtype=torch.float32, device=device) / D))
    ang = torch.arange(first, first + n, dtype=torch.float32, device=device)[:, None] * inv
    ang = torch.cat([ang, ang], dim=-1)[None]
    return ang.cos().half(), ang.sin().half()


def _kv(c, T, seed, layer=0):
    """Token-major K and V [T, B, Hkv, D], and queries [B, Hq, D] of unit variance."""
    k, v, q = make_kv(T, c["B"], c["Hkv"], D, seed=seed, layer=layer, device="cuda", Hq=c["Hkv"] * c["G"])
    if c["kmode"] == "BlockQuant":
        # a unit spans all channels: one channel far beyond every other can push a block past the stream format's 8191 bytes
        k.clamp_(-24.0, 24.0)
    return k, v, (q.float() * math.sqrt(D)).half()


def _heads_first(x):
    return x.permute(1, 2, 0, 3).contiguous()            # [B, Hkv, T, D], as a model's projections leave it


def prepare(case, seed):
    c = case
    cfg = KVCompCacheConfigStatic.config = _config(c)
    B, H, T = c["B"], c["Hkv"], c["T"]
    s = dict(case=c, cfg=cfg, kind=c["kind"])
    if c["kind"] == "attend":
        # keys as they lie in the cache: no further rotation on the way in
        k, v, q = _kv(c, T, seed)
        one, zero = torch.ones(1, T, D, dtype=torch.float16, device="cuda"), torch.zeros(1, T, D, dtype=torch.float16, device="cuda")
        s["cache"] = KVCompCache(B, H * c["G"], D, 1)
        s["cache"].append(_heads_first(k), _heads_first(v), 0, {"cos": one, "sin": zero})
        s["q"] = q.unsqueeze(2)
    elif c["kind"] == "prefill":
        k, v, _ = _kv(c, T, seed)
        s["k"], s["v"] = _heads_first(k), _heads_first(v)
        s["cos"], s["sin"] = _rotation(0, T)
        s["pools"] = _pools(c, 1, T)
    elif c["kind"] == "generate":
        L, n = c["layers"], c["steps"]
        s["prompt"], s["steps"] = [], [[] for _ in range(n)]
        s["pools"] = _pools(c, L, T + n) if c["api"] == "attend" else None
        s["rot"] = [_rotation(0, T)] + [_rotation(T + i, 1) for i in range(n)]
        for layer in range(L):
            k, v, _ = _kv(c, T + n, seed, layer)
            q = torch.randn(n, B, H * c["G"], 1, D, device="cuda",
                            generator=torch.Generator(device="cuda").manual_seed(seed * 7 + layer)).half()
            s["prompt"].append((_heads_first(k[:T]), _heads_first(v[:T])))
            for i in range(n):
                s["steps"][i].append((_heads_first(k[T + i:T + i + 1]), _heads_first(v[T + i:T + i + 1]), q[i].contiguous()))
    elif c["kind"] in ("readback", "matvec"):
        k, v, q = _kv(c, T, seed)
        s["kc"], s["vc"] = KVCompCtx(True, B, H, D, c["krel"]), KVCompCtx(False, B, H, D, c["vrel"])
        s["kc"].store(k)
        s["vc"].store(v)
        if c["kind"] == "matvec":
            s["q"] = q
            g = torch.Generator(device="cuda").manual_seed(seed)
            s["p"] = torch.softmax(2.5 * torch.randn(B, H, T, device="cuda", generator=g), dim=-1).half()
    else:                                                # operators
        k, v, q = _kv(c, T, seed)
        for name, x, is_k, mode, rel in (("k", k, True, ops.MODE_BLOCK, c["krel"]), ("v", v, False, ops.MODE_TOKEN, c["vrel"])):
            codes, mi, sc, _, _ = ops.quantize(x, mode, 64, rel)
            codes = codes.view(-1, 64 if is_k else 128, B, H, D)
            _, enc, dec = kvcomp_cuda.build_codebook([codes])
            bsz, tsz, isz, n = kvcomp_cuda.calculate_buffer_size(codes, is_k, H, D)
            s[name] = dict(codes=codes, mi=mi, sc=sc, enc=enc.cuda(), dec=dec.cuda(),
                           bi=torch.empty(bsz, dtype=torch.uint8, device="cuda"), ti=torch.empty(tsz, dtype=torch.uint8, device="cuda"),
                           idx=torch.zeros(isz, dtype=torch.uint8, device="cuda"), stream=torch.zeros(n, dtype=torch.uint8, device="cuda"),
                           back=torch.empty_like(codes))
        s["q"] = q
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["p"] = torch.softmax(2.5 * torch.randn(B, H, T, device="cuda", generator=g), dim=-1).half()
        s["scores"] = torch.empty(B, H, T, dtype=torch.float16, device="cuda")
        s["parts"] = torch.empty(T // 128, B, H, D, dtype=torch.float16, device="cuda")
    return s


# ---- one pass ---------------------------------------------------------------------------------------
def _stored(cache, pools):
    """Everything a cache holds of its layers: tables, unit parameters, recent windows, and the streams, whose length
    depends on the values, in the caller's pool."""
    got = []
    for i, x in enumerate(x for pair in zip(cache.k_ctx, cache.v_ctx) for x in pair):
        stream = x.encoded_data
        if stream is not None:
            pools[i][:stream.numel()].copy_(stream)
        got.append([pools[i], x.block_infos, x.thread_infos, x.quant_min_ints, x.quant_scales, x.buffer])
    return got


def _pools(c, layers, T):
    return [torch.zeros(T * c["B"] * c["Hkv"] * D, dtype=torch.uint8, device="cuda") for _ in range(2 * layers)]


def run(s):
    c, kind = s["case"], s["kind"]
    KVCompCacheConfigStatic.config = s["cfg"]            # one process serves one configuration; here each case has its own
    if kind == "attend":
        return s["cache"].attend(s["q"], 0)
    if kind == "prefill":
        cache = KVCompCache(c["B"], c["Hkv"] * c["G"], D, 1)
        cache.append(s["k"], s["v"], 0, {"cos": s["cos"], "sin": s["sin"]})
        return _stored(cache, s["pools"])
    if kind == "generate":
        cache = KVCompCache(c["B"], c["Hkv"] * c["G"], D, c["layers"])
        fused, out = c["api"] == "attend", []
        rot = dict(zip(("cos", "sin"), s["rot"][0]))
        for layer, (k, v) in enumerate(s["prompt"]):
            (cache.append if fused else cache.update)(k, v, layer, rot)
        for i, step in enumerate(s["steps"]):
            rot = dict(zip(("cos", "sin"), s["rot"][1 + i]))
            for layer, (k, v, q) in enumerate(step):
                if fused:
                    cache.append(k, v, layer, rot)
                    out.append(cache.attend(q, layer))
                else:
                    kept = cache.update(k, v, layer, rot)
        # the fused path: every step's attention output and what the cache holds in the end; the other: the last update's values
        return {"out": torch.cat(out, dim=2), "stored": _stored(cache, s["pools"])} if fused else list(kept)
    if kind == "readback":
        return s["kc"].get()[0], s["vc"].get()[0]
    if kind == "matvec":
        return s["kc"].mat_vec_mul(s["q"])[0], s["vc"].mat_vec_mul(s["p"])[0]
    H, out = c["Hkv"], []
    for name in ("k", "v"):
        x = s[name]
        enc, dec, mul = (getattr(kvcomp_cuda, name + f) for f in (
            "_entropy_encode_cuda_export", "_entropy_decode_cuda_export", "_decode_and_mat_vec_mul_cuda_export"))
        stream, bi, ti = enc(x["codes"], x["enc"], x["bi"], x["ti"], x["idx"], x["stream"], 0, H, D)
        dec(stream, bi, ti, x["dec"], x["back"], H, D)
        mul(x["dec"], bi, ti, stream, x["mi"], x["sc"], s["q"] if name == "k" else s["p"], s["scores"] if name == "k" else s["parts"], H, D)
        out += [x["stream"], bi, ti, x["back"]]
    return out + [s["scores"], s["parts"]]


# ---- what a pass cannot do without ---------------------------------------------------------------------
def _bits(c, is_k):
    """Bits per symbol of the stream, from the entropy of a normal variable in steps of rel x range: the range of n
    normal values is about 2 * sqrt(2 ln n) - 1 deviations; a K block spans channels of very different spread."""
    rel, mode = (c["krel"], c["kmode"]) if is_k else (c["vrel"], c["vmode"])
    if mode == "BlockQuant":
        return max(1.1, 2.1 + math.log2(0.05 / rel))
    n = {"ChannelQuant": c["block"], "VectorQuant": D, "TokenQuant": c["Hkv"] * D}[mode]
    spread = 1.0 / (rel * (2 * math.sqrt(2 * math.log(n)) - 1))
    return max(1.1, math.log2(spread) + 2.1)


def _compressed(c, T, is_k):
    """Bytes of T compressed tokens of one tensor: stream, block and vector tables, unit parameters."""
    n = T * c["B"] * c["Hkv"] * D
    mode, B, H = c["kmode"] if is_k else c["vmode"], c["B"], c["Hkv"]
    units = {"BlockQuant": T / c["block"] * B, "ChannelQuant": T / c["block"] * B * H * D, "TokenQuant": T * B, "VectorQuant": T * B * H}[mode]
    return n * _bits(c, is_k) / 8 + n / 8192 * 8 + n / 128 * 2 + units * 4


def work(case):
    c = case
    B, H, T = c["B"], c["Hkv"], c["T"]
    row = B * H * D                                      # values of one token's keys (or values)
    Tc = max(0, (T - c["recent"]) // 128 * 128)          # tokens in the streams, the rest are fp16 rows
    packed = _compressed(c, Tc, True) + _compressed(c, Tc, False)
    dot = 4.0 * row * c["G"]                             # operations per cached token of one attention step
    if c["kind"] == "attend":
        return {"bytes": packed + 4.0 * (T - Tc) * row + 4.0 * row * c["G"], "flops": dot * T}
    if c["kind"] == "prefill":
        return {"bytes": 4.0 * T * row + packed + 4.0 * (T - Tc) * row, "flops": 0.0}
    if c["kind"] == "generate":
        n, L = c["steps"], c["layers"]
        fill = 4.0 * T * row + packed + 4.0 * (T - Tc) * row
        each = packed + 4.0 * (T - Tc) * row             # a step reads the compressed cache and the window
        if c["api"] == "attend":
            return {"bytes": L * (fill + n * (each + 8.0 * row)), "flops": L * n * dot * T}
        return {"bytes": L * (fill + (n + 1) * (each + 4.0 * T * row)), "flops": 0.0}
    if c["kind"] == "readback":
        return {"bytes": packed + 4.0 * (T - Tc) * row + 4.0 * T * row, "flops": 0.0}
    if c["kind"] == "matvec":
        return {"bytes": packed + 4.0 * row + 4.0 * B * H * T, "flops": dot * T}
    # codes in, stream out; stream in, codes out; stream in, products out
    return {"bytes": 4.0 * T * row + 3 * packed + 4.0 * row + 4.0 * B * H * T + 2.0 * T / 128 * row, "flops": dot * T}


def tolerance(case):
    # bytes, codes and dequantised values are exact; attention outputs and products are fp16 (half a step is 2.4e-4 of
    # a value at most, about half of that on average) over sums whose order is free
    if case["kind"] in ("prefill", "readback") or (case["kind"] == "generate" and case["api"] == "update"):
        return "exact"
    return {"rel": 1e-3, "max": 1e-2}


# ---- the same in 64 bits -------------------------------------------------------------------------------
def _dequantised(c, x, is_k, shared):
    """x [T,B,H,D] as the compressed cache holds it, in 64 bits: round(x / step) * step, the quotient in 16 bits,
    step = rel * range in 16 bits.  shared: a unit spans the sequences."""
    rel, mode = (c["krel"], c["kmode"]) if is_k else (c["vrel"], c["vmode"])
    T, B, H, _ = x.shape
    n = c["block"] if mode in ("BlockQuant", "ChannelQuant") else 1
    u = x.view(T // n, n, B, H, D)
    dims = {"BlockQuant": (1, 3, 4), "ChannelQuant": (1,), "TokenQuant": (3, 4), "VectorQuant": (4,)}[mode]
    dims += (2,) if shared else ()
    step = ((u.amax(dims, keepdim=True) - u.amin(dims, keepdim=True)).float() * torch.tensor(rel, dtype=torch.float32)).half()
    return ((u / step).round().double() * step.double()).view(T, B, H, D)


def exact(case, seed):
    c = case
    if c["kind"] not in ("attend", "matvec", "operators"):       # bytes and 16-bit rows, exact as they are
        return None
    B, H, G, T = c["B"], c["Hkv"], c["G"], c["T"]
    k, v, q = _kv(c, T, seed)
    if c["kind"] == "attend":
        over = T + c["block"] - T % c["block"] - c["recent"]      # whole blocks beyond the recent window are compressed
        n = min(max(0, over) // c["block"] * c["block"], T) // c["block"] * c["block"]
        out = torch.empty(B, H * G, 1, D, dtype=torch.float64, device="cuda")
        for b in range(B):
            kb, vb = (torch.cat([_dequantised(c, x[:n, b:b + 1], is_k, False), x[n:, b:b + 1].double()])[:, 0].transpose(0, 1)
                      for x, is_k in ((k, True), (v, False)))      # [H, T, D]
            s = torch.matmul(q[b].double().view(H, G, D), kb.transpose(1, 2)) / math.sqrt(D)
            out[b] = torch.matmul(torch.softmax(s, dim=-1), vb).view(H * G, 1, D)
        return out
    p = torch.softmax(2.5 * torch.randn(B, H, T, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)), dim=-1).half()
    scores = torch.empty(B, H, T, dtype=torch.float64, device="cuda")
    parts = torch.empty(T // 128, B, H, D, dtype=torch.float64, device="cuda")
    for t in range(0, T, 128):                                    # 128 is a whole number of units of either tensor
        kt, vt = _dequantised(c, k[t:t + 128], True, True), _dequantised(c, v[t:t + 128], False, True)
        scores[:, :, t:t + 128] = torch.einsum("tbhd,bhd->bht", kt, q.double())
        parts[t // 128] = torch.einsum("tbhd,bht->bhd", vt, p[:, :, t:t + 128].double())
    if c["kind"] == "matvec":
        return scores, parts.sum(dim=0, keepdim=True)
    return [None] * 8 + [scores, parts]
