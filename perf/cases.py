"""Performance cases of the attention framework: the calls its users make, over the sizes they make them at.

``listed()`` holds twelve calls, ``draw(rng)`` gives more of the same ranges.  A case is a dict of plain values;
its ``kind`` says which entry points it runs:

* ``decode``   one token per sequence over a KV cache (``DecodeCache.update`` + ``mha`` with ``KVLenMask``, or
               ``decode_paged`` over a page pool);
* ``latent_decode``  one token per sequence over the compressed cache (absorbed ``mla``);
* ``attend``   ``flex_attention``, forward only or forward and backward, with the mask and bias objects of the package;
* ``layer``    a prefill attention layer: ``linear`` projections, ``rope_interleaved``, causal ``flex_attention``, output
               projection; returns the layer's output and the keys and values it would put into the cache;
* ``latent``   latent attention over materialized keys and values (``mla`` with ``wk`` / ``wv``), forward only or
               forward and backward.

Sizes are the five configurations of the benchmark (``oracle/inputs.py``, ``bench.py``), scaled up and down.
"""

import math

import torch

import probjax_b200 as pj

_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


# ------------------------------------------------------------------------------------------------ cases


def listed():
    return [
        # A chat with one user: every token appends to the cache and attends over about 1500 tokens.  The smallest
        # call: latency, launches and host work count.
        dict(name="decode_chat", kind="decode", B=1, Hq=32, Hkv=8, D=128, cap=4096, lo=1500, hi=1500, append=True,
             page=0, dtype="bf16"),
        # A serving batch with ragged contexts of 1k to 32k tokens (the decode configuration of the benchmark).
        dict(name="decode_ragged", kind="decode", B=16, Hq=32, Hkv=8, D=128, cap=32768, lo=1024, hi=32768, append=False,
             page=0, dtype="bf16"),
        # The same for a model that caches a latent of rank 512 plus a rotary key of 64.
        dict(name="latent_decode", kind="latent_decode", B=16, H=16, R=576, cap=32768, lo=2048, hi=32768, dtype="bf16"),
        # An encoder over full sequences: the headline prefill configuration, no mask.
        dict(name="encoder_full", kind="attend", B=4, Lq=4096, Lkv=4096, Hq=32, Hkv=8, D=128, mask="none", docs=0, window=0,
             bias="none", dropout=0.0, grad=False, dtype="bf16"),
        # Prefill of a prompt through a whole attention layer of width 4096, causal.
        dict(name="prefill_layer", kind="layer", B=1, L=4096, Hq=32, Hkv=8, D=128, width=4096, dtype="bf16"),
        # A few short prompts of unequal length, padded to an odd common length, in fp16 with head width 64.
        dict(name="prefill_ragged", kind="attend", B=3, Lq=777, Lkv=777, Hq=16, Hkv=4, D=64, mask="causal_len", docs=0,
             window=0, bias="none", dropout=0.0, grad=False, dtype="f16"),
        # Prefill of a latent-attention layer (the latent configuration of the benchmark), causal.
        dict(name="latent_prefill", kind="latent", B=8, L=2048, H=16, nope=128, rope=64, Dv=128, R=512, grad=False,
             dtype="bf16"),
        # Training step of a causal language model with grouped heads: forward and gradients of q, k, v.
        dict(name="train_causal", kind="attend", B=2, Lq=4096, Lkv=4096, Hq=32, Hkv=8, D=128, mask="causal", docs=0, window=0,
             bias="none", dropout=0.0, grad=True, dtype="bf16"),
        # Training on packed documents of unequal length, causal inside each, with ALiBi.
        dict(name="train_packed", kind="attend", B=1, Lq=4096, Lkv=4096, Hq=32, Hkv=8, D=128, mask="packed", docs=8, window=0,
             bias="alibi", dropout=0.0, grad=True, dtype="bf16"),
        # Training with a learnable fp32 bias per head and key padding (the bias configuration of the benchmark):
        # gradients of q, k, v and of the bias.
        dict(name="train_bias", kind="attend", B=8, Lq=1024, Lkv=1024, Hq=16, Hkv=16, D=64, mask="len", docs=0, window=0,
             bias="dense", dropout=0.0, grad=True, dtype="bf16"),
        # Training of latent attention: gradients of the queries, the latent and both up-projections.
        dict(name="train_latent", kind="latent", B=2, L=2048, H=16, nope=128, rope=64, Dv=128, R=512, grad=True, dtype="bf16"),
        # A small fp32 transformer (the first configuration of the benchmark, at an odd length), forward and backward.
        dict(name="train_fp32", kind="attend", B=2, Lq=250, Lkv=250, Hq=4, Hkv=4, D=64, mask="causal", docs=0, window=0,
             bias="none", dropout=0.0, grad=True, dtype="f32"),
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of its range; half of them odd, the others multiples of 64."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n | 1 if rng.random() < 0.5 else (n + 63) // 64 * 64))


def draw(rng):
    kind = rng.choice(["decode", "decode", "latent_decode", "attend", "attend", "attend", "train", "train", "train",
                       "layer", "latent", "latent_train"])
    half = rng.choice(["bf16", "bf16", "f16"])
    if kind == "decode":
        Hq, Hkv = rng.choice([(32, 8), (32, 8), (16, 16), (16, 4), (32, 2), (8, 1)])
        B = rng.choice([1, 2, 3, 4, 8, 16, 21, 32])
        D = rng.choice([128, 128, 64])
        cap = _size(rng, 256, min(32768, (1 << 28) // (B * Hkv * D)))
        hi = max(1, int(cap * rng.uniform(0.5, 1.0)) - 1)
        page = rng.choice([0, 0, 64, 256])
        if page:
            cap = (cap + page - 1) // page * page
        return dict(kind="decode", B=B, Hq=Hq, Hkv=Hkv, D=D, cap=cap, lo=max(1, int(hi * rng.uniform(0.05, 1.0))),
                    hi=hi, append=page == 0 and B * cap <= 65536, page=page, dtype=half)
    if kind == "latent_decode":
        B = rng.choice([1, 2, 4, 7, 16, 32])
        cap = _size(rng, 512, min(32768, 524288 // B))
        hi = max(1, int(cap * rng.uniform(0.5, 1.0)))
        return dict(kind="latent_decode", B=B, H=rng.choice([16, 16, 32, 64]), R=rng.choice([576, 576, 512]), cap=cap,
                    lo=max(1, int(hi * rng.uniform(0.05, 1.0))), hi=hi, dtype=half)
    if kind == "layer":
        Hq, Hkv, width = rng.choice([(32, 8, 4096), (16, 4, 2048), (16, 16, 2048)])
        L = _size(rng, 128, 4096)
        return dict(kind="layer", B=rng.randint(1, max(1, min(8, 4096 // L))), L=L, Hq=Hq, Hkv=Hkv, D=128, width=width, dtype=half)
    if kind in ("latent", "latent_train"):
        L = _size(rng, 128, 2048)
        tokens = 4096 if kind == "latent_train" else 16384
        return dict(kind="latent", B=rng.randint(1, max(1, min(16, tokens // L))), L=L, H=rng.choice([8, 16]), nope=128, rope=64,
                    Dv=128, R=512, grad=kind == "latent_train", dtype=half)
    grad = kind == "train"
    if rng.random() < 0.2:  # fp32: small models
        L = _size(rng, 64, 1024)
        return dict(kind="attend", B=rng.randint(1, max(1, min(16, 2048 // L))), Lq=L, Lkv=L, Hq=4, Hkv=4, D=rng.choice([32, 64]),
                    mask=rng.choice(["none", "causal", "len"]), docs=0, window=0, bias="none", dropout=0.0, grad=grad, dtype="f32")
    D, Hq, Hkv = rng.choice([(128, 32, 8), (128, 16, 16), (64, 16, 16), (64, 16, 4)])
    bias = rng.choice(["none", "none", "none", "alibi", "t5", "dense"])
    L = _size(rng, 128, 1536 if bias == "dense" else 4096)
    area = (8 << 20) if bias == "dense" else (16 << 20) if grad else (32 << 20)  # a dense bias is [H, L, L] in fp32
    B = rng.randint(1, max(1, min(8, area // (L * L), 8192 // L)))
    mask = rng.choice(["none", "len"] if bias == "dense" else ["none", "causal", "causal", "causal_len", "len", "window", "packed"])
    return dict(kind="attend", B=B, Lq=L, Lkv=L, Hq=Hq, Hkv=Hkv, D=D, mask=mask, docs=rng.randint(2, 8) if mask == "packed" else 0,
                window=min(1024, max(64, L // 4)) if mask == "window" else 0, bias=bias,
                dropout=0.1 if grad and bias == "none" and rng.random() < 0.15 else 0.0, grad=grad, dtype=half)


# ------------------------------------------------------------------------------------------------ inputs


def _spread(lo, hi, n):
    """n whole numbers spread evenly over [lo, hi] (their order is drawn, their sum is not)."""
    if n == 1:
        return [hi]
    return [lo + (hi - lo) * i // (n - 1) for i in range(n)]


def _doc_lengths(total, docs):
    """Lengths of `docs` documents in the proportion 1 : 2 : ... : docs that fill `total` tokens."""
    weight = docs * (docs + 1) // 2
    out = [max(1, total * (i + 1) // weight) for i in range(docs)]
    out[-1] += total - sum(out)
    return out


def _lengths(case):
    """Key lengths of the sequences of an ``attend`` case, before shuffling: a quarter of the length to all of it."""
    return _spread(max(1, case["Lkv"] // 4), case["Lkv"], case["B"])


def prepare(case, seed):
    dev = torch.device("cuda")
    dt = _DTYPES[case["dtype"]]
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    gh = torch.Generator()
    gh.manual_seed(seed)

    def normal(*shape, dtype=dt, std=1.0):
        return (torch.randn(*shape, generator=g, device=dev, dtype=torch.float32) * std).to(dtype)

    def cache_rows(*shape):  # large: drawn in the cache's own type
        return torch.randn(*shape, generator=g, device=dev, dtype=dt)

    def shuffled(values):
        order = torch.randperm(len(values), generator=gh).tolist()
        return [values[i] for i in order]

    def lengths_tensor(values):
        return torch.tensor(shuffled(values), dtype=torch.int32, device=dev)

    s = {"case": case}
    kind = case["kind"]
    if kind == "decode":
        B, Hq, Hkv, D, cap = case["B"], case["Hq"], case["Hkv"], case["D"], case["cap"]
        s["q"] = normal(B, 1, Hq, D)
        s["scale"] = 1.0 / math.sqrt(D)
        lengths = lengths_tensor(_spread(case["lo"], case["hi"], B))
        if case["page"]:
            pages = cap // case["page"]
            s["k_pool"], s["v_pool"] = (cache_rows(B * pages, case["page"], Hkv, D) for _ in range(2))
            s["table"] = torch.randperm(B * pages, generator=g, device=dev).to(torch.int32).view(B, pages)
            s["lengths"] = lengths
        elif case["append"]:
            cache = pj.DecodeCache(B, cap, Hkv, D, dtype=dt, device=dev)
            cache.cached_key.copy_(cache_rows(B, cap, Hkv, D))
            cache.cached_value.copy_(cache_rows(B, cap, Hkv, D))
            cache.reset(lengths)
            s["cache"] = cache
            s["k"], s["v"] = normal(B, 1, Hkv, D), normal(B, 1, Hkv, D)
            s["mask"] = pj.KVLenMask(lengths + 1)  # the new token sees itself
        else:
            s["kc"], s["vc"] = cache_rows(B, cap, Hkv, D), cache_rows(B, cap, Hkv, D)
            s["mask"] = pj.KVLenMask(lengths)
    elif kind == "latent_decode":
        B, H, R = case["B"], case["H"], case["R"]
        s["q"] = normal(B, 1, H, R)
        s["latent"] = cache_rows(B, case["cap"], R)
        s["mask"] = pj.KVLenMask(lengths_tensor(_spread(case["lo"], case["hi"], B)))
        s["scale"] = 1.0 / math.sqrt(192.0)  # of the head width before absorption
    elif kind == "layer":
        B, L, Hq, Hkv, D, W = (case[n] for n in ("B", "L", "Hq", "Hkv", "D", "width"))
        s["x"] = normal(B, L, W)
        for name, heads in (("wq", Hq), ("wk", Hkv), ("wv", Hkv)):
            s[name] = normal(heads * D, W, std=1.0 / math.sqrt(W))
        s["wo"] = normal(W, Hq * D, std=1.0 / math.sqrt(Hq * D))
    elif kind == "latent":
        B, L, H, Dv, R, nope, rope = (case[n] for n in ("B", "L", "H", "Dv", "R", "nope", "rope"))
        D = nope + rope
        s["q"] = normal(B, L, H, D)
        s["latent"] = normal(B, L, R + rope)
        # the per-head key weights pass the rotary columns of the latent through
        wk = torch.zeros(H, D, R + rope, dtype=dt, device=dev)
        wk[:, :nope, :R] = normal(H, nope, R, std=1.0 / math.sqrt(R))
        wk[:, nope:, R:] = torch.eye(rope, dtype=dt, device=dev)
        wv = torch.zeros(H, Dv, R + rope, dtype=dt, device=dev)
        wv[:, :, :R] = normal(H, Dv, R, std=1.0 / math.sqrt(R))
        s["wk"], s["wv"] = wk, wv
        s["mask"] = pj.CausalMask()
        s["scale"] = 1.0 / math.sqrt(D)
        if case["grad"]:
            s["g"] = normal(B, L, H, Dv)
            s["inputs"] = [s[n].requires_grad_(True) for n in ("q", "latent", "wk", "wv")]
    else:
        B, Lq, Lkv, Hq, Hkv, D = (case[n] for n in ("B", "Lq", "Lkv", "Hq", "Hkv", "D"))
        s["q"], s["k"], s["v"] = normal(B, Lq, Hq, D), normal(B, Lkv, Hkv, D), normal(B, Lkv, Hkv, D)
        mask = case["mask"]
        if mask == "none":
            s["mask"] = None
        elif mask == "causal":
            s["mask"] = pj.CausalMask()
        elif mask == "len":
            s["mask"] = pj.KVLenMask(lengths_tensor(_lengths(case)))
        elif mask == "causal_len":
            s["mask"] = pj.CausalMask() & pj.KVLenMask(lengths_tensor(_lengths(case)))
        elif mask == "window":
            s["mask"] = pj.CausalLocalWindowMask(case["window"])
        else:
            rows = []
            for _ in range(B):
                docs = shuffled(_doc_lengths(Lq, case["docs"]))
                rows.append(torch.repeat_interleave(torch.arange(len(docs), dtype=torch.int32), torch.tensor(docs)))
            s["mask"] = pj.BlockDiagonalCausalMask(torch.stack(rows).to(dev))
        bias = case["bias"]
        learnable = []
        if bias == "alibi":
            s["bias"] = pj.CausalAlibiBias()
        elif bias == "t5":
            s["bias"] = pj.T5RelativePositionBias(normal(Hq, 32, dtype=torch.float32), num_buckets=32, max_distance=128,
                                                  bidirectional=mask in ("none", "len"))
        elif bias == "dense":
            s["dense"] = normal(1, Hq, Lq, Lkv, dtype=torch.float32)
            learnable = [s["dense"]]
        else:
            s["bias"] = None
        s["dropout"] = case["dropout"]
        s["rng"] = [seed & 0xFFFFFFFF, 7]
        if case["grad"]:
            s["g"] = normal(B, Lq, Hq, D)
            s["inputs"] = [x.requires_grad_(True) for x in [s["q"], s["k"], s["v"], *learnable]]
        if bias == "dense":
            s["bias"] = pj.DenseBias(s["dense"])
    return s


# ------------------------------------------------------------------------------------------------ one pass


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode":
        if case["page"]:
            return pj.decode_paged(s["q"], s["k_pool"], s["v_pool"], s["table"], s["lengths"], sm_scale=s["scale"])
        if case["append"]:
            cache = s["cache"]
            cache.update(s["k"], s["v"], advance=False)
            o = pj.mha(s["q"], cache.cached_key, cache.cached_value, mask=s["mask"], sm_scale=s["scale"])
            return o, cache.cached_key, cache.cached_value
        return pj.mha(s["q"], s["kc"], s["vc"], mask=s["mask"], sm_scale=s["scale"])
    if kind == "latent_decode":
        return pj.mla(s["q"], s["latent"], mask=s["mask"], sm_scale=s["scale"])
    if kind == "layer":
        x, D = s["x"], case["D"]
        B, L = x.shape[:2]
        q = pj.rope_interleaved(pj.linear(x, s["wq"]).view(B, L, -1, D))
        k = pj.rope_interleaved(pj.linear(x, s["wk"]).view(B, L, -1, D))
        v = pj.linear(x, s["wv"]).view(B, L, -1, D)
        o = pj.flex_attention(q, k, v, mask=pj.CausalMask(), enable_gqa=True)
        return pj.linear(o.view(B, L, -1), s["wo"]), k, v
    if kind == "latent":
        o = pj.mla(s["q"], s["latent"], s["wk"], s["wv"], mask=s["mask"], sm_scale=s["scale"])
    else:
        o = pj.flex_attention(s["q"], s["k"], s["v"], mask=s["mask"], bias=s["bias"], dropout_rng=s["rng"],
                              dropout_rate=s["dropout"], deterministic=s["dropout"] == 0.0, enable_gqa=True)
    if not case["grad"]:
        return o
    grads = torch.autograd.grad(o, s["inputs"], s["g"])
    return (o.detach(), *grads)


# ------------------------------------------------------------------------------------------------ floors


def _pairs(case):
    """Visible (query, key) pairs of an ``attend`` case, summed over the batch."""
    B, L, n = case["B"], case["Lq"], case["Lkv"]
    tri = L * (L + 1) // 2
    mask = case["mask"]
    if mask == "none":
        return B * L * n
    if mask == "causal":
        return B * tri
    if mask == "len":
        return L * sum(_lengths(case))
    if mask == "causal_len":
        return sum(m * (m + 1) // 2 + (L - m) * m for m in _lengths(case))
    if mask == "window":
        w = min(case["window"], L - 1)
        return B * (w * (w + 1) // 2 + (L - w) * (w + 1))
    return B * sum(m * (m + 1) // 2 for m in _doc_lengths(L, case["docs"]))


def work(case):
    es = 4 if case["dtype"] == "f32" else 2
    kind = case["kind"]
    if kind == "decode":
        B, Hq, Hkv, D = case["B"], case["Hq"], case["Hkv"], case["D"]
        keys = sum(_spread(case["lo"], case["hi"], B))
        io = 2 * B * Hq * D * es + (4 * B * Hkv * D * es if case["append"] else 0)
        return {"bytes": 2 * keys * Hkv * D * es + io, "flops": 4 * keys * Hq * D}
    if kind == "latent_decode":
        B, H, R = case["B"], case["H"], case["R"]
        keys = sum(_spread(case["lo"], case["hi"], B))
        return {"bytes": keys * R * es + 2 * B * H * R * es, "flops": 4 * keys * H * R}
    if kind == "layer":
        B, L, Hq, Hkv, D, W = (case[n] for n in ("B", "L", "Hq", "Hkv", "D", "width"))
        heads = 2 * Hq + 2 * Hkv
        return {"bytes": es * (2 * B * L * W + heads * D * W + 2 * B * L * Hkv * D),
                "flops": 2 * B * L * heads * D * W + 2 * B * Hq * D * L * (L + 1)}
    if kind == "latent":
        B, L, H, Dv, R = (case[n] for n in ("B", "L", "H", "Dv", "R"))
        D, Rr = case["nope"] + case["rope"], case["R"] + case["rope"]
        pairs = B * H * L * (L + 1) // 2
        up = 2 * B * L * H * (D + Dv) * Rr
        ins = B * L * H * D + B * L * Rr + H * (D + Dv) * Rr
        out = B * L * H * Dv
        if not case["grad"]:
            return {"bytes": es * (ins + out), "flops": up + 2 * pairs * (D + Dv)}
        # backward: scores again, dP, dV, dQ, dK; both gradients of the two up-projections
        return {"bytes": es * (2 * ins + 2 * out), "flops": 3 * up + 2 * pairs * (D + Dv) + 2 * pairs * (3 * D + 2 * Dv)}
    B, Lq, Lkv, Hq, Hkv, D = (case[n] for n in ("B", "Lq", "Lkv", "Hq", "Hkv", "D"))
    ins = es * (B * Lq * Hq * D + 2 * B * Lkv * Hkv * D) + (4 * Hq * Lq * Lkv if case["bias"] == "dense" else 0)
    out = es * B * Lq * Hq * D
    pairs = _pairs(case) * Hq
    if not case["grad"]:
        return {"bytes": ins + out, "flops": 4 * pairs * D}
    return {"bytes": 2 * ins + 2 * out, "flops": 14 * pairs * D}


def tolerance(case):
    # Largest errors of outputs and gradients against float64 of the same formula, at up to 1024 keys (2-norm of the
    # error over the norm, largest error over the larger of value and root mean square): bf16 3.4e-3 and 0.067 (the
    # latent gradients), fp16 4.2e-4 and 0.0072, fp32 4.9e-7 and 4.6e-6.  Four times that; twice more for fp32, whose
    # sums grow with the length.
    return {"bf16": {"rel": 1.4e-2, "max": 0.27}, "f16": {"rel": 1.7e-3, "max": 0.03}, "f32": {"rel": 4e-6, "max": 4e-5}}[case["dtype"]]
