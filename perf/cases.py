"""What this framework is used for, as cases that can be timed: decoder models on the megakernel, its FP8 / expert / latent attention
blocks, hybrid models, online sessions and the allocation-free attention call, from one request to full batches.

    listed()             the cases; draw(rng) gives further ones of the same ranges
    prepare(case, seed)  what a program holds before the call: weights, caches, the compiled graph, the batch
    run(state)           one call through the public entry points, and its outputs
    work(case)           bytes and floating-point operations that a call cannot do without
    tolerance(case)      how far another correct implementation of the same precision may be off
    exact(case, seed)    the outputs of run() in 64 bits, from plain torch

Graphs whose batch the caller describes (mode "online_notoken") process the same tokens at the same positions on every call, so a
call can be repeated: the cache rows it appends are the ones it appended before.  Recurrent state moves on with every call.
"""
import gc
import math

import torch

import mirage_b200 as mi

DEV = "cuda"
PAGE = 64

# Layer sizes of the benchmark's decoder (width 4096) and of its smaller relatives; feed-forwards are three times the width.
DECODERS = {
    1024: dict(heads=8, kv=4, ff=3072),
    2048: dict(heads=16, kv=8, ff=6144),
    4096: dict(heads=32, kv=8, ff=12288),
}
# Hybrid models of the benchmark: heads of the attention and of the matrix memories, feed-forward widths.
HYBRIDS = {
    2048: dict(heads=16, kv=8, dim=128, ff=8192, gff=6144, mheads=4, mdim=256, mvdim=512, blocks=8),
    4096: dict(heads=32, kv=8, dim=128, ff=16384, gff=12288, mheads=8, mdim=256, mvdim=512, blocks=16),
}
HYBRID_VOCAB = 32768
RANK, ROT, LDIM = 512, 64, 128          # latent rows, their rotated part, unrotated head size
CACHE = 1 << 25                         # caches up to so many values are outputs beside the logits


def _decoder(name, layers, width, vocab, requests, tokens, lo, hi, fp8=False):
    """`requests` requests at contexts from `lo` to `hi` (before the call), `tokens` tokens in all (decode: one each)."""
    return {"name": name, "kind": "decoder", "layers": layers, "width": width, "vocab": vocab, "requests": requests,
            "tokens": tokens, "ctx_lo": lo, "ctx_hi": hi, "fp8": fp8}


def listed():
    return [
        # attention of three requests between a host program's own kernels: the smallest call there is
        {"name": "attention_3", "kind": "attention", "requests": 3, "heads": 32, "kv": 8, "ctx_lo": 90, "ctx_hi": 700},
        # interactive decoding of a small model, one request: latency of the task groups
        _decoder("decode_small_1", 8, 2048, 32768, 1, 1, 300, 300),
        # the headline: one request on the 36-layer decoder, bound by the weights
        _decoder("decode_1", 36, 4096, 151936, 1, 1, 1024, 1024),
        # a handful of users at unequal contexts: still the weight-streaming path
        _decoder("decode_5", 36, 4096, 151936, 5, 5, 37, 2000),
        # a serving batch at ragged contexts: the tensor path
        _decoder("decode_16", 36, 4096, 151936, 16, 16, 512, 4000),
        # a full batch: weights, keys and values both count
        _decoder("decode_64", 36, 4096, 151936, 64, 64, 512, 1536),
        # prompts entering the cache, 64 tokens a launch, two prompts sharing it
        _decoder("prefill_64", 36, 4096, 151936, 2, 64, 200, 1000),
        # the FP8 form of the decoder (block-scaled weights, quantised activations) at a full batch
        _decoder("fp8_decode_64", 6, 4096, 151936, 64, 64, 1024, 2048, fp8=True),
        # the routed experts of one layer of a large mixture-of-experts model: routing, both projections, weighted sum
        {"name": "experts_32", "kind": "experts", "tokens": 32, "experts": 256, "hidden": 7168, "ff": 2048},
        # absorbed latent attention over the paged cache, a rank's 16 heads
        {"name": "latent_32", "kind": "latent", "requests": 32, "heads": 16, "ctx_lo": 4096, "ctx_hi": 4096},
        # a serving batch on a hybrid model: matrix memories, attention beside a diagonal recurrence
        {"name": "hybrid_decode_16", "kind": "hybrid", "width": 4096, "layers": 8, "requests": 16, "ctx_lo": 700, "ctx_hi": 1400},
        # prompts scored through an online session: the scheduler, portions of 64 tokens, logits read back by the host
        {"name": "session_3", "kind": "session", "width": 2048, "layers": 6, "requests": 3, "len_lo": 45, "len_hi": 200},
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["attention", "decoder", "decoder", "decoder", "decoder", "experts", "latent", "hybrid", "session"])
    if kind == "attention":
        kv = rng.choice([2, 4, 8])
        return {"kind": kind, "requests": log(1, 48), "heads": kv * rng.choice([1, 2, 4, 8]), "kv": kv, "ctx_lo": log(1, 300), "ctx_hi": log(301, 4000)}
    if kind == "experts":
        # a launch reads every expert that some token chose; smaller models have fewer and narrower ones
        hidden, ff = rng.choice([(7168, 2048), (4096, 1536), (2048, 1024)])
        return {"kind": kind, "tokens": log(1, 64), "experts": rng.choice([64, 128, 256]), "hidden": hidden, "ff": ff}
    if kind == "latent":
        lo = log(33, 2000)
        return {"kind": kind, "requests": log(1, 32), "heads": 16, "ctx_lo": lo, "ctx_hi": lo + log(1, 2096)}
    if kind == "hybrid":
        lo = log(20, 1200)
        return {"kind": kind, "width": rng.choice(sorted(HYBRIDS)), "layers": 4 * rng.randint(1, 2), "requests": log(1, 48), "ctx_lo": lo, "ctx_hi": lo + log(1, 800)}
    if kind == "session":
        lo = log(5, 150)
        return {"kind": kind, "width": rng.choice(sorted(HYBRIDS)), "layers": rng.randint(2, 6), "requests": log(1, 4), "len_lo": lo, "len_hi": lo + log(1, 100)}
    width = rng.choice(sorted(DECODERS))
    prompts = rng.random() < 0.3
    tokens = log(9, 64) if prompts else log(1, 64)
    requests = rng.randint(1, 4) if prompts else tokens
    lo = log(16, 1500)
    fp8 = not prompts and width > 1024 and rng.random() < 0.3
    return {"kind": kind, "layers": log(2, 6) if fp8 else log(4, 24) if width == 4096 else log(4, 36), "width": width, "vocab": rng.choice([32768, 65544, 151936]),
            "requests": requests, "tokens": tokens, "ctx_lo": lo, "ctx_hi": lo + log(1, 1000), "fp8": fp8}


# ---------------------------------------------------------------------------------------------------- inputs
def _spread(case, n, lo, hi):
    """`n` sizes from lo to hi that depend on the case alone (what a call costs does not depend on the seed)."""
    lo, hi = min(lo, hi), max(lo, hi)
    return [lo + (hi - lo) * ((i * 37 + 11) % 64) // 63 for i in range(n)] if n > 1 else [hi]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _normal(g, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    return torch.empty(*shape, dtype=dtype, device=DEV).normal_(mean, std, generator=g)


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _batch(case, seed):
    """Page tables of a batch: (lengths with the call's tokens, new tokens per request, pages, description)."""
    n = case["requests"]
    tokens = case.get("tokens", n)
    ctx = _spread(case, n, case["ctx_lo"], case["ctx_hi"])
    new = [tokens // n + (1 if r < tokens % n else 0) for r in range(n)]
    lens = [c + t for c, t in zip(ctx, new)]
    need = [-(-l // PAGE) for l in lens]
    pool = torch.randperm(sum(need) + 3, generator=torch.Generator().manual_seed(int(seed) + 1)).tolist()
    indptr, qo = [0], [0]
    for k, t in zip(need, new):
        indptr.append(indptr[-1] + k)
        qo.append(qo[-1] + t)
    d = {"qo_indptr_buffer": qo, "paged_kv_indptr_buffer": indptr, "paged_kv_indices_buffer": pool[:indptr[-1]],
         "paged_kv_last_page_len_buffer": [(l - 1) % PAGE + 1 for l in lens]}
    return lens, new, len(pool), d


def _keep(owner, outputs):
    """Views of memory that the library owns: each keeps the kernel that it belongs to."""
    for t in outputs.values():
        t.owner = owner
    return outputs


def _describe(meta, d):
    for key, values in d.items():
        meta[key][:len(values)].copy_(_i32(values))


def _pages_of(d, r):
    return d["paged_kv_indices_buffer"][d["paged_kv_indptr_buffer"][r]:d["paged_kv_indptr_buffer"][r + 1]]


def _decoder_inputs(case, seed):
    z, D, L = DECODERS[case["width"]], case["width"], case["layers"]
    H, G, F = z["heads"], z["kv"], z["ff"]
    g = _gen(seed)
    lin = lambda n, k: _normal(g, n, k, std=0.02)
    one = lambda n: _normal(g, n, std=0.02, mean=1.0)
    # projections that join the stream are scaled with the depth, as decoders are initialised: the stream neither vanishes nor explodes.
    # Its length at the start decides how much of a layer's error it carries on; e4m3 steps are ten times those of bf16.
    join = 1.0 / math.sqrt(2 * L)
    w, fp8 = {"model.embed_tokens.weight": _normal(g, case["vocab"], D, std=8.0 if case["fp8"] else 2.0), "model.norm.weight": one(D), "lm_head.weight": lin(case["vocab"], D)}, {}
    for i in range(L):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = one(D), one(D)
        w[p + "self_attn.q_norm.weight"], w[p + "self_attn.k_norm.weight"] = one(128), one(128)
        for name, n, k in (("self_attn.q_proj", H * 128, D), ("self_attn.k_proj", G * 128, D), ("self_attn.v_proj", G * 128, D),
                           ("self_attn.o_proj", D, H * 128), ("mlp.gate_proj", F, D), ("mlp.up_proj", F, D), ("mlp.down_proj", D, F)):
            std = 0.02 * (join if name.endswith(("o_proj", "down_proj")) else 1.0)
            if not case["fp8"]:
                w[p + name + ".weight"] = _normal(g, n, k, std=std)
                continue
            # a checkpoint's form: e4m3 values of full range and one float32 scale per 128 x 128 block
            scale = 0.01 * std * torch.exp(torch.empty(n // 128, k // 128, device=DEV).normal_(0, 0.2, generator=g))
            fp8[p + name + ".weight"] = (_normal(g, n, k, std=100.0).clamp_(-448, 448).to(torch.float8_e4m3fn), scale)
    lens, new, pages, d = _batch(case, seed)
    ids = torch.randint(0, case["vocab"], (sum(new), 1), generator=g, device=DEV)
    # keys as they stand in a cache: normed and rotated; values as projected
    k = _normal(g, L, pages, PAGE, G, 128)
    v = _normal(g, L, pages, PAGE, G, 128, std=0.02 * math.sqrt(D))
    return w, fp8, lens, new, pages, d, ids, k, v


def _prepare_decoder(case, seed):
    from mirage_b200.builders.runner import DecoderShape, Qwen3Runner
    z = DECODERS[case["width"]]
    w, fp8, lens, new, pages, d, ids, k, v = _decoder_inputs(case, seed)
    span = -(-max(lens) // PAGE) * PAGE
    shape = DecoderShape(case["layers"], case["width"], z["heads"], z["kv"], 128, z["ff"], case["vocab"], max_position=max(span, 4096))
    r = Qwen3Runner(shape, w, total_num_requests=case["requests"], max_seq_length=span, max_num_batched_requests=case["requests"],
                    max_num_batched_tokens=case["tokens"], max_num_pages=pages, page_size=PAGE, mode="online_notoken", fp8_state_dict=fp8 or None)
    r.k_cache.copy_(k)
    r.v_cache.copy_(v)
    _describe(r.meta, d)
    r.meta["input_tokens"].copy_(ids)
    caches = {"k_cache": r.k_cache, "v_cache": r.v_cache} if k.numel() <= CACHE else {}
    return {"kind": "graph", "kernel": r.mpk, "owner": r, "out": _keep(r, {"logits": r.logits, **caches})}


# Palarax of the benchmark's sizes: every fourth layer has attention beside a diagonal recurrence, the others a matrix memory
def _palarax_inputs(case, seed):
    z, D, L = HYBRIDS[case["width"]], case["width"], case["layers"]
    H, d, dv, W, F = z["mheads"], z["mdim"], z["mvdim"], case["width"], z["ff"]
    g = _gen(seed)
    rnd = lambda *s, std=None, mean=0.0: _normal(g, *s, std=s[-1] ** -0.5 if std is None else std, mean=mean)
    mlp = {"kind": "dense", "ff": F}
    ml = {"type": "mlstm", "mlp": mlp, "mixer": {"heads": H, "dim": d, "vdim": dv, "gate_cap": 15.0}}
    pa = {"type": "parallel", "mlp": mlp, "mixer": {
        "left": {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["dim"], "scale": z["dim"] ** -0.5, "softcap": 50.0,
                 "rot": {"base": 1e6, "dims": z["dim"]}},
        "right": {"width": W, "blocks": z["blocks"], "conv": 4}, "left_scale": 0.7, "right_scale": 0.7}}
    c = {"architecture": "Palarax", "vocab": HYBRID_VOCAB, "width": D, "norm": {"eps": 1e-6}, "layers": [pa if n % 4 == 3 else ml for n in range(L)]}
    w = {"embed": rnd(HYBRID_VOCAB, D, std=1.0), "final.norm": rnd(D, std=0.1)}
    for n, layer in enumerate(c["layers"]):
        p = f"l{n}."
        for nm in ("norm1", "norm1b", "norm2", "norm2b"):
            w[p + nm] = rnd(D, std=0.1)
        w[p + "mlp.up"], w[p + "mlp.down"] = rnd(F, D), rnd(D, F)
        if layer["type"] == "mlstm":
            for nm, rows in (("q", H * d), ("k", H * d), ("v", H * dv), ("g", H * dv), ("i", H), ("f", H)):
                w[p + "mix." + nm] = rnd(rows, D)
            w[p + "mix.o"], w[p + "mix.norm"] = rnd(D, H * dv), rnd(H * dv, std=0.1, mean=1.0)
            w[p + "mix.i.b"], w[p + "mix.f.b"] = rnd(H, std=1.0), rnd(H, std=1.0, mean=4.0)
        else:
            l, r = p + "mix.left.", p + "mix.right."
            w[l + "q"], w[l + "k"], w[l + "o"] = rnd(z["heads"] * z["dim"], D), rnd(z["kv"] * z["dim"], D), rnd(D, z["heads"] * z["dim"])
            for nm in ("y", "x"):
                w[r + nm], w[r + nm + ".b"] = rnd(W, D), rnd(W, std=0.3)
            w[r + "conv"], w[r + "conv.b"], w[r + "o"], w[r + "lam"] = rnd(W, 4, std=0.5), rnd(W, std=0.2), rnd(D, W), rnd(W, mean=-5.0, std=1.0)
            for nm in ("ra", "ri"):
                s = W // z["blocks"]
                w[r + nm], w[r + nm + ".b"] = rnd(z["blocks"], s, s), rnd(z["blocks"], s, std=0.5)
    lens, new, pages, desc = _batch(case, seed)
    ids = torch.randint(0, HYBRID_VOCAB, (sum(new), 1), generator=g, device=DEV)
    R, state = case["requests"], []
    f32 = lambda *s, std=1.0: _normal(g, *s, std=std, dtype=torch.float32)
    for layer in c["layers"]:
        # what earlier tokens left: memory, normaliser and running maximum (zero), or cache rows, convolution inputs and the recurrence
        if layer["type"] == "mlstm":
            state.append({"memory": f32(R, H, d, dv, std=8.0), "normaliser": f32(R, H, d, std=8.0)})      # some hundred updates
        else:
            state.append({"k": _normal(g, pages, PAGE, z["kv"], z["dim"]), "v": _normal(g, pages, PAGE, z["kv"], z["dim"]),
                          "conv": f32(R, 3, W), "diag": f32(R, W)})
    return c, w, lens, new, pages, desc, ids, state


def _prepare_hybrid(case, seed):
    from mirage_b200.builders.palarax import PalaraxConfig
    from mirage_b200.builders.runner import PalaraxRunner
    c, w, lens, new, pages, d, ids, state = _palarax_inputs(case, seed)
    r = PalaraxRunner(PalaraxConfig.from_dict(c), w, total_num_requests=case["requests"], max_seq_length=-(-max(lens) // PAGE) * PAGE,
                      max_num_batched_requests=case["requests"], max_num_batched_tokens=sum(new), max_num_pages=pages, page_size=PAGE,
                      mode="online_notoken")
    out = {"logits": r.logits}
    for n, (mine, given) in enumerate(zip(r.state, state)):
        for key, t in given.items():
            if key == "normaliser":      # every part of a head has a copy, followed by the running maximum
                mine[key][..., :-1].copy_(t[:, :, None])
                mine[key][..., -1].zero_()
            else:
                mine[key].copy_(t)
        for key in ("memory", "conv", "diag"):
            if key in mine:
                out[f"{key}_{n}"] = mine[key]
    _describe(r.meta, d)
    r.meta["input_tokens"].copy_(ids)
    return {"kind": "graph", "kernel": r.mpk, "owner": r, "out": _keep(r, out)}


# Lofirax with dense feed-forwards: gated linear attention, every third layer latent attention; the first two layers run twice
def _lofirax_inputs(case, seed):
    z, D, L = HYBRIDS[case["width"]], case["width"], case["layers"]
    H, d, dv, F, LH = z["mheads"], z["mdim"], z["mvdim"], z["gff"], z["heads"]
    g = _gen(seed)
    rnd = lambda *s, std=None, mean=0.0: _normal(g, *s, std=s[-1] ** -0.5 if std is None else std, mean=mean)
    gla = {"type": "gla", "mixer": {"heads": H, "dim": d, "vdim": dv, "tau": 16.0}}
    lat = {"type": "latent_attention", "mixer": {"heads": LH, "dim": LDIM, "rot_dim": ROT, "vdim": LDIM, "kv_rank": RANK,
                                                 "scale": (LDIM + ROT) ** -0.5, "rot": {"base": 1e6, "dims": ROT}}}
    c = {"architecture": "Lofirax", "vocab": HYBRID_VOCAB, "width": D, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
         "logit_softcap": 30.0, "loop": {"start": 0, "stop": 2, "times": 2},
         "layers": [dict(lat if n % 3 == 2 else gla, mlp={"kind": "dense", "ff": F}) for n in range(L)]}
    w = {"embed": rnd(HYBRID_VOCAB, D, std=1.0), "head": rnd(HYBRID_VOCAB, D), "loop.step": rnd(2, D, std=0.1)}
    for n in [f"l{n}.norm{k}" for n in range(L) for k in (1, 2)] + ["final.norm"]:
        w[n], w[n + ".b"] = rnd(D, std=0.1, mean=1.0), rnd(D, std=0.1)
    for n, layer in enumerate(c["layers"]):
        p = f"l{n}.mix."
        if layer["type"] == "gla":
            for nm, rows in (("q", H * d), ("k", H * d), ("v", H * dv), ("g", H * dv), ("a1", 16)):
                w[p + nm] = rnd(rows, D)
            w[p + "a2"], w[p + "a2.b"], w[p + "norm"], w[p + "o"] = rnd(H * d, 16), rnd(H * d, std=1.0, mean=2.0), rnd(dv, std=0.1, mean=1.0), rnd(D, H * dv)
        else:
            w[p + "q"], w[p + "dkv"], w[p + "dkv.norm"], w[p + "sink"] = rnd(LH * (LDIM + ROT), D), rnd(RANK + ROT, D), rnd(RANK, std=0.1, mean=1.0), rnd(LH, std=1.0)
            w[p + "uk"], w[p + "uv"], w[p + "o"] = rnd(LH * LDIM, RANK), rnd(LH * LDIM, RANK), rnd(D, LH * LDIM)
        m = f"l{n}.mlp."
        w[m + "gate"], w[m + "up"], w[m + "down"] = rnd(F, D), rnd(F, D), rnd(D, F)
    lens = _spread(case, case["requests"], case["len_lo"], case["len_hi"])
    prompts = [torch.randint(0, HYBRID_VOCAB, (n,), generator=g, device=DEV).tolist() for n in lens]
    return c, w, prompts


def _prepare_session(case, seed):
    from mirage_b200.builders.lofirax import LofiraxConfig
    from mirage_b200.builders.runner import LofiraxRunner
    c, w, prompts = _lofirax_inputs(case, seed)
    span = -(-(max(map(len, prompts)) + 2) // PAGE) * PAGE
    r = LofiraxRunner(LofiraxConfig.from_dict(c), w, total_num_requests=2 * len(prompts), max_seq_length=span, max_num_batched_requests=len(prompts),
                      max_num_batched_tokens=64, max_num_pages=2 * len(prompts) * (span // PAGE), page_size=PAGE, mode="online")
    return {"kind": "session", "session": mi.OnlineSession(r), "entries": [(k, p, [len(p) - 1]) for k, p in enumerate(prompts)]}


def _expert_inputs(case, seed):
    E, H, I, B = case["experts"], case["hidden"], case["ff"], case["tokens"]
    g = _gen(seed)
    w13 = torch.empty(E, 2 * I, H, dtype=torch.float8_e4m3fn, device=DEV)
    w2 = torch.empty(E, H, I, dtype=torch.float8_e4m3fn, device=DEV)
    for e in range(E):
        w13[e] = _normal(g, 2 * I, H, std=0.5).to(torch.float8_e4m3fn)
        w2[e] = _normal(g, H, I, std=0.5).to(torch.float8_e4m3fn)
    power = lambda *s: torch.exp2(torch.randint(-8, -4, s, generator=g, device=DEV).float())
    s13, s2 = power(E, 2 * I, H // 128), power(E, H, I // 128)
    return dict(w13=w13, w2=w2, s13=s13, s2=s2, x=_normal(g, B, H), logits=_normal(g, B, E), bias=_normal(g, E, std=0.1, dtype=torch.float32))


def _test_kernel(tokens, **kw):
    params = mi.PersistentKernel.get_default_init_parameters()
    params.update(test_mode=True, num_workers=0, max_num_batched_tokens=tokens, max_num_batched_requests=tokens, **kw)
    return mi.PersistentKernel(**params)


def _prepare_experts(case, seed):
    E, H, I, B, top = case["experts"], case["hidden"], case["ff"], case["tokens"], 8
    t = _expert_inputs(case, seed)
    pk = _test_kernel(B)
    new = lambda dims, dt, name: pk.new_tensor(dims=dims, dtype=dt, name=name)
    logits = t["logits"].clone()
    grid = dict(grid_dim=(B, 1, 1), block_dim=(128, 1, 1))
    att = {k: pk.attach_input(t[k], name=k) for k in ("w13", "w2", "s13", "s2", "x", "bias")}
    routing = (new((B, top), mi.float32, "weights"), new((E, B), mi.int32, "slots"), new((E + 1,), mi.int32, "active"))
    xq, xs = new((B, H), mi.float8_e4m3, "xq"), new((B, H // 128), mi.float32, "xs")
    mid, act = new((B, top, 2 * I), mi.bfloat16, "mid"), new((B, top, I), mi.bfloat16, "act")
    aq, asc = new((B, top, I), mi.float8_e4m3, "aq"), new((B, top, I // 128), mi.float32, "as")
    down, y = new((B, top, H), mi.bfloat16, "down"), torch.zeros(B, H, dtype=torch.bfloat16, device=DEV)
    pk.moe_topk_sigmoid_routing_layer(input=pk.attach_input(logits, name="logits"), bias=att["bias"], output=routing, **grid)
    pk.quantize_fp8_layer(input=att["x"], output_fp8=xq, output_scale=xs, scale_ue8m0=False, **grid)
    pk.moe_w13_fp8_layer(input_fp8=xq, input_scale=xs, weight_fp8=att["w13"], weight_scale=att["s13"], moe_routing_indices=routing[1],
                         moe_mask=routing[2], output=mid, **grid)
    pk.moe_silu_mul_layer(input=mid, output=act, grid_dim=(B, top, 1), block_dim=(128, 1, 1))
    pk.quantize_fp8_layer(input=act, output_fp8=aq, output_scale=asc, scale_ue8m0=False, **grid)
    pk.moe_w2_fp8_layer(input_fp8=aq, input_scale=asc, weight_fp8=att["w2"], weight_scale=att["s2"], moe_routing_indices=routing[1],
                        moe_mask=routing[2], output=down, **grid)
    pk.moe_mul_sum_add_layer(input=down, weight=routing[0], residual=att["x"], output=pk.attach_input(y, name="y"), **grid)
    pk.compile()
    return {"kind": "experts", "kernel": pk, "logits": logits, "source": t["logits"],
            "out": _keep(pk, {"y": y, "weights": pk.tensor_as_torch(routing[0]), "slots": pk.tensor_as_torch(routing[1])})}


def _latent_inputs(case, seed):
    g = _gen(seed)
    R, H = case["requests"], case["heads"]
    lens, new, pages, d = _batch(case, seed)
    rnd = lambda *s: _normal(g, *s, std=0.3)
    return lens, pages, d, dict(cache=rnd(pages, PAGE, RANK + ROT), latent=rnd(R, RANK), rotated=rnd(R, 128), q=rnd(R, H * (RANK + ROT)))


def _prepare_latent(case, seed):
    R, H = case["requests"], case["heads"]
    lens, pages, d, t = _latent_inputs(case, seed)
    span = -(-max(lens) // PAGE) * PAGE
    pk = _test_kernel(R, max_num_pages=pages, page_size=PAGE, max_seq_length=span, meta_tensors={k: _i32(v) for k, v in d.items()})
    att = {k: pk.attach_input(v, name=k) for k, v in t.items()}
    splits = -(-span // 128)
    rows = pk.new_tensor(dims=(8, RANK + ROT), dtype=mi.bfloat16, name="rows")
    part = pk.new_tensor(dims=(R * H * splits, RANK), dtype=mi.bfloat16, name="part")
    lse = pk.new_tensor(dims=(R * H * splits,), dtype=mi.float32, name="lse")
    out = torch.zeros(R, H * RANK, dtype=torch.bfloat16, device=DEV)
    pk.mla_kv_gather_layer(c_latent_new=att["latent"], k_pe_new=att["rotated"], paged_cache=att["cache"], contiguous_kv=rows,
                           mla_params=(RANK + ROT, RANK, PAGE), grid_dim=(R, 1, 1), block_dim=(128, 1, 1))
    pk.mla_mtp_decode_layer(att["q"], rows, part, lse, R, span, sm_scale=(128 + ROT) ** -0.5)
    pk.mla_mtp_reduce_layer(part, lse, pk.attach_input(out, name="out"), R, span)
    pk.compile()
    return {"kind": "graph", "kernel": pk, "out": _keep(pk, {"attention": out, "cache": t["cache"]})}


def _attention_inputs(case, seed):
    g = _gen(seed)
    R, H, G = case["requests"], case["heads"], case["kv"]
    lens, new, pages, d = _batch(case, seed)
    qkv = _normal(g, R, (H + 2 * G) * 128)
    return lens, d, qkv, _normal(g, pages, PAGE, G, 128), _normal(g, pages, PAGE, G, 128)


def _prepare_attention(case, seed):
    lens, d, qkv, k, v = _attention_inputs(case, seed)
    out = torch.zeros(case["requests"], case["heads"] * 128, dtype=torch.bfloat16, device=DEV)
    args = (qkv, k, v, out, _i32(d["paged_kv_indptr_buffer"]), _i32(d["paged_kv_indices_buffer"]), _i32(d["paged_kv_last_page_len_buffer"]),
            case["heads"], case["kv"])
    return {"kind": "attention", "args": args, "out": {"attention": out, "k_cache": k, "v_cache": v}}


def prepare(case, seed):
    # a program that replaces a model gives the old one's memory back first: the library allocates beside torch's pool
    gc.collect()
    torch.cuda.empty_cache()
    return {"attention": _prepare_attention, "decoder": _prepare_decoder, "experts": _prepare_experts, "latent": _prepare_latent,
            "hybrid": _prepare_hybrid, "session": _prepare_session}[case["kind"]](case, seed)


def run(state):
    if state["kind"] == "attention":
        mi.paged_decode_attention_noalloc(*state["args"])
    elif state["kind"] == "session":
        entries = state["entries"]
        return state["session"].step(entries, end=[rid for rid, _, _ in entries])
    else:
        if state["kind"] == "experts":
            state["logits"].copy_(state["source"])       # the routing task clears its logits
        state["kernel"]()
    return state["out"]


# ---------------------------------------------------------------------------------------------------- work
def work(case):
    k = case["kind"]
    if k == "session":
        z, D, L = HYBRIDS[case["width"]], case["width"], case["layers"]
        lens = _spread(case, case["requests"], case["len_lo"], case["len_hi"])
        n = sum(lens)
        runs = list(range(L)) + [0, 1]
        gla = D * z["mheads"] * (2 * z["mdim"] + 3 * z["mvdim"])
        lat = D * (z["heads"] * (2 * LDIM + ROT) + RANK + ROT) + 2 * z["heads"] * LDIM * RANK
        mixer = lambda i: lat if i % 3 == 2 else gla
        params = sum(mixer(i) + 3 * D * z["gff"] for i in range(L))
        token = sum(mixer(i) + 3 * D * z["gff"] + (0 if i % 3 == 2 else 4 * z["mheads"] * z["mdim"] * z["mvdim"] // 2) for i in runs)
        attended = sum(l * (l + 1) // 2 for l in lens) * sum(i % 3 == 2 for i in runs) * z["heads"] * (2 * RANK + ROT)
        head = D * HYBRID_VOCAB
        state = case["requests"] * sum(i % 3 != 2 for i in runs) * z["mheads"] * z["mdim"] * z["mvdim"] * 4
        return {"bytes": 2 * (params + head + n * D) + state + 4 * case["requests"] * HYBRID_VOCAB,
                "flops": 2 * (token * n + attended + head * case["requests"])}
    if k == "experts":
        # distinct experts a batch chooses, on average: choices of different tokens fall independently
        E, H, I, B = case["experts"], case["hidden"], case["ff"], case["tokens"]
        active = E * (1 - (1 - 8 / E) ** B)
        return {"bytes": active * (3 * I * H + 4 * (2 * I * (H // 128) + H * (I // 128))) + 4 * B * H, "flops": 2 * B * 8 * 3 * I * H}
    lens, new, _, _ = _batch(case, 0)
    ctx, n = sum(lens), sum(new)
    attended = sum(t * l - t * (t - 1) // 2 for l, t in zip(lens, new))
    if k == "attention":
        H, G = case["heads"], case["kv"]
        return {"bytes": 2 * 128 * (2 * G * ctx + n * (2 * H + 2 * G)), "flops": 4 * 128 * H * ctx}
    if k == "latent":
        H = case["heads"]
        return {"bytes": 2 * ((RANK + ROT) * (ctx + n * H) + n * H * RANK), "flops": 2 * H * ctx * (2 * RANK + ROT)}
    if k == "hybrid":
        z, D, L = HYBRIDS[case["width"]], case["width"], case["layers"]
        pa = L // 4
        ml = L - pa
        memory = z["mheads"] * z["mdim"] * z["mvdim"]
        params = ml * D * z["mheads"] * (2 * z["mdim"] + 3 * z["mvdim"]) + pa * D * (2 * z["heads"] + z["kv"]) * 128 + pa * 3 * D * D \
            + pa * 2 * D * D // z["blocks"] + L * 2 * D * z["ff"] + D * HYBRID_VOCAB
        return {"bytes": 2 * params + 8 * ml * n * memory + 4 * pa * z["kv"] * 128 * ctx + 32 * pa * n * D + n * (2 * D + 4 * HYBRID_VOCAB),
                "flops": 2 * params * n + 4 * ml * n * memory + 4 * pa * z["heads"] * 128 * attended}
    z, D, L, V = DECODERS[case["width"]], case["width"], case["layers"], case["vocab"]
    layer = D * 128 * (2 * z["heads"] + 2 * z["kv"]) + 3 * D * z["ff"]
    return {"bytes": (1 if case["fp8"] else 2) * L * layer + 2 * D * V + 4 * 128 * z["kv"] * ctx * L + n * 2 * (V + D),
            "flops": 2 * n * (L * layer + D * V) + 4 * 128 * z["heads"] * attended * L}


def tolerance(case):
    # bf16 results of bf16 operands: one rounding of the output
    if case["kind"] in ("attention", "latent"):
        return {"rel": 1e-2}
    # two e4m3 quantisations: a bf16 step in front of one moves a few values by an e4m3 step
    if case["kind"] == "experts":
        return {"rel": 1e-2}
    # whole models: bf16 roundings (in the FP8 form e4m3 steps as well) add up over the layers.  One bf16 step on 0.05 % of the
    # inputs' entries moves the 36-layer logits by 0.014, those of 6 FP8 layers by 0.011
    if case["kind"] == "decoder":
        return {"rel": 3e-2}
    # (float32 streams; 0.005 to 0.008 off 64 bits)
    return {"rel": 2e-2}


# ---------------------------------------------------------------------------------------------------- 64 bits
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, pos, base, dims):
    """x [tokens, heads, size]: component i < dims / 2 turns with component i + dims / 2."""
    half = dims // 2
    f = float(base) ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / dims)
    a = pos.double()[:, None] * f
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _gather(cache, pages, length):
    return cache[torch.tensor(pages, device=cache.device)].flatten(0, 1)[:length].double()


def _attend(q, k, v, scale, softcap=0.0, sink=None):
    """q [t, H, d] at the last t of k's positions, k [n, G, d], v [n, G, dv]; sink [H]: a logit that joins the denominators."""
    t, H, n = q.shape[0], q.shape[1], k.shape[0]
    rep = H // k.shape[1]
    s = torch.einsum("thd,nhd->htn", q, k.repeat_interleave(rep, 1)) * scale
    if softcap:
        s = softcap * torch.tanh(s / softcap)
    late = torch.arange(n, device=q.device)[None] > torch.arange(n - t, n, device=q.device)[:, None]
    s = s.masked_fill(late[None], -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.view(H, 1, 1).expand(H, t, 1)], -1)
    return torch.einsum("htn,nhd->thd", torch.softmax(s, -1)[..., :n], v.repeat_interleave(rep, 1))


def _paged_attention(q, k, v, kc, vc, lens, new, d, **kw):
    """New rows k, v follow the cached ones; q, k [tokens, heads, size] in batch order."""
    out, row = [], 0
    for r, (l, t) in enumerate(zip(lens, new)):
        pages = _pages_of(d, r)
        kk = torch.cat([_gather(kc, pages, l - t), k[row:row + t]])
        vv = torch.cat([_gather(vc, pages, l - t), v[row:row + t]])
        out.append(_attend(q[row:row + t], kk, vv, **kw))
        row += t
    return torch.cat(out)


def _positions(lens, new):
    return torch.cat([torch.arange(l - t, l) for l, t in zip(lens, new)]).to(DEV)


def _ue8m0(x):
    """What an FP8 linear reads of x: e4m3 values by the smallest power of two that holds 448 of them, per 128 columns."""
    g = x.float().unflatten(-1, (-1, 128))
    s = torch.exp2(torch.ceil(torch.log2(g.abs().amax(-1, keepdim=True).clamp(min=1e-12) / 448.0)))
    return ((g / s).to(torch.float8_e4m3fn).double() * s.double()).flatten(-2)


def _exact_decoder(case, seed):
    z = DECODERS[case["width"]]
    w, fp8, lens, new, pages, d, ids, kc, vc = _decoder_inputs(case, seed)
    H, G = z["heads"], z["kv"]
    pos, eps = _positions(lens, new), 1e-6

    def weight(name):
        if name not in fp8:
            return w[name].double()
        q, s = fp8[name]
        return _ue8m0((q.float().view(s.shape[0], 128, s.shape[1], 128) * s[:, None, :, None]).view(q.shape))

    # the FP8 form quantises the (bf16) input of every projection
    lin = lambda x, name: (_ue8m0(x.bfloat16()) if fp8 else x) @ weight(name).T

    norm = lambda x, name: _rms(x, eps) * w[name].double()
    x = w["model.embed_tokens.weight"][ids[:, 0]].double()
    keys = [(torch.tensor(_pages_of(d, r), device=DEV)[torch.arange(l - t, l, device=DEV) // PAGE], torch.arange(l - t, l, device=DEV) % PAGE)
            for r, (l, t) in enumerate(zip(lens, new))]
    at = torch.cat([a for a, _ in keys]), torch.cat([b for _, b in keys])     # page and place of every new row
    whole = (kc.double(), vc.double()) if kc.numel() <= CACHE else None
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = norm(x, p + "input_layernorm.weight")
        turn = lambda nm, heads: _rotate(norm(lin(h, f"{p}self_attn.{nm}_proj.weight").view(-1, heads, 128), f"{p}self_attn.{nm}_norm.weight"),
                                         pos, 1e6, 128)
        v = lin(h, p + "self_attn.v_proj.weight").view(-1, G, 128)
        k = turn("k", G)
        o = _paged_attention(turn("q", H), k, v, kc[i], vc[i], lens, new, d, scale=128 ** -0.5)
        if whole:
            whole[0][i][at], whole[1][i][at] = k, v
        x = x + lin(o.flatten(1), p + "self_attn.o_proj.weight")
        h = norm(x, p + "post_attention_layernorm.weight")
        u = torch.nn.functional.silu(lin(h, p + "mlp.gate_proj.weight")) * lin(h, p + "mlp.up_proj.weight")
        x = x + lin(u, p + "mlp.down_proj.weight")
    logits = norm(x, "model.norm.weight") @ w["lm_head.weight"].double().T
    return {"logits": logits, "k_cache": whole[0], "v_cache": whole[1]} if whole else {"logits": logits}


def _exact_hybrid(case, seed):
    c, w, lens, new, pages, d, ids, state = _palarax_inputs(case, seed)
    eps, pos, out = 1e-6, _positions(lens, new), {}
    W = lambda name: w[name].double()
    lin = lambda x, name: x @ W(name).T
    norm = lambda x, name: _rms(x, eps) * (1 + W(name))
    x = W("embed")[ids[:, 0]]
    for n, layer in enumerate(c["layers"]):
        p, m, st = f"l{n}.mix.", layer["mixer"], state[n]
        h = norm(x, f"l{n}.norm1")
        if layer["type"] == "mlstm":
            H, dk, dv, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
            q, k, v = lin(h, p + "q").view(-1, H, dk) * dk ** -0.5, lin(h, p + "k").view(-1, H, dk), lin(h, p + "v").view(-1, H, dv)
            i = cap * torch.tanh((lin(h, p + "i") + W(p + "i.b")) / cap)
            f = torch.nn.functional.logsigmoid(cap * torch.tanh((lin(h, p + "f") + W(p + "f.b")) / cap))
            top = torch.maximum(f, i)                                  # the running maximum was zero
            keep, add = torch.exp(f - top)[..., None], torch.exp(i - top)[..., None]
            S = keep[..., None] * st["memory"].double() + add[..., None] * k[..., :, None] * v[..., None, :]
            nrm = keep * st["normaliser"].double() + add * k
            o = torch.einsum("thd,thdv->thv", q, S) / (torch.maximum((nrm * q).sum(-1).abs(), torch.exp(-top)) + 1e-6)[..., None]
            y = lin(_rms(o, eps).flatten(1) * W(p + "norm") * torch.sigmoid(lin(h, p + "g")), p + "o")
            out[f"memory_{n}"] = S
        else:
            l, r, pl, pr = m["left"], m["right"], p + "left.", p + "right."
            v = lin(h, pl + "k").view(-1, l["kv_heads"], l["dim"])
            turn = lambda t: _rms(_rotate(t, pos, l["rot"]["base"], l["rot"]["dims"]), eps)
            q = turn(lin(h, pl + "q").view(-1, l["heads"], l["dim"]))
            zero = torch.zeros(l["heads"], dtype=torch.float64, device=DEV)
            o = _paged_attention(q, turn(v), v, st["k"], st["v"], lens, new, d, scale=l["scale"], softcap=l["softcap"], sink=zero)
            left = lin(o.flatten(1), pl + "o")
            gate = torch.nn.functional.gelu(lin(h, pr + "y") + W(pr + "y.b"), approximate="tanh")
            into = lin(h, pr + "x") + W(pr + "x.b")
            seen = torch.cat([st["conv"].double(), into[:, None]], 1)                          # [requests, taps, width], oldest first
            u = (seen * W(pr + "conv").T[None]).sum(1) + W(pr + "conv.b")
            block = lambda nm: torch.sigmoid(torch.einsum("tbk,bok->tbo", u.view(u.shape[0], r["blocks"], -1), W(pr + nm)) + W(pr + nm + ".b")).flatten(1)
            a = -8.0 * block("ra") * torch.nn.functional.softplus(W(pr + "lam"))
            S = torch.exp(a) * st["diag"].double() + torch.sqrt(-torch.expm1(2 * a)) * block("ri") * u
            y = m["left_scale"] * left + m["right_scale"] * lin(S * gate, pr + "o")
            out[f"conv_{n}"], out[f"diag_{n}"] = seen[:, 1:].contiguous(), S
        x = x + norm(y, f"l{n}.norm1b")
        y = lin(torch.relu(lin(norm(x, f"l{n}.norm2"), f"l{n}.mlp.up")) ** 2, f"l{n}.mlp.down")
        x = x + norm(y, f"l{n}.norm2b")
    out["logits"] = lin(norm(x, "final.norm"), "embed")
    return out


def _exact_session(case, seed):
    c, w, prompts = _lofirax_inputs(case, seed)
    eps, out = 1e-5, []
    W = lambda name: w[name].double()
    lin = lambda x, name: x @ W(name).T

    def norm(x, name):
        e = x - x.mean(-1, keepdim=True)
        return e / torch.sqrt((e * e).mean(-1, keepdim=True) + eps) * W(name) + W(name + ".b")

    def gla(p, m, h):
        T, H, dk, dv = h.shape[0], m["heads"], m["dim"], m["vdim"]
        q, k, v = lin(h, p + "q").view(T, H, dk) * dk ** -0.5, lin(h, p + "k").view(T, H, dk), lin(h, p + "v").view(T, H, dv)
        keep = torch.sigmoid(lin(lin(h, p + "a1"), p + "a2") + W(p + "a2.b")).view(T, H, dk) ** (1.0 / m["tau"])
        S, o = torch.zeros(H, dk, dv, dtype=torch.float64, device=DEV), []
        for t in range(T):
            S = keep[t][..., None] * S + k[t][..., None] * v[t][:, None]
            o.append(torch.einsum("hd,hdv->hv", q[t], S))
        o = _rms(torch.stack(o), eps) * W(p + "norm")
        return lin(o.flatten(1) * torch.nn.functional.silu(lin(h, p + "g")), p + "o")

    def latent(p, m, h):
        T, H, dim, rot = h.shape[0], m["heads"], m["dim"], m["rot_dim"]
        pos = torch.arange(T, device=DEV)
        q, down = lin(h, p + "q").view(T, H, dim + rot), lin(h, p + "dkv")
        lat = _rms(down[:, :m["kv_rank"]], eps) * W(p + "dkv.norm")
        k_rot = _rotate(down[:, None, m["kv_rank"]:], pos, m["rot"]["base"], rot).expand(T, H, rot)
        k = torch.cat([lin(lat, p + "uk").view(T, H, dim), k_rot], -1)
        q = torch.cat([q[..., :dim], _rotate(q[..., dim:], pos, m["rot"]["base"], rot)], -1)
        o = _attend(q, k, lin(lat, p + "uv").view(T, H, -1), m["scale"], sink=W(p + "sink"))
        return lin(o.flatten(1), p + "o")

    runs = [(0, 0), (1, None), (0, 1), (1, None)] + [(n, None) for n in range(2, len(c["layers"]))]
    for prompt in prompts:
        first = W("embed")[torch.tensor(prompt, device=DEV)]
        x = first.clone()
        for n, t in runs:
            if t is not None:
                x = x + W("loop.step")[t] + (first if t else 0.0)
            layer, p = c["layers"][n], f"l{n}."
            x = x + (gla if layer["type"] == "gla" else latent)(p + "mix.", layer["mixer"], norm(x, p + "norm1"))
            h = norm(x, p + "norm2")
            x = x + lin(torch.nn.functional.gelu(lin(h, p + "mlp.gate"), approximate="tanh") * lin(h, p + "mlp.up"), p + "mlp.down")
        out.append(30.0 * torch.tanh(lin(norm(x[-1:], "final.norm"), "head") / 30.0))
    return out


def _quantised(x):
    """What the expert projections read of x: e4m3 values by the group's amax / 448, multiplied by the power of two below that scale."""
    g = x.bfloat16().float().unflatten(-1, (-1, 128))
    s = (g.abs().amax(-1, keepdim=True) / 448.0).clamp(min=1e-10)
    return ((g / s).to(torch.float8_e4m3fn).double() * torch.exp2(torch.floor(torch.log2(s.double())))).flatten(-2)


def _exact_experts(case, seed):
    E, B = case["experts"], case["tokens"]
    t = _expert_inputs(case, seed)
    score = torch.sigmoid(t["logits"].double())
    choice = score + t["bias"].double()
    groups = choice.view(B, 8, E // 8)
    kept = torch.zeros(B, 8, dtype=torch.bool, device=DEV).scatter_(1, groups.topk(2, -1).values.sum(-1).topk(4, -1).indices, True)
    chosen = choice.masked_fill(~kept.repeat_interleave(E // 8, 1), -1e4).topk(8, -1).indices
    picked = score.gather(1, chosen)
    weights = 2.5 * picked / picked.sum(-1, keepdim=True)
    xq = _quantised(t["x"])
    y = t["x"].double()
    for e in chosen.unique().tolist():
        tok, slot = (chosen == e).nonzero(as_tuple=True)
        full = lambda w, s: (w.double().unflatten(-1, (-1, 128)) * s.double()[..., None]).flatten(-2)
        mid = (xq[tok] @ full(t["w13"][e], t["s13"][e]).T).bfloat16().double()
        gate, up = mid.chunk(2, -1)
        o = _quantised(torch.nn.functional.silu(gate) * up) @ full(t["w2"][e], t["s2"][e]).T
        y.index_add_(0, tok, weights[tok, slot][:, None] * o)
    return {"y": y, "weights": weights, "slots": None}


def _exact_latent(case, seed):
    lens, pages, d, t = _latent_inputs(case, seed)
    R, H = case["requests"], case["heads"]
    cache, rows = t["cache"].double(), []
    row = torch.cat([t["latent"], t["rotated"][:, :ROT]], -1).double()
    q = t["q"].double().view(R, H, RANK + ROT)
    for r, l in enumerate(lens):
        cache[_pages_of(d, r)[-1], (l - 1) % PAGE] = row[r]
        k = _gather(cache, _pages_of(d, r), l)
        p = torch.softmax(q[r] @ k.T * (128 + ROT) ** -0.5, -1)
        rows.append((p @ k[:, :RANK]).flatten())
    return {"attention": torch.stack(rows), "cache": cache}


def _exact_attention(case, seed):
    lens, d, qkv, kc, vc = _attention_inputs(case, seed)
    R, H, G = case["requests"], case["heads"], case["kv"]
    x = qkv.double().view(R, G, H // G + 2, 128)
    q, k, v = x[:, :, :-2].reshape(R, H, 128), x[:, :, -2], x[:, :, -1]
    o = _paged_attention(q, k, v, kc, vc, lens, [1] * R, d, scale=128 ** -0.5)
    kc, vc = kc.double(), vc.double()
    for r, l in enumerate(lens):
        at = _pages_of(d, r)[-1], (l - 1) % PAGE
        kc[at], vc[at] = k[r], v[r]
    return {"attention": o.flatten(1), "k_cache": kc, "v_cache": vc}


def exact(case, seed):
    return {"attention": _exact_attention, "decoder": _exact_decoder, "experts": _exact_experts, "latent": _exact_latent,
            "hybrid": _exact_hybrid, "session": _exact_session}[case["kind"]](case, seed)
