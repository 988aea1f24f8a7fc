"""Workloads by which the speed of this package is followed, each with its inputs, its arithmetic in 64 bits and the work it cannot do without.

Three models and one training loop carry the package's use, at the sizes of its own configurations:

* ``dense``    the Gemma-4-12B-style decoder (hidden 3840, 16 query / 8 kv heads of 256, five layers with a window of 1024 and one global
               layer, feed-forward 15360, vocabulary 262144): whole prompts, and decode steps over the paged cache in bf16 or 8 bits
* ``mla``      the latent-attention half of a layer of the K3-class decoder (hidden 7168, 64 heads, latent rows of 512 + 64)
* ``experts``  the feed-forward half of a layer with NVFP4 experts: ``k3`` (384 experts of 2048, sigmoid router in groups, the shared expert among
               them) or ``inkling`` (hidden 4096, 128 experts of 1536, softmax router, a bf16 shared expert)
* ``lora``     loss and adapter gradients of the LoRA fine-tuning step (rank 16 on every projection) on two layers of the dense decoder

A dense model is cut to one period of its layer pattern; every other size is the configuration's.  Decode-sized passes replay a CUDA graph, as the
package's fixed-batch decoder does; prompts and training steps are launched call by call, prompts with the batch built for every call, as the
engine does."""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

# dense decoder, one period of its layers
H, NQ, NKV, D, F, V, WINDOW, CAP, EPS = 3840, 16, 8, 256, 15360, 262144, 1024, 30.0, 1e-6
LAYERS, GLOBAL, PAGE = 6, 5, 16
THETA = {True: 1e6, False: 1e4}                 # by: global layer
LORA_LAYERS, RANK, ALPHA = 2, 16, 32.0
PROJECTIONS = ("q_proj", "k_proj", "v_proj", "o_proj", "gate_proj", "up_proj", "down_proj")
# latent attention
MH, MQ, ML, MR, MN, MHEADS, MPAGE, MTHETA = 7168, 1536, 512, 64, 128, 64, 32, 1e6
# expert layers: hidden, experts, expert width, experts per token, groups, groups kept, scale of the routed sum
EXPERTS = {"k3": (7168, 384, 2048, 8, 8, 4, 2.5), "inkling": (4096, 128, 1536, 8, 1, 1, 1.0)}


def listed():
    return [
        # one user's reply, token by token: latency
        {"name": "decode 1 x 777", "kind": "dense", "phase": "decode", "seqs": 1, "tokens": 777, "kv": "bf16"},
        # a batch of replies behind 2048-token prompts: the decoder's serving workload
        {"name": "decode 32 x 2048", "kind": "dense", "phase": "decode", "seqs": 32, "tokens": 2048, "kv": "bf16"},
        # longer contexts of unequal lengths in an 8-bit cache
        {"name": "decode 24 x 4000 int8", "kind": "dense", "phase": "decode", "seqs": 24, "tokens": 4000, "kv": "int8"},
        # one short question
        {"name": "prefill 1 x 217", "kind": "dense", "phase": "prefill", "seqs": 1, "tokens": 217, "kv": "bf16"},
        # prompts of unequal lengths that arrive together
        {"name": "prefill 3 x 701", "kind": "dense", "phase": "prefill", "seqs": 3, "tokens": 701, "kv": "bf16"},
        # the serving workload's prompts, four at a time
        {"name": "prefill 4 x 2048", "kind": "dense", "phase": "prefill", "seqs": 4, "tokens": 2048, "kv": "bf16"},
        # attention of the headline decode step: 128 sequences, the pending token and two drafts each
        {"name": "mla decode 128 x 4096", "kind": "mla", "phase": "decode", "seqs": 128, "tokens": 4096, "rows": 3},
        # attention of the headline prompt
        {"name": "mla prefill 1 x 4096", "kind": "mla", "phase": "prefill", "seqs": 1, "tokens": 4096, "rows": 1},
        # experts of the headline decode step: 128 sequences, three rows each
        {"name": "k3 experts 384", "kind": "experts", "model": "k3", "rows": 384},
        # experts of the 64-sequence decode step
        {"name": "inkling experts 64", "kind": "experts", "model": "inkling", "rows": 64},
        # experts of a prompt batch
        {"name": "inkling experts 4096", "kind": "experts", "model": "inkling", "rows": 4096},
        # one fine-tuning sequence
        {"name": "lora 1 x 4096", "kind": "lora", "seqs": 1, "tokens": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["dense decode", "dense prefill", "mla decode", "mla prefill", "k3", "inkling", "lora"])
    if what == "dense decode":
        tokens = _log(rng, 64, 4000)
        return {"kind": "dense", "phase": "decode", "seqs": _log(rng, 1, min(48, 98304 // tokens)), "tokens": tokens, "kv": rng.choice(["bf16", "bf16", "int8"])}
    if what == "dense prefill":
        seqs = rng.choice([1, 1, 2, 3, 4])
        return {"kind": "dense", "phase": "prefill", "seqs": seqs, "tokens": _log(rng, 48, 8000 // seqs), "kv": "bf16"}
    if what == "mla decode":
        return {"kind": "mla", "phase": "decode", "seqs": _log(rng, 1, 128), "tokens": _log(rng, 64, 4096), "rows": rng.choice([1, 3])}
    if what == "mla prefill":
        return {"kind": "mla", "phase": "prefill", "seqs": 1, "tokens": _log(rng, 64, 4096), "rows": 1}
    if what == "lora":
        return {"kind": "lora", "seqs": rng.choice([1, 1, 2]), "tokens": _log(rng, 128, 2048)}
    return {"kind": "experts", "model": what, "rows": _log(rng, 1, 4096)}


def _lengths(case):
    """Context or prompt lengths of a batch: the named one, the other sequences up to a third shorter (equal where they fill whole pages)."""
    n, t = case["seqs"], case["tokens"]
    return [t if t % 64 == 0 else t - (i * 97) % (t // 3 + 1) for i in range(n)]


# ------------------------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    return torch.empty(*shape, dtype=dtype, device="cuda").normal_(mean, std, generator=g)


def _dense_weights(g, layers):
    """Weights of the dense decoder as a trained one has them: matrices of 0.02, gains about 1, head gains that keep scores of order one."""
    w = {"embed": _normal(g, V, H, std=0.02), "norm": _normal(g, H, std=0.1, mean=1.0), "layers": []}
    for _ in range(layers):
        w["layers"].append({
            "w_qkv": _normal(g, (NQ + 2 * NKV) * D, H, std=0.02), "w_o": _normal(g, H, NQ * D, std=0.02), "w_gu": _normal(g, 2 * F, H, std=0.02),
            "w_down": _normal(g, H, F, std=0.02), "q_norm": _normal(g, D, std=0.03, mean=0.3), "k_norm": _normal(g, D, std=0.03, mean=0.3),
            **{n: _normal(g, H, std=0.1, mean=1.0) for n in ("ln_in", "ln_post_attn", "ln_pre_ffn", "ln_post_ffn")}})
    return w


def _batch(case, seed, page):
    """Query lengths, lengths after the pass, a page table over a pool whose pages are handed out in no order, and the pool's size."""
    decode = case["phase"] == "decode"
    kv = _lengths(case)
    q = [case.get("rows", 1)] * len(kv) if decode else list(kv)
    need = [-(-n // page) for n in kv]
    total = sum(need)
    order = np.random.default_rng(seed).permutation(total + 4)[:total].astype(np.int32)
    table = np.zeros((len(kv), max(need)), dtype=np.int32)
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = order[at:at + n]
        at += n
    return q, kv, table, total + 4


def _slots(table, s, n, page):
    """Flat cache slots of positions ``0 .. n - 1`` of sequence ``s``."""
    p = np.arange(n)
    return torch.from_numpy(table[s, p // page].astype(np.int64) * page + p % page).cuda()


def _dense_inputs(case, seed):
    g = _gen(seed)
    w = _dense_weights(g, LAYERS)
    q, kv, table, pages = _batch(case, seed, PAGE)
    ids = torch.randint(0, V, (sum(q),), generator=g, device="cuda", dtype=torch.int32)
    caches = []
    if case["phase"] == "decode":               # what earlier passes left: keys of normed heads, values of unit size
        for _ in range(LAYERS):
            caches.append((_normal(g, pages, PAGE, NKV, D, std=0.3), _normal(g, pages, PAGE, NKV, D)))
    return w, q, kv, table, pages, ids, caches


def _mla_inputs(case, seed):
    g = _gen(seed)
    w = {"w_qa_kva": _normal(g, MQ + ML + MR, MH, std=0.02), "qa_norm": _normal(g, MQ, std=0.1, mean=1.0), "kv_norm": _normal(g, ML, std=0.1, mean=1.0),
         "w_qb": _normal(g, MHEADS * (MN + MR), MQ, std=0.02), "w_uk": _normal(g, MHEADS, ML, MN, std=0.02), "w_uv": _normal(g, MHEADS, MN, ML, std=0.02),
         "w_o": _normal(g, MH, MHEADS * MN, std=0.02)}
    q, kv, table, pages = _batch(case, seed, MPAGE)
    x = _normal(g, sum(q), MH)
    cache = _normal(g, pages, MPAGE, ML + MR) if case["phase"] == "decode" else torch.zeros(pages, MPAGE, ML + MR, dtype=torch.bfloat16, device="cuda")
    return w, q, kv, table, pages, x, cache


_CODES = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0]


def _fp4_matrix(g, experts, rows, cols):
    """E2M1 codes, E4M3 block scales (in the tensor core's block order) and f32 second-level scales as blocks of 16 of a normal distribution
    have them: codes of normal values whose largest of 16 sits at 6, scales spread as those maxima are."""
    probs = np.diff([0.5 * (1 + math.erf(t * 0.31 / math.sqrt(2))) for t in (0.0, 0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 99.0)]) * 2
    nib = np.repeat(np.arange(8), np.maximum(1, np.round(probs * 128)).astype(int))[:128]
    nib = np.concatenate([np.pad(nib, (0, 128 - len(nib)), constant_values=1)] * 2) | (np.arange(256) // 128 * 8)
    lut = torch.from_numpy((nib[None, :] | (nib[:, None] << 4)).astype(np.uint8).reshape(-1)).cuda()
    codes = torch.empty(experts * rows, cols // 2, dtype=torch.uint8, device="cuda")
    step = max(1, (64 << 20) // (cols // 2))
    for i in range(0, codes.shape[0], step):
        part = codes[i:i + step]
        part.copy_(lut[torch.randint(0, 65536, part.shape, generator=g, device="cuda", dtype=torch.int32)])
    scales = torch.empty(experts * rows // 128, cols // 64, 512, dtype=torch.float32, device="cuda").normal_(150.0, 30.0, generator=g)
    sf = scales.clamp_(40.0, 400.0).to(torch.float8_e4m3fn).view(torch.uint8)
    s2 = torch.empty(experts, dtype=torch.float32, device="cuda").uniform_(0.9, 1.1, generator=g) * (0.02 / (3.2 * 150.0))
    return codes, sf, s2


def _experts_inputs(case, seed):
    g = _gen(seed)
    h, e, f, k, *_ = EXPERTS[case["model"]]
    slots = e + (1 if case["model"] == "k3" else 0)
    w = {"w13": _fp4_matrix(g, slots, 2 * f, h), "w2": _fp4_matrix(g, slots, h, f), "w_router": _normal(g, e, h, std=0.02), "next": _normal(g, h, std=0.1, mean=1.0)}
    if case["model"] == "k3":
        w["bias"] = _normal(g, e, std=0.002, dtype=torch.float32)       # small beside the scores: the load is balanced, as the bias is there for
    else:
        w["shared_gu"], w["shared_down"] = _normal(g, 2 * f, h, std=0.02), _normal(g, h, f, std=0.02)
    return w, _normal(g, case["rows"], h), _normal(g, case["rows"], h)


def _lora_inputs(case, seed):
    g = _gen(seed)
    w = _dense_weights(g, LORA_LAYERS)
    sizes = {"q_proj": (H, NQ * D), "k_proj": (H, NKV * D), "v_proj": (H, NKV * D), "o_proj": (NQ * D, H), "gate_proj": (H, F), "up_proj": (H, F),
             "down_proj": (F, H)}
    ad = {}
    for i in range(LORA_LAYERS):
        for p in PROJECTIONS:                   # adapters some way into their training: both factors filled
            fin, fout = sizes[p]
            bound = math.sqrt(3.0 / fin)
            a = torch.empty(RANK, fin, dtype=torch.float32, device="cuda").uniform_(-bound, bound, generator=g)
            ad[f"{i}_{p}"] = (a, _normal(g, fout, RANK, std=0.01, dtype=torch.float32))
    return w, ad, torch.randint(0, V, (case["seqs"], case["tokens"]), generator=g, device="cuda")


# ------------------------------------------------------------------------------------------------------------------ passes
def _dense_model(w, layers):
    from mary_b200.models.gemma4 import Gemma4Model, gemma_12b_config
    cfg = gemma_12b_config()
    cfg.num_hidden_layers = layers
    cfg.layer_types = cfg.layer_types[:layers]
    model = Gemma4Model(cfg, dtype=torch.bfloat16, device="cuda")
    model.embed.data, model.norm.data = w["embed"], w["norm"]
    for layer, lw in zip(model.layers, w["layers"]):
        for n, t in lw.items():
            getattr(layer, n).data = t
    return model


def _captured(step):
    """``step()`` as a CUDA graph, warmed up on a side stream first; returns the graph and the buffers that it fills."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), torch.no_grad():
        for _ in range(2):
            step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(graph):
        out = step()
    return graph, out


def _prepare_dense(case, seed):
    from mary_b200.runtime.batch import BatchMeta
    from mary_b200.runtime.kv_cache import PagedKVCache, Q8Pages
    w, q, kv, table, pages, ids, caches = _dense_inputs(case, seed)
    model = _dense_model(w, LAYERS)
    int8 = case["kv"] == "int8"
    cache = PagedKVCache(LAYERS, pages, PAGE, NKV, D, dtype=torch.bfloat16, device="cuda", kv_dtype="int8" if int8 else None)
    for i, rows in enumerate(caches):
        for t, r in zip((cache.k[i], cache.v[i]), rows):
            if int8:
                t.codes, t.sz = Q8Pages.quantize(r)
            else:
                t.copy_(r)
    kept = [t for l in range(LAYERS) for t in (cache.k[l], cache.v[l])]
    kept = [x for t in kept for x in ((t.codes, t.sz) if int8 else (t,))]
    state = {"kind": "dense", "phase": case["phase"], "model": model, "cache": cache, "kept": kept, "q": q, "kv": kv, "table": table, "ids": ids}
    if case["phase"] == "decode":
        meta = state["meta"] = BatchMeta.build(q, kv, table, PAGE, "cuda")      # the graph reads its tensors: they live with it
        state["graph"], state["out"] = _captured(lambda: model(ids, meta, cache))
    return state


def _prepare_mla(case, seed):
    from mary_b200.models.moe import k3_class_config
    from mary_b200.models.moe.model import MLAAttention, NoParallel
    from mary_b200.runtime.batch import BatchMeta
    from mary_b200.runtime.kv_cache import PagedKVCache
    w, q, kv, table, pages, x, rows = _mla_inputs(case, seed)
    attn = MLAAttention(k3_class_config(), 0, NoParallel(), torch.bfloat16, "cuda")
    for n, t in w.items():
        getattr(attn, n).data = t
    cache = PagedKVCache(1, pages, MPAGE, 1, ML + MR, dtype=torch.bfloat16, device="cuda", latent_dim=ML + MR)
    cache.k[0].copy_(rows)
    state = {"kind": "mla", "phase": case["phase"], "attn": attn, "cache": cache, "q": q, "kv": kv, "table": table, "x": x}
    if case["phase"] == "decode":
        meta = state["meta"] = BatchMeta.build(q, kv, table, MPAGE, "cuda")
        state["graph"], state["out"] = _captured(lambda: attn(x, meta, cache))
    return state


def _prepare_experts(case, seed):
    from mary_b200.models.moe import inkling_style_config, k3_class_config
    from mary_b200.models.moe.model import MoEFFN, NoParallel
    from mary_b200.ops.moe import NVFP4Experts
    w, x, h = _experts_inputs(case, seed)
    cfg = k3_class_config() if case["model"] == "k3" else inkling_style_config()
    ffn = MoEFFN(cfg, NoParallel(), torch.bfloat16, "cuda")
    ffn.w_router.data = w["w_router"]
    if "bias" in w:
        ffn.router_bias.data = w["bias"]
    else:
        ffn.shared.w_gu.data, ffn.shared.w_down.data = w["shared_gu"], w["shared_down"]
    hid, f = EXPERTS[case["model"]][0], EXPERTS[case["model"]][2]
    ffn.experts = NVFP4Experts(w["w13"][2].numel(), hid, f, *w["w13"], *w["w2"], act=cfg.act)
    state = {"kind": "experts", "ffn": ffn, "x": x, "h": h, "next": w["next"]}
    if case["rows"] <= 512:
        state["graph"], state["out"] = _captured(lambda: _feed_forward(state))
    return state


def _feed_forward(s):
    """The feed-forward half of a decoder layer: ``h += ffn(x)`` and the next layer's normed input."""
    from mary_b200 import ops
    ffn, x, h = s["ffn"], s["x"], s["h"].clone()
    fused = ffn.fused_ctx(x)
    if fused is not None:
        return ffn.forward_fused(fused, x, h, s["next"])
    return ops.add_rmsnorm(ffn(x), h, s["next"], EPS)


def _prepare_lora(case, seed):
    from mary_b200.train.lora import Gemma4LoraForward, LoraWeights
    w, adapters, ids = _lora_inputs(case, seed)
    model = _dense_model(w, LORA_LAYERS)
    lora = LoraWeights.init_gemma4(model, RANK, ALPHA)
    for n, (a, b) in adapters.items():
        lora.adapters[n].A.data, lora.adapters[n].B.data = a, b
    return {"kind": "lora", "fwd": Gemma4LoraForward(model, lora), "lora": lora, "ids": ids}


def prepare(case, seed):
    return {"dense": _prepare_dense, "mla": _prepare_mla, "experts": _prepare_experts, "lora": _prepare_lora}[case["kind"]](case, seed)


def run(state):
    kind = state["kind"]
    if "graph" in state:
        state["graph"].replay()
        out = state["out"]
    elif kind == "dense":
        from mary_b200.runtime.batch import BatchMeta
        with torch.no_grad():
            meta = BatchMeta.build(state["q"], state["kv"], state["table"], PAGE, "cuda")
            out = state["model"](state["ids"], meta, state["cache"], (meta.q_start[1:] - 1).long())
    elif kind == "mla":
        from mary_b200.runtime.batch import BatchMeta
        with torch.no_grad():
            out = state["attn"](state["x"], BatchMeta.build(state["q"], state["kv"], state["table"], MPAGE, "cuda"), state["cache"])
    elif kind == "experts":
        with torch.no_grad():
            out = _feed_forward(state)
    else:
        params = {f"{n}_{m}": p for n, ad in state["lora"].adapters.items() for m, p in (("A", ad.A), ("B", ad.B))}
        for p in params.values():
            p.grad = None
        loss = state["fwd"].loss(state["ids"])
        loss.backward()
        return {"loss": loss.detach(), "grads": {n: p.grad for n, p in params.items()}}
    if kind == "dense":
        return {"logits": out, "cache": state["kept"]}
    if kind == "mla":
        return {"out": out, "cache": state["cache"].k[0]}
    return {"next": out[0], "h": out[1]}


# ------------------------------------------------------------------------------------------------------------------ the work
def _pairs(kv, q, window):
    """(query, key) pairs that causal attention with this window forms."""
    total = 0
    for n, m in zip(kv, q):
        p = np.arange(n - m, n) + 1
        total += int(np.minimum(p, window).sum() if window else p.sum())
    return total


def _read_rows(kv, q, window):
    """Cache rows that a pass cannot do without."""
    return sum(min(n, window + m - 1) if window else n for n, m in zip(kv, q))


def work(case):
    kind = case["kind"]
    if kind == "dense":
        kv = _lengths(case)
        decode = case["phase"] == "decode"
        q = [1] * len(kv) if decode else kv
        t, b = sum(q), len(kv)
        per = (NQ + 2 * NKV) * D * H + H * NQ * D + 3 * F * H
        rows = sum(_read_rows(kv, q, 0 if l == GLOBAL else WINDOW) for l in range(LAYERS)) if decode else LAYERS * t
        row = 2 * NKV * (D + 8 if case["kv"] == "int8" else 2 * D)
        flops = 2 * LAYERS * per * t + 2 * V * H * b + sum(4 * NQ * D * _pairs(kv, q, 0 if l == GLOBAL else WINDOW) for l in range(LAYERS))
        return {"bytes": 2 * (LAYERS * per + V * H) + rows * row + 4 * b * V, "flops": flops}
    if kind == "mla":
        kv = _lengths(case)
        decode = case["phase"] == "decode"
        q = [case["rows"]] * len(kv) if decode else kv
        t = sum(q)
        mats = (MQ + ML + MR) * MH + MHEADS * (MN + MR) * MQ + 2 * MHEADS * ML * MN + MH * MHEADS * MN
        wide = (ML + MR + ML) if decode else (MN + MR + MN)      # scores and sums in the latent space, or over expanded keys and values
        return {"bytes": 2 * mats + 4 * t * MH + 2 * (ML + MR) * sum(kv), "flops": 2 * mats * t + 2 * MHEADS * wide * _pairs(kv, q, 0)}
    if kind == "experts":
        h, e, f, k, *_ = EXPERTS[case["model"]]
        t = case["rows"]
        hit = e * (1 - (1 - k / e) ** t) + (1 if case["model"] == "k3" else 0)
        k3 = case["model"] == "k3"
        return {"bytes": hit * 3 * h * f * 9 / 16 + 2 * e * h + (0 if k3 else 6 * h * f) + 8 * t * h, "flops": 2 * t * (3 * h * f * (k + 1) + e * h)}
    t = case["seqs"] * case["tokens"]
    per = (NQ + 2 * NKV) * D * H + H * NQ * D + 3 * F * H
    ranks = RANK * ((NQ + 2 * NKV) * D + 3 * H + NQ * D + H + 2 * (F + H) + F + H)
    flops = 4 * LORA_LAYERS * per * t + 6 * LORA_LAYERS * ranks * t + 4 * V * H * t
    flops += LORA_LAYERS * 14 * NQ * D * case["seqs"] * _pairs([case["tokens"]], [case["tokens"]], WINDOW)
    return {"bytes": 2 * (LORA_LAYERS * per + V * H) + 8 * LORA_LAYERS * ranks, "flops": flops}


def tolerance(case):
    """About four times what bf16 activations were seen to give against 64 bits: 0.015 after six dense layers, 0.005 for one attention half, 0.0035
    for one expert half, 0.016 for adapter gradients.  Two runs of one dense decode step differ by up to 0.009 (sums whose order is not fixed)."""
    return {"dense": {"rel": 5e-2, "max": 0.3, "differ": 2e-3}, "mla": {"rel": 2e-2}, "experts": {"rel": 1.5e-2}, "lora": {"rel": 6e-2}}[case["kind"]]


# ------------------------------------------------------------------------------------------------------------------ 64 bits
def _rms(x, w=None):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w.double()


def _turn(x, pos, theta):
    """Rotation of the pairs ``(i, i + D / 2)`` of ``x [T, heads, D]``."""
    d = x.shape[-1]
    a = pos.double()[:, None] * (theta ** (-2.0 * torch.arange(d // 2, dtype=torch.float64, device=x.device) / d))[None]
    c, s = a.cos()[:, None], a.sin()[:, None]
    x1, x2 = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([x1 * c - x2 * s, x1 * s + x2 * c], -1)


def _mul(x, w):
    return x @ w.double().t()


def _attend(q, k, v, pos, window, scale):
    """``q [T, Hq, d]`` at ``pos`` over the keys at ``0 .. L - 1``, in runs of rows and kv head by kv head."""
    g, out = q.shape[1] // k.shape[1], torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=q.dtype, device=q.device)
    at = torch.arange(k.shape[0], device=q.device)
    for r in range(0, q.shape[0], 1024):
        p = pos[r:r + 1024, None]
        hidden = (at[None] > p) | ((p - at[None] >= window) if window else torch.zeros_like(at[None] > p))
        for j in range(k.shape[1]):
            s = torch.einsum("tgd,ld->gtl", q[r:r + 1024, j * g:(j + 1) * g], k[:, j]) * scale
            out[r:r + 1024, j * g:(j + 1) * g] = torch.einsum("gtl,ld->tgd", torch.softmax(s.masked_fill(hidden[None], -math.inf), -1), v[:, j])
    return out


def _geglu(gu):
    n = gu.shape[-1] // 2
    return torch.nn.functional.gelu(gu[..., :n], approximate="tanh") * gu[..., n:]


def _q8(x):
    lo, hi = x.amin(-1, keepdim=True), x.amax(-1, keepdim=True)
    sc = torch.where(hi > lo, (hi - lo) / 255.0, torch.ones_like(lo))
    return torch.floor((x - lo) / sc + 0.5).clamp(0, 255) * sc + lo


def _exact_dense(case, seed):
    w, q, kv, table, pages, ids, caches = _dense_inputs(case, seed)
    pos = torch.cat([torch.arange(n - m, n) for n, m in zip(kv, q)]).cuda()
    h = w["embed"][ids.long()].double() * math.sqrt(H)
    kept = []
    for l, lw in enumerate(w["layers"]):
        x = _mul(_rms(h, lw["ln_in"]), lw["w_qkv"]).view(-1, NQ + 2 * NKV, D)
        theta, window = THETA[l == GLOBAL], 0 if l == GLOBAL else WINDOW
        xq = _turn(_rms(x[:, :NQ], lw["q_norm"]), pos, theta)
        xk, xv = _turn(_rms(x[:, NQ:NQ + NKV], lw["k_norm"]), pos, theta), _rms(x[:, NQ + NKV:])
        kc, vc = (t.double() for t in caches[l]) if caches else (torch.zeros(pages, PAGE, NKV, D, dtype=torch.float64, device="cuda") for _ in range(2))
        if case["kv"] == "int8":
            kc, vc, xk, xv = _q8(kc.float()).double(), _q8(vc.float()).double(), _q8(xk), _q8(xv)
        o = torch.empty_like(xq)
        at = 0
        for s, (n, m) in enumerate(zip(kv, q)):
            slots = _slots(table, s, n, PAGE)
            for c, rows in ((kc, xk), (vc, xv)):
                c.view(-1, NKV, D)[slots[n - m:]] = rows[at:at + m]
            o[at:at + m] = _attend(xq[at:at + m], kc.view(-1, NKV, D)[slots], vc.view(-1, NKV, D)[slots], pos[at:at + m], window, 1.0)
            at += m
        kept += [None] * 4 if case["kv"] == "int8" else [kc, vc]
        h = h + _rms(_mul(o.flatten(1), lw["w_o"]), lw["ln_post_attn"])
        y = torch.cat([_mul(_geglu(_mul(_rms(p, lw["ln_pre_ffn"]), lw["w_gu"])), lw["w_down"]) for p in h.split(2048)])
        h = h + _rms(y, lw["ln_post_ffn"])
    rows = torch.tensor(np.cumsum(q) - 1, device="cuda")
    x = _rms(h, w["norm"])[rows]
    logits = torch.cat([_mul(x, part) for part in w["embed"].split(65536)], 1)
    return {"logits": CAP * torch.tanh(logits / CAP), "cache": kept}


def _exact_mla(case, seed):
    w, q, kv, table, pages, x, cache = _mla_inputs(case, seed)
    pos = torch.cat([torch.arange(n - m, n) for n, m in zip(kv, q)]).cuda()
    y = _mul(x.double(), w["w_qa_kva"])
    qb = _mul(_rms(y[:, :MQ], w["qa_norm"]), w["w_qb"]).view(-1, MHEADS, MN + MR)
    row = torch.cat([_rms(y[:, MQ:MQ + ML], w["kv_norm"]), _turn(y[:, None, MQ + ML:], pos, MTHETA)[:, 0]], -1)
    qr = _turn(qb[..., MN:], pos, MTHETA)
    cache = cache.double()
    o = torch.empty(x.shape[0], MHEADS, MN, dtype=torch.float64, device="cuda")
    at = 0
    for s, (n, m) in enumerate(zip(kv, q)):
        slots = _slots(table, s, n, MPAGE)
        cache.view(-1, ML + MR)[slots[n - m:]] = row[at:at + m]
        lat = cache.view(-1, ML + MR)[slots]
        for j in range(0, MHEADS, 16):
            uk, uv = w["w_uk"][j:j + 16].double(), w["w_uv"][j:j + 16].double()
            if m == n:                          # a prompt: over expanded keys and values
                k = torch.cat([torch.einsum("lk,hkn->lhn", lat[:, :ML], uk), lat[:, None, ML:].expand(n, 16, MR)], -1)
                v = torch.einsum("lk,hnk->lhn", lat[:, :ML], uv)
                qq = torch.cat([qb[at:at + m, j:j + 16, :MN], qr[at:at + m, j:j + 16]], -1)
                o[at:at + m, j:j + 16] = _attend(qq, k, v, pos[at:at + m], 0, (MN + MR) ** -0.5)
            else:
                qq = torch.cat([torch.einsum("thn,hkn->thk", qb[at:at + m, j:j + 16, :MN], uk), qr[at:at + m, j:j + 16]], -1)
                a = _attend(qq, lat[:, None], lat[:, None, :ML], pos[at:at + m], 0, (MN + MR) ** -0.5)
                o[at:at + m, j:j + 16] = torch.einsum("thk,hnk->thn", a, uv)
        at += m
    return {"out": _mul(o.flatten(1), w["w_o"]), "cache": cache}


def _fp4_blocks(x):
    """The activation rule in blocks of 16: E4M3 scale of the largest magnitude over 6, then the nearest E2M1 value."""
    b = x.float().unflatten(-1, (-1, 16))
    s = (b.abs().amax(-1) / 6.0).clamp(max=448.0).to(torch.float8_e4m3fn).float()
    m = b / torch.where(s > 0, s, torch.ones_like(s))[..., None]
    step = torch.bucketize(m.abs(), torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=x.device), right=True)
    v = torch.tensor(_CODES, dtype=torch.float64, device=x.device)[step] * torch.sign(m).double() * s[..., None].double()
    return v.flatten(-2)


def _fp4_dense(parts, e, rows, cols):
    codes, sf, s2 = parts
    c = codes[e * rows:(e + 1) * rows]
    table = torch.tensor(_CODES + [-v for v in _CODES], dtype=torch.float64, device=c.device)
    v = table[torch.stack([c & 15, c >> 4], -1).reshape(rows, cols).int()]
    b = sf[e * rows // 128:(e + 1) * rows // 128].view(rows // 128, cols // 64, 32, 4, 4).permute(0, 3, 2, 1, 4).reshape(rows, cols // 16)
    return (v.view(rows, cols // 16, 16) * b.contiguous().view(torch.float8_e4m3fn).double()[..., None]).view(rows, cols) * s2[e].double()


def _swiglu(gu):
    n = gu.shape[-1] // 2
    return torch.nn.functional.silu(gu[..., :n]) * gu[..., n:]


def _exact_experts(case, seed):
    w, x, h = _experts_inputs(case, seed)
    hid, e, f, k, groups, keep, scale = EXPERTS[case["model"]]
    logits = _mul(x.double(), w["w_router"])
    if case["model"] == "k3":
        p = torch.sigmoid(logits)
        pick = p + w["bias"].double()
        best = pick.view(-1, groups, e // groups).topk(2, -1).values.sum(-1).topk(keep, -1).indices
        mask = torch.zeros(x.shape[0], groups, dtype=torch.bool, device="cuda").scatter_(1, best, True)
        idx = pick.masked_fill(~mask.repeat_interleave(e // groups, 1), -math.inf).topk(k, -1).indices
    else:
        p = torch.softmax(logits, -1)
        idx = p.topk(k, -1).indices
    wt = p.gather(1, idx)
    wt = wt / wt.sum(-1, keepdim=True) * scale
    if case["model"] == "k3":                   # the shared expert: one more, which every row visits with weight 1
        idx = torch.cat([idx, torch.full_like(idx[:, :1], e)], 1)
        wt = torch.cat([wt, torch.ones_like(wt[:, :1])], 1)
        y = torch.zeros_like(logits[:, :1].expand(-1, hid)).contiguous()
    else:
        y = _mul(_swiglu(_mul(x.double(), w["shared_gu"])), w["shared_down"])
    xq = _fp4_blocks(x)
    for j in idx.unique().tolist():
        t, c = (idx == j).nonzero(as_tuple=True)
        a = _swiglu(xq[t] @ _fp4_dense(w["w13"], j, 2 * f, hid).t())
        y.index_add_(0, t, (_fp4_blocks(a.to(torch.bfloat16)) @ _fp4_dense(w["w2"], j, hid, f).t()) * wt[t, c][:, None])
    out = h.double() + y
    return {"next": _rms(out, w["next"]), "h": out}


def _exact_lora(case, seed):
    w, adapters, ids = _lora_inputs(case, seed)
    b, n = ids.shape
    ad = {name: (a.double().requires_grad_(), c.double().requires_grad_()) for name, (a, c) in adapters.items()}
    pos = torch.arange(n, device="cuda")

    def lin(x, base, i, names):
        y, parts = _mul(x, base), []
        for p in names:
            a, c = ad[f"{i}_{p}"]
            parts.append((x @ a.t()) @ c.t() * (ALPHA / RANK))
        return y + torch.cat(parts, -1)

    def attend(q, k, v, window):
        hidden = (pos[None] > pos[:, None]) | (pos[:, None] - pos[None] >= window)
        outs = []
        for j in range(NQ):
            s = (q[:, j] @ k[:, j // 2].t()).masked_fill(hidden, -math.inf)
            outs.append(torch.softmax(s, -1) @ v[:, j // 2])
        return torch.stack(outs, 1)

    total = 0.0
    for r in range(b):                          # sequence by sequence: the gradients add up
        h = w["embed"][ids[r]].double() * math.sqrt(H)
        for i, lw in enumerate(w["layers"]):
            x = lin(_rms(h, lw["ln_in"]), lw["w_qkv"], i, PROJECTIONS[:3]).view(n, NQ + 2 * NKV, D)
            xq, xk = _turn(_rms(x[:, :NQ], lw["q_norm"]), pos, THETA[False]), _turn(_rms(x[:, NQ:NQ + NKV], lw["k_norm"]), pos, THETA[False])
            o = checkpoint(attend, xq, xk, _rms(x[:, NQ + NKV:]), WINDOW, use_reentrant=False)
            h = h + _rms(lin(o.flatten(1), lw["w_o"], i, ("o_proj",)), lw["ln_post_attn"])
            gu = lin(_rms(h, lw["ln_pre_ffn"]), lw["w_gu"], i, ("gate_proj", "up_proj"))
            h = h + _rms(lin(_geglu(gu), lw["w_down"], i, ("down_proj",)), lw["ln_post_ffn"])
        x = _rms(h, w["norm"])[:-1]
        head = w["embed"].double()
        grad = torch.zeros_like(x)
        for c in range(0, n - 1, 512):
            part = x[c:c + 512].detach().requires_grad_()
            loss = torch.nn.functional.cross_entropy(CAP * torch.tanh(part @ head.t() / CAP), ids[r, c + 1:c + 513][:part.shape[0]], reduction="sum") / (b * (n - 1))
            total += float(loss.detach())
            grad[c:c + 512] = torch.autograd.grad(loss, part)[0]
        del head
        x.backward(grad)
    return {"loss": torch.tensor(total, dtype=torch.float64), "grads": {f"{name}_{m}": p.grad for name, pair in ad.items() for m, p in zip("AB", pair)}}


def exact(case, seed):
    return {"dense": _exact_dense, "mla": _exact_mla, "experts": _exact_experts, "lora": _exact_lora}[case["kind"]](case, seed)
