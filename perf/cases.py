"""What this framework is timed on: the calls its users make, on models of the shapes this repository is configured, tested and benchmarked with.

A case is a model (a cut of `layers` of its layers, or all of them) and one thing done with it:

  generate  the whole loop of a small program: a prompt, then greedy tokens, through `generate`
  decode    a conversation whose cache is there (`context` rows) goes on for `tokens` tokens, fed back on the device
  prompt    a prompt of `tokens` tokens, behind `context` cached ones, up to its last row's logits and sample
  batch     `batch` conversations of `context` cached rows advance together by `tokens` tokens
  both      a prompt of `context` tokens, then `tokens` tokens fed back on the device

Weights are drawn on the GPU from the seed.  Linear layers are normal and, for Q8_0 models, quantised here; the vocabulary projection holds,
for every token, the embedding of the token before it in a random order, and what the layers add is of the embedding's own size.  So the
best token stands out as clearly as a trained model's does, and a sum in another order never changes which token is fed back.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("oneiron-luminal_b200")

# Decoders of `CONFIGS`; what a draw may cut them to.
PLAIN = ["llama3_8b_q8", "qwen3_4b_q8", "gpt_oss_20b_q8"]
SMALL = ["tiny_f32", "small_q8", "small_oss", "small_q8_odd"]
# Layers described one by one, at the sizes of the benchmark's comparisons.
MADIPEL = {
    "madipel_4096": dict(width=4096, heads=32, kv=8, dim=128, ff=21504, window=4096),
    "madipel_2560": dict(width=2560, heads=32, kv=8, dim=128, ff=14592, window=1024),
    "madipel_2048": dict(width=2048, heads=16, kv=4, dim=128, ff=12288, window=512),
}
REDENEX = {
    "redenex_2560": dict(width=2560, lru=2560, blocks=10, heads=20, kv=4, dim=64, vdim=128, ff=7680, chunk=2048),
    "redenex_2048": dict(width=2048, lru=2560, blocks=10, heads=16, kv=2, dim=64, vdim=128, ff=6144, chunk=1024),
}
BLOCK_VOCAB = 32768


def listed():
    return [
        # the smallest call: a toy decoder in 32 bits, where launches and the way to the GPU are all there is
        dict(name="tiny-generate", do="generate", model="tiny_f32", layers=2, context=16, tokens=16, batch=1),
        # one user talking to the headline model: a reply of some words behind a short conversation
        dict(name="llama-decode", do="decode", model="llama3_8b_q8", layers=32, context=512, tokens=16, batch=1),
        # a document as prompt, and a follow-up question (a ragged number of tokens) behind a conversation
        dict(name="llama-prompt-4096", do="prompt", model="llama3_8b_q8", layers=32, context=0, tokens=4096, batch=1),
        dict(name="llama-prompt-387", do="prompt", model="llama3_8b_q8", layers=32, context=1021, tokens=387, batch=1),
        # a server: many long conversations with one system prompt, and a few short ones on a paged cache
        dict(name="llama-batch-32", do="batch", model="llama3_8b_q8", layers=32, context=2048, tokens=8, batch=32),
        dict(name="llama-batch-5", do="batch", model="llama3_8b_q8", layers=32, context=301, tokens=8, batch=5, page=64),
        # a smaller model (head norms, tied bf16 head) far into a conversation, its tokens drawn and not the best ones taken
        dict(name="qwen-decode", do="decode", model="qwen3_4b_q8", layers=36, context=3000, tokens=16, batch=1, temperature=0.8),
        # routed experts, sliding windows, sinks
        dict(name="oss-decode", do="decode", model="gpt_oss_20b_q8", layers=24, context=700, tokens=16, batch=1),
        # dense bf16 layers described one by one: a long prompt, and decoding
        dict(name="madipel-prompt", do="prompt", model="madipel_4096", layers=4, context=0, tokens=4096, batch=1),
        dict(name="madipel-decode", do="decode", model="madipel_2560", layers=8, context=2500, tokens=16, batch=1),
        # recurrences over residual streams: their state comes from the prompt
        dict(name="redenex-both", do="both", model="redenex_2048", layers=9, context=1000, tokens=16, batch=1),
    ]


def draw(rng):
    def size(a, b):
        return min(b, max(a, int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))))

    do = rng.choice(["generate", "decode", "decode", "prompt", "prompt", "batch", "batch", "both"])
    if do == "generate":
        model = rng.choice(SMALL)
        n = pkg.CONFIGS[model].max_seq
        context = size(1, n // 2)
        return dict(do=do, model=model, layers=pkg.CONFIGS[model].n_layers, context=context, tokens=rng.randint(2, n - context), batch=1)
    if do == "both":
        return dict(do=do, model=rng.choice(sorted(REDENEX)), layers=3 * rng.randint(1, 3), context=size(8, 3000), tokens=rng.randint(2, 24), batch=1)
    if do == "batch":
        c = dict(do=do, model="llama3_8b_q8", layers=rng.randint(2, 8), context=size(1, 3000), tokens=rng.randint(2, 10), batch=rng.randint(2, 32))
        if rng.random() < 0.5:
            c["page"] = rng.choice([64, 128])
        return c
    model = rng.choice(PLAIN + PLAIN + sorted(MADIPEL))
    if do == "prompt":
        if model == "gpt_oss_20b_q8":
            model = "qwen3_4b_q8"                     # (its prompts are taken token by token: what `decode` measures)
        tokens = size(4, 4000)
        return dict(do=do, model=model, layers=rng.randint(2, 6), context=size(1, 4096 - tokens) if rng.random() < 0.4 else 0, tokens=tokens, batch=1)
    c = dict(do=do, model=model, layers=rng.randint(2, 8), context=size(1, 4000), tokens=rng.randint(2, 24), batch=1)
    if rng.random() < 0.3:
        c["temperature"] = 0.8
    return c


# ---------------------------------------------------------------------------------------------------------------- models

def spec_of(case):
    """(ModelDesc, layer descriptors or None, configuration of layers described one by one)."""
    L, name, page = case["layers"], case["model"], case.get("page", 0)
    if name in MADIPEL:
        z = MADIPEL[name]
        mixer = {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["dim"], "scale": z["dim"] ** -0.5, "v_mix": True, "mask": {"size": z["window"]}}
        cfg = {"architecture": "Madipel", "layers": [{"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": z["ff"]}}] * L, "width": z["width"],
               "vocab": BLOCK_VOCAB, "residual_mult": 0.5, "logit_scale": 1.0, "norm": {"eps": 1e-5}}
    elif name in REDENEX:
        z = REDENEX[name]
        mlp = {"kind": "dense", "ff": z["ff"], "limit": 7.0}
        rec = {"type": "rglru", "mixer": {"width": z["lru"], "blocks": z["blocks"], "conv": 4}, "mlp": mlp}
        att = {"type": "attention", "mlp": mlp, "mixer": {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["vdim"], "conv": 4, "diff": 0.5,
               "scale": z["dim"] ** -0.5, "rot": {"dims": z["dim"], "base": 10000.0}, "mask": {"size": z["chunk"]}}}
        cfg = {"architecture": "Redenex", "layers": [(rec, rec, att)[i % 3] for i in range(L)], "width": z["width"], "vocab": BLOCK_VOCAB, "streams": 4,
               "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6}}
    else:
        return pkg.CONFIGS[name].copy(n_layers=L, max_batch=case["batch"], kv_page_rows=page), None, None
    spec = pkg.models.from_config(cfg, dtype="bfloat16", max_seq=4096)
    return spec.desc, spec.layers, cfg


class Draws:
    """Normal numbers by (seed, what, layer): the same whoever asks."""

    def __init__(self, seed):
        self.seed = seed

    def generator(self, what, layer):
        key = (self.seed * 1000003 + layer * 911 + sum((i + 1) * 131 * ord(c) for i, c in enumerate(what))) & 0x7FFFFFFFFFFF
        return torch.Generator(device="cuda").manual_seed(key)

    def normal(self, what, layer, shape, std=1.0, mean=0.0):
        return torch.randn(shape, generator=self.generator(what, layer), device="cuda").mul_(std).add_(mean)

    def uniform(self, what, layer, shape, a, b):
        return torch.rand(shape, generator=self.generator(what, layer), device="cuda").mul_(b - a).add_(a)

    def next_token(self, vocab):
        """next[t]: the token the vocabulary projection puts behind t."""
        return torch.randperm(vocab, generator=self.generator("order", 0), device="cuda")


def q8_blocks(w):
    """[n, k] -> Q8_0 wire blocks [n, k / 32, 34]: a binary16 scale, 32 quants."""
    b = w.view(w.shape[0], -1, 32)
    out = torch.empty((*b.shape[:2], 34), dtype=torch.uint8, device=w.device)
    d = b.abs().amax(-1).div_(127).half()
    out[..., :2] = d.unsqueeze(-1).view(torch.uint8)
    s = d.float().clamp_(min=1e-8).reciprocal_().unsqueeze(-1)
    out[..., 2:] = (b * s).round_().clamp_(-127, 127).to(torch.int8).view(torch.uint8)
    return out


def q8_values(blocks):
    """Q8_0 wire blocks -> [n, k] in 64 bits."""
    d = blocks[..., :2].contiguous().view(torch.float16).double()
    return (blocks[..., 2:].view(torch.int8).double() * d).view(blocks.shape[0], -1)


def plain_tensors(d, r):
    """(slot, layer, tensor) of a decoder of `CONFIGS`; uint8: Q8_0 blocks, bfloat16 or float32: values."""
    H, F, V, E = d.hidden, d.ffn, d.vocab, d.n_experts
    qd, kvd = d.n_q_heads * d.head_dim, d.n_kv_heads * d.head_dim
    q8 = d.weight_dtype == pkg.DTYPE["q8_0"]
    small = torch.bfloat16 if d.embed_dtype == pkg.DTYPE["bf16"] else torch.float32
    lin = q8_blocks if q8 else (lambda w: w)
    e = 0.05 if d.tied_head else 1.0                                  # a tied table is small, or its logits would be huge
    added = e * 3.5 / math.sqrt(d.n_layers)                           # what all layers add is about as large as the embedding
    embed = r.normal("embed", 0, (V, H), e).to(small)
    yield "embed", 0, embed
    for l in range(d.n_layers):
        yield "attn_norm", l, r.normal("attn_norm", l, (H,), 0.1, 1.0).to(small)
        yield "mlp_norm", l, r.normal("mlp_norm", l, (H,), 0.1, 1.0).to(small)
        for s, n in (("q", qd), ("k", kvd), ("v", kvd)):
            yield s, l, lin(r.normal(s, l, (n, H), (0.7 if s == "v" else 1.0) / math.sqrt(H)))
        yield "o", l, lin(r.normal("o", l, (H, qd), added / math.sqrt(qd)))
        if d.qk_norm:
            for s in ("q_norm", "k_norm"):
                yield s, l, r.normal(s, l, (d.head_dim,), 0.1, 1.0).to(small)
        if d.proj_bias:
            for s, n in (("q_bias", qd), ("k_bias", kvd), ("v_bias", kvd), ("o_bias", H)):
                yield s, l, r.normal(s, l, (n,), 0.1).to(small)
        if d.attn_sinks:
            yield "sinks", l, r.normal("sinks", l, (d.n_q_heads,)).to(small)
        if E:
            yield "router", l, r.normal("router", l, (E, H), 3.0 / math.sqrt(H)).to(small)
            yield "router_bias", l, r.normal("router_bias", l, (E,), 0.1).to(small)
            yield "exp_gate_up", l, q8_blocks(r.normal("exp_gate_up", l, (E * 2 * F, H), 1 / math.sqrt(H)))
            yield "exp_gate_up_bias", l, r.normal("exp_gate_up_bias", l, (E * 2 * F,), 0.1).to(small)
            yield "exp_down", l, q8_blocks(r.normal("exp_down", l, (E * H, F), added / math.sqrt(F)))
            yield "exp_down_bias", l, r.normal("exp_down_bias", l, (E * H,), 0.1 * e).to(small)
        else:
            for s in ("gate", "up"):
                yield s, l, lin(r.normal(s, l, (F, H), 1 / math.sqrt(H)))
            yield "down", l, lin(r.normal("down", l, (H, F), added / math.sqrt(F)))
    yield "final_norm", 0, r.normal("final_norm", 0, (H,), 0.1, 1.0).to(small)
    if not d.tied_head:
        head = torch.empty((V, H), device="cuda")
        head[r.next_token(V)] = embed.float() / math.sqrt(H)
        yield "lm_head", 0, lin(head)


def block_tensors(cfg, r):
    """The same for layers described one by one (all bf16)."""
    D, V, bf = cfg["width"], cfg["vocab"], torch.bfloat16

    def lin(s, l, n, k, g=1.0):
        return s, l, r.normal(s, l, (n, k), g / math.sqrt(k)).to(bf)

    def vec(s, l, n, std, mean=0.0):
        return s, l, r.normal(s, l, (n,) if isinstance(n, int) else n, std, mean).to(bf)

    def taps(s, l, channels, n):
        w = r.normal(s, l, (channels, n), 0.4)
        w[:, -1] += 1.0
        return s, l, w.to(bf)

    embed = r.normal("embed", 0, (V, D)).to(bf)
    yield "embed", 0, embed
    head = torch.empty((V, D), device="cuda")
    head[r.next_token(V)] = embed.float() / math.sqrt(D)
    yield "lm_head", 0, head.to(bf)
    if cfg["architecture"] == "Madipel":
        yield vec("final_norm", 0, D, 0.1, 1.0)
        yield vec("final_norm_bias", 0, D, 0.1)
        for l, layer in enumerate(cfg["layers"]):
            m, F = layer["mixer"], layer["mlp"]["ff"]
            nq, nk, nv = m["heads"] * m["dim"], m["kv_heads"] * m["dim"], m["kv_heads"] * m["vdim"]
            yield vec("attn_norm", l, D, 0.1, 1.0)
            yield vec("attn_norm_bias", l, D, 0.1)
            yield lin("q", l, nq, D)
            yield lin("k", l, nk, D)
            yield lin("v", l, nv, D)
            yield lin("o", l, D, m["heads"] * m["vdim"], 0.5)
            yield vec("q_norm", l, nq, 0.2, 1.0)
            yield vec("k_norm", l, nk, 0.2, 1.0)
            for s, a, b in (("temp", 0.5, 1.5), ("dist_r1", 0.05, 1.0), ("dist_r2", 0.05, 0.6)):
                yield s, l, r.uniform(s, l, (m["heads"],), a, b).to(bf)
            yield "v_mix", l, r.uniform("v_mix", l, (1,), 0.2, 0.8).to(bf)
            yield lin("up", l, F, D, 1.2)
            yield lin("down", l, D, F, 0.2)
            yield "act", l, (torch.tensor([0.6, -0.4], device="cuda") + r.normal("act", l, (2,), 0.1)).to(bf)
        return
    S = cfg["streams"]
    yield vec("final_norm", 0, D, 0.1)
    for l, layer in enumerate(cfg["layers"]):
        m, F = layer["mixer"], layer["mlp"]["ff"]
        for q, norm in (("hc1", "attn_norm"), ("hc2", "mlp_norm")):
            yield vec(norm, l, D, 0.1)
            yield vec(q + "_in", l, S, 0.1, 1.0 / S)
            yield vec(q + "_out", l, S, 0.1, 0.4)
            yield q + "_mix", l, (torch.eye(S, device="cuda") + r.normal(q + "_mix", l, (S, S), 0.03)).to(bf)
        if layer["type"] == "rglru":
            w, b = m["width"], m["blocks"]
            n = w // b
            yield lin("rec_y", l, w, D)
            yield vec("rec_y_bias", l, w, 0.3)
            yield lin("rec_x", l, w, D)
            yield vec("rec_x_bias", l, w, 0.3)
            yield taps("rec_conv", l, w, m["conv"])
            yield vec("rec_conv_bias", l, w, 0.2)
            for s in ("rec_ra", "rec_ri"):
                yield vec(s, l, (b, n, n), 1 / math.sqrt(n))
                yield vec(s + "_bias", l, (b, n), 0.5)
            yield "rec_lam", l, r.uniform("rec_lam", l, (w,), -8.0, 0.5).to(bf)
            yield lin("o", l, D, w)
        else:
            H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            for s, n in (("q", H * 2 * dk), ("k", G * 2 * dk), ("v", G * dv)):
                yield lin(s, l, n, D)
                yield vec(s + "_bias", l, n, 0.3)
                yield taps(s + "_conv", l, n, m["conv"])
            yield vec("q_norm", l, dk, 0.2, 1.0)
            yield vec("k_norm", l, dk, 0.2, 1.0)
            for s in ("lq1", "lk1", "lq2", "lk2"):
                yield vec(s, l, dk, 0.5 / math.sqrt(dk))
            yield lin("o", l, D, H * dv)
        yield lin("gate", l, F, D, 1.5)
        yield lin("up", l, F, D, 1.5)
        yield lin("down", l, D, F)


def tensors(case, r):
    d, layers, cfg = spec_of(case)
    return plain_tensors(d, r) if cfg is None else block_tensors(cfg, r)


def cached_rows(case, d, layers, r):
    """(layer, "k" or "v", rows) of the conversation so far, as the cache holds them."""
    kv = torch.bfloat16 if d.kv_dtype == pkg.DTYPE["bf16"] else torch.float32
    for l in range(d.n_layers):
        g = layers[l] if layers else None
        nk, nv = (g.n_kv_heads * g.qk_dim, g.n_kv_heads * g.v_dim) if g else (d.n_kv_heads * d.head_dim,) * 2
        yield l, "k", r.normal("cache k", l, (case["context"], nk)).to(kv)
        yield l, "v", r.normal("cache v", l, (case["context"], nv), 0.7).to(kv)


def first_tokens(case, seed, vocab):
    """What the user sends: a prompt, or one token per conversation."""
    n = {"generate": case["context"], "both": case["context"], "prompt": case["tokens"], "decode": 1, "batch": case["batch"]}[case["do"]]
    return [int(t) for t in np.random.default_rng(seed).integers(0, vocab, n)]


# ------------------------------------------------------------------------------------------------------------------ runs

def prepare(case, seed):
    d, layers, _ = spec_of(case)
    r = Draws(seed)
    rt = pkg.B200Runtime.initialize()
    rt.load_model(d, layers)
    kind = {torch.uint8: "q8_0", torch.bfloat16: "bf16", torch.float32: "f32"}
    for slot, layer, t in tensors(case, r):
        torch.cuda.current_stream().synchronize()      # the library copies from the tensor on its own stream
        rc = rt._lib.lum_model_set_weight(rt._h, pkg.SLOT[slot], layer, ctypes.c_void_p(t.data_ptr()), t.numel() * t.element_size(), pkg.DTYPE[kind[t.dtype]])
        if rc:
            raise pkg.LumError(rc, "%s of layer %d: %s" % (slot, layer, rt._lib.lum_last_error(rt._h).decode()))
        del t
    rt.synchronize()
    if case["do"] in ("decode", "batch", "prompt") and case["context"]:
        for layer, which, rows in cached_rows(case, d, layers, r):
            rt.kv_load(layer, which, case["context"], rows.view(torch.uint8).cpu().numpy())
        for b in range(1, case["batch"]):
            rt.kv_copy(0, b, case["context"])
    if case.get("temperature"):
        rt.set_sampling(temperature=case["temperature"], top_k=64, top_p=0.95, seed=seed)
    rt.synchronize()
    torch.cuda.empty_cache()
    return {"rt": rt, "case": dict(case), "tokens": first_tokens(case, seed, d.vocab)}


def run(state):
    rt, case, tokens = state["rt"], state["case"], state["tokens"]
    n, p = case["tokens"], case["context"]
    if case["do"] == "generate":
        got = rt.generate(tokens, n)
        return {"tokens": np.asarray(got, np.int32), "logits": rt.get_f32()}
    if case["do"] == "batch":
        rt.batch_begin(tokens, [p] * len(tokens))
        rt.batch_decode(n)
        return {"tokens": rt.batch_get_decoded(n), "logits": np.stack([rt.batch_get_logits(b) for b in range(len(tokens))])}
    if case["do"] == "prompt":
        rt.set_data(tokens)
        rt.execute({"s": n, "p": p})
        return {"tokens": np.asarray([rt.get_token()], np.int32), "logits": rt.get_f32()}
    rt.decode_reset()
    rt.set_data(tokens)
    rt.execute({"s": len(tokens), "p": p if case["do"] == "decode" else 0})
    rt.decode_greedy(n - 1)
    return {"tokens": rt.get_decoded(n - 1), "logits": rt.get_f32()}


def work(case):
    d, layers, cfg = spec_of(case)
    n, p, B = case["tokens"], case["context"], case["batch"]
    if cfg is None:
        qd, kvd = d.n_q_heads * d.head_dim, d.n_kv_heads * d.head_dim
        q8 = 34 / 32 if d.weight_dtype == pkg.DTYPE["q8_0"] else 4
        eb, kb = (2 if d.embed_dtype == pkg.DTYPE["bf16"] else 4), (2 if d.kv_dtype == pkg.DTYPE["bf16"] else 4)
        ff = 3 * d.hidden * d.ffn * max(1, d.top_k)
        per = 2 * d.hidden * (qd + kvd) + ff
        weights, head = d.n_layers * per * q8, d.vocab * d.hidden * (eb if d.tied_head else q8)
        flops, head_flops = 2.0 * d.n_layers * per, 2.0 * d.vocab * d.hidden
        reach = [d.sliding_window if d.sliding_window and l % 2 == 0 else 1 << 30 for l in range(d.n_layers)]
        att = [(4.0 * qd, 2 * kvd * kb, w, 0) for w in reach]
    else:
        weights = 2 * (pkg.models.ModelSpec(cfg["architecture"], d, layers).weight_elems_per_token() - d.vocab * d.hidden)
        head, flops, head_flops = 2 * d.vocab * d.hidden, float(weights), 2.0 * d.vocab * d.hidden
        att = [(2.0 * g.n_q_heads * max(1, g.maps) * (g.qk_dim + g.v_dim), 2 * g.n_kv_heads * (max(1, g.maps) * g.qk_dim + g.v_dim), g.window or 1 << 30, g.chunk)
               for g in layers if g.mixer == 0]

    def rows(first, count):
        """Bytes of cache read once for these positions taken together, written ones included, and flops of their attention."""
        nbytes = nflops = 0.0
        for f, row, window, chunk in att:
            low = max(0, first - window + 1)
            if chunk:
                low = max(low, first // chunk * chunk)
            nbytes += row * (first + count - low)
            if chunk:
                nflops += f * sum((i % chunk) + 1 for i in range(first, first + count))
            else:
                seen = [min(window, i + 1) for i in (first, first + count - 1)]
                nflops += f * count * (seen[0] + seen[1]) / 2
        return nbytes, nflops

    if case["do"] == "prompt":
        kv, fl = rows(p, n)
        return {"bytes": weights + head + kv, "flops": flops * n + head_flops + fl}
    total, ops = 0.0, 0.0
    at, steps = p, n
    if case["do"] in ("generate", "both"):            # the prompt's own pass gives the first token
        kv, fl = rows(0, p)
        total, ops = weights + head + kv, flops * p + head_flops + fl
        steps = n - 1
    for i in range(steps):
        kv, fl = rows(at + i, 1)
        total += weights + head + B * kv
        ops += B * (flops + head_flops + fl)
    return {"bytes": total, "flops": ops}


def tolerance(case):
    # About four times what is seen against 64 bits, or between two orders of the sums.  Whole numbers (tokens) agree: see the top of this
    # file for why no near-tie decides one.
    if case["model"] == "tiny_f32":
        return {"rel": 5e-6}                          # 32 bits throughout (4e-7 seen)
    if case["model"] in MADIPEL or case["model"] in REDENEX:
        return {"rel": 4e-3, "max": 0.1}              # operands rounded to bf16 on the way (8e-4 seen)
    if "oss" in case["model"]:
        return {"rel": 1e-2, "max": 0.3}              # as the next line, and a router's near-tie may fall the other way in a row of the cache
    return {"rel": 3e-3, "max": 0.05}                 # 32-bit sums over a cache of bf16 values, whose roundings may fall the other way (7e-4 seen)


# ----------------------------------------------------------------------------------------------------------------- exact

def values(t):
    return q8_values(t) if t.dtype == torch.uint8 else t.double()


def rms(x, g, eps):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt() * g


def six(v):
    """A graph's constants travel as text with six decimals."""
    return float("%.6f" % v)


def turn(x, pos, d):
    """x [..., rows, heads, dim], rotated by the rows' positions."""
    n = d.head_dim
    i = torch.arange(n // 2, device=x.device, dtype=torch.float64)
    pos, fac = pos.double(), 1.0
    if d.rope_style == 0:
        inv = torch.exp2(-(2 * i * six(1.0 / n)) * six(math.log(d.rope_theta)) * six(1.0 / math.log(2.0)))
    elif d.rope_style == 1:
        inv = d.rope_theta ** (-2 * i / n)
    else:
        def corr(rot):
            return n * math.log(d.yarn_orig_max_pos / (rot * 2 * math.pi)) / (2 * math.log(d.rope_theta))
        low, high = corr(d.yarn_beta_fast), corr(d.yarn_beta_slow)
        t = ((i - low) / (high - low)).clamp(0, 1)
        pf = d.rope_theta ** (2 * i / n)
        inv, fac = t / (d.yarn_factor * pf) + (1 - t) / pf, 0.1 * math.log(d.yarn_factor) + 1.0
    a = (pos[:, None] * inv)[:, None, :]
    c, s = a.cos() * fac, a.sin() * fac
    if d.rope_style == 0:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, u * s + v * c], -1).flatten(-2)
    u, v = x[..., : n // 2], x[..., n // 2:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def attend(q, k, v, pos, kpos, scale, window=0, sinks=None, bias=None, chunk=0):
    """q [B, n, heads, dim], k and v [B, m, kv heads, dim] (B = 1: shared) -> [B, n, heads * vdim]."""
    B, n, H, _ = q.shape
    G = k.shape[2]
    see = kpos[None, :] <= pos[:, None]
    if window:
        see &= pos[:, None] - kpos[None, :] < window
    if chunk:
        see &= pos[:, None] // chunk == kpos[None, :] // chunk
    out = torch.empty(B, n, H, v.shape[-1], dtype=q.dtype, device=q.device)
    for h in range(H):
        kh, vh = k[:, :, h // (H // G)], v[:, :, h // (H // G)]
        s = (q[:, :, h] @ kh.transpose(1, 2)) * (scale if not isinstance(scale, torch.Tensor) else scale[h])
        if bias is not None:
            s = s - bias(h, (pos[:, None] - kpos[None, :]).clamp(min=0).double())
        s = s.masked_fill_(~see, -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks[h].expand(B, n, 1)], -1)
            out[:, :, h] = s.softmax(-1)[..., :-1] @ vh
        else:
            out[:, :, h] = s.softmax(-1) @ vh
    return out.flatten(2)


def experts(x, W, d):
    flat = x.reshape(-1, d.hidden)
    top, which = (flat @ W["router"].T + W["router_bias"]).topk(d.top_k, -1)
    share = top.softmax(-1)
    out = torch.zeros_like(flat)
    F, H = d.ffn, d.hidden
    for e in which.unique().tolist():
        row, k = (which == e).nonzero(as_tuple=True)
        gu = flat[row] @ q8_values(W["exp_gate_up"][e * 2 * F:(e + 1) * 2 * F]).T + W["exp_gate_up_bias"][e * 2 * F:(e + 1) * 2 * F]
        g, u = gu[:, 0::2].clamp(max=d.swiglu_limit), gu[:, 1::2].clamp(-d.swiglu_limit, d.swiglu_limit)
        y = ((u + 1) * g * torch.sigmoid(1.702 * g)) @ q8_values(W["exp_down"][e * H:(e + 1) * H]).T + W["exp_down_bias"][e * H:(e + 1) * H]
        out.index_add_(0, row, share[row, k, None] * y)
    return out.view_as(x)


def plain_forward(case, d, r, tokens, first, last_only):
    """Logits of `tokens` [B, n] at positions first .. (behind the cached rows, if any)."""
    B, n = tokens.shape
    pos = torch.arange(first, first + n, device="cuda")
    old = dict(((l, w), t) for l, w, t in cached_rows(case, d, None, r)) if first else {}
    kpos = torch.arange(0, first + n, device="cuda")
    x, W, at, embed = None, {}, 0, None

    def cache(l, which, new):
        if d.kv_dtype == pkg.DTYPE["bf16"]:
            new = new.bfloat16().double()             # what a cache of that type holds
        if not first:
            return new
        return torch.cat([old[l, which].double().view(1, first, d.n_kv_heads, d.head_dim).expand(B, -1, -1, -1), new], 1)

    def layer(l, x):
        q, k, v = (rms(x, W["attn_norm"], six(d.rms_eps)) @ W[s].T + (W[s + "_bias"] if d.proj_bias else 0) for s in "qkv")
        q, k, v = q.view(B, n, -1, d.head_dim), k.view(B, n, -1, d.head_dim), v.view(B, n, -1, d.head_dim)
        if d.qk_norm:
            q, k = rms(q, W["q_norm"], d.rms_eps), rms(k, W["k_norm"], d.rms_eps)
        window = d.sliding_window if d.sliding_window and (not d.window_even_layers or l % 2 == 0) else 0
        a = attend(turn(q, pos, d), cache(l, "k", turn(k, pos, d)), cache(l, "v", v), pos, kpos, d.head_dim ** -0.5, window, W.get("sinks"))
        x = x + a @ W["o"].T + (W["o_bias"] if d.proj_bias else 0)
        h = rms(x, W["mlp_norm"], six(d.rms_eps))
        if d.n_experts:
            return x + experts(h, W, d)
        g = h @ W["gate"].T
        return x + (g / (1 + torch.exp2(-g * six(1.0 / math.log(2.0)))) * (h @ W["up"].T)) @ W["down"].T

    for slot, l, t in plain_tensors(d, r):
        if slot == "embed":
            embed, x = t, t[tokens].double()
            continue
        if (l != at or slot == "final_norm") and "o" in W:
            x, W = layer(at, x), {}
        at = l
        if slot == "final_norm":
            x = rms(x[:, -1:] if last_only else x, t.double(), six(d.rms_eps))
        elif slot == "lm_head":
            return x @ values(t).T
        else:
            W[slot] = t if slot in ("exp_gate_up", "exp_down") else values(t)
    return x @ embed.double().T


def madipel_forward(case, d, layers, cfg, r, tokens, first, last_only):
    n, D = tokens.shape[1], cfg["width"]
    pos, kpos = torch.arange(first, first + n, device="cuda"), torch.arange(0, first + n, device="cuda")
    old = dict(((l, w), t) for l, w, t in cached_rows(case, d, layers, r)) if first else {}
    W = {(s, l): t for s, l, t in block_tensors(cfg, r)}
    e = torch.arange(D, device="cuda")
    ang = pos.double()[:, None] * 10000.0 ** (-(2.0 * (e // 2)) / D)
    x = W["embed", 0][tokens].double() + torch.where(e % 2 == 0, ang.sin(), ang.cos())
    eps, v_first = cfg["norm"]["eps"], None

    def norm(x, g, b):
        c = x - x.mean(-1, keepdim=True)
        return c * (c.square().mean(-1, keepdim=True) + eps).rsqrt() * g.double() + b.double()

    for l, y in enumerate(cfg["layers"]):
        m = y["mixer"]
        w = {s: t.double() for (s, k), t in W.items() if k == l and s not in ("embed", "lm_head", "final_norm", "final_norm_bias")}
        h = norm(x, w["attn_norm"], w["attn_norm_bias"])
        q, k, v = rms(h @ w["q"].T, w["q_norm"], eps), rms(h @ w["k"].T, w["k_norm"], eps), h @ w["v"].T
        v_first = v if v_first is None else v_first
        v = v if l == 0 else (1 - w["v_mix"]) * v + w["v_mix"] * v_first
        if first:
            k, v = torch.cat([old[l, "k"].double()[None], k], 1), torch.cat([old[l, "v"].double()[None], v], 1)
        a = attend(q.view(1, n, m["heads"], -1), k.view(1, first + n, m["kv_heads"], -1), v.view(1, first + n, m["kv_heads"], -1), pos, kpos, m["scale"] * w["temp"],
                   m["mask"]["size"], bias=lambda h, dist: w["dist_r1"][h] * torch.log1p(w["dist_r2"][h] * dist))
        z = h @ w["up"].T
        sp = torch.nn.functional.softplus(w["act"])
        neg = z.clamp(max=0)
        z = torch.where(z > 0, sp[0] * z * z, (0.5 + sp[1]) * (torch.expm1(neg) - neg)) + z / 2
        x = x + cfg["residual_mult"] * (a @ w["o"].T + z @ w["down"].T)
    x = norm(x[:, -1:] if last_only else x, W["final_norm", 0], W["final_norm_bias", 0])
    return x @ W["lm_head", 0].double().T * cfg["logit_scale"]


def redenex_forward(cfg, r, tokens):
    """Logits of every row of a whole sequence [n]."""
    W = {(s, l): t for s, l, t in block_tensors(cfg, r)}
    n, eps, F = len(tokens), cfg["norm"]["eps"], torch.nn.functional
    pos = torch.arange(n, device="cuda")

    def norm(x, g):
        return rms(x, 1.0 + g, eps)

    def conv(u, w):
        t = w.shape[1]
        p = torch.cat([u.new_zeros(t - 1, u.shape[1]), u])
        return sum(p[j:j + n] * w[:, j] for j in range(t))

    def recurrence(h, w):
        y = F.gelu(h @ w["rec_y"].T + w["rec_y_bias"], approximate="tanh")
        u = conv(h @ w["rec_x"].T + w["rec_x_bias"], w["rec_conv"]) + w["rec_conv_bias"]
        b = w["rec_ra"].shape[0]
        gate = [torch.sigmoid(torch.einsum("nbk,bok->nbo", u.view(n, b, -1), w[s]) + w[s + "_bias"]).reshape(n, -1) for s in ("rec_ra", "rec_ri")]
        log_a = -8.0 * gate[0] * F.softplus(w["rec_lam"])
        a, add = log_a.exp(), (-torch.expm1(2 * log_a)).sqrt() * gate[1] * u
        s, out = torch.zeros_like(u[0]), torch.empty_like(u)
        for t in range(n):
            s = torch.addcmul(add[t], a[t], s)
            out[t] = s
        return (out * y) @ w["o"].T

    def attention(h, w, m):
        q, k, v = (conv(h @ w[c].T + w[c + "_bias"], w[c + "_conv"]) for c in "qkv")
        H, G, dim = m["heads"], m["kv_heads"], m["dim"]
        half = m["rot"]["dims"] // 2
        ang = (pos.double()[:, None] * m["rot"]["base"] ** (-2.0 * torch.arange(half, device="cuda").double() / (2 * half)))[:, None, :]

        def rot(x):
            a, b = x[..., :half], x[..., half:2 * half]
            return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin(), x[..., 2 * half:]], -1)

        q = rot(rms(q.view(n, H * 2, dim), w["q_norm"], eps)).view(1, n, H, 2, dim)
        k = rot(rms(k.view(n, G * 2, dim), w["k_norm"], eps)).view(1, n, G, 2, dim)
        lam = (w["lq1"] @ w["lk1"]).exp() - (w["lq2"] @ w["lk2"]).exp() + m["diff"]
        a = [attend(q[:, :, :, i], k[:, :, :, i], v.view(1, n, G, -1), pos, pos, m["scale"], chunk=m["mask"]["size"]).view(n, H, -1) for i in (0, 1)]
        o = rms(a[0] - lam * a[1], 1.0, eps) * (1.0 - m["diff"])
        return o.reshape(n, -1) @ w["o"].T

    xs = (W["embed", 0][tokens].double() * cfg["embedding"]["scale"])[None].expand(cfg["streams"], -1, -1)
    for l, y in enumerate(cfg["layers"]):
        w = {s: t.double() for (s, k), t in W.items() if k == l and s not in ("embed", "lm_head", "final_norm")}
        h = norm(torch.einsum("s,snd->nd", w["hc1_in"], xs), w["attn_norm"])
        z = recurrence(h, w) if y["type"] == "rglru" else attention(h, w, y["mixer"])
        xs = torch.einsum("st,snd->tnd", w["hc1_mix"], xs) + w["hc1_out"][:, None, None] * z
        h, lim = norm(torch.einsum("s,snd->nd", w["hc2_in"], xs), w["mlp_norm"]), y["mlp"]["limit"]
        g, u = (h @ w["gate"].T).clamp(max=lim), (h @ w["up"].T).clamp(-lim, lim)
        z = (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w["down"].T
        xs = torch.einsum("st,snd->tnd", w["hc2_mix"], xs) + w["hc2_out"][:, None, None] * z
    return norm(xs.sum(0), W["final_norm", 0].double()) @ W["lm_head", 0].double().T


def exact(case, seed):
    d, layers, cfg = spec_of(case)
    r, do, n = Draws(seed), case["do"], case["tokens"]
    tokens = torch.tensor(first_tokens(case, seed, d.vocab), device="cuda")
    after = torch.arange(d.vocab, device="cuda") if d.tied_head else r.next_token(d.vocab)
    if do == "prompt":
        rows = tokens[None]
    else:                                             # the tokens that will be fed back are known: all rows in one pass
        rows = tokens[:, None] if do in ("decode", "batch") else tokens[None]
        for _ in range(n - 1):
            rows = torch.cat([rows, after[rows[:, -1:]]], 1)
    first = case["context"] if do in ("decode", "batch", "prompt") else 0
    with torch.no_grad():
        if cfg is None:
            logits = plain_forward(case, d, r, rows, first, do == "prompt")
        elif cfg["architecture"] == "Madipel":
            logits = madipel_forward(case, d, layers, cfg, r, rows, first, do == "prompt")
        else:
            logits = redenex_forward(cfg, r, rows[0])[None]
    best = logits.argmax(-1)
    if do == "prompt":
        return {"tokens": best[0].int().cpu().numpy(), "logits": logits[0, -1].cpu().numpy()}
    if do == "batch":
        return {"tokens": best.T.int().cpu().numpy(), "logits": logits[:, -1].cpu().numpy()}
    best = best[0, -n:] if do == "generate" else best[0, 1 - n:]
    return {"tokens": best.int().cpu().numpy(), "logits": logits[0, -1].cpu().numpy()}
