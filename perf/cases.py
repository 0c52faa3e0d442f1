"""The work a user of this framework has it do, as cases that can be timed and compared.

Four kinds of case, each through the public entry points:

* ``linear``  -- one packed linear called eagerly, as a module written against ``torch.ops.alloy`` calls it
  (``gguf_*_mm`` or the fused gate/up ``gguf_*_silu``), from one token to a long prompt;
* ``attention`` -- one cache-attention op (``attention_cache``, ``_q8``, ``_q8_paged``): a decode token or a short
  verification chunk per sequence over a filled cache, the new K/V rows appended by the call;
* ``decode``  -- one step of ``QuantLlamaDecoder`` replayed from its captured graph, the serving loop's inner call;
* ``prefill`` -- a prompt chunk through ``QuantLlamaDecoder.prefill``.

Shapes are the repository's benchmark shapes (8B: hidden 4096, FFN 14336, 32/8 heads; 70B: hidden 8192, FFN 28672,
64/8 heads; head_dim 128, vocab 128256; fp16 cache at 2048 tokens, paged q8_0 pools at 4096-32768) and generic ones
of the same ranges.
"""

from __future__ import annotations

import math

import torch

from alloy_b200 import llama, synth
from alloy_b200.kv import PagedKVPool, alloc_quantized_kv

VOCAB = 128256
SHAPES = {  # name of the shape: hidden, ffn, heads, kv_heads
    "8b": (4096, 14336, 32, 8),
    "70b": (8192, 28672, 64, 8),
    "small": (2048, 5632, 16, 4),
}
D = 128          # head_dim of every shape above
ROW_BYTES = D // 32 * 34        # one q8_0 token row of one head
W_BYTES = {"q4_k": 144 / 256, "q6_k": 210 / 256, "q8_0": 34 / 32}


def listed():
    return [
        # The smallest call: one token through one square projection, called eagerly (an o_proj of a module model).
        {"name": "linear q4k 4096x4096 m1", "kind": "linear", "fmt": "q4_k", "gated": False, "n": 4096, "k": 4096, "m": 1,
         "dtype": "f16"},
        # A Q8_0 checkpoint's gate/up pair for one token of bf16 activations (bf16 modules on a Q8_0 file).
        {"name": "gated q80 14336x4096 m1", "kind": "linear", "fmt": "q8_0", "gated": True, "n": 14336, "k": 4096, "m": 1,
         "dtype": "bf16"},
        # A down projection (Q6_K in the Q4_K_M mix) over an odd-sized prompt chunk.
        {"name": "linear q6k 4096x14336 m333", "kind": "linear", "fmt": "q6_k", "gated": False, "n": 4096, "k": 14336,
         "m": 333, "dtype": "f16"},
        # A gate or up projection over a long prompt: the dense contraction of prefill.
        {"name": "linear q4k 14336x4096 m4096", "kind": "linear", "fmt": "q4_k", "gated": False, "n": 14336, "k": 4096,
         "m": 4096, "dtype": "bf16"},
        # Long-context serving: one token for each of 64 sequences over ragged paged q8_0 contexts.
        {"name": "attention paged b64 4k-32k", "kind": "attention", "kv": "paged", "batch": 64, "heads": 32, "kv_heads": 8,
         "lo": 4096, "hi": 32768, "queries": 1},
        # Chat with one user, and with 4, 16 and 32 users at once: the full 8B step at a filled context of 2048.
        {"name": "decode 8b b1", "kind": "decode", "shape": "8b", "layers": 32, "batch": 1, "context": 2048, "kv": "f16"},
        {"name": "decode 8b b4", "kind": "decode", "shape": "8b", "layers": 32, "batch": 4, "context": 2048, "kv": "f16"},
        {"name": "decode 8b b16", "kind": "decode", "shape": "8b", "layers": 32, "batch": 16, "context": 2048, "kv": "f16"},
        {"name": "decode 8b b32", "kind": "decode", "shape": "8b", "layers": 32, "batch": 32, "context": 2048, "kv": "f16"},
        # The large model's layers with the paged q8_0 pool: ten of its eighty layers, an odd batch, an odd context.
        {"name": "decode 70b/8 b7 paged", "kind": "decode", "shape": "70b", "layers": 10, "batch": 7, "context": 4101,
         "kv": "q8_paged"},
        # A whole prompt in one chunk: time to first token.
        {"name": "prefill 8b 2048", "kind": "prefill", "shape": "8b", "layers": 32, "batch": 1, "tokens": 2048, "start": 0,
         "kv": "f16"},
        # The next turn of a conversation: an odd number of new tokens behind a cached history in the paged pool.
        {"name": "prefill 8b 77 after 1500", "kind": "prefill", "shape": "8b", "layers": 32, "batch": 1, "tokens": 77,
         "start": 1500, "kv": "q8_paged"},
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], uniform over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "attention", "decode", "decode", "prefill"])
    if kind == "linear":
        fmt = rng.choice(["q4_k", "q4_k", "q6_k", "q8_0"])
        n = _log(rng, 512, 28672)
        return {"kind": kind, "fmt": fmt, "gated": fmt != "q6_k" and rng.random() < 0.4,
                "n": n if rng.random() < 0.25 else -(-n // 64) * 64, "k": 256 * _log(rng, 4, 56), "m": _log(rng, 1, 4096),
                "dtype": rng.choice(["f16", "bf16"])}
    if kind == "attention":
        heads, kv_heads = rng.choice([(32, 8), (64, 8), (16, 4), (32, 32), (28, 4)])
        batch = _log(rng, 1, 64)
        hi = _log(rng, 128, max(256, min(32768, (1 << 20) // batch)))
        return {"kind": kind, "kv": rng.choice(["f16", "q8", "paged"]), "batch": batch, "heads": heads, "kv_heads": kv_heads,
                "lo": max(64, hi // rng.choice([1, 2, 8])), "hi": hi, "queries": 1 if rng.random() < 0.7 else rng.randint(2, 16)}
    shape = rng.choice(["8b", "8b", "70b", "small"])
    layers = rng.randint(2, {"8b": 16, "70b": 5, "small": 24}[shape])
    kv = rng.choice(["f16", "q8_paged"])
    if kind == "decode":
        batch = _log(rng, 1, 64)
        return {"kind": kind, "shape": shape, "layers": layers, "batch": batch,
                "context": _log(rng, 128, min(8192, 131072 // batch)), "kv": kv}
    batch = rng.choice([1, 1, 1, 3])
    tokens = _log(rng, 8, 1500 // batch)
    return {"kind": kind, "shape": shape, "layers": layers, "batch": batch, "tokens": tokens, "start": _log(rng, tokens, 4096),
            "kv": kv}


# ------------------------------------------------------------------------------------------- what a program has in hand


def _q8_rows(shape, gen):
    """q8_0 codes and scales of N(0, 1) rows."""
    x = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(generator=gen).view(*shape[:-1], shape[-1] // 32, 32)
    s = (x.abs().amax(-1) / 127).half()
    codes = torch.round(x / s.float().unsqueeze(-1)).clamp_(-127, 127).to(torch.int8)
    return codes.view(shape), s


def _fill_pool(pool, gen):
    """A pool's pages as quantised N(0, 1) rows, some thousand pages at a time."""
    rows = pool.pool.view(-1, pool.row_bytes)
    for lo in range(0, rows.shape[0], 1 << 20):
        part = rows[lo:lo + (1 << 20)]
        codes, s = _q8_rows((part.shape[0], pool.head_dim), gen)
        blocks = part.view(part.shape[0], -1, 34)
        blocks[:, :, 2:] = codes.view(torch.uint8).view(part.shape[0], -1, 32)
        blocks[:, :, :2] = s.view(torch.uint8).view(part.shape[0], -1, 2)


def _prepare_linear(c, gen):
    n, k = c["n"], c["k"]
    make = {"q4_k": lambda: (synth.q4k_blocks_device(n, k, gen),), "q6_k": lambda: (synth.q6k_blocks_device(n, k, gen),),
            "q8_0": lambda: synth.q8_0_weight_device(n, k, gen)}[c["fmt"]]
    weights = make() + make() if c["gated"] else make()
    # a gate's products of about one, where SiLU bends; N(0, 1) activations elsewhere
    scale = {"q4_k": 3.0, "q8_0": 12.0}[c["fmt"]] / math.sqrt(k) if c["gated"] else 1.0
    x = torch.empty((c["m"], k), dtype=torch.float32, device="cuda").normal_(0, scale, generator=gen)
    op = getattr(torch.ops.alloy, "gguf_%s_%s" % (c["fmt"], "silu" if c["gated"] else "mm"))
    return {"op": op, "x": x.to(torch.float16 if c["dtype"] == "f16" else torch.bfloat16), "w": weights}


def _prepare_attention(c, gen):
    b, h, kv_h, s = c["batch"], c["heads"], c["kv_heads"], c["queries"]
    # the same lengths for every seed, dealt to the sequences in another order: the pool keeps its size
    lens = torch.randint(c["lo"], c["hi"] + 1, (b,), generator=torch.Generator().manual_seed(b))
    lens = lens[torch.randperm(b, generator=torch.Generator().manual_seed(gen.initial_seed()))]
    half = lambda *sh: torch.empty(sh, dtype=torch.float32, device="cuda").normal_(generator=gen).half()
    st = {"kv": c["kv"], "q": half(b, h, s, D), "k": half(b, kv_h, s, D), "v": half(b, kv_h, s, D)}
    if c["kv"] == "paged":
        pages = [(int(n) + s + 15) // 16 for n in lens]
        order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(gen.initial_seed() + 1)).tolist()
        pool = PagedKVPool(sum(pages), kv_h, D, b, max(pages), "cuda", free_order=order)
        for i in range(b):
            pool.reserve(i, int(lens[i]) + s)
        _fill_pool(pool, gen)
        st.update(pos=lens.to(torch.int32).cuda(), cache=(pool.page_table, pool.pool))
        return st
    # the contiguous caches have one position for the whole batch
    rows = c["hi"] + s
    st["pos"] = torch.tensor([c["hi"]], dtype=torch.int32, device="cuda")
    if c["kv"] == "f16":
        st["cache"] = (half(b, kv_h, rows, D), half(b, kv_h, rows, D))
    else:
        cache = alloc_quantized_kv(b, kv_h, rows, D, "cuda")
        for codes, scales in (cache[:2], cache[2:]):
            for i in range(b):
                codes[i], scales[i] = _q8_rows(tuple(codes.shape[1:]), gen)
        st["cache"] = cache
    return st


def _prepare_model(c, gen, seed):
    hidden, ffn, heads, kv_heads = SHAPES[c["shape"]]
    shape = llama.LlamaShape(layers=c["layers"], hidden=hidden, ffn=ffn, heads=heads, kv_heads=kv_heads, head_dim=D, vocab=VOCAB)
    context = c["context"] if c["kind"] == "decode" else c["start"] + c["tokens"]
    # zero-mean weights of a trained model's size keep a deep random stack inside fp16
    dec = llama.QuantLlamaDecoder(shape, c["batch"], context, seed=seed, kv=c["kv"], d_scale=0.1, centered=True)
    for pool in dec.pools:
        _fill_pool(pool, gen)
    if c["kind"] == "prefill":
        ids = torch.randint(0, VOCAB, (c["batch"], c["tokens"]), generator=gen, device="cuda")
        return {"dec": dec, "ids": ids, "start": c["start"]}
    dec.ids.copy_(torch.randint(0, VOCAB, (c["batch"],), generator=gen, device="cuda"))
    if c["kv"] == "q8_paged":       # sequences of different lengths, the longest at the full context
        dec.seq_pos.copy_(torch.randint(context // 2, context, (c["batch"],), generator=gen, device="cuda").to(torch.int32))
        dec.seq_pos[0] = context - 1
    dec.capture()
    return {"dec": dec}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "linear":
        state = _prepare_linear(case, gen)
    elif case["kind"] == "attention":
        state = _prepare_attention(case, gen)
    else:
        state = _prepare_model(case, gen, seed)
    state["kind"] = case["kind"]
    return state


# ------------------------------------------------------------------------------------------- one pass


def _model_outputs(dec):
    """Logits and the first layer's cache.  The tokens are the logits' argmax and are left out: two rows of a random
    model can be close enough for a rounding to swap them."""
    cache = (dec.k_cache[0], dec.v_cache[0]) if dec.kv_kind == "f16" else (dec.pools[0].pool,)
    return (dec.logits,) + cache


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["op"](state["x"], *state["w"])
    if kind == "attention":
        if state["kv"] == "f16":
            out = torch.ops.alloy.attention_cache(state["q"], state["k"], state["v"], state["pos"], *state["cache"], -1.0)
        else:
            op = torch.ops.alloy.attention_cache_q8 if state["kv"] == "q8" else torch.ops.alloy.attention_cache_q8_paged
            out = op(state["q"], state["k"], state["v"], state["pos"], *state["cache"])
        return (out,) + state["cache"]
    if kind == "decode":
        state["dec"].step()
    else:
        state["dec"].prefill(state["ids"], state["start"])
    return _model_outputs(state["dec"])


# ------------------------------------------------------------------------------------------- its size and its accuracy


def _kv_bytes(kv, kv_heads):
    """Cache bytes of one token, K and V."""
    return 2 * kv_heads * (2 * D if kv == "f16" else ROW_BYTES)


def work(case):
    c = case
    if c["kind"] == "linear":
        mats = 2 if c["gated"] else 1
        return {"bytes": mats * c["n"] * c["k"] * W_BYTES[c["fmt"]] + 2 * c["m"] * (c["n"] + c["k"]),
                "flops": 2.0 * mats * c["m"] * c["n"] * c["k"]}
    if c["kind"] == "attention":
        b, h, s = c["batch"], c["heads"], c["queries"]
        tokens = b * (c["hi"] if c["kv"] != "paged" else (c["lo"] + c["hi"]) / 2)
        return {"bytes": (tokens + 2 * b * s) * _kv_bytes(c["kv"], c["kv_heads"]) + 4 * b * h * s * D,
                "flops": 4.0 * h * D * s * (tokens + b * (s + 1) / 2)}
    hidden, ffn, heads, kv_heads = SHAPES[c["shape"]]
    shape = llama.LlamaShape(c["layers"], hidden, ffn, heads, kv_heads, D, VOCAB)
    b, s = c["batch"], c.get("tokens", 1)
    if c["kind"] == "decode":       # paged sequences are between half and all of the context long
        tokens, pairs = b * c["context"] * (0.75 if c["kv"] != "f16" else 1.0), 0.0
        pairs = tokens
    else:
        tokens, pairs = b * (c["start"] + s), b * s * (c["start"] + (s + 1) / 2)
    return {"bytes": shape.weight_bytes() + c["layers"] * (tokens + b * s) * _kv_bytes(c["kv"], kv_heads) + 2 * b * VOCAB,
            "flops": 2.0 * b * s * shape.layer_weight_elems() + 2.0 * b * hidden * VOCAB + 4.0 * c["layers"] * heads * D * pairs}


def tolerance(case):
    """About four times what the path differs by from the same sums in 64 bits (linear, attention) or from another
    kernel of the library for the same step (models).

    Measured: fp16 linears 2.1e-4 (weights in fp32) to 3.2e-4 (weights rounded to fp16), bf16 ones 1.7e-3 to 2.4e-3,
    the largest element 1.3e-3 and 1.1e-2; decode attention 2.1e-4 and 4.9e-4; the logits of 8 and 32 layers 1.7e-3 and
    3.8e-3 (one launch against op by op), those of a batch of 32 against the same token alone 7.0e-3 and 3.5e-2.  A
    chunk reads q8_0 rows rounded to fp16.  A q8_0 pool's bytes move where an fp16 rounding of K or V moves a scale."""
    if case["kind"] == "linear":
        return {"rel": 1.2e-3, "max": 6e-3} if case["dtype"] == "f16" else {"rel": 1e-2, "max": 4.5e-2}
    if case["kind"] == "attention":
        return {"rel": 1e-3, "max": 2.5e-3} if case["queries"] == 1 else {"rel": 2e-3, "max": 2e-2}
    deep = math.sqrt(case["layers"])
    return {"rel": 5e-3 * deep, "max": 2.5e-2 * deep, "differ": 0.01 if case["kv"] != "f16" else 0.0}


# ------------------------------------------------------------------------------------------- the same in 64 bits


def _block(w, nbytes):
    """Packed rows as (N, super-blocks, bytes)."""
    return w.reshape(w.shape[0], -1, nbytes)


def _f16_at(blk, at):
    return blk[..., at:at + 2].contiguous().view(torch.float16).double()


def _weights64(fmt, w, scales=None):
    """A packed matrix in 64 bits, (N, K)."""
    if fmt == "q8_0":
        return (w.double().view(w.shape[0], -1, 32) * scales.double().unsqueeze(-1)).view(w.shape)
    if fmt == "q4_k":
        blk = _block(w, 144)
        s = blk[..., 4:16].int()
        a, b, c = s[..., :4], s[..., 4:8], s[..., 8:]
        scale = torch.cat([a & 63, (c & 15) | (a >> 6 << 4)], -1).double() * _f16_at(blk, 0)
        least = torch.cat([b & 63, (c >> 4) | (b >> 6 << 4)], -1).double() * _f16_at(blk, 2)
        qs = blk[..., 16:].unflatten(-1, (4, 32))
        codes = torch.stack([qs & 15, qs >> 4], -2).flatten(-3, -2)
        return (codes.double() * scale.unsqueeze(-1) - least.unsqueeze(-1)).flatten(1)
    blk = _block(w, 210)
    low = blk[..., :128].unflatten(-1, (2, 2, 32))
    low = torch.cat([low & 15, low >> 4], -2)
    high = blk[..., 128:192].unflatten(-1, (2, 1, 32))
    high = torch.cat([(high >> s) & 3 for s in (0, 2, 4, 6)], -2)
    codes = (low | high << 4).double() - 32
    scale = blk[..., 192:208].contiguous().view(torch.int8).double() * _f16_at(blk, 208)
    return (codes.flatten(-3).unflatten(-1, (16, 16)) * scale.unsqueeze(-1)).flatten(1)


def _product64(x, w, fmt, scales=None):
    """x W^T in 64 bits, some rows of W at a time."""
    part = max(1, (1 << 27) // x.shape[-1])
    return torch.cat([x @ _weights64(fmt, w[i:i + part], None if scales is None else scales[i:i + part]).T
                      for i in range(0, w.shape[0], part)], -1)


def _stored64(rows, kv):
    """New K or V rows as a cache holds them: a q8_0 cache rounds them to its codes."""
    if kv == "f16":
        return rows
    x = rows.half().float().unflatten(-1, (-1, 32))
    s = (x.abs().amax(-1, keepdim=True) / 127).half().double()
    return (torch.round(x.double() / s.clamp_min(1e-30)).clamp(-127, 127) * s).flatten(-2)


def _cached64(kv, cache, i, n):
    """The first n K and V rows of sequence i, (kv_heads, n, D) each."""
    if kv == "f16":
        return [c[i, :, :n].double() for c in cache]
    if kv == "q8":
        return [(cache[j][i, :, :n].double().unflatten(-1, (-1, 32)) * cache[j + 1][i, :, :n].double().unsqueeze(-1)).flatten(-2)
                for j in (0, 2)]
    table, pool = cache
    pages = pool[table[i, :(n + 15) // 16].long()].unflatten(-1, (-1, 34))
    rows = pages[..., 2:].contiguous().view(torch.int8).double() * _f16_at(pages, 0)
    return [rows[:, j].flatten(-2).transpose(0, 1).flatten(1, 2)[:, :n] for j in (0, 1)]


def _attention64(q, k, v, kv, cache, starts):
    """Causal attention of new rows (batch, heads, tokens, D) over the cached ones before `starts` and themselves."""
    out = []
    for i, start in enumerate(starts):
        ck, cv = (torch.cat([c, _stored64(new[i], kv)], 1) for c, new in zip(_cached64(kv, cache, i, start), (k, v)))
        s, kv_h = q.shape[2], k.shape[1]
        mask = torch.arange(start + s, device="cuda") > start + torch.arange(s, device="cuda").unsqueeze(1)
        heads = []
        for g in range(kv_h):
            p = q[i].unflatten(0, (kv_h, -1))[g] @ ck[g].T / math.sqrt(D)
            heads.append(p.masked_fill(mask, -math.inf).softmax(-1) @ cv[g])
        out.append(torch.cat(heads))
    return torch.stack(out)


def _norm64(x, w, eps):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt() * w.double()


def _rope64(x, pos, inv_freq):
    angle = (pos.float().unsqueeze(-1) * inv_freq).double().unsqueeze(1)        # (batch, 1, tokens, D / 2)
    a, b = x.chunk(2, -1)
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], -1)


def _model64(c, dec, ids, pos):
    """Logits of each sequence's last token; ids and pos are (batch, tokens)."""
    s, (b, n) = dec.shape, ids.shape
    x = _weights64("q4_k", dec.embed[ids.flatten()])
    split = lambda t: t.view(b, n, -1, D).transpose(1, 2)
    kv = "f16" if c["kv"] == "f16" else "paged"
    for i, lw in enumerate(dec.layers):
        y = _norm64(x, lw.norm_in, s.eps)
        q, k, v = (split(_product64(y, w, fmt)) for w, fmt in ((lw.wq, "q4_k"), (lw.wk, "q4_k"), (lw.wv, "q6_k")))
        q, k = _rope64(q, pos, dec.inv_freq), _rope64(k, pos, dec.inv_freq)
        cache = (dec.k_cache[i], dec.v_cache[i]) if kv == "f16" else (dec.pools[i].page_table, dec.pools[i].pool)
        a = _attention64(q, k, v, kv, cache, pos[:, 0].tolist())
        x = x + _product64(a.transpose(1, 2).reshape(b * n, -1), lw.wo, "q4_k")
        y = _norm64(x, lw.norm_post, s.eps)
        y = torch.nn.functional.silu(_product64(y, lw.wg, "q4_k")) * _product64(y, lw.wu, "q4_k")
        x = x + _product64(y, lw.wd, "q6_k")
    return _product64(_norm64(x.view(b, n, -1)[:, -1], dec.norm_final, s.eps), dec.head, "q6_k")


def exact(case, seed):
    """What `run` returns, in 64 bits; the caches hold copies and codes and have no such value."""
    c, st = case, prepare(case, seed)
    if c["kind"] == "linear":
        x, w = st["x"].double(), st["w"]
        if c["fmt"] == "q8_0":
            y = [_product64(x, w[i], "q8_0", w[i + 1]) for i in range(0, len(w), 2)]
        else:
            y = [_product64(x, m, c["fmt"]) for m in w]
        return torch.nn.functional.silu(y[0]) * y[1] if c["gated"] else y[0]
    if c["kind"] == "attention":
        starts = st["pos"].tolist() * (1 if c["kv"] == "paged" else c["batch"])
        out = _attention64(*(st[n].double() for n in "qkv"), c["kv"], st["cache"], starts)
        return (out,) + (None,) * len(st["cache"])
    dec, b = st["dec"], c["batch"]
    if c["kind"] == "prefill":
        ids, first = st["ids"], torch.full((b, 1), c["start"], device="cuda")
    else:
        ids, first = dec.ids.view(b, 1), (dec.pos.expand(b) if c["kv"] == "f16" else dec.seq_pos).view(b, 1)
    logits = _model64(c, dec, ids, first + torch.arange(ids.shape[1], device="cuda"))
    return (logits,) + (None,) * (2 if c["kv"] == "f16" else 1)
