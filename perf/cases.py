"""The performance cases of this library: what a program that serves a model with the ``efficient_kascade`` attention
has it do, through the public entry points of :class:`kascade_b200.EfficientKascadeStrategy`.

Four kinds of case, all with 32 query heads, 8 KV heads and head dimension 128:

* ``prefill``      the attention of a prompt, layer by layer, as the Hugging Face attention modules call it
                   (``attention_forward``); optionally a left-padded batch with its 4-D mask
* ``hf_decode``    one generated token over a contiguous Hugging Face cache (``attention_forward``), optionally padded
* ``paged_decode`` one generated token per sequence over a paged cache (``paged_decode_forward``), fp16, bf16 or FP8
* ``append``       rotary embedding, optional QK norm and the append of new rows to a paged cache (``append_kv``)

A model has 32 to 36 layers, 5 of them anchors; a case runs its first few layers, which holds every kind of layer
(layer 0 is dense and selects, layer 2 is an anchor, the others reuse).  Rows of Q and K have unit RMS, as in models
with QK norm: logits then spread over a few units and 1 % of the keys draw a large part of the attention.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

from kascade_b200 import EfficientKascadeStrategy
from kascade_b200.strategy import topk_budget

H, G, D, TILE, PAGE = 32, 8, 128, 32, 16
ANCHORS = (0, 2)
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
SCALE = D ** -0.5
SEQUENCES_SEED = 77          # lengths belong to the case, not to the seed of its values


def listed():
    return [
        # a short chat turn: below 129 tokens the strategy is plain dense attention; launches and host time count
        {"name": "prefill_96", "kind": "prefill", "batch": 1, "length": 96, "layers": 8, "dtype": "fp16", "pct": 10,
         "rolling": True, "padded": False},
        # an ordinary prompt (the single-operator check's length)
        {"name": "prefill_2k", "kind": "prefill", "batch": 1, "length": 2048, "layers": 8, "dtype": "fp16", "pct": 10,
         "rolling": True, "padded": False},
        # a batch of prompts of different lengths, left-padded by the tokenizer to an odd length
        {"name": "prefill_padded_4x3001", "kind": "prefill", "batch": 4, "length": 3001, "layers": 8, "dtype": "bf16",
         "pct": 10, "rolling": False, "padded": True},
        # the benchmark's prompt: a long document, the first eight layers of a 32-layer model
        {"name": "prefill_32k", "kind": "prefill", "batch": 1, "length": 32768, "layers": 8, "dtype": "fp16", "pct": 10,
         "rolling": True, "padded": False},
        # the long-prompt configuration's length on one GPU
        {"name": "prefill_131k", "kind": "prefill", "batch": 1, "length": 131072, "layers": 4, "dtype": "bf16", "pct": 10,
         "rolling": True, "padded": False},
        # interactive generation of one sequence through the Hugging Face cache
        {"name": "hf_decode_1x4k", "kind": "hf_decode", "batch": 1, "context": 4097, "layers": 8, "dtype": "fp16",
         "pct": 10, "padded": False},
        # one long reasoning trace on a server
        {"name": "paged_decode_1x131k", "kind": "paged_decode", "batch": 1, "context": 131072, "ragged": False, "layers": 8,
         "dtype": "bf16", "pct": 10},
        # the benchmark's decode step: batch 64 at context 32768
        {"name": "paged_decode_64x32k", "kind": "paged_decode", "batch": 64, "context": 32768, "ragged": False, "layers": 8,
         "dtype": "fp16", "pct": 10},
        # long-reasoning decode: contexts spread over a factor of sixteen
        {"name": "paged_decode_ragged_24", "kind": "paged_decode", "batch": 24, "context": 65536, "ragged": True, "layers": 8,
         "dtype": "fp16", "pct": 10},
        # the same server with a quantised cache
        {"name": "paged_decode_fp8_32x16k", "kind": "paged_decode", "batch": 32, "context": 16000, "ragged": False,
         "layers": 8, "dtype": "fp8", "pct": 10},
        # hand-off of a prompt to the paged cache, QK-norm model
        {"name": "append_32k", "kind": "append", "batch": 1, "tokens": 32768, "start": 0, "norm": True, "dtype": "bf16"},
        # the new token of every running sequence, once per layer and step
        {"name": "append_64x1", "kind": "append", "batch": 64, "tokens": 1, "start": 511, "norm": False, "dtype": "fp16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, sizes spread over the logarithm of its range (odd ones among them), and the options."""
    kind = rng.choice(["prefill", "prefill", "prefill", "hf_decode", "paged_decode", "paged_decode", "append"])
    pct = rng.choice([5, 10, 10, 10, 20])
    if kind == "prefill":
        length = _log_int(rng, 64, 131071)
        room = max(1, int(min(65536 // length, 8)))          # prompts of a batch hold at most 65536 tokens together
        batch = _log_int(rng, 1, room)
        return {"kind": kind, "batch": batch, "length": length, "layers": 4 if length > 40000 else 8,
                "dtype": rng.choice(["fp16", "bf16"]), "pct": pct if length <= 65536 else min(pct, 10),
                "rolling": rng.random() < 0.5, "padded": batch > 1 and rng.random() < 0.7}
    if kind == "hf_decode":
        context = _log_int(rng, 100, 65536)
        batch = _log_int(rng, 1, max(1, min(16, 262144 // context)))
        return {"kind": kind, "batch": batch, "context": context, "layers": 8, "dtype": rng.choice(["fp16", "bf16"]),
                "pct": pct, "padded": batch > 1 and rng.random() < 0.5}
    if kind == "paged_decode":
        context = _log_int(rng, 200, 131072)
        batch = _log_int(rng, 1, max(1, min(256, 2 ** 21 // context)))
        return {"kind": kind, "batch": batch, "context": context, "ragged": batch > 1 and rng.random() < 0.5, "layers": 8,
                "dtype": rng.choice(["fp16", "bf16", "fp8"]), "pct": pct}
    if rng.random() < 0.5:                                   # a prompt's rows
        tokens = _log_int(rng, 64, 65536)
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, min(8, 65536 // tokens))), "tokens": tokens, "start": 0,
                "norm": rng.random() < 0.5, "dtype": rng.choice(["fp16", "bf16"])}
    return {"kind": kind, "batch": _log_int(rng, 1, 256), "tokens": rng.randint(1, 4), "start": rng.randint(1, 600),
            "norm": rng.random() < 0.5, "dtype": rng.choice(["fp16", "bf16"])}


# ---- sizes -----------------------------------------------------------------------------------------------------------
def _is_anchor(layer):
    return layer in ANCHORS


def _lengths(case):
    """Tokens of every sequence of the case (cached tokens for a decode step)."""
    batch = case["batch"]
    longest = case.get("length") or case.get("context")
    if not (case.get("padded") or case.get("ragged")):
        return [longest] * batch
    g = torch.Generator().manual_seed(SEQUENCES_SEED + batch + longest)
    lo = max(1, longest // (16 if case.get("ragged") else 3))
    lens = torch.randint(lo, longest + 1, (batch,), generator=g).tolist()
    lens[batch // 2] = longest                               # the longest sequence sets the padded length
    return lens


def _head_mapping(layers):
    g = torch.Generator().manual_seed(1234)
    return [list(range(G)) if _is_anchor(i) else torch.randint(0, G, (G,), generator=g).tolist() for i in range(layers)]


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _unit_rms(x):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6)


def _keys(shape, u, gen, dev):
    """Rows of N(0, 1) with 1 % of them moved along the direction `u` that the queries share; unit RMS."""
    k = torch.randn(*shape, generator=gen, device=dev) / D ** 0.5
    hot = torch.rand(*shape[:-1], 1, generator=gen, device=dev) < 0.01
    return _unit_rms(k + 2.5 * u * hot)


def _queries(shape, u, gen, dev):
    return _unit_rms(torch.randn(*shape, generator=gen, device=dev) / D ** 0.5 + 0.5 * u)


def _direction(gen, dev):
    u = torch.randn(D, generator=gen, device=dev)
    return u / u.norm()


def _strategy(case):
    return EfficientKascadeStrategy(list(ANCHORS), "synthetic/model", k=case["pct"], tile_size=TILE,
                                    rolling_prefill=bool(case.get("rolling", True)),
                                    head_mapping=_head_mapping(case["layers"]), register=False)


def _prepare_prefill(case, gen, dev):
    dtype, B, L = DTYPES[case["dtype"]], case["batch"], case["length"]
    layers = []
    for i in range(case["layers"]):
        u = _direction(gen, dev)
        # queries as the projection leaves them (token-major), keys and values as the cache holds them
        q = _queries((B, L, H, D), u, gen, dev).to(dtype).transpose(1, 2)
        k = _keys((B, G, L, D), u, gen, dev).to(dtype)
        v = torch.randn(B, G, L, D, generator=gen, device=dev).to(dtype)
        layers.append((SimpleNamespace(layer_idx=i), q, k, v))
    mask = None
    if case["padded"]:
        first = torch.tensor([L - n for n in _lengths(case)], device=dev)
        keep = torch.arange(L, device=dev)[None, :] >= first[:, None]                     # left padding
        causal = torch.ones(L, L, dtype=torch.bool, device=dev).tril()
        mask = causal[None, None] & keep[:, None, None, :]
    return {"kind": "prefill", "strategy": _strategy(case), "layers": layers, "mask": mask}


def _prepare_hf_decode(case, gen, dev):
    dtype, B, L = DTYPES[case["dtype"]], case["batch"], case["context"]
    layers = []
    for i in range(case["layers"]):
        u = _direction(gen, dev)
        q = _queries((B, H, 1, D), u, gen, dev).to(dtype)
        k = _keys((B, G, L, D), u, gen, dev).to(dtype)
        v = torch.randn(B, G, L, D, generator=gen, device=dev).to(dtype)
        layers.append((SimpleNamespace(layer_idx=i), q, k, v))
    mask = None
    if case["padded"]:
        first = torch.tensor([L - n for n in _lengths(case)], device=dev)
        mask = (torch.arange(L, device=dev)[None, :] >= first[:, None])[:, None, None, :]
    return {"kind": "hf_decode", "strategy": _strategy(case), "layers": layers, "mask": mask}


def _prepare_paged_decode(case, gen, dev):
    B, lens = case["batch"], _lengths(case)
    fp8 = case["dtype"] == "fp8"
    dtype = torch.float16 if fp8 else DTYPES[case["dtype"]]
    per_seq = [-(-n // PAGE) for n in lens]
    n_pages = sum(per_seq)
    table = torch.zeros(B, max(per_seq), dtype=torch.int32)
    order = torch.randperm(n_pages, generator=torch.Generator().manual_seed(SEQUENCES_SEED)).to(torch.int32)
    at = 0
    for b, n in enumerate(per_seq):
        table[b, :n] = order[at:at + n]
        at += n
    # two layer caches in turn: those of all layers would not fit beside each other
    caches, directions = [], []
    for _ in range(2):
        u = _direction(gen, dev)
        shape = (n_pages, PAGE, G, D)
        store = torch.float8_e4m3fn if fp8 else dtype
        k, v = torch.empty(shape, dtype=store, device=dev), torch.empty(shape, dtype=store, device=dev)
        ks = vs = None
        if fp8:                                              # one scale per (page, KV head)
            ks, vs = (torch.empty(n_pages, G, dtype=torch.float32, device=dev) for _ in range(2))
        for s in range(0, n_pages, 16384):
            e = min(n_pages, s + 16384)
            new_k = _keys((e - s, PAGE, G, D), u, gen, dev)
            new_v = torch.randn(e - s, PAGE, G, D, generator=gen, device=dev)
            for new, cache, scale in ((new_k, k, ks), (new_v, v, vs)):
                if fp8:
                    scale[s:e] = new.abs().amax(dim=(1, 3)) / 448.0
                    new = new / scale[s:e, None, :, None]
                cache[s:e] = new.to(store)
        caches.append((k, v, ks, vs))
        directions.append(u)
    queries = [_queries((B, H, D), directions[i & 1], gen, dev).to(dtype) for i in range(case["layers"])]
    return {"kind": "paged_decode", "strategy": _strategy(case), "queries": queries, "caches": caches, "table": table.to(dev),
            "seq_lens": torch.tensor(lens, dtype=torch.int32, device=dev), "max_len": max(lens),
            "mean_len": sum(lens) / len(lens) if case["ragged"] else None}


def _prepare_append(case, gen, dev):
    dtype, B, T, start = DTYPES[case["dtype"]], case["batch"], case["tokens"], case["start"]
    pages = -(-(start + T) // PAGE)
    order = torch.randperm(B * pages, generator=torch.Generator().manual_seed(SEQUENCES_SEED)).to(torch.int32)
    # q, k, v as the fused projection leaves them: slices of one row per token
    qkv = torch.randn(B, T, H + 2 * G, D, generator=gen, device=dev).to(dtype)
    gains = [(1 + 0.1 * torch.randn(D, generator=gen, device=dev)).to(dtype) for _ in range(2)] if case["norm"] else [None, None]
    cache = torch.randn(2, B * pages, PAGE, G, D, generator=gen, device=dev, dtype=dtype)
    inv_freq = 500000.0 ** (-torch.arange(0, D, 2, dtype=torch.float32, device=dev) / D)
    return {"kind": "append", "q": qkv[:, :, :H], "k": qkv[:, :, H:H + G], "v": qkv[:, :, H + G:], "k_cache": cache[0],
            "v_cache": cache[1], "table": order.view(B, pages).to(dev), "gains": gains, "inv_freq": inv_freq,
            "start": torch.full((B,), start, dtype=torch.int32, device=dev)}


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    make = {"prefill": _prepare_prefill, "hf_decode": _prepare_hf_decode, "paged_decode": _prepare_paged_decode,
            "append": _prepare_append}[case["kind"]]
    return make(case, gen, dev)


# ---- one pass --------------------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind in ("prefill", "hf_decode"):
        strategy, mask = state["strategy"], state["mask"]
        if mask is not None:
            mask = mask[:]                                   # every forward of a model brings a mask of its own
        return [strategy.attention_forward(module, q, k, v, mask, SCALE)[0] for module, q, k, v in state["layers"]]
    if kind == "paged_decode":
        strategy, out = state["strategy"], []
        for layer, q in enumerate(state["queries"]):
            k, v, k_scale, v_scale = state["caches"][layer & 1]
            out.append(strategy.paged_decode_forward(layer, q, k, v, state["table"], state["seq_lens"], SCALE,
                                                     state["max_len"], k_scale, v_scale, mean_seq_len=state["mean_len"]))
        return out
    q_out = EfficientKascadeStrategy.append_kv(state["k"], state["v"], state["k_cache"], state["v_cache"], state["table"],
                                               state["start"], query=state["q"], q_norm_weight=state["gains"][0],
                                               k_norm_weight=state["gains"][1], inv_freq=state["inv_freq"])
    return q_out, state["k_cache"], state["v_cache"]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _prefill_work(case):
    flops = nbytes = 0.0
    for n in _lengths(case):
        qk = 2.0 * H * D * n * n / 2                         # one causal Q.K^T
        if n <= 128:
            sparse = 0.0
        else:
            budget = topk_budget(case["pct"], n, TILE)
            keys = 0
            for t in range(-(-n // TILE)):
                start = t * TILE
                k = min(budget, max(128, int(case["pct"] * start // 100))) if case["rolling"] else budget
                keys += min(k, start) + TILE
            sparse = 4.0 * TILE * H * D * keys
        for i in range(case["layers"]):
            # the scores of a tile need every row's normaliser first: an anchor's Q.K^T runs twice
            flops += 2 * qk if n <= 128 else (3 * qk if i == 0 else 2 * qk + sparse if _is_anchor(i) else sparse)
            nbytes += n * D * (2 * H + 2 * G) * 2.0
    return {"bytes": nbytes, "flops": flops}


def _decode_work(case):
    row = D * (1 if case["dtype"] == "fp8" else 2)
    flops = nbytes = 0.0
    for n in _lengths(case):
        k = n if n <= 128 else topk_budget(case["pct"], n, TILE)
        for i in range(case["layers"]):
            dense = G * n * row * (2 if i == 0 or n <= 128 else 1)
            sparse = G * k * (2 * row + 4)
            nbytes += (dense if i == 0 or n <= 128 else dense + sparse if _is_anchor(i) else sparse) + 2 * H * D * 2
            flops += 2.0 * H * D * (2 * n if i == 0 or n <= 128 else n + 2 * k if _is_anchor(i) else 2 * k)
    return {"bytes": nbytes, "flops": flops}


def work(case):
    if case["kind"] == "prefill":
        return _prefill_work(case)
    if case["kind"] == "append":
        rows = case["batch"] * case["tokens"] * (H + 2 * G)
        return {"bytes": rows * D * 2 * 2.0, "flops": rows * D * 4.0}
    return _decode_work(case)


def tolerance(case):
    """Outputs are rounded to fp16 (2^-11) or bf16 (2^-8), and so are the probabilities before P.V.  Where keys are
    selected, two whose scores are equal to fp32 rounding may change places, which moves a whole row."""
    if case["kind"] == "append":
        # rotations round twice per element in the storage type, sin and cos may differ by one unit in its last place
        return {"rel": 1e-3 if case["dtype"] == "fp16" else 8e-3, "max": 2e-2 if case["dtype"] == "fp16" else 1e-1}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 4e-3, "max": 0.9}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------
EXACT_MAX_PROMPT = 8192      # longer prompts: the [heads, L, L] scores in 64 bits would take too long and too much memory


def _select(pooled, k):
    """Positions of the k largest of the last dimension (the lowest ones of equal scores), ascending."""
    order = torch.sort(pooled, dim=-1, descending=True, stable=True).indices[..., :k]
    return torch.sort(order, dim=-1).values


def _exact_sequence(case, layers, heads, padded):
    """Outputs [n, H, D] of every layer for one prompt; layers: q [H, n, D], k / v [G, n, D] in 64 bits."""
    outs, chosen = [], None
    n = layers[0][0].shape[1]
    dense_only = n <= 128 and not padded
    tiles = -(-n // TILE)
    budget = max(0, min(max(128, int(case["pct"] / 100 * n)), n) - TILE)
    rolling = case["rolling"] and n > 128
    budgets = [min(budget, max(128, int(case["pct"] * t * TILE / 100))) if rolling else budget for t in range(tiles)]
    for i, (q, k, v) in enumerate(layers):
        dev = q.device
        out = torch.zeros(H, n, D, dtype=torch.float64, device=dev)
        if dense_only or _is_anchor(i):
            chosen = [] if not dense_only else None
            causal = torch.ones(n, n, dtype=torch.bool, device=dev).tril()
            for g in range(G):
                s = (q[g * 4:g * 4 + 4] @ k[g].T) * SCALE
                p = torch.softmax(s.masked_fill(~causal, -math.inf), dim=-1)
                del s
                if dense_only or i == 0:
                    out[g * 4:g * 4 + 4] = p @ v[g]
                if not dense_only:
                    chosen.append([_select(p[:, t * TILE:(t + 1) * TILE, :t * TILE].sum((0, 1)), min(budgets[t], t * TILE))
                                   for t in range(tiles)])
                del p
        if not dense_only and i > 0:
            for g in range(G):
                rows = chosen[g if _is_anchor(i) else heads[i][g]]
                for t in range(tiles):
                    a, e = t * TILE, min((t + 1) * TILE, n)
                    keys = torch.cat([rows[t], torch.arange(a, e, device=dev)])
                    s = (q[g * 4:g * 4 + 4, a:e] @ k[g, keys].T) * SCALE
                    later = keys[None, :] > torch.arange(a, e, device=dev)[:, None]
                    out[g * 4:g * 4 + 4, a:e] = torch.softmax(s.masked_fill(later, -math.inf), dim=-1) @ v[g, keys]
        outs.append(out.transpose(0, 1))
    return outs


def _exact_prefill(case, state):
    if case["length"] > EXACT_MAX_PROMPT:
        return None
    L, lens = case["length"], _lengths(case)
    heads = _head_mapping(case["layers"])
    outs = [torch.zeros(case["batch"], L, H, D, dtype=torch.float64, device=state["layers"][0][1].device)
            for _ in range(case["layers"])]
    padded = any(n != L for n in lens)                       # a batch in which nothing is padded runs as any other
    for b, n in enumerate(lens):
        layers = [[x[b, :, L - n:].double() for x in (q, k, v)] for _, q, k, v in state["layers"]]
        for out, one in zip(outs, _exact_sequence(case, layers, heads, padded)):
            out[b, L - n:] = one
    return outs


def _exact_token(case, layers, n, longest):
    """Outputs [H, D] of every layer for one new token over n cached ones; layers: q [H, D], k / v [G, n, D]."""
    outs, chosen = [], None
    heads = _head_mapping(case["layers"])
    budget = n if n <= 128 else min(max(128, int(case["pct"] / 100 * n)), n) - TILE
    for i, (q, kv) in enumerate(layers):
        k, v = kv()
        q = q.view(G, 4, D)
        if longest <= 128 or _is_anchor(i):
            p = torch.softmax((q @ k.transpose(1, 2)) * SCALE, dim=-1)
            chosen = _select(p.sum(1), budget) if longest > 128 else None
        if longest <= 128 or i == 0:
            out = p @ v
        else:
            rows = chosen if _is_anchor(i) else chosen[heads[i]]
            rows = rows[:, :, None].expand(-1, -1, D)
            out = torch.softmax((q @ k.gather(1, rows).transpose(1, 2)) * SCALE, dim=-1) @ v.gather(1, rows)
        outs.append(out.reshape(H, D))
    return outs


def _exact_hf_decode(case, state):
    L, per_sequence = case["context"], []
    lens = _lengths(case)
    for b, n in enumerate(lens):
        layers = [(q[b, :, 0].double(), lambda k=k, v=v: (k[b, :, L - n:].double(), v[b, :, L - n:].double()))
                  for _, q, k, v in state["layers"]]
        per_sequence.append(_exact_token(case, layers, n, max(lens)))
    return [torch.stack(rows).unsqueeze(1) for rows in zip(*per_sequence)]


def _exact_paged_decode(case, state):
    per_sequence = []
    lens = _lengths(case)
    for b, n in enumerate(lens):
        pages = state["table"][b, :-(-n // PAGE)].long()

        def rows(cache, scale):
            x = cache[pages].double()
            if scale is not None:
                x = x * scale[pages].double()[:, None, :, None]
            return x.reshape(-1, G, D)[:n].transpose(0, 1)

        layers = [(q[b].double(), lambda c=state["caches"][i & 1]: (rows(c[0], c[2]), rows(c[1], c[3])))
                  for i, q in enumerate(state["queries"])]
        per_sequence.append(_exact_token(case, layers, n, max(lens)))
    return [torch.stack(rows) for rows in zip(*per_sequence)]


def _exact_append(case, state):
    B, T, start = case["batch"], case["tokens"], case["start"]
    pos = start + torch.arange(T, device=state["q"].device)
    angle = pos.double()[:, None] * state["inv_freq"].double()
    cos, sin = (f(torch.cat([angle, angle], -1))[None, :, None] for f in (torch.cos, torch.sin))

    def turned(x, gain):
        x = x.double()
        if gain is not None:
            x = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * gain.double()
        return x * cos + torch.cat([-x[..., D // 2:], x[..., :D // 2]], -1) * sin

    page, slot = state["table"].long()[:, pos // PAGE], (pos % PAGE).expand(B, T)
    caches = []
    for cache, new in ((state["k_cache"], turned(state["k"], state["gains"][1])), (state["v_cache"], state["v"].double())):
        cache = cache.double()
        cache[page, slot] = new
        caches.append(cache)
    return turned(state["q"], state["gains"][0]), caches[0], caches[1]


def exact(case, seed):
    """What `run` returns for these inputs, in 64 bits and without the library's kernels; None for a case that would take
    too long.  Keys whose scores differ by less than the library's rounding may be selected differently."""
    state = prepare(case, seed)
    return {"prefill": _exact_prefill, "hf_decode": _exact_hf_decode, "paged_decode": _exact_paged_decode,
            "append": _exact_append}[case["kind"]](case, state)
