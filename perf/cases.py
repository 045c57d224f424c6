"""Performance cases of the attention library: what an engine has it do, through the public entry points.

Every case is one call site of the engine with the buffers such a program keeps (caches, workspaces, outputs, recorded
steps) made in ``prepare`` and the per-step calls in ``run``.  Seven kinds:

  decode   one dense sequence, a decode step (1 token) or an MTP-verify step (2 tokens): ``mla_decode``
  serve    a batch of paged sequences, one serving step: ``rope_kv_append`` of the new rows, then ``mla_decode``
  layer    one layer's step with host buffers: ``MlaDecodeLayer.step`` (recorded graph, input and output page-locked)
  sparse   a decode or MTP-verify step beyond top_k positions, as the engine issues it: KV-append (f16 or Q8 rows),
           ``gs_idx_pool``, ``gs_idx_score``, ``gs_idx_select``, ``gs_mla_attn`` over the selected rows
  list     ``gs_mla_attn`` of a prefill chunk (up to 256 queries, one split) over given position lists, f16 or Q8 cache
  index    the indexer of a prefill chunk: ``gs_idx_pool``, ``gs_idx_score``, ``gs_idx_select``
  prefill  RoPE of the new Q and K rows, then ``prefill_attn``, with or without prior context
"""
import importlib
import math
import random
from types import SimpleNamespace

import torch

pkg = importlib.import_module("glm-ssd_b200")

D_V, D_ROPE, PAGE = 512, 64, 64
LATENT = 512                              # row width of the engine's own latent cache
IDX_HEADS, IDX_DIM, KPOOL, TOP_K = 32, 128, 4, 512
SEL_STRIDE = (TOP_K + 1) * KPOOL          # 2052 listed positions at most
SCALE = 1.0 / 16.0
SPLITS = {1: 16, 2: 4}                    # the engine's split counts for decode and MTP verify; a chunk has one


def listed():
    return [
        # the smallest call: one token over a 4K context; launches and host work count
        {"name": "decode_4k", "kind": "decode", "rows": 4096, "tokens": 1, "heads": 20, "d_qk": 576},
        # the headline call: MTP verify at 32K
        {"name": "verify_32k", "kind": "decode", "rows": 32768, "tokens": 2, "heads": 20, "d_qk": 576},
        # a long context on one GPU
        {"name": "decode_128k", "kind": "decode", "rows": 131072, "tokens": 1, "heads": 20, "d_qk": 576},
        # batched serving: 64 long sequences over a shuffled page pool
        {"name": "serve_64_long", "kind": "serve", "seqs": 64, "min_ctx": 1024, "max_ctx": 65536, "tokens": 1, "heads": 20},
        # a handful of young, ragged sequences with a draft token each
        {"name": "serve_7_ragged", "kind": "serve", "seqs": 7, "min_ctx": 2, "max_ctx": 3000, "tokens": 2, "heads": 20},
        # the call-site mirror end to end: host rows in, host output back
        {"name": "layer_32k", "kind": "layer", "rows": 32768, "tokens": 2, "heads": 20},
        # the engine's decode step once the context is longer than top_k, 64 heads
        {"name": "sparse_decode_32k", "kind": "sparse", "rows": 32768, "tokens": 1, "heads": 64, "cache": "f16"},
        # the same with a draft token and the Q8 cache at the engine's default-size long context
        {"name": "sparse_verify_64k_q8", "kind": "sparse", "rows": 65536, "tokens": 2, "heads": 64, "cache": "q8"},
        # attention of one 256-query prefill block over its selected rows
        {"name": "list_chunk_256", "kind": "list", "rows": 32768, "tokens": 256, "heads": 64, "cache": "f16"},
        # the selection for such a block
        {"name": "index_chunk_256", "kind": "index", "rows": 32768, "tokens": 256},
        # a full prefill pass, the largest arithmetic
        {"name": "prefill_8k", "kind": "prefill", "tokens": 8192, "context": 0, "heads": 20, "f16_out": False},
        # the ragged last chunk of a long prompt
        {"name": "prefill_tail", "kind": "prefill", "tokens": 1000, "context": 7168, "heads": 20, "f16_out": True},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "serve", "layer", "sparse", "list", "index", "prefill"])
    if kind == "decode":
        return {"kind": kind, "rows": _log(rng, 64, 131072), "tokens": rng.choice([1, 2]), "heads": rng.choice([16, 20, 32, 64]),
                "d_qk": rng.choice([512, 576, 576])}
    if kind == "serve":
        seqs = _log(rng, 2, 64)
        top = _log(rng, 256, 65536)
        return {"kind": kind, "seqs": seqs, "min_ctx": max(2, top // rng.choice([2, 16, 64])), "max_ctx": top, "tokens": rng.choice([1, 2]),
                "heads": rng.choice([16, 20])}
    if kind == "layer":
        return {"kind": kind, "rows": _log(rng, 256, 131072), "tokens": rng.choice([1, 2]), "heads": rng.choice([16, 20])}
    if kind == "sparse":
        return {"kind": kind, "rows": _log(rng, 2304, 131072), "tokens": rng.choice([1, 2]), "heads": rng.choice([16, 32, 64]),
                "cache": rng.choice(["f16", "q8"])}
    if kind == "list":
        return {"kind": kind, "rows": _log(rng, 2304, 131072), "tokens": _log(rng, 16, 256), "heads": rng.choice([16, 32, 64]),
                "cache": rng.choice(["f16", "f16", "q8"])}
    if kind == "index":
        return {"kind": kind, "rows": _log(rng, 2304, 65536), "tokens": _log(rng, 16, 256)}
    tokens = _log(rng, 32, 8192)
    room = max(0, (8192 * 8192 // 2) // tokens - tokens // 2)  # no more (query, key) pairs than the full 8192-token pass
    return {"kind": kind, "tokens": tokens, "context": min(room, rng.choice([0, _log(rng, 64, 32768)])), "heads": rng.choice([16, 20]),
            "f16_out": rng.choice([False, True])}


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, shape, sigma=1.0):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * sigma


def _randn_f16(g, shape, sigma=1.0):
    out = torch.empty(shape, dtype=torch.float16, device="cuda")
    flat = out.view(-1)
    for i in range(0, flat.numel(), 1 << 28):
        part = flat[i:i + (1 << 28)]
        part.copy_(torch.randn(part.numel(), generator=g, device="cuda", dtype=torch.float32).mul_(sigma))
    return out


def _contexts(case):
    """The batch's context lengths, uniform over the case's range and the same for every seed."""
    r = random.Random(case["seqs"] * 1000003 + case["max_ctx"])
    return [r.randint(case["min_ctx"], case["max_ctx"]) for _ in range(case["seqs"])]


def _first_position(case):
    """Position of the first new row: the last pool of kpool positions completes with the last new row."""
    return max(SEL_STRIDE, case["rows"] // KPOOL * KPOOL) - case["tokens"]


def _latent_cache(g, rows, kind):
    """The engine's latent cache: f16 rows, or int8 rows with one f16 scale per 32 values."""
    c = _randn_f16(g, (rows, LATENT), 0.5)
    if kind == "f16":
        return c, None
    q8 = torch.empty((rows, LATENT), dtype=torch.int8, device="cuda")
    sc = torch.empty((rows, LATENT // 32), dtype=torch.float16, device="cuda")
    pkg.quant_q8_rows(c.float(), q8, sc, rows * LATENT)
    return q8, sc


def _indexer(g, p0, tokens, ctx):
    """What the indexer keeps (pooled keys, rings) and gets (keys, gates, queries, weights of the new positions)."""
    s = SimpleNamespace()
    s.pools = ctx // KPOOL + 1
    s.kc, s.gc = _randn(g, (tokens, IDX_DIM)), _randn(g, (tokens, IDX_DIM))
    s.rk, s.rg = _randn(g, (KPOOL, IDX_DIM)), _randn(g, (KPOOL, IDX_DIM))
    s.ape = _randn(g, (KPOOL, IDX_DIM), 0.3)
    s.pooled = _randn(g, (s.pools, IDX_DIM), 0.6)
    s.qi, s.wi = _randn(g, (tokens, IDX_HEADS, IDX_DIM)), _randn(g, (tokens, IDX_HEADS))
    s.score = torch.zeros((tokens, s.pools), dtype=torch.float32, device="cuda")
    s.sel = torch.zeros((tokens, SEL_STRIDE), dtype=torch.int32, device="cuda")
    s.cnt = torch.zeros(tokens, dtype=torch.int32, device="cuda")
    # the three calls as the engine issues them: raw pointers and sizes, an error code back
    s.pool_args = [t.data_ptr() for t in (s.kc, s.gc, s.rk, s.rg, s.ape, s.pooled)] + [p0, tokens, IDX_DIM, KPOOL]
    s.score_args = [t.data_ptr() for t in (s.qi, s.wi, s.pooled, s.score)] + [s.pools, p0, tokens, KPOOL, IDX_HEADS, IDX_DIM,
                                                                             1.0 / math.sqrt(IDX_DIM)]
    s.select_args = [s.score.data_ptr(), s.pools, p0, tokens, KPOOL, TOP_K, s.sel.data_ptr(), SEL_STRIDE, s.cnt.data_ptr()]
    return s


def _prepare_decode(case, seed):
    g, s = _gen(seed), SimpleNamespace()
    n, T, H, d = case["rows"], case["tokens"], case["heads"], case["d_qk"]
    s.rows = n
    s.q = _randn_f16(g, (1, T, H, d))
    s.cache = _randn_f16(g, (n, d), 0.5)
    s.lens = torch.tensor([n], dtype=torch.int32, device="cuda")
    s.out = torch.empty((1, T, H, D_V), dtype=torch.float32, device="cuda")
    s.workspace = pkg.new_workspace(1, T, H, D_V)
    return s


def _run_decode(s):
    return pkg.mla_decode(s.q, s.cache, s.lens, out=s.out, workspace=s.workspace, max_seq_len=s.rows)


def _prepare_serve(case, seed):
    g, s = _gen(seed), SimpleNamespace()
    n, T, H = case["seqs"], case["tokens"], case["heads"]
    ctx = _contexts(case)
    pages = [-(-c // PAGE) for c in ctx]
    pool_pages = sum(pages) + 1
    s.pool = _randn_f16(g, (pool_pages * PAGE, 576), 0.5)
    order = torch.randperm(pool_pages, generator=g, device="cuda").to(torch.int32)
    s.pages = torch.zeros((n, max(pages)), dtype=torch.int32, device="cuda")
    at = 0
    for b, k in enumerate(pages):
        s.pages[b, :k] = order[at:at + k]
        at += k
    s.longest = max(ctx)
    s.lens = torch.tensor(ctx, dtype=torch.int32, device="cuda")
    s.pos = s.lens - T
    s.kv = _randn(g, (n, T, 576), 0.5)
    s.q = _randn_f16(g, (n, T, H, 576))
    s.out = torch.empty((n, T, H, D_V), dtype=torch.float32, device="cuda")
    s.workspace = pkg.new_workspace(n, T, H, D_V)
    return s


def _run_serve(s):
    pkg.rope_kv_append(s.kv, s.pool, s.pos, page_table=s.pages)
    pkg.mla_decode(s.q, s.pool, s.lens, page_table=s.pages, out=s.out, workspace=s.workspace, max_seq_len=s.longest)
    return s.out, s.pool


def _prepare_layer(case, seed):
    g, s = _gen(seed), SimpleNamespace()
    n, T, H = case["rows"], case["tokens"], case["heads"]
    s.layer = pkg.MlaDecodeLayer(ctx=n, H=H, T_max=T, use_graph=True)
    s.layer.cache.copy_(_randn_f16(g, (n, 576), 0.5))
    s.q = _randn_f16(g, (T, H, 576)).cpu().pin_memory()
    s.kv = _randn(g, (T, 576), 0.5).cpu().pin_memory()
    s.pos = n - T
    torch.cuda.synchronize()
    _run_layer(s)  # the step is recorded on its first use, once in the life of a layer
    return s


def _run_layer(s):
    s.layer.pos = s.pos
    return s.layer.step(s.q, s.kv), s.layer.cache


def _prepare_sparse(case, seed):
    g = _gen(seed)
    T, H = case["tokens"], case["heads"]
    p0 = _first_position(case)
    s = _indexer(g, p0, T, p0 + T)
    s.heads = H
    s.tokens, s.new_values = T, T * LATENT
    s.cache, s.scales = _latent_cache(g, p0 + T, case["cache"])
    s.new_rows = s.cache[p0:]
    s.new_scales = None if s.scales is None else s.scales[p0:]
    s.kv = _randn(g, (T, LATENT), 0.5)
    s.q = _randn(g, (T, H, LATENT))
    s.out = torch.empty((T, H, LATENT), dtype=torch.float32, device="cuda")
    s.part = torch.zeros(T * H * SPLITS[T] * (LATENT + 2), dtype=torch.float32, device="cuda")
    return s


def _select(s):
    lib, stream = pkg._lib.load(), torch.cuda.current_stream().cuda_stream
    pkg._lib.check(lib.gs_idx_pool(*s.pool_args, stream), "gs_idx_pool")
    pkg._lib.check(lib.gs_idx_score(*s.score_args, stream), "gs_idx_score")
    pkg._lib.check(lib.gs_idx_select(*s.select_args, stream), "gs_idx_select")


def _run_sparse(s):
    if s.scales is None:
        pkg.f32_to_f16(s.kv, s.new_rows, s.new_values)
    else:
        pkg.quant_q8_rows(s.kv, s.new_rows, s.new_scales, s.new_values)
    _select(s)
    pkg.mla_attn(s.q, s.cache, s.scales, s.sel, SEL_STRIDE, s.cnt, SCALE, s.out, s.part, s.tokens, s.heads, LATENT, SPLITS[s.tokens])
    return s.out, s.cache, s.scales, s.sel, s.cnt, s.score, s.pooled


def _prepare_list(case, seed):
    g, s = _gen(seed), SimpleNamespace()
    s.tokens, s.heads = case["tokens"], case["heads"]
    ctx = case["rows"]
    s.cache, s.scales = _latent_cache(g, ctx, case["cache"])
    s.q = _randn(g, (s.tokens, s.heads, LATENT))
    # lists as gs_idx_select makes them: top_k pools of kpool consecutive positions in ascending order, then the tail
    pools = (ctx - s.tokens) // KPOOL
    picked = torch.rand((s.tokens, pools), generator=g, device="cuda").topk(TOP_K, dim=1).indices.sort(dim=1).values
    rows = picked.unsqueeze(2) * KPOOL + torch.arange(KPOOL, device="cuda")
    s.sel = torch.zeros((s.tokens, SEL_STRIDE), dtype=torch.int32, device="cuda")
    s.sel[:, :TOP_K * KPOOL] = rows.reshape(s.tokens, -1)
    t = torch.arange(s.tokens, device="cuda")
    first_tail = (ctx - s.tokens + t) // KPOOL * KPOOL
    s.sel[:, TOP_K * KPOOL:] = torch.minimum(first_tail[:, None] + torch.arange(KPOOL, device="cuda"), torch.tensor(ctx - 1, device="cuda"))
    s.cnt = (TOP_K * KPOOL + (ctx - s.tokens + t) % KPOOL).to(torch.int32)
    s.out = torch.empty((s.tokens, s.heads, LATENT), dtype=torch.float32, device="cuda")
    return s


def _run_list(s):
    pkg.mla_attn(s.q, s.cache, s.scales, s.sel, SEL_STRIDE, s.cnt, SCALE, s.out, None, s.tokens, s.heads, LATENT, 1)
    return s.out


def _prepare_index(case, seed):
    p0 = _first_position(case)
    return _indexer(_gen(seed), p0, case["tokens"], p0 + case["tokens"])


def _run_index(s):
    _select(s)
    return s.sel, s.cnt, s.score, s.pooled, s.rk, s.rg


def _prepare_prefill(case, seed):
    g, s = _gen(seed), SimpleNamespace()
    S, p0, H = case["tokens"], case["context"], case["heads"]
    s.p0 = p0
    s.q = _randn_f16(g, (S, H, 256))
    s.k, s.v = _randn_f16(g, (p0 + S, H, 256)), _randn_f16(g, (p0 + S, H, 256))
    s.new_k = s.k[p0:]
    s.out = torch.empty((S, H, 256), dtype=torch.float16 if case["f16_out"] else torch.float32, device="cuda")
    return s


def _run_prefill(s):
    pkg.rope_f16_inplace(s.q, pos0=s.p0)
    pkg.rope_f16_inplace(s.new_k, pos0=s.p0)
    return pkg.prefill_attn(s.q, s.k, s.v, p0=s.p0, out=s.out), s.q, s.new_k


_KINDS = {
    "decode": (_prepare_decode, _run_decode), "serve": (_prepare_serve, _run_serve), "layer": (_prepare_layer, _run_layer),
    "sparse": (_prepare_sparse, _run_sparse), "list": (_prepare_list, _run_list), "index": (_prepare_index, _run_index),
    "prefill": (_prepare_prefill, _run_prefill),
}


def prepare(case, seed):
    make, run_kind = _KINDS[case["kind"]]
    return run_kind, make(case, seed)


def run(state):
    run_kind, s = state
    return run_kind(s)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

def _index_work(p0, T):
    pools = (p0 + T) // KPOOL
    return (4 * (pools * IDX_DIM + T * IDX_HEADS * (IDX_DIM + 1) + T * pools + T * SEL_STRIDE + 2 * T * IDX_DIM),
            2 * T * pools * IDX_HEADS * (IDX_DIM + 1))


def _list_work(case, T, ctx, listed_rows):
    H = case["heads"]
    unique = ctx * (1.0 - (1.0 - min(1.0, listed_rows / ctx)) ** T)
    row_bytes = 2 * LATENT if case["cache"] == "f16" else LATENT + LATENT // 16
    return unique * row_bytes + 2 * 4 * T * H * LATENT + 4 * T * listed_rows, 4 * T * H * listed_rows * LATENT


def work(case):
    kind = case["kind"]
    T = case["tokens"]
    if kind in ("decode", "layer"):
        n, H, d = case["rows"], case["heads"], case.get("d_qk", 576)
        return {"bytes": 2 * n * d + T * H * (2 * d + 4 * D_V), "flops": 2 * T * H * n * (d + D_V)}
    if kind == "serve":
        n = sum(_contexts(case))
        H, b = case["heads"], case["seqs"]
        return {"bytes": 2 * n * 576 + b * T * (H * (2 * 576 + 4 * D_V) + 6 * 576), "flops": 2 * T * H * n * (576 + D_V)}
    if kind == "sparse":
        p0 = _first_position(case)
        ib, fi = _index_work(p0, T)
        lb, fl = _list_work(case, T, p0 + T, SEL_STRIDE)
        return {"bytes": ib + lb, "flops": fi + fl}
    if kind == "list":
        b, f = _list_work(case, T, case["rows"], SEL_STRIDE)
        return {"bytes": b, "flops": f}
    if kind == "index":
        b, f = _index_work(_first_position(case), T)
        return {"bytes": b, "flops": f}
    p0, H = case["context"], case["heads"]
    out = 2 if case["f16_out"] else 4
    pairs = T * p0 + T * (T + 1) // 2
    # q, k, v read once; the rotated columns of q and the new keys, and the result, written once
    return {"bytes": H * (512 * (T + 2 * (p0 + T)) + 2 * 2 * D_ROPE * T + 256 * out * T), "flops": 4 * 256 * H * pairs}


def tolerance(case):
    if case["kind"] == "index":
        # 32-bit sums; a score that rounds the other way at the k-th largest swaps one pool of a query's list
        return {"rel": 1e-5, "differ": 0.01}
    # f16 rows and probabilities, 32-bit accumulation
    return {"rel": 1e-3, "differ": 0.01} if case["kind"] == "sparse" else {"rel": 1e-3}
