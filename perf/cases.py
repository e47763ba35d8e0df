"""The work users have this library do, as cases that can be timed: decode-step attention over sealed pages, the prompt
batches before it, and the sealing that fills the pages, through the Python store and through the C ABIs that
llama.cpp-side callers link.

A case is a dict of plain values; "op" says which entry points it goes through:

  decode         SealedKvLayer.attention: one query token per sequence over its sealed pages and its unsealed tail
  shared         the same over sequences forked from one prompt, whose sealed pages are stored once
  ingest         cf_b200_seal_pages_async over whole prompts, then the first decode step over what was sealed
  prefill        cf_device_kv_attention_async: the query tokens of a prompt batch over everything stored so far
  server_decode  cf_llama_server_execute_batch_async: one token for every slot of a server
  server_prompt  a request's life in a server: slot_create, append_layer of the prompt, execute_batch, slot_reset
  adapter        cf_llama_kv_attention over the adapter's default pages (int4 / int8, scales per channel and token)
  adapter_prompt cf_llama_kv_clear, then a prompt in batches: cf_llama_kv_append per kv head, cf_llama_kv_attention

K/V codes are discretised Laplace (scale `spread`, in code units) or two-sided geometric (p = `spread`), as the library's
own workloads draw them; queries are N(0, 1). Every state owns its output buffers.
"""
import ctypes as C
import math

import numpy as np
import torch

from chromofold_b200 import _native as N
from chromofold_b200.cache import SealedKvLayer
from chromofold_b200.workloads import CODERS, build_sealed_layer, geometric_codes, laplace_codes, tiles_from_codes

DEVICE = "cuda:0"
PAGE = 16                 # tokens of a sealed page of the Python store
LARGEST_TOKENS = 1 << 20  # cached tokens of the largest listed case (8 x 131072)


# ---- the cases -------------------------------------------------------------------------------------------------------
def listed():
    decode = dict(op="decode", head_dim=128, block=64, dist="laplace", spread=12.0, tails=True, queries="f16", window=0)
    return [
        # one chat on one GPU, no grouped heads: nothing to batch, the latency of a token counts
        dict(decode, name="decode_one", coder="rans", q_heads=8, kv_heads=8, seqs=1, ctx_lo=4096, ctx_hi=4096),
        # the decode step of a busy server, mixed context lengths: the benchmark's headline shape and default coder
        dict(decode, name="decode_batch", coder="rans4", q_heads=32, kv_heads=8, seqs=64, ctx_lo=2048, ctx_hi=32768,
             tails=False),
        # a batch at one context length with the one-step-per-code Huffman pages and skewed codes (the coder sweep)
        dict(decode, name="decode_huffman", coder="huffman", q_heads=32, kv_heads=8, seqs=32, ctx_lo=8192, ctx_hi=8192,
             dist="geometric", spread=0.2),
        # long documents on a model with 64 query heads: the largest case
        dict(decode, name="decode_long", coder="rans", q_heads=64, kv_heads=8, seqs=8, ctx_lo=131072, ctx_hi=131072,
             tails=False),
        # a small model, 14 query heads on 2 kv heads of 64 channels, ragged contexts, fp32 queries
        dict(decode, name="decode_dim64", coder="huffman4", q_heads=14, kv_heads=2, head_dim=64, seqs=8, ctx_lo=700,
             ctx_hi=9000, queries="f32"),
        # many requests over one system prompt: the prompt's pages are shared, each request owns a short suffix
        dict(op="shared", name="shared_prompt", coder="rans4", q_heads=32, kv_heads=8, seqs=256, prefix=16384, suffix=512),
        # a batch of prompts that arrives whole: 64 prompts of 512 tokens are sealed, then every one decodes a token
        dict(op="ingest", name="ingest_prompts", coder="rans4", q_heads=32, kv_heads=8, head_dim=128, block=64, seqs=64,
             tokens=512),
        # the last batch of a long prompt: 500 query tokens after 16384 tokens, its own rows stored before it attends
        dict(op="prefill", name="prefill_chunk", q_heads=32, kv_heads=8, head_dim=128, page=128, history=16384, rows=500),
        # one token for each of 32 slots of a server, contexts as they come
        dict(op="server_decode", name="server_decode", q_heads=32, kv_heads=8, head_dim=128, page=64, seqs=32, ctx_lo=900,
             ctx_hi=8200),
        # a request from its prompt to its first token
        dict(op="server_prompt", name="server_prompt", q_heads=32, kv_heads=8, head_dim=128, page=64, tokens=2000),
        # a token of a single chat through the llama.cpp adapter, default pages
        dict(op="adapter", name="adapter_decode", q_heads=32, kv_heads=8, head_dim=128, page=128, bits=4, ctx=8200, rows=1),
        # a prompt through the llama.cpp adapter, in batches of 512 tokens
        dict(op="adapter_prompt", name="adapter_prompt", q_heads=32, kv_heads=8, head_dim=128, page=128, bits=4, tokens=1000,
             batch=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


HEADS = [(8, 8), (32, 8), (32, 8), (64, 8), (14, 2), (16, 16), (12, 4)]


def draw(rng):
    op = rng.choice(["decode"] * 5 + ["shared", "ingest", "prefill", "server_decode", "server_prompt", "adapter", "adapter_prompt"])
    q_heads, kv_heads = rng.choice(HEADS)
    head_dim = rng.choice([128, 128, 128, 64])
    if op == "decode":
        head_dim = rng.choice([128, 128, 128, 128, 64, 64, 96, 80, 32])
        geometric = rng.random() < 0.3
        seqs = _log(rng, 1, 96)
        most = LARGEST_TOKENS // 2 if head_dim in (128, 96, 64, 32) else LARGEST_TOKENS // 8
        hi = _log(rng, 100, min(131072, max(most * 8 // (kv_heads * seqs), 200)))
        return dict(op=op, coder=rng.choice(sorted(CODERS)), q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim,
                    block=rng.choice([64, 64, 64, 128, 256]) if head_dim == 128 else 64, seqs=seqs,
                    ctx_lo=max(PAGE, int(hi * rng.uniform(0.05, 1.0))), ctx_hi=hi, dist="geometric" if geometric else "laplace",
                    spread=rng.choice([0.05, 0.1, 0.2, 0.4, 0.7]) if geometric else 12.0, tails=rng.random() < 0.7,
                    queries=rng.choice(["f16", "f16", "f32"]), window=rng.choice([0, 0, 0, 0, _log(rng, 256, 8192)]))
    if op == "shared":
        q_heads, kv_heads = rng.choice([(8, 8), (32, 8), (64, 8)])
        return dict(op=op, coder=rng.choice(["rans4", "huffman4", "rans"]), q_heads=q_heads, kv_heads=kv_heads,
                    seqs=_log(rng, 8, 256), prefix=PAGE * _log(rng, 16, 1024), suffix=rng.randint(1, 512))
    if op == "ingest":
        seqs = _log(rng, 1, 128)
        return dict(op=op, coder=rng.choice(sorted(CODERS)), q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim,
                    block=64, seqs=seqs, tokens=PAGE * _log(rng, 1, max(1, min(256, 4096 // seqs))))
    if op == "prefill":
        page = rng.choice([16, 64, 128, 256])
        history = _log(rng, 256, 16384 if page >= 64 else 4096)
        return dict(op=op, q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, page=page, history=history,
                    rows=_log(rng, 2, 512))
    if op == "server_decode":
        hi = _log(rng, 200, 8192)
        return dict(op=op, q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, page=rng.choice([16, 64, 128, 256]),
                    seqs=_log(rng, 1, 32), ctx_lo=max(1, int(hi * rng.uniform(0.1, 1.0))), ctx_hi=hi)
    if op == "server_prompt":
        return dict(op=op, q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, page=rng.choice([16, 64, 128, 256]),
                    tokens=_log(rng, 20, 4096))
    q_heads, kv_heads = rng.choice([(14, 2), (32, 8), (8, 8)])
    if op == "adapter":
        return dict(op=op, q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, page=rng.choice([64, 128, 256]),
                    bits=rng.choice([4, 8]), ctx=_log(rng, 200, 16384), rows=rng.choice([1, _log(rng, 2, 64)]))
    return dict(op=op, q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, page=rng.choice([64, 128, 256]),
                bits=rng.choice([4, 8]), tokens=_log(rng, 50, 2000), batch=rng.choice([256, 512]))


# ---- what a caller has in hand -----------------------------------------------------------------------------------------
class KvOptions(C.Structure):        # cf_llama_kv_options
    _fields_ = [(n, C.c_uint32) for n in ("struct_size", "backend", "layer_count", "kv_head_count", "query_head_count",
                                          "head_dim", "page_size", "gqa_group_size", "kv_bits")]


class DeviceKvConfig(C.Structure):   # cf_device_kv_config
    _fields_ = [(n, C.c_uint32) for n in ("layer_count", "kv_head_count", "query_head_count", "head_dim", "page_size",
                                          "gqa_group_size", "use_async_allocator")]


class Handle:
    """A handle of one of the C ABIs, destroyed with the state that owns it."""

    def __init__(self, value, destroy, *extra):
        if not value:
            raise RuntimeError("the library refused the configuration")
        self.value, self._destroy, self._extra = C.c_void_p(value), destroy, extra

    def __del__(self):
        torch.cuda.synchronize()
        self._destroy(self.value, *self._extra)


_ready = None


def _lib():
    global _ready
    if _ready is None:
        _ready = N.lib()
        for name in ("cf_llama_kv_create", "cf_device_kv_create", "cf_llama_server_runtime_create"):
            getattr(_ready, name).restype = C.c_void_p
        for name in ("cf_llama_kv_last_error", "cf_device_kv_last_error", "cf_llama_server_last_error"):
            getattr(_ready, name).restype = C.c_char_p
    return _ready


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ok(rc, handle=None, last_error=None):
    if rc != 0:
        raise RuntimeError(last_error(handle.value).decode() if last_error else "status %d" % rc)


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _queries(c, rows, gen, f32=True):
    q = torch.randn((rows, c["q_heads"], c["head_dim"]), generator=gen, device=DEVICE)
    return q if f32 else q.half()


def _rows(c, tokens, gen):
    """fp32 K or V rows [token][kv head][channel] as a model's projections come: Laplace values, the odd large one."""
    return laplace_codes((tokens, c["kv_heads"], c["head_dim"]), 12.0, gen, DEVICE) * 0.01


def _contexts(c, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(c["ctx_lo"], c["ctx_hi"] + 1, c["seqs"]).astype(np.int64)


def _scale(c):
    return 1.0 / math.sqrt(c["head_dim"])


def _prepare_decode(c, seed):
    contexts = _contexts(c, seed)
    sealed = contexts // PAGE * PAGE
    layer, _ = build_sealed_layer(sealed, query_heads=c["q_heads"], kv_heads=c["kv_heads"], head_dim=c["head_dim"],
                                  page_tokens=PAGE, block_size=c["block"], coder=c["coder"], dist=(c["dist"], c["spread"]),
                                  seed=seed, device=DEVICE) if sealed.sum() else (_empty_layer(c), None)
    gen = _generator(seed + 1)
    if c["tails"]:
        shape = (1, c["kv_heads"], PAGE, c["head_dim"])
        for s, n in enumerate(contexts - sealed):
            if n:
                k, v = (torch.randn(shape, generator=gen, device=DEVICE) * 0.2 for _ in range(2))
                layer.fill_tails([s], k, v, int(n))
    q = _queries(c, c["seqs"], gen, c["queries"] == "f32")
    return {"c": c, "layer": layer, "q": q, "out": torch.zeros(q.shape, device=DEVICE)}


def _empty_layer(c):
    return SealedKvLayer(kv_heads=c["kv_heads"], query_heads=c["q_heads"], head_dim=c["head_dim"], page_tokens=PAGE,
                         block_size=c["block"], coder=CODERS[c["coder"]], max_sequences=c["seqs"], max_pages_per_sequence=2,
                         max_pages=2 * c["seqs"] + 2, arena_bytes=1 << 20, device=DEVICE)


def _prepare_shared(c, seed):
    n, own = c["seqs"], c["suffix"] // PAGE
    shape = dict(c, head_dim=128)
    layer, _ = build_sealed_layer(np.array([c["prefix"]] + [0] * (n - 1)), query_heads=c["q_heads"], kv_heads=c["kv_heads"],
                                  coder=c["coder"], seed=seed, device=DEVICE, extra_pages_per_sequence=own + 2,
                                  reserve_pages=n * (own + 2))
    for s in range(1, n):
        layer.copy_sequence(0, s)
    gen = _generator(seed + 1)
    for p in range(own):   # every sequence's private suffix, a page of all of them at a time
        tiles = [tiles_from_codes(laplace_codes((n, c["kv_heads"], PAGE, 128), 12.0, gen, DEVICE), 0.005, 0.02, gen) for _ in range(2)]
        layer.seal_tiles(np.arange(n), *tiles)
        torch.cuda.synchronize()
    left = c["suffix"] % PAGE
    if left:
        k, v = (torch.randn((n, c["kv_heads"], PAGE, 128), generator=gen, device=DEVICE) * 0.2 for _ in range(2))
        layer.fill_tails(np.arange(n), k, v, left)
    q = _queries(shape, n, gen, False)
    return {"c": c, "layer": layer, "q": q, "out": torch.zeros(q.shape, device=DEVICE)}


def _prepare_ingest(c, seed):
    """The tiles of every prompt (binary16, page by page), a calibrated store, and the seal descriptor a caller keeps. The
    prompts are sealed once here, so that the store's page table names their pages; a pass seals them into the same ids."""
    n, pages = c["seqs"], c["tokens"] // PAGE
    gen = _generator(seed)
    layer = build_sealed_layer(np.array([PAGE] + [0] * (n - 1)), query_heads=c["q_heads"], kv_heads=c["kv_heads"],
                               head_dim=c["head_dim"], block_size=c["block"], coder=c["coder"], seed=seed, device=DEVICE)[0]
    fresh = SealedKvLayer(kv_heads=c["kv_heads"], query_heads=c["q_heads"], head_dim=c["head_dim"], page_tokens=PAGE,
                          block_size=c["block"], coder=CODERS[c["coder"]], max_sequences=n, max_pages_per_sequence=pages,
                          max_pages=n * pages + 1,
                          arena_bytes=n * pages * c["kv_heads"] * (16 + 2 * c["head_dim"] * PAGE) + 4096, device=DEVICE)
    fresh.k_tables.copy_(layer.k_tables)
    fresh.v_tables.copy_(layer.v_tables)
    fresh.host_tables, fresh._codebooks_set = layer.host_tables, True
    shape = (n * pages, c["kv_heads"], PAGE, c["head_dim"])
    k, v = (tiles_from_codes(laplace_codes(shape, 12.0, gen, DEVICE), 0.005, 0.02, gen) for _ in range(2))
    fresh.seal_tiles(np.repeat(np.arange(n), pages), k, v)
    d = N.SealDesc()
    d.struct_size, d.abi_version = C.sizeof(N.SealDesc), N.ABI_VERSION
    d.kv_head_count, d.head_dim, d.page_tokens, d.block_size = c["kv_heads"], c["head_dim"], PAGE, c["block"]
    d.coder, d.codebook_id = CODERS[c["coder"]], 0
    d.k_tables, d.v_tables = fresh.k_tables.data_ptr(), fresh.v_tables.data_ptr()
    d.tail_k, d.tail_v = k.data_ptr(), v.data_ptr()
    tiles = torch.arange(n * pages, dtype=torch.int32, device=DEVICE)
    ids = tiles + 1
    d.job_slots, d.job_pages, d.job_count = tiles.data_ptr(), ids.data_ptr(), n * pages
    d.arena, d.arena_units = fresh.arena.data_ptr(), fresh.arena_units
    d.arena_cursor_units, d.page_dir, d.status = fresh.cursor.data_ptr(), fresh.page_dir.data_ptr(), fresh.status.data_ptr()
    q = _queries(c, n, gen, False)
    return {"c": c, "layer": fresh, "desc": d, "keep": (k, v, tiles, ids), "q": q, "out": torch.zeros(q.shape, device=DEVICE)}


def _view(t):
    """A dense fp32 [token][head][channel] tensor as the C ABIs describe it."""
    n, h, d = t.shape
    return N.TensorView(t.data_ptr(), N.F32, n, h, d, h * d * 4, d * 4, 4, 0)


def _prepare_prefill(c, seed):
    lib, gen = _lib(), _generator(seed)
    cfg = DeviceKvConfig(1, c["kv_heads"], c["q_heads"], c["head_dim"], c["page"], c["q_heads"] // c["kv_heads"], 1)
    kv = Handle(lib.cf_device_kv_create(C.byref(cfg)), lib.cf_device_kv_destroy, None)
    tokens = c["history"] + c["rows"]
    k, v = _rows(c, tokens, gen), _rows(c, tokens, gen)
    for begin in range(0, tokens, c["page"]):
        end = min(begin + c["page"], tokens)
        _ok(lib.cf_device_kv_append_async(kv.value, 0, begin, C.byref(_view(k[begin:end])), C.byref(_view(v[begin:end])), _stream()),
            kv, lib.cf_device_kv_last_error)
        _ok(lib.cf_device_kv_seal_full_pages_async(kv.value, _stream()), kv, lib.cf_device_kv_last_error)
    q = _queries(c, c["rows"], gen)
    return {"c": c, "kv": kv, "q": q, "out": torch.zeros(q.shape, device=DEVICE)}


def _server(c):
    lib = _lib()
    cfg = N.LlamaServerConfig(1, c["q_heads"], c["kv_heads"], c["head_dim"], c["page"], 64, 1 << 20, c["q_heads"] // c["kv_heads"],
                              0, 1, None, b"local", b"0" * 64)
    return Handle(lib.cf_llama_server_runtime_create(C.byref(cfg)), lib.cf_llama_server_runtime_destroy, None)


def _append_prompt(server, slot, k, v):
    lib = _lib()
    _ok(lib.cf_llama_server_append_layer_async(server.value, C.c_int64(slot), 0, 0, C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()),
                                               C.c_uint32(k.shape[0]), _stream()), server, lib.cf_llama_server_last_error)


def _batch(c, q, out, positions):
    """One attention item per slot, slots numbered from 1."""
    items = (N.SequenceAttentionItem * len(positions))()
    hq, d = c["q_heads"], c["head_dim"]
    for i, (it, at) in enumerate(zip(items, positions)):
        it.sequence_id, it.layer, it.query = i + 1, 0, _view(q[i:i + 1])
        it.output, it.output_type = out[i].data_ptr(), N.F32
        it.output_token_stride_bytes, it.output_head_stride_bytes, it.output_element_stride_bytes = hq * d * 4, d * 4, 4
        it.query_token_begin, it.softmax_scale, it.causal_window = int(at), _scale(c), 0
    return N.LlamaServerBatch(None, 0, C.cast(items, C.c_void_p), len(items)), items


def _prepare_server_decode(c, seed):
    lib, gen, server = _lib(), _generator(seed), _server(c)
    contexts = _contexts(c, seed)
    for i, n in enumerate(contexts):
        _ok(lib.cf_llama_server_slot_create(server.value, C.c_int64(i + 1)), server, lib.cf_llama_server_last_error)
        _append_prompt(server, i + 1, _rows(c, int(n), gen), _rows(c, int(n), gen))
    q = _queries(c, c["seqs"], gen)
    out = torch.zeros(q.shape, device=DEVICE)
    batch, items = _batch(c, q, out, contexts)
    return {"c": c, "server": server, "q": q, "out": out, "batch": batch, "items": items}


def _prepare_server_prompt(c, seed):
    gen, server = _generator(seed), _server(c)
    k, v, q = _rows(c, c["tokens"], gen), _rows(c, c["tokens"], gen), _queries(c, 1, gen)
    out = torch.zeros(q.shape, device=DEVICE)
    batch, items = _batch(c, q, out, [c["tokens"]])
    return {"c": c, "server": server, "k": k, "v": v, "q": q, "out": out, "batch": batch, "items": items}


def _adapter(c):
    lib = _lib()
    opt = KvOptions(C.sizeof(KvOptions), 1, 1, c["kv_heads"], c["q_heads"], c["head_dim"], c["page"], c["q_heads"] // c["kv_heads"],
                    c["bits"])
    return Handle(lib.cf_llama_kv_create(C.byref(opt)), lib.cf_llama_kv_destroy)


def _host_rows(c, tokens, gen):
    """Rows as the adapter takes them: host fp32 [kv head][token][channel]."""
    return _rows(c, tokens, gen).permute(1, 0, 2).contiguous().cpu().numpy()


def _adapter_append(c, kv, k, v, begin, end):
    lib = _lib()
    for h in range(c["kv_heads"]):
        _ok(lib.cf_llama_kv_append(kv.value, 0, h, begin, C.c_void_p(k[h, begin:].ctypes.data), C.c_void_p(v[h, begin:].ctypes.data),
                                   end - begin, _stream()), kv, lib.cf_llama_kv_last_error)


def _adapter_attention(c, kv, q, out, begin):
    lib = _lib()
    _ok(lib.cf_llama_kv_attention(kv.value, 0, C.c_void_p(q.data_ptr()), C.c_void_p(out.data_ptr()), q.shape[0], c["q_heads"],
                                  c["q_heads"] // c["kv_heads"], begin, C.c_float(_scale(c)), 0, _stream()),
        kv, lib.cf_llama_kv_last_error)


def _prepare_adapter(c, seed):
    gen, kv = _generator(seed), _adapter(c)
    _adapter_append(c, kv, _host_rows(c, c["ctx"], gen), _host_rows(c, c["ctx"], gen), 0, c["ctx"])
    q = _queries(c, c["rows"], gen)
    return {"c": c, "kv": kv, "q": q, "out": torch.zeros(q.shape, device=DEVICE)}


def _prepare_adapter_prompt(c, seed):
    gen, kv = _generator(seed), _adapter(c)
    k, v = _host_rows(c, c["tokens"], gen), _host_rows(c, c["tokens"], gen)
    q = _queries(c, c["tokens"], gen)
    return {"c": c, "kv": kv, "k": k, "v": v, "q": q, "out": torch.zeros(q.shape, device=DEVICE)}


def prepare(case, seed):
    state = globals()["_prepare_" + case["op"]](case, seed)
    torch.cuda.synchronize()
    return state


# ---- one pass -----------------------------------------------------------------------------------------------------------
def run(state):
    c = state["c"]
    op = c["op"]
    if op == "decode":
        return state["layer"].attention(state["q"], out=state["out"], causal_window=c["window"])
    if op == "shared":
        return state["layer"].attention(state["q"], out=state["out"], shared_prefix_pages=c["prefix"] // PAGE)
    if op == "ingest":
        layer = state["layer"]
        layer.cursor.zero_()
        N.check("seal_pages", layer.lib.cf_b200_seal_pages_async(C.byref(state["desc"]), _stream()))
        return layer.attention(state["q"], out=state["out"])
    lib = _lib()
    if op == "prefill":
        kv, rows = state["kv"], c["rows"]
        _ok(lib.cf_device_kv_attention_async(kv.value, 0, C.c_void_p(state["q"].data_ptr()), C.c_void_p(state["out"].data_ptr()), rows,
                                             c["history"], C.c_float(_scale(c)), 0, _stream()), kv, lib.cf_device_kv_last_error)
    elif op == "server_decode":
        server = state["server"]
        _ok(lib.cf_llama_server_execute_batch_async(server.value, C.byref(state["batch"]), _stream()), server,
            lib.cf_llama_server_last_error)
    elif op == "server_prompt":
        server = state["server"]
        _ok(lib.cf_llama_server_slot_create(server.value, C.c_int64(1)), server, lib.cf_llama_server_last_error)
        _append_prompt(server, 1, state["k"], state["v"])
        _ok(lib.cf_llama_server_execute_batch_async(server.value, C.byref(state["batch"]), _stream()), server,
            lib.cf_llama_server_last_error)
        _ok(lib.cf_llama_server_slot_reset_async(server.value, C.c_int64(1), _stream()), server, lib.cf_llama_server_last_error)
    elif op == "adapter":
        _adapter_attention(c, state["kv"], state["q"], state["out"], c["ctx"] - c["rows"])
    else:   # adapter_prompt
        kv = state["kv"]
        _ok(lib.cf_llama_kv_clear(kv.value), kv, lib.cf_llama_kv_last_error)
        for begin in range(0, c["tokens"], c["batch"]):
            end = min(begin + c["batch"], c["tokens"])
            _adapter_append(c, kv, state["k"], state["v"], begin, end)
            _adapter_attention(c, kv, state["q"][begin:end], state["out"][begin:end], begin)
    return state["out"]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------
def _code_bits(coder, dist, spread):
    """Bits a coded value takes at least: the entropy of the codes; with the nibble-split coders the raw low nibble and
    the entropy of the high one."""
    x = np.arange(-128, 129)
    if dist == "laplace":
        cdf = lambda t: np.where(t < 0, 0.5 * np.exp(np.minimum(t, 0) / spread), 1 - 0.5 * np.exp(-np.maximum(t, 0) / spread))
        p = cdf(x[1:] - 0.5) - cdf(x[:-1] - 0.5)
    else:
        p = (1 - spread) ** np.abs(x[:-1])
    p = p / p.sum()
    h = lambda q: float(-(q[q > 0] * np.log2(q[q > 0])).sum())
    if coder == "fixed8":
        return 8.0
    return 4.0 + h(p.reshape(16, 16).sum(1)) if coder.endswith("4") else h(p)


def work(case):
    c = case
    hq, hkv, d = c["q_heads"], c["kv_heads"], c.get("head_dim", 128)
    bits = _code_bits(c.get("coder", "rans4"), c.get("dist", "laplace"), c.get("spread", 12.0))
    kv = lambda tokens, b=bits: tokens * hkv * 2 * d * b / 8     # coded K and V of so many tokens
    io = lambda rows, q_bytes: rows * hq * d * (q_bytes + 4)     # queries in, outputs (fp32) back
    flops = lambda pairs: 4 * d * hq * pairs                     # pairs of (query token, visible token)
    op = c["op"]
    if op in ("decode", "server_decode"):
        mean = (c["ctx_lo"] + c["ctx_hi"]) / 2
        seen = c["seqs"] * (min(mean, c["window"]) if c.get("window") else mean)
        return {"bytes": kv(seen) + io(c["seqs"], 4 if c.get("queries", "f32") == "f32" else 2), "flops": flops(seen)}
    if op == "shared":
        return {"bytes": kv(c["prefix"] + c["seqs"] * c["suffix"]) + io(c["seqs"], 2),
                "flops": flops(c["seqs"] * (c["prefix"] + c["suffix"]))}
    if op == "ingest":
        tokens = c["seqs"] * c["tokens"]
        return {"bytes": tokens * hkv * 2 * d * 2 + kv(tokens) + io(c["seqs"], 2), "flops": flops(tokens)}
    if op == "prefill":
        rows = c["rows"]
        return {"bytes": kv(c["history"] + rows) + io(rows, 4), "flops": flops(rows * c["history"] + rows * (rows + 1) // 2)}
    if op == "server_prompt":
        return {"bytes": c["tokens"] * hkv * 2 * d * 4 + kv(c["tokens"]) + io(1, 4), "flops": flops(c["tokens"])}
    if op == "adapter":
        return {"bytes": kv(c["ctx"], c["bits"]) + io(c["rows"], 4), "flops": flops(c["rows"] * c["ctx"])}
    tokens = c["tokens"]
    return {"bytes": tokens * hkv * 2 * d * 4 + kv(tokens, c["bits"]) + io(tokens, 4), "flops": flops(tokens * (tokens + 1) // 2)}


def tolerance(case):
    """Codes are exact; scores, softmax and weighted sums are kept to fp32 accuracy, in whatever order they are added."""
    return {"rel": 2e-5, "max": 1e-3}
