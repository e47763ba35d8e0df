"""cf_kv_paged_attention_async at head_dim 128 and 64 (csrc/compat_paged_mma.cu) against fp64 softmax over the dequantised
rows, where the tiles and branches of the tensor-core form begin and end: row counts around the 16-row tile, page sizes
around the 16-token group, windows, tails, every code width it loads directly, and the ones it decodes first."""
import ctypes as C

import numpy as np
import pytest

from compat_types import DevicePage, PagedAttentionDesc
from test_gpu_compat import _read_device

pytestmark = pytest.mark.gpu


def _pack(sym, bits):
    """Symbols MSB-first in u32 words, two words of slack."""
    per = 32 // bits
    s = np.concatenate([sym.astype(np.uint64).ravel(), np.zeros(-sym.size % per, np.uint64)]).reshape(-1, per)
    shifts = (32 - bits - bits * np.arange(per)).astype(np.uint64)
    return np.concatenate([(s << shifts).sum(1).astype(np.uint32), np.zeros(2, np.uint32)])


# (bits, head_dim, q heads, kv heads, page sizes, tail, query tokens, window, zero point, what is special)
CASES = [
    (4, 128, 4, 1, [16], 0, 1, 0, 8, ""),
    (4, 128, 32, 8, [128] * 9, 5, 1, 0, 8, ""),
    (4, 64, 14, 2, [1, 15, 17, 31], 1, 3, 0, 8, ""),
    (8, 128, 8, 8, [33, 16, 128], 17, 16, 0, 128, ""),
    (8, 64, 16, 1, [64, 2], 0, 5, 20, 128, ""),
    (4, 128, 5, 1, [128, 128, 128], 127, 7, 100, 8, ""),
    (4, 128, 4, 1, [], 40, 9, 0, 8, ""),
    (8, 128, 2, 2, [48], 16, 60, 33, 128, ""),
    (4, 128, 32, 8, [40, 24], 3, 2, 0, 8, "unaligned"),
    (2, 64, 4, 2, [20, 12], 2, 1, 0, 1, ""),
    (0, 128, 8, 2, [40, 9], 4, 3, 0, 128, ""),
    (0, 64, 7, 1, [100], 0, 1, 30, 128, ""),
    (8, 128, 4, 1, [32, 32], 6, 2, 0, 2000, ""),
    (4, 128, 4, 1, [64, 64], 6, 2, 0, 8, "magnitudes"),
]


@pytest.mark.parametrize("case", CASES, ids=str)
def test_paged_attention_on_the_tensor_cores(native, oracle, case):
    import torch
    from helpers import hist_of, laplace_codes
    from test_gpu_compat import _softmax_attention
    bits, d, hq, hkv, sizes, tail, nq, window, zp, special = case
    rng = np.random.default_rng(CASES.index(case))
    dev = lambda a: torch.from_numpy(np.array(a, copy=True)).cuda()
    pages, keep, begin, sealed = [], [], 0, sum(sizes)
    dense_k, dense_v = np.zeros((hkv, sealed, d)), np.zeros((hkv, sealed, d))
    for tokens in sizes:
        for h in range(hkv):
            ks, vs = rng.uniform(0.005, 0.02, d).astype(np.float32), rng.uniform(0.005, 0.02, tokens).astype(np.float32)
            if zp == 2000:
                ks, vs = ks / 2000, vs / 2000
            if special == "magnitudes":
                ks, vs = ks * 10.0 ** rng.uniform(-5, 1, d).astype(np.float32), vs * 10.0 ** rng.uniform(-6, 4, tokens).astype(np.float32)
            n = tokens * d
            if bits:
                syms = [rng.integers(0, 1 << bits, n).astype(np.uint8) for _ in range(2)]
                words, offs, luts = [_pack(s, bits) for s in syms], [np.zeros((n + 63) // 64, np.int32)] * 2, [np.zeros(1 << bits, np.int32)] * 2
            else:
                syms = [(laplace_codes(rng, n, b).astype(np.int16) + 128).astype(np.uint8) for b in (9.0, 14.0)]
                cbs = [oracle.codebook_from_hist(hist_of(s)) for s in syms]
                coded = [oracle.huff_encode(s, 64, cb) for s, cb in zip(syms, cbs)]
                words, offs, luts = [np.concatenate([w, np.zeros(2, np.uint32)]) for w, _ in coded], [o for _, o in coded], [cb.np("lut") for cb in cbs]
            dense_k[h, begin:begin + tokens] = (syms[0].reshape(tokens, d).astype(np.float64) - zp) * ks[None, :]
            dense_v[h, begin:begin + tokens] = (syms[1].reshape(tokens, d).astype(np.float64) - zp) * vs[:, None]
            shift = 1 if special == "unaligned" else 0
            held = [dev(np.concatenate([np.zeros(shift, np.uint32), w]).view(np.int32)) for w in words] + [dev(x) for x in (*offs, *luts, ks, vs)]
            keep.append(held)
            pg = DevicePage()
            pg.k_words, pg.v_words = held[0].data_ptr() + 4 * shift, held[1].data_ptr() + 4 * shift
            pg.k_block_offsets, pg.v_block_offsets, pg.k_lut, pg.v_lut, pg.k_scales, pg.v_scales = [x.data_ptr() for x in held[2:]]
            pg.token_begin, pg.token_count, pg.head_dim, pg.block_size = begin, tokens, d, 64
            pg.k_max_code_length = pg.v_max_code_length = bits or 12
            pg.zero_point, pg.kv_head, pg.fixed_code_length = zp, h, bits
            pages.append(pg)
        begin += tokens
    q = rng.standard_normal((nq, hq, d)).astype(np.float32)
    tk, tv = (rng.standard_normal((max(tail, 1), hkv, d)).astype(np.float32) for _ in range(2))
    if special == "magnitudes":
        tv *= 1e3
    out = torch.full((nq, hq, d), 3.0, device="cuda")
    d_q, d_tk, d_tv = dev(q), dev(tk), dev(tv)
    desc = PagedAttentionDesc()
    desc.struct_size, desc.abi_version = C.sizeof(desc), 0
    if pages:
        d_pages = dev(np.frombuffer(bytes((DevicePage * len(pages))(*pages)), np.uint8))
        desc.pages, desc.page_count = d_pages.data_ptr(), len(pages)
    desc.kv_head_count, desc.query_head_count, desc.gqa_group_size = hkv, hq, hq // hkv
    desc.active_k, desc.active_v, desc.active_token_begin, desc.active_token_count = d_tk.data_ptr(), d_tv.data_ptr(), sealed, tail
    first = sealed + tail - nq
    desc.queries, desc.output, desc.query_token_begin, desc.query_count = d_q.data_ptr(), out.data_ptr(), first, nq
    desc.head_dim, desc.causal_window, desc.softmax_scale = d, window, 1.0 / np.sqrt(d)
    for _ in range(2):   # twice: the splits' arrival counters are left at zero
        out.fill_(3.0)
        assert native.lib().cf_kv_paged_attention_async(C.byref(desc), None) == 0
    torch.cuda.synchronize()
    pos = [first + i for i in range(nq)]
    want = _softmax_attention(np.concatenate([dense_k, tk[:tail].transpose(1, 0, 2)], axis=1),
                              np.concatenate([dense_v, tv[:tail].transpose(1, 0, 2)], axis=1), q, pos,
                              [max(0, p + 1 - window) if window else 0 for p in pos], 1.0 / np.sqrt(d), hq // hkv)
    got = out.cpu().numpy()
    assert np.isfinite(got).all()
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max(), np.abs(got - want).max() / np.abs(want).max()


def _tail_only(native, q, k, v, first, pages=None, sealed=0):
    """cf_kv_paged_attention_async over an fp32 tail [token][kv head][D] (and pages in front of it), one query head per kv head."""
    import torch
    dev = lambda a: torch.from_numpy(np.array(a, copy=True)).cuda()
    out = torch.full(q.shape, 3.0, device="cuda")
    d_q, d_k, d_v = dev(q), dev(k), dev(v)
    desc = PagedAttentionDesc()
    desc.struct_size, desc.abi_version = C.sizeof(desc), 0
    if pages:
        table = dev(np.frombuffer(bytes((DevicePage * len(pages))(*pages)), np.uint8))
        desc.pages, desc.page_count = table.data_ptr(), len(pages)
    desc.kv_head_count, desc.query_head_count, desc.gqa_group_size = k.shape[1], q.shape[1], q.shape[1] // k.shape[1]
    desc.active_k, desc.active_v, desc.active_token_begin, desc.active_token_count = d_k.data_ptr(), d_v.data_ptr(), sealed, k.shape[0]
    desc.queries, desc.output, desc.query_token_begin, desc.query_count = d_q.data_ptr(), out.data_ptr(), first, q.shape[0]
    desc.head_dim, desc.softmax_scale = q.shape[2], 1.0 / np.sqrt(q.shape[2])
    assert native.lib().cf_kv_paged_attention_async(C.byref(desc), None) == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("d,hq,hkv,tokens,nq", [(128, 4, 1, 21, 1), (64, 2, 2, 40, 1), (128, 4, 1, 33, 20), (64, 16, 1, 16, 9)], ids=str)
def test_infinities_and_nan_in_the_tail_stay_where_fp32_puts_them(native, d, hq, hkv, tokens, nq):
    rng = np.random.default_rng(d + nq)
    q = rng.standard_normal((nq, hq, d)).astype(np.float32)
    k, v = (rng.standard_normal((tokens, hkv, d)).astype(np.float32) for _ in range(2))
    first, group = tokens - nq, hq // hkv
    q[..., 5] = np.abs(q[..., 5]) + 0.1
    k[0, :, 5] = -np.inf                        # a score of -inf: the token weighs nothing
    v[2, :, 3], v[3, :, 60] = np.inf, -np.inf   # of visible tokens: the channels become infinite, no other does
    if nq > 1:                                  # tokens that the first rows do not see
        k[first + 2, :, 7], v[first + 2, :, 11] = np.nan, np.nan
        v[first + 1, :, 20] = np.inf
    got = _tail_only(native, q, k, v, first)
    with np.errstate(invalid="ignore"):
        for i in range(nq):
            for h in range(hq):
                kk, vv = (x[:first + i + 1, h // group].astype(np.float64) for x in (k, v))
                s = kk @ q[i, h].astype(np.float64) / np.sqrt(d)
                if np.isnan(s).any():
                    continue
                w = np.exp(s - s.max())
                want = np.where(w[:, None] == 0, 0, w[:, None] * vv).sum(0) / w.sum()
                finite = np.isfinite(want)
                assert np.array_equal(np.isnan(want), np.isnan(got[i, h])) and np.array_equal(want[~finite], got[i, h][~finite], equal_nan=True)
                if finite.any():
                    assert np.abs(got[i, h] - want)[finite].max() <= 2e-5 * np.abs(want[finite]).max()


@pytest.mark.parametrize("scale", [1e-36, 0.0, 1e34])
def test_a_tail_behind_pages_of_any_scale(native, scale):
    """V scales far from the tail's magnitudes: neither side of the sum overflows or vanishes."""
    import torch
    d, page = 128, 16
    rng = np.random.default_rng(8)
    dev = lambda a: torch.from_numpy(np.array(a, copy=True)).cuda()
    held = [dev(rng.integers(0, 1 << 32, page * d // 4, dtype=np.uint32).view(np.int32)), dev(np.full(d, 1e-3, np.float32)), dev(np.full(page, scale, np.float32)),
            dev(np.zeros(page * d // 64, np.int32))]
    pg = DevicePage()
    pg.k_words = pg.v_words = held[0].data_ptr()
    pg.k_scales, pg.v_scales = held[1].data_ptr(), held[2].data_ptr()
    pg.k_block_offsets = pg.v_block_offsets = pg.k_lut = pg.v_lut = held[3].data_ptr()
    pg.token_count, pg.head_dim, pg.block_size = page, d, 64
    pg.k_max_code_length = pg.v_max_code_length = pg.fixed_code_length = 8
    pg.zero_point = 128
    codes = held[0].cpu().numpy().view(np.uint32)
    codes = np.stack([(codes >> s) & 255 for s in (24, 16, 8, 0)], 1).reshape(page, d).astype(np.float64) - 128
    tail = 30
    q, k, v = (rng.standard_normal((n, 1, d)).astype(np.float32) for n in (1, tail, tail))
    v *= 1e5 if scale < 1 else 1.0
    got = _tail_only(native, q, k, v, page + tail - 1, [pg], page)[0, 0]
    s = np.concatenate([codes * np.float64(np.float32(1e-3)), k[:, 0]]) @ q[0, 0].astype(np.float64) / np.sqrt(d)
    w = np.exp(s - s.max())
    want = (w[:, None] * np.concatenate([codes * np.float64(np.float32(scale)), v[:, 0]])).sum(0) / w.sum()
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


def test_paged_attention_from_several_threads(native):
    """Callers on streams of their own share the slots in which splits leave their partials: every call, whatever its number of
    splits, gives what it gives alone."""
    import threading
    import torch
    lib, d, hq, hkv, page, threads, calls = native.lib(), 128, 8, 2, 32, 12, 250
    rng = np.random.default_rng(11)
    dev = lambda a: torch.from_numpy(np.array(a, copy=True)).cuda()
    most = 40
    held = [dev(rng.integers(0, 1 << 32, page * d // 8, dtype=np.uint32).view(np.int32)) for _ in range(2 * hkv * most)]
    scales = dev(rng.uniform(0.005, 0.02, max(d, page)).astype(np.float32))
    spare = dev(np.zeros(page * d // 64, np.int32))
    jobs = []
    for i in range(threads):
        pages = (DevicePage * ((3 + 3 * i) * hkv))()
        for n, pg in enumerate(pages):
            pg.k_words, pg.v_words = held[2 * (n % (hkv * most))].data_ptr(), held[2 * (n % (hkv * most)) + 1].data_ptr()
            pg.k_block_offsets = pg.v_block_offsets = pg.k_lut = pg.v_lut = spare.data_ptr()
            pg.k_scales = pg.v_scales = scales.data_ptr()
            pg.token_begin, pg.token_count, pg.head_dim, pg.block_size = n // hkv * page, page, d, 64
            pg.k_max_code_length = pg.v_max_code_length = pg.fixed_code_length = 4
            pg.zero_point, pg.kv_head = 8, n % hkv
        table = dev(np.frombuffer(bytes(pages), np.uint8))
        q = dev(rng.standard_normal((1 + i % 3, hq, d)).astype(np.float32))
        out = torch.zeros((calls, *q.shape), device="cuda")
        desc = PagedAttentionDesc()
        desc.struct_size, desc.abi_version = C.sizeof(desc), 0
        desc.pages, desc.page_count = table.data_ptr(), len(pages)
        desc.kv_head_count, desc.query_head_count, desc.gqa_group_size = hkv, hq, hq // hkv
        desc.queries, desc.query_token_begin, desc.query_count = q.data_ptr(), page * len(pages) // hkv, q.shape[0]
        desc.head_dim, desc.softmax_scale = d, d ** -0.5
        jobs.append((desc, out, torch.cuda.Stream(), table, q))
    alone = []
    for desc, out, *_ in jobs:
        desc.output = out[0].data_ptr()
        assert lib.cf_kv_paged_attention_async(C.byref(desc), None) == 0
        torch.cuda.synchronize()
        alone.append(out[0].clone())
        out.zero_()
    torch.cuda.synchronize()
    failed = []

    def work(desc, out, stream):
        for n in range(calls):
            desc.output = out.data_ptr() + n * out[0].numel() * 4
            if lib.cf_kv_paged_attention_async(C.byref(desc), C.c_void_p(stream.cuda_stream)) != 0:
                failed.append(n)

    runners = [threading.Thread(target=work, args=job[:3]) for job in jobs]
    for t in runners:
        t.start()
    for t in runners:
        t.join()
    torch.cuda.synchronize()
    assert not failed
    for want, (_, out, *_) in zip(alone, jobs):   # the same splits, merged in the same order
        assert torch.equal(out, want.expand_as(out))


# ---- the adapter's page quantiser (csrc/adapter.cu): several pages per launch --------------------------------------------
def _quantised(x, axis, bits):
    """The reference fixture's rule (src/runtime/kv_gpu_fixture.cpp:12-16, 46-95) in fp32: one scale along `axis`."""
    qmax = (1 << (bits - 1)) - 1
    m = np.abs(x).max(axis=axis, keepdims=True)
    scale = np.where(m == 0, np.float32(1), m / np.float32(qmax)).astype(np.float32)
    return (np.clip(np.rint(x / scale), -(qmax + 1), qmax) + (1 << (bits - 1))).astype(np.uint8), scale.ravel()


def _adapter(native, heads, d, page, bits):
    from compat_types import LlamaKvOptions
    lib = native.lib()
    lib.cf_llama_kv_create.restype = C.c_void_p
    opt = LlamaKvOptions(C.sizeof(LlamaKvOptions), 1, 1, heads, heads, d, page, 1, bits)
    handle = C.c_void_p(lib.cf_llama_kv_create(C.byref(opt)))
    assert handle.value
    return lib, handle


def _append(lib, handle, head, begin, k, v):
    return lib.cf_llama_kv_append(handle, 0, head, begin, C.c_void_p(k.ctypes.data), C.c_void_p(v.ctypes.data), k.shape[0], None)


@pytest.mark.parametrize("d,page,bits,pieces", [(128, 128, 4, [1, 500, 300]), (64, 16, 8, [1100]), (48, 32, 4, [31, 1, 33]), (30, 16, 4, [50]),
                                                (128, 256, 8, [255, 2, 600])], ids=str)
def test_adapter_pages_of_multi_page_appends_are_exact(native, d, page, bits, pieces):
    import torch
    rng = np.random.default_rng(d + page)
    lib, handle = _adapter(native, 2, d, page, bits)
    total = sum(pieces)
    k = (rng.standard_normal((2, total, d)) * 10.0 ** rng.uniform(-3, 2, (1, total, 1))).astype(np.float32)
    v = (rng.standard_normal((2, total, d)) * 10.0 ** rng.uniform(-3, 2, (1, 1, d))).astype(np.float32)
    k[0, :, 3] = 0.0
    at = 0
    for n in pieces:
        for h in range(2):
            kk, vv = np.ascontiguousarray(k[h, at:at + n]), np.ascontiguousarray(v[h, at:at + n])
            assert _append(lib, handle, h, at, kk, vv) == 0
        at += n
    seen = {0: 0, 1: 0}
    for i in range(2 * (total // page)):
        pg = DevicePage()
        assert lib.cf_b200_llama_kv_reference_page(handle, 0, i, C.byref(pg)) == 0
        h = pg.kv_head
        assert pg.token_begin == seen[h] and pg.token_count == page
        rows = slice(seen[h], seen[h] + page)
        seen[h] += page
        ks, kscale = _quantised(k[h, rows], 0, bits)
        vs, vscale = _quantised(v[h, rows], 1, bits)
        words = (page * d * bits + 31) // 32
        for ptr, want in ((pg.k_words, _pack(ks, bits)[:words]), (pg.v_words, _pack(vs, bits)[:words])):
            assert np.array_equal(_read_device(ptr, words, np.uint32), want)
        assert np.array_equal(_read_device(pg.k_scales, d, np.float32), kscale) and np.array_equal(_read_device(pg.v_scales, page, np.float32), vscale)
    assert lib.cf_b200_llama_kv_reference_page(handle, 0, 2 * (total // page), C.byref(DevicePage())) == -1
    lib.cf_llama_kv_destroy(handle)


def test_adapter_append_keeps_the_pages_before_a_refused_one(native):
    """Five pages in one append, NaN in the fourth: the first three are sealed, the fourth's rows are the full tail and every
    further append fails, as when the rows came page by page."""
    from compat_types import LlamaKvStats
    rng = np.random.default_rng(3)
    lib, handle = _adapter(native, 1, 64, 16, 4)
    lib.cf_llama_kv_last_error.restype = C.c_char_p
    k, v = (rng.standard_normal((85, 64)).astype(np.float32) for _ in range(2))
    v[3 * 16 + 2, 7] = np.nan
    assert _append(lib, handle, 0, 0, k[:5], v[:5]) == 0
    assert _append(lib, handle, 0, 5, k[5:], v[5:]) == -1 and lib.cf_llama_kv_last_error(handle) == b"invalid quantization input"
    stats = LlamaKvStats()
    assert lib.cf_llama_kv_get_stats(handle, C.byref(stats)) == 0
    assert (stats.sealed_pages, stats.sealed_tokens, stats.active_tokens) == (3, 48, 16)
    assert _append(lib, handle, 0, 64, k[64:66], v[64:66]) == -1
    assert lib.cf_llama_kv_clear(handle) == 0 and _append(lib, handle, 0, 0, k[:48], v[:48]) == 0
    pg = DevicePage()
    assert lib.cf_b200_llama_kv_reference_page(handle, 0, 2, C.byref(pg)) == 0 and pg.token_begin == 32
    ks, _ = _quantised(k[32:48], 0, 4)
    assert np.array_equal(_read_device(pg.k_words, 128, np.uint32), _pack(ks, 4)[:128])
    lib.cf_llama_kv_destroy(handle)


def _attend(lib, handle, q, begin, stream=None):
    import torch
    out = torch.full(q.shape, 5.0, device="cuda")
    hq = q.shape[1]
    assert lib.cf_llama_kv_attention(handle, 0, C.c_void_p(q.data_ptr()), C.c_void_p(out.data_ptr()), q.shape[0], hq, 1, begin,
                                     C.c_float(q.shape[2] ** -0.5), 0, C.c_void_p(stream.cuda_stream) if stream else None) == 0
    return out


def test_adapter_append_that_runs_out_of_memory_leaves_no_page_behind(native):
    """The page memory ends in the middle of a launch's pages: the pages before that launch stay, none of its own is named, and the
    same rows go in once there is memory again."""
    import torch
    lib, handle = _adapter(native, 1, 128, 128, 8)
    rng = np.random.default_rng(5)
    block = 2 * 128 * 128 + 4 * 256 + 2 * 4 * 256
    pages = (32 << 20) // ((block + 255) // 256 * 256)       # of the first chunk
    rows = np.tile(rng.standard_normal((128 * 16, 128)).astype(np.float32), ((pages + 40) // 16 + 1, 1))[:128 * (pages + 40)]
    k, v = rows, np.ascontiguousarray(rows[::-1])
    assert lib.cf_b200_test_llama_kv_chunk_limit(handle, 1) == 0
    assert _append(lib, handle, 0, 0, k, v) == -1 and lib.cf_b200_llama_kv_reserved_bytes(handle) == 32 << 20
    named = 0
    while lib.cf_b200_llama_kv_reference_page(handle, 0, named, C.byref(DevicePage())) == 0:
        named += 1
    launch = (1 << 20) // (4 * 128 * 128)                    # pages of a launch
    assert pages % launch != 0 and named == pages // launch * launch
    q = torch.from_numpy(rng.standard_normal((2, 1, 128)).astype(np.float32)).cuda()
    few = _attend(lib, handle, q, 128 * named - 1)
    other_lib, other = _adapter(native, 1, 128, 128, 8)
    assert _append(lib, other, 0, 0, k[:128 * named], v[:128 * named]) == 0
    assert torch.equal(few, _attend(lib, other, q, 128 * named - 1))
    assert lib.cf_b200_test_llama_kv_chunk_limit(handle, 2) == 0
    for h in (handle, other):
        assert _append(lib, h, 0, 128 * named, k[128 * named:], v[128 * named:]) == 0
    assert torch.equal(_attend(lib, handle, q, len(k) - 1), _attend(lib, other, q, len(k) - 1))
    for h in (handle, other):
        lib.cf_llama_kv_destroy(h)
