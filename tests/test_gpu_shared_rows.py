"""The shared-prefix kernel and the combine forms at the edges of their ranges: query groups that do not divide a row tile, both
head_dims, a chunk of query tokens that sees its own pages in part, groups of more than four heads of fp32 queries."""
import ctypes as C

import numpy as np
import pytest

from compat_types import DeviceKvConfig, TensorView
from helpers import attention_close
from test_gpu_device_engine import _expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim,coder,pages,seqs,f32", [
    ((14, 2), 128, "rans4", 8, 9, False), ((12, 4), 64, "huffman4", 33, 7, True), ((8, 8), 64, "rans", 17, 130, False),
    ((14, 2), 64, "huffman", 24, 19, True), ((32, 8), 64, "fixed8", 9, 40, False), ((48, 4), 128, "rans4", 16, 11, True)])
def test_shared_pages_give_what_each_sequence_alone_gives(native, heads, dim, coder, pages, seqs, f32):
    import torch
    from chromofold_b200.workloads import build_sealed_layer
    hq, hkv = heads
    layer, _ = build_sealed_layer(np.array([16 * pages] + [0] * (seqs - 1)), query_heads=hq, kv_heads=hkv, head_dim=dim, coder=coder, seed=5,
                                  extra_pages_per_sequence=pages + 2, reserve_pages=4 * seqs)
    for s in range(1, seqs):
        layer.copy_sequence(0, s)
    g = torch.Generator(device="cuda")
    g.manual_seed(6)
    for _ in range(19):     # a private page and a tail for every sequence
        k, v = ((torch.randn((seqs, hkv, dim), generator=g, device="cuda") * 0.7).half() for _ in range(2))
        layer.append(list(range(seqs)), k, v)
        layer.seal_full_pages()
    q = torch.randn((seqs, hq, dim), generator=g, device="cuda")
    q = q if f32 else q.half()
    before = native.lib().cf_b200_shared_prefix_launches()
    shared = layer.attention(q, shared_prefix_pages=pages).cpu().numpy()
    assert native.lib().cf_b200_shared_prefix_launches() == before + 1
    alone = layer.attention(q).cpu().numpy()
    assert layer.device_status() == 0
    ok, err = attention_close(shared, alone, rel=2e-5, abs_=2e-5)
    assert ok, err


@pytest.mark.parametrize("heads,dim,page,history,rows", [
    ((8, 2), 128, 128, 0, 150), ((32, 8), 128, 16, 130, 301), ((14, 2), 64, 64, 300, 70), ((12, 4), 128, 256, 1, 255), ((8, 8), 64, 32, 515, 129)])
def test_a_chunk_of_query_tokens_sees_each_token_up_to_its_own(native, oracle, heads, dim, page, history, rows):
    import torch
    lib = native.lib()
    lib.cf_device_kv_create.restype = C.c_void_p
    lib.cf_device_kv_last_error.restype = C.c_char_p
    hq, hkv = heads
    cfg = DeviceKvConfig(1, hkv, hq, dim, page, hq // hkv, 0)
    kv = C.c_void_p(lib.cf_device_kv_create(C.byref(cfg)))
    rng = np.random.default_rng(rows)
    tokens = history + rows
    k, v = (rng.standard_normal((tokens, hkv, dim)).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((rows, hq, dim)).astype(np.float32)
    dk, dv, dq = (torch.from_numpy(x).cuda() for x in (k, v, q))
    def view(t):
        return TensorView(t.data_ptr(), native.F32, *t.shape, hkv * dim * 4, dim * 4, 4, 0)

    for begin in range(0, tokens, page):
        end = min(begin + page, tokens)
        assert lib.cf_device_kv_append_async(kv, 0, begin, C.byref(view(dk[begin:end])), C.byref(view(dv[begin:end])), None) == 0
        assert lib.cf_device_kv_seal_full_pages_async(kv, None) == 0, lib.cf_device_kv_last_error(kv)
    out = torch.full((rows, hq, dim), 7.0, device="cuda")
    scale = dim ** -0.5
    assert lib.cf_device_kv_attention_async(kv, 0, C.c_void_p(dq.data_ptr()), C.c_void_p(out.data_ptr()), rows, history, C.c_float(scale), 0,
                                            None) == 0, lib.cf_device_kv_last_error(kv)
    torch.cuda.synchronize()
    some = sorted({0, 1, 15, 16, rows // 2, rows - 2, rows - 1})
    want = _expected(oracle, k, v, tokens // page * page, 16, q[some], [history + i for i in some], 0, scale, hq // hkv)
    ok, err = attention_close(out.cpu().numpy()[some], want)
    assert ok, err
    lib.cf_device_kv_destroy(kv, None)


@pytest.mark.parametrize("heads,dim,coder,f32,window", [
    ((8, 8), 80, "rans4", False, 0), ((32, 8), 80, "huffman4", True, 200), ((14, 2), 80, "rans", True, 0), ((40, 4), 80, "huffman", False, 0),
    ((6, 1), 80, "fixed8", True, 0), ((64, 8), 128, "rans4", True, 0), ((16, 1), 64, "rans", True, 77), ((24, 4), 96, "huffman4", True, 0)])
def test_lane_kernels_agree_with_the_any_geometry_kernel(native, heads, dim, coder, f32, window):
    import torch
    from chromofold_b200.workloads import build_sealed_layer
    hq, hkv = heads
    layer, _ = build_sealed_layer(np.array([16, 16 * 70, 16 * 9, 16 * 33]), query_heads=hq, kv_heads=hkv, head_dim=dim, coder=coder, seed=9)
    g = torch.Generator(device="cuda")
    g.manual_seed(10)
    tails = torch.randn((4, hkv, 16, dim), generator=g, device="cuda").half()
    layer.fill_tails([0, 1, 2, 3], tails, tails.flip(0).contiguous(), 5)
    q = torch.randn((4, hq, dim), generator=g, device="cuda")
    q = q if f32 else q.half()
    fast = layer.attention(q, kernel=native.KERNEL_LANES, causal_window=window).cpu().numpy()
    slow = layer.attention(q, kernel=native.KERNEL_GENERIC, causal_window=window).cpu().numpy()
    assert layer.device_status() == 0
    ok, err = attention_close(fast, slow, rel=2e-5, abs_=2e-5)
    assert ok, err


@pytest.mark.parametrize("heads,dim,f32,shift,shared", [
    ((8, 2), 80, True, 4, 0), ((8, 2), 80, False, 2, 0), ((14, 2), 64, True, 8, 12), ((14, 2), 64, False, 2, 12), ((8, 8), 128, True, 4, 9),
    ((32, 8), 128, False, 8, 9), ((6, 2), 96, True, 12, 0)])
def test_queries_that_begin_anywhere(native, heads, dim, f32, shift, shared):
    """The kernels that read queries 4, 8 or 16 bytes at a time are only given rows that lie so."""
    import torch
    from chromofold_b200.workloads import build_sealed_layer
    hq, hkv = heads
    layer, _ = build_sealed_layer(np.array([16 * 13, 0, 0, 0, 0]), query_heads=hq, kv_heads=hkv, head_dim=dim, seed=3, extra_pages_per_sequence=2)
    for s in range(1, 5):
        layer.copy_sequence(0, s)
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    q = torch.randn((5, hq, dim), generator=g, device="cuda")
    q = q if f32 else q.half()
    offset = shift // q.element_size()
    room = torch.zeros(q.numel() + offset, dtype=q.dtype, device="cuda")
    moved = room[offset:].view_as(q)
    moved.copy_(q)
    assert moved.data_ptr() % 16 == shift
    a, b = (layer.attention(x, shared_prefix_pages=shared).cpu().numpy() for x in (q, moved))
    assert layer.device_status() == 0
    ok, err = attention_close(b, a, rel=2e-5, abs_=2e-5)
    assert ok, err


@pytest.mark.parametrize("heads,dim,seqs,slots,coder", [((8, 2), 128, 40, 40, "rans4"), ((64, 8), 128, 24, 31, "huffman"), ((14, 2), 64, 300, 420, "rans"),
                                                        ((4, 4), 48, 30, 33, "rans4"), ((8, 8), 128, 1, 1, "rans4")])
def test_a_small_workspace_still_gives_every_sequence_a_unit(native, heads, dim, seqs, slots, coder):
    """Room for `slots` partials per query head, the fewest that are accepted or a few more: the work is cut into no fewer units than
    there are sequences, and the results are those of an ample workspace."""
    import torch
    from chromofold_b200.workloads import build_sealed_layer
    hq, hkv = heads
    rng = np.random.default_rng(seqs)
    layer, _ = build_sealed_layer(16 * rng.integers(8, 60, seqs), query_heads=hq, kv_heads=hkv, head_dim=dim, coder=coder, seed=2)
    q = torch.from_numpy(rng.standard_normal((seqs, hq, dim)).astype(np.float32)).cuda().half()
    want = layer.attention(q).cpu().numpy()
    bytes_ = (64 + 4 * (seqs + 1) + 255) // 256 * 256 + 32 * (seqs + 1) + slots * 4 * (dim + 2) * hq
    layer.workspace = torch.zeros(bytes_ + 512, dtype=torch.uint8, device="cuda")
    skip = -layer.workspace.data_ptr() % 256
    layer.workspace = layer.workspace[skip:skip + bytes_]
    got = layer.attention(q).cpu().numpy()
    assert layer.device_status() == 0
    header = layer.workspace[:28].cpu().numpy().view(np.uint32)      # positions, pages per position, stretches, ...
    assert min(seqs, 444) <= header[2] and header[2] <= max(slots, seqs)
    ok, err = attention_close(got, want, rel=2e-5, abs_=2e-5)
    assert ok, err
