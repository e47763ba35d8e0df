"""cf_llama_server_append_layer_async with whole prompts: what is stored must not depend on how the rows were cut into calls
(one call takes the bulk sealer, calls that stop short of a page the tail), a page with NaN is refused by the call that
brings it with the pages before it kept, and a server that only resets its slots reuses their memory."""
import ctypes as C

import numpy as np
import pytest

from compat_types import LlamaServerBatch, LlamaServerConfig, MsBatchItem, TensorView

pytestmark = pytest.mark.gpu
i64 = C.c_int64


class Server:
    def __init__(self, native, hq, hkv, d, page, layers=1):
        self.lib, self.hq, self.d = native.lib(), hq, d
        self.lib.cf_llama_server_runtime_create.restype = C.c_void_p
        self.lib.cf_llama_server_last_error.restype = C.c_char_p
        cfg = LlamaServerConfig(layers, hq, hkv, d, page, 64, 1 << 20, hq // hkv, 0, 1, None, b"test", b"0" * 64)
        self.rt = C.c_void_p(self.lib.cf_llama_server_runtime_create(C.byref(cfg)))
        assert self.rt.value

    def append(self, slot, k, v, begin, layer=0):
        return self.lib.cf_llama_server_append_layer_async(self.rt, i64(slot), layer, begin, C.c_void_p(k[begin:].data_ptr()),
                                                           C.c_void_p(v[begin:].data_ptr()), k.shape[0] - begin, None)

    def attend(self, slot, q, position, layer=0):
        import torch
        out = torch.full_like(q, 7.0)
        it = MsBatchItem()
        it.sequence_id, it.layer = slot, layer
        it.query = TensorView(q.data_ptr(), 3, q.shape[0], self.hq, self.d, self.hq * self.d * 4, self.d * 4, 4, 0)
        it.output, it.output_type = out.data_ptr(), 3
        it.output_token_stride_bytes, it.output_head_stride_bytes, it.output_element_stride_bytes = self.hq * self.d * 4, self.d * 4, 4
        it.query_token_begin, it.softmax_scale, it.causal_window = position, 1.0 / np.sqrt(self.d), 0
        batch = LlamaServerBatch(None, 0, C.cast(C.byref(it), C.c_void_p), 1)
        assert self.lib.cf_llama_server_execute_batch_async(self.rt, C.byref(batch), None) == 0, self.error()
        torch.cuda.synchronize()
        return out

    def error(self):
        return self.lib.cf_llama_server_last_error(self.rt)


def _rows(n, hkv, d, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return [torch.randn((n, hkv, d), generator=g, device="cuda") for _ in range(2)]


@pytest.mark.parametrize("shape", [(8, 2, 128, 64), (14, 2, 64, 16), (4, 4, 128, 16), (4, 2, 96, 32), (4, 2, 48, 32)], ids=str)
def test_one_call_stores_what_many_calls_store(native, shape):
    import torch
    hq, hkv, d, page = shape
    tokens = 9 * page + 5
    k, v = _rows(tokens, hkv, d, 3)
    server = Server(native, hq, hkv, d, page)
    cuts = {1: [tokens], 2: [page // 2, 3 * page, 3 * page + 1, tokens], 3: list(range(page // 4, tokens, page // 4)) + [tokens]}
    q = torch.randn((1, hq, d), device="cuda")
    outs = []
    for slot, ends in cuts.items():
        assert server.lib.cf_llama_server_slot_create(server.rt, i64(slot)) == 0
        begin = 0
        for end in ends:
            assert server.append(slot, k[:end], v[:end], begin) == 0, server.error()
            begin = end
        outs.append(server.attend(slot, q, tokens))
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert server.append(1, k, v, tokens - 1) == -1   # not contiguous
    server.lib.cf_llama_server_runtime_destroy(server.rt, None)


def test_a_refused_page_keeps_the_pages_before_it(native):
    import torch
    hq, hkv, d, page = 8, 2, 128, 16
    k, v = _rows(8 * page, hkv, d, 4)
    bad = v.clone()
    bad[5 * page + 3, 1, 17] = float("inf")
    server = Server(native, hq, hkv, d, page)
    for slot in (1, 2):
        assert server.lib.cf_llama_server_slot_create(server.rt, i64(slot)) == 0
    assert server.append(1, k, bad, 0) == -1 and server.error() == b"page contains NaN or Inf"
    assert server.append(2, k[:5 * page], v[:5 * page], 0) == 0
    q = torch.randn((1, hq, d), device="cuda")
    assert torch.equal(server.attend(1, q, 5 * page - 1), server.attend(2, q, 5 * page - 1))   # the refused rows come later
    assert server.append(1, k, v, 6 * page) == -1   # its page is full and was not sealed
    server.lib.cf_llama_server_runtime_destroy(server.rt, None)


def test_reset_slots_are_reused_without_a_reclaim_call(native):
    import torch
    hq, hkv, d, page = 8, 8, 128, 64
    k, v = _rows(4 * page, hkv, d, 5)
    server = Server(native, hq, hkv, d, page)
    q, first = torch.randn((1, hq, d), device="cuda"), None
    free = None
    for i in range(120):   # 120 requests of 0.5 MB: the 16 MB the arena starts with, many times over
        assert server.lib.cf_llama_server_slot_create(server.rt, i64(1)) == 0
        assert server.append(1, k, v, 0) == 0, server.error()
        out = server.attend(1, q, 4 * page)
        first = out if first is None else first
        assert torch.equal(out, first)
        assert server.lib.cf_llama_server_slot_reset_async(server.rt, i64(1), None) == 0
        if i == 60:
            free = torch.cuda.mem_get_info()[0]
    assert torch.cuda.mem_get_info()[0] >= free - (4 << 20)
    server.lib.cf_llama_server_runtime_destroy(server.rt, None)


@pytest.mark.parametrize("shift", [1, 2, 0])
def test_outputs_may_overlap_the_queries_of_the_batch(native, shift):
    """Queries and outputs in one buffer, `shift` rows apart: every query is read before any output is written."""
    import torch
    hq, hkv, d, page, layers = 8, 2, 128, 16, 4
    server = Server(native, hq, hkv, d, page, layers)
    assert server.lib.cf_llama_server_slot_create(server.rt, i64(1)) == 0
    for layer in range(layers):
        k, v = _rows(40, hkv, d, 20 + layer)
        assert server.append(1, k, v, 0, layer) == 0, server.error()
    g = torch.Generator(device="cuda")
    g.manual_seed(6)
    q = torch.randn((layers, hq, d), generator=g, device="cuda")
    alone = torch.cat([server.attend(1, q[layer:layer + 1].contiguous(), 40, layer) for layer in range(layers)])
    room = torch.zeros((layers + shift, hq, d), device="cuda")
    room[:layers] = q
    items = (MsBatchItem * layers)()
    for i, it in enumerate(items):
        it.sequence_id, it.layer = 1, i
        it.query = TensorView(room[i].data_ptr(), 3, 1, hq, d, hq * d * 4, d * 4, 4, 0)
        it.output, it.output_type = room[i + shift].data_ptr(), 3
        it.output_token_stride_bytes, it.output_head_stride_bytes, it.output_element_stride_bytes = hq * d * 4, d * 4, 4
        it.query_token_begin, it.softmax_scale, it.causal_window = 40, 1.0 / np.sqrt(d), 0
    batch = LlamaServerBatch(None, 0, C.cast(items, C.c_void_p), layers)
    assert server.lib.cf_llama_server_execute_batch_async(server.rt, C.byref(batch), None) == 0, server.error()
    torch.cuda.synchronize()
    assert torch.equal(room[shift:], alone)
    server.lib.cf_llama_server_runtime_destroy(server.rt, None)


@pytest.mark.parametrize("rows,position", [(1, 0xffffffff), (8, 3_000_000_000), (40, 0x7fffffe0), (2, 0xfffffffe)])
def test_positions_far_beyond_the_context_see_all_of_it(native, rows, position):
    import torch
    hq, hkv, d, page = 8, 2, 128, 16
    server = Server(native, hq, hkv, d, page)
    assert server.lib.cf_llama_server_slot_create(server.rt, i64(1)) == 0
    k, v = _rows(300, hkv, d, 30)
    assert server.append(1, k, v, 0) == 0, server.error()
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    q = torch.randn((rows, hq, d), generator=g, device="cuda")
    near, far = server.attend(1, q, 300), server.attend(1, q, position)
    assert torch.equal(near, far)
    server.lib.cf_llama_server_runtime_destroy(server.rt, None)
