"""The llama.cpp adapter called on several streams: whatever stream a call names, it comes after the appends before it, and an append
after the attention calls before it."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_paged_mma import _adapter

pytestmark = pytest.mark.gpu
HEADS, D, PAGE = 2, 64, 16


class _Calls:
    """One adapter and a fixed sequence of rows; `late` puts 40 ms of other work in front of the calls that ask for it, and then
    nothing waits for the GPU; otherwise every call ends before the next."""

    def __init__(self, native, late):
        import torch
        self.torch, self.late = torch, late
        self.lib, self.handle = _adapter(native, HEADS, D, PAGE, 8)
        self.streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        rng = np.random.default_rng(2)
        self.k, self.v = (rng.standard_normal((HEADS, 400, D)).astype(np.float32) for _ in range(2))
        self.q = torch.from_numpy(rng.standard_normal((1, HEADS, D)).astype(np.float32)).cuda()
        self.outs, self.at = [], 0
        torch.cuda.synchronize()

    def _delay(self, stream, late):
        if self.late and late:
            with self.torch.cuda.stream(stream):
                self.torch.cuda._sleep(80_000_000)

    def append(self, on, rows, late=False):
        s = self.streams[on]
        self._delay(s, late)
        for h in range(HEADS):
            kk, vv = self.k[h, self.at:], self.v[h, self.at:]
            assert self.lib.cf_llama_kv_append(self.handle, 0, h, self.at, C.c_void_p(kk.ctypes.data), C.c_void_p(vv.ctypes.data), rows,
                                               C.c_void_p(s.cuda_stream)) == 0
        self.at += rows
        if not self.late:
            self.torch.cuda.synchronize()

    def attend(self, on, late=False):
        s = self.streams[on]
        out = self.torch.zeros_like(self.q)
        s.wait_stream(self.torch.cuda.current_stream())   # for the zeros
        self._delay(s, late)
        assert self.lib.cf_llama_kv_attention(self.handle, 0, C.c_void_p(self.q.data_ptr()), C.c_void_p(out.data_ptr()), 1, HEADS, 1, self.at - 1,
                                              C.c_float(D ** -0.5), 0, C.c_void_p(s.cuda_stream)) == 0
        self.outs.append(out)
        if not self.late:
            self.torch.cuda.synchronize()


STORIES = {
    "a tail row on one stream, attention on the other": [("append", 0, 20), ("append", 0, 1, True), ("attend", 1)],
    "a tail row on one stream, the page it belongs to filled on the other": [("append", 0, 20), ("append", 0, 3, True), ("append", 1, 12), ("attend", 1)],
    "pages on one stream, attention on the other": [("append", 0, 5), ("append", 0, 90, True), ("attend", 1)],
    "attention on one stream, the tail it reads replaced on the other": [("append", 0, 20), ("attend", 0, True), ("append", 1, 30), ("attend", 1)],
    "two readers, then a writer on neither's turn": [("append", 0, 9), ("attend", 1, True), ("attend", 0), ("append", 0, 39), ("attend", 1)],
}


@pytest.mark.parametrize("story", STORIES)
def test_calls_on_two_streams_take_effect_in_their_order(native, story):
    import torch
    got, want = _Calls(native, True), _Calls(native, False)
    for calls in (want, got):
        for name, *args in STORIES[story]:
            getattr(calls, name)(*args)
        torch.cuda.synchronize()
        calls.lib.cf_llama_kv_destroy(calls.handle)
    for a, b in zip(got.outs, want.outs):
        assert torch.equal(a, b)


def test_attention_after_an_append_on_another_stream_can_be_captured(native):
    import torch
    calls = _Calls(native, True)
    calls.append(0, 20, late=True)
    out = torch.zeros_like(calls.q)
    graph, side = torch.cuda.CUDAGraph(), calls.streams[1]
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        graph.capture_begin()
        rc = calls.lib.cf_llama_kv_attention(calls.handle, 0, C.c_void_p(calls.q.data_ptr()), C.c_void_p(out.data_ptr()), 1, HEADS, 1, 19,
                                             C.c_float(D ** -0.5), 0, C.c_void_p(side.cuda_stream))
        graph.capture_end()
    assert rc == 0
    graph.replay()
    torch.cuda.synchronize()
    calls.attend(1)
    torch.cuda.synchronize()
    # one launch under capture, splits outside of it: the same sums in another order
    assert torch.allclose(out, calls.outs[0], rtol=1e-5, atol=1e-6) and float(out.abs().max()) > 0
    calls.append(0, 30)      # the captured call left nothing behind that a later one would trip over
    calls.attend(0)
    torch.cuda.synchronize()
    calls.lib.cf_llama_kv_destroy(calls.handle)


@pytest.mark.parametrize("rows", [[1, 14, 1], [3, 45], [70], [5, 2]], ids=str)
def test_rows_in_pinned_memory_are_read_in_stream_order(native, rows):
    """Rows that the stream's earlier work is still to put into pinned memory (a copy from the GPU, as a model's projections come)."""
    import torch
    calls, want = _Calls(native, True), _Calls(native, False)
    stream, held = calls.streams[0], []
    for n in rows:
        want.append(0, n)
        for h in range(HEADS):
            source = [torch.from_numpy(x[h, calls.at:calls.at + n]).cuda() for x in (calls.k, calls.v)]
            pinned = [torch.full((n, D), float("nan")).pin_memory() for _ in source]
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                torch.cuda._sleep(20_000_000)
                for a, b in zip(pinned, source):
                    a.copy_(b, non_blocking=True)
            held.append((source, pinned))
            assert calls.lib.cf_llama_kv_append(calls.handle, 0, h, calls.at, C.c_void_p(pinned[0].data_ptr()), C.c_void_p(pinned[1].data_ptr()), n,
                                                C.c_void_p(stream.cuda_stream)) == 0
        calls.at += n
    for c in (calls, want):
        c.attend(0)
        assert c.lib.cf_llama_kv_flush(c.handle, C.c_void_p(c.streams[0].cuda_stream)) == 0
        c.attend(0)
        torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(calls.outs, want.outs))
    bad = torch.zeros((40, D)).pin_memory()          # pages before a refused one stay, as with rows in pageable memory
    bad[25, 3] = float("inf")
    for c, rows in ((calls, bad.data_ptr()), (want, bad.numpy().copy())):
        ptr = C.c_void_p(rows if c is calls else rows.ctypes.data)
        begin = c.at
        assert c.lib.cf_llama_kv_append(c.handle, 0, 0, begin, ptr, ptr, 40, C.c_void_p(c.streams[0].cuda_stream)) == -1
    from compat_types import LlamaKvStats
    stats = [LlamaKvStats() for _ in range(2)]
    assert calls.lib.cf_llama_kv_get_stats(calls.handle, C.byref(stats[0])) == 0 and calls.lib.cf_llama_kv_get_stats(want.handle, C.byref(stats[1])) == 0
    assert bytes(stats[0]) == bytes(stats[1])
    for c in (calls, want):
        c.lib.cf_llama_kv_destroy(c.handle)


def test_rows_in_device_memory_are_taken_too(native):
    import torch
    calls, want = _Calls(native, False), _Calls(native, False)
    k, v = (torch.from_numpy(x).cuda() for x in (calls.k, calls.v))
    for n in (3, 40):
        want.append(0, n)
        for h in range(HEADS):
            assert calls.lib.cf_llama_kv_append(calls.handle, 0, h, calls.at, C.c_void_p(k[h, calls.at:].data_ptr()), C.c_void_p(v[h, calls.at:].data_ptr()),
                                                n, C.c_void_p(calls.streams[0].cuda_stream)) == 0
        calls.at += n
    for c in (calls, want):
        c.attend(0)
        c.lib.cf_llama_kv_destroy(c.handle)
    assert torch.equal(calls.outs[0], want.outs[0])
