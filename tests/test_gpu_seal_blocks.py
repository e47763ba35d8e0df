"""The warp-per-page sealer (csrc/seal_blocks.cu) byte for byte against the oracle where its branches begin and end: every
head_dim it is built for, ragged rows, streams that fall back to fixed width, quotients next to a half-integer, scales in the
binary16 denormals (the clamp decides), more pages than one pass of the grid."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(rng, kind, shape):
    if kind == "noise":          # incompressible: the entropy coders give way to fixed width
        return (rng.integers(-127, 128, shape) * 0.01).astype(np.float32)
    if kind == "halves":         # quotients on and next to half-integers
        x = (rng.integers(-120, 120, shape) + 0.5 + rng.choice([0, 1e-5, -1e-5, 3e-5], shape)) * 0.0078125
        x.reshape(-1)[0] = 127 * 0.0078125
        return x.astype(np.float32)
    if kind == "tiny":           # absmax / 127 far below the smallest normal binary16
        return (rng.standard_normal(shape) * 3e-6).astype(np.float32)
    return (np.rint(rng.laplace(0, 9, shape)).clip(-127, 127) * 0.01).astype(np.float32)


@pytest.mark.parametrize("d", [128, 96, 80, 64, 32])
@pytest.mark.parametrize("coder", range(5))
def test_blocks_are_sealed_byte_for_byte(native, oracle, d, coder):
    import torch
    from chromofold_b200.cache import SealedKvLayer
    from helpers import hist_for_coder, laplace_codes
    rng = np.random.default_rng(10 * d + coder)
    kinds, hkv = ["codes", "noise", "halves", "tiny", "codes"], 3
    rows = [16, 16, 16, 7, 1]
    n = len(kinds)
    hist = hist_for_coder(laplace_codes(rng, 1 << 15, 9.0).astype(np.int16) + 128, coder)
    kcb = oracle.codebook_from_hist(hist)
    layer = SealedKvLayer(kv_heads=hkv, query_heads=3, head_dim=d, page_tokens=16, block_size=64, coder=coder, max_sequences=n,
                          max_pages_per_sequence=4, max_pages=64, arena_bytes=2 << 20)
    layer.set_codebooks(hist, hist)
    for f32 in (True, False):
        k, v = (np.stack([_values(rng, kind, (hkv, 16, d)) for kind in kinds]) for _ in range(2))
        if not f32:
            k, v = k.astype(np.float16).astype(np.float32), v.astype(np.float16).astype(np.float32)
        dk, dv = (torch.from_numpy(x if f32 else x.astype(np.float16)).cuda() for x in (k, v))
        desc = layer._seal_desc(torch.arange(n, dtype=torch.int32, device="cuda"), torch.arange(1, n + 1, dtype=torch.int32, device="cuda"),
                                torch.as_tensor(rows, dtype=torch.int32, device="cuda"))
        desc.tail_k, desc.tail_v, desc.tail_type = dk.data_ptr(), dv.data_ptr(), native.F32 if f32 else native.F16
        assert native.lib().cf_b200_seal_pages_async(C.byref(desc), None) == 0
        torch.cuda.synchronize()
        assert layer.device_status() == 0
        for s in range(n):
            for h in range(hkv):
                want = oracle.seal_record(k[s, h, :rows[s]], v[s, h, :rows[s]], rows[s], d, 16, 64, coder, 0, kcb, kcb)[0]
                assert np.array_equal(layer.record_bytes(s + 1, h), want), (f32, kinds[s], h)


def test_more_pages_than_warps_and_odd_head_counts(native):
    """Every page-head of a launch is sealed exactly once whatever the grid's stride: all decode to the symbols they hold."""
    import torch
    from chromofold_b200.cache import SealedKvLayer
    n, hkv, d = 1100, 7, 128
    layer = SealedKvLayer(kv_heads=hkv, query_heads=7, head_dim=d, page_tokens=16, block_size=64, coder=0, max_sequences=1,
                          max_pages_per_sequence=n, max_pages=n + 1, arena_bytes=n * hkv * 4112 + 4096)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    codes = torch.randint(-126, 127, (2, n, hkv, 16, d), generator=g, device="cuda").float()
    codes[:, :, :, 0, 0] = 127
    layer.seal_tiles(np.zeros(n, np.int64), (codes[0] * 0.0078125).half(), (codes[1] * 0.0078125).half())
    assert layer.device_status() == 0
    k, v = layer.decode_pages(np.arange(1, n + 1))
    assert torch.equal(k, (codes[0] + 128).to(torch.uint8).reshape(n, hkv, -1))
    assert torch.equal(v, (codes[1] + 128).to(torch.uint8).transpose(-1, -2).reshape(n, hkv, -1))


@pytest.mark.parametrize("coder", range(5))
@pytest.mark.parametrize("f32", [False, True])
def test_few_page_heads_and_many_are_sealed_alike(native, coder, f32):
    """Two warps share a page-head where a launch has few of them: the same records as of a launch with many, refusals (NaN in K or V
    alone, no rows, no room in the arena) included."""
    import torch
    from chromofold_b200.cache import SealedKvLayer
    from helpers import hist_for_coder, laplace_codes
    n, hkv, d = 400, 8, 128
    rng = np.random.default_rng(coder)
    hist = hist_for_coder(laplace_codes(rng, 1 << 15, 9.0).astype(np.int16) + 128, coder)
    kinds = ["codes", "noise", "halves", "tiny"]
    k, v = (np.stack([_values(rng, kinds[i % 4], (hkv, 16, d)) for i in range(n)]) for _ in range(2))
    k[10, 3, 2, 5], v[11, 0, 15, 127] = np.nan, np.inf
    rows = rng.integers(1, 17, n)
    rows[[10, 11]], rows[12] = 16, 0
    dk, dv = (torch.from_numpy(x if f32 else x.astype(np.float16)).cuda() for x in (k, v))
    layers = []
    for step in (n, 29, 1):
        layer = SealedKvLayer(kv_heads=hkv, query_heads=hkv, head_dim=d, page_tokens=16, block_size=64, coder=coder, max_sequences=1,
                              max_pages_per_sequence=n, max_pages=n + 1, arena_bytes=n * hkv * 4112 + 4096)
        layer.set_codebooks(hist, hist)
        for begin in range(0, n if step > 1 else 40, step):
            jobs = torch.arange(begin, min(begin + step, n), dtype=torch.int32, device="cuda")
            desc = layer._seal_desc(jobs, jobs + 1, torch.as_tensor(rows[begin:begin + step], dtype=torch.int32, device="cuda"))
            desc.tail_k, desc.tail_v, desc.tail_type = dk.data_ptr(), dv.data_ptr(), native.F32 if f32 else native.F16
            assert native.lib().cf_b200_seal_pages_async(C.byref(desc), None) == 0
        torch.cuda.synchronize()
        assert layer.device_status() == native.DEVSTAT_NONFINITE
        layers.append(layer)
    directory = [layer.page_dir.cpu().numpy().reshape(-1, hkv) for layer in layers]
    missing = {(11, 3), (12, 0)} | {(13, h) for h in range(hkv)}
    for page in list(range(1, 41)) + [57, 399, 400]:
        for h in range(hkv):
            there = [bool(x[page, h]) for x in directory[:2]] + [bool(directory[2][page, h])] * (page <= 40)
            assert all(t == ((page, h) not in missing) for t in there), (page, h)
            if there[0]:
                records = [layer.record_bytes(page, h) for layer in layers[:2 + (page <= 40)]]
                assert all(np.array_equal(records[0], r) for r in records[1:])
    layer = layers[2]      # room for some of the records of one more launch
    layer.status.zero_()
    layer.cursor.fill_(layer.arena_units - 1000)
    layer.page_dir.zero_()
    jobs = torch.arange(20, dtype=torch.int32, device="cuda")
    desc = layer._seal_desc(jobs, jobs + 1, torch.full((20,), 16, dtype=torch.int32, device="cuda"))
    desc.tail_k, desc.tail_v, desc.tail_type = dk.data_ptr(), dv.data_ptr(), native.F32 if f32 else native.F16
    assert native.lib().cf_b200_seal_pages_async(C.byref(desc), None) == 0
    torch.cuda.synchronize()
    assert layer.device_status() & native.DEVSTAT_ARENA_FULL
    entries = layer.page_dir.cpu().numpy()
    assert 0 < np.count_nonzero(entries) < 20 * hkv
