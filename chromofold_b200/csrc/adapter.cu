// adapter.cu — the llama.cpp-facing KV adapter (include/chromofold_b200/compat_adapter.h) on top of the sealed-KV
// entry points. Host logic mirrors the reference's adapter and single-sequence cache
// (integrations/llama.cpp/chromofold_kv_adapter.cpp, src/runtime/compressed_kv_cache.cu) — same checks, same error
// strings where a caller could match on them — while every byte of KV lives on the GPU: appended rows go straight
// into a device tail, full tiles are sealed by cf_b200_seal_pages_async, attention is cf_b200_sealed_attention_async.

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "attention_params.cuh"
#include "copy_helpers.h"
#include "host_rows.h"
#include "chromofold_b200/compat_adapter.h"
#include "chromofold_b200/compat_kv.h"
#include "chromofold_b200/sealed_kv.h"

namespace {

void cuda_check(cudaError_t e, const char *what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

template <class T>
struct DeviceBuffer {  // grow-only device array; growing copies the old contents (set-up and append path only)
    T *ptr = nullptr;
    size_t count = 0;
    ~DeviceBuffer() { if (ptr) cudaFree(ptr); }
    void ensure(size_t wanted, cudaStream_t s) {
        if (wanted <= count) return;
        size_t next = std::max(wanted, count ? count * 2 : wanted);
        T *fresh = nullptr;
        cuda_check(cudaMalloc(reinterpret_cast<void **>(&fresh), next * sizeof(T)), "cudaMalloc");
        cuda_check(cudaMemsetAsync(fresh, 0, next * sizeof(T), s), "cudaMemsetAsync");
        if (ptr) {
            cuda_check(cudaMemcpyAsync(fresh, ptr, count * sizeof(T), cudaMemcpyDeviceToDevice, s), "cudaMemcpyAsync");
            cuda_check(cudaStreamSynchronize(s), "cudaStreamSynchronize");
            cudaFree(ptr);
        }
        ptr = fresh;
        count = next;
    }
};

// ---- the reference's own page quantiser on the GPU ---------------------------------------------------------------
// What the reference's adapter stores for kv_bits 4 / 8 (integrations/llama.cpp/chromofold_kv_adapter.cpp:30-31) is what
// gpu_fixture::encode_int{4,8}_page makes on the host (src/runtime/kv_gpu_fixture.cpp:46-95): K with one fp32 scale per
// channel, V with one per token, scale = absmax / qmax (1 when the row or column is all zero), symbol =
// clamp(lrint(x / scale), -(qmax+1), qmax) + 2^(bits-1), symbols packed MSB-first at `bits` bits, block offsets
// b * 64 * bits, the LUT s | bits << 8. The kernel below makes the same page, bit for bit, from rows already on the GPU.
struct KiviLayout {
    size_t k_words, v_words, k_scales, v_scales, k_offsets, v_offsets, total;   // byte offsets inside a page block
    uint32_t word_count, block_count;
};
inline KiviLayout kivi_layout(uint32_t tokens, uint32_t dim, uint32_t bits) {
    KiviLayout l{};
    const uint64_t symbols = static_cast<uint64_t>(tokens) * dim;
    l.word_count = static_cast<uint32_t>((symbols * bits + 31u) / 32u);
    l.block_count = static_cast<uint32_t>((symbols + 63u) / 64u);
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t here = at; at += (bytes + 15u) / 16u * 16u; return here; };
    l.k_words = take(4ull * l.word_count);
    l.v_words = take(4ull * l.word_count);
    l.k_scales = take(4ull * dim);
    l.v_scales = take(4ull * tokens);
    l.k_offsets = take(4ull * l.block_count);
    l.v_offsets = take(4ull * l.block_count);
    l.total = at;
    return l;
}

// The pages of one append: rows are numbered from the first unsealed one; the first tail_rows of them are already in the
// tail ([token][row_stride floats], this head's `dim` values first in each row), the others just arrived in the stage
// ([token][dim]). CTA p makes page p of rows p * tokens ..; the rows after the last page become the new tail.
constexpr uint32_t kKiviPagesPerLaunch = 64;
struct KiviJob {
    const float *stage_k, *stage_v;
    float *tail_k, *tail_v;
    uint32_t row_stride, tail_rows, tokens, dim, bits, pages, rest_rows;
    cf_kv_device_page *pages_out;              // descriptor of page p goes to pages_out[p]
    cf_kv_device_page page;                    // what those of all pages have in common; token_begin is page 0's
    uint8_t *block[kKiviPagesPerLaunch];
};

// Bound: latency of two passes over a page (64 KB + 64 KB at 128 x 128, the second out of L1) and, on one SM per page, an
// IEEE division per value. 32 warps, a token per warp and four channels per lane, so that a pass is a handful of
// independent 16-byte loads per thread: 50 us with 256 threads that walked the tokens of a channel one by one, 14 us now.
__global__ void __launch_bounds__(1024) kivi_quantise_kernel(const __grid_constant__ KiviJob job, KiviLayout lay) {
    extern __shared__ uint32_t magnitudes[];   // [dim] K | [tokens] V absmax as float bits, then the scales in their place
    const uint32_t tokens = job.tokens, dim = job.dim, bits = job.bits, page = blockIdx.x, first_row = page * tokens;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    uint32_t *k_mag = magnitudes, *v_mag = magnitudes + dim;
    const int qmax = (1 << (bits - 1)) - 1, zero = 1 << (bits - 1);
    auto k_row = [&](uint32_t t) {
        const uint32_t r = first_row + t;
        return r < job.tail_rows ? job.tail_k + static_cast<size_t>(r) * job.row_stride : job.stage_k + static_cast<size_t>(r - job.tail_rows) * dim;
    };
    auto v_row = [&](uint32_t t) {
        const uint32_t r = first_row + t;
        return r < job.tail_rows ? job.tail_v + static_cast<size_t>(r) * job.row_stride : job.stage_v + static_cast<size_t>(r - job.tail_rows) * dim;
    };
    for (uint32_t i = threadIdx.x; i < dim; i += blockDim.x) k_mag[i] = 0u;
    __syncthreads();
    const bool quads = dim % 4u == 0 && dim <= 128u;   // rows are 16-byte aligned then
    if (quads) {
        uint32_t km[4] = {0u, 0u, 0u, 0u};
#pragma unroll 4
        for (uint32_t t = warp; t < tokens; t += warps) {
            uint32_t vm = 0u;
            if (4u * lane < dim) {
                const uint4 k = *reinterpret_cast<const uint4 *>(k_row(t) + 4u * lane), v = *reinterpret_cast<const uint4 *>(v_row(t) + 4u * lane);
                km[0] = max(km[0], k.x & 0x7fffffffu), km[1] = max(km[1], k.y & 0x7fffffffu);
                km[2] = max(km[2], k.z & 0x7fffffffu), km[3] = max(km[3], k.w & 0x7fffffffu);
                vm = max(max(v.x & 0x7fffffffu, v.y & 0x7fffffffu), max(v.z & 0x7fffffffu, v.w & 0x7fffffffu));
            }
            vm = __reduce_max_sync(0xffffffffu, vm);
            if (lane == 0) v_mag[t] = vm;
        }
        if (4u * lane < dim)
            for (int j = 0; j < 4; ++j) atomicMax(&k_mag[4u * lane + j], km[j]);
    } else {
        for (uint32_t t = warp; t < tokens; t += warps) {
            uint32_t vm = 0u;
            for (uint32_t d = lane; d < dim; d += 32u) {
                atomicMax(&k_mag[d], __float_as_uint(k_row(t)[d]) & 0x7fffffffu);
                vm = max(vm, __float_as_uint(v_row(t)[d]) & 0x7fffffffu);
            }
            vm = __reduce_max_sync(0xffffffffu, vm);
            if (lane == 0) v_mag[t] = vm;
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < dim + tokens; i += blockDim.x) {   // dim K channels, then tokens V rows
        const uint32_t m = magnitudes[i];
        const float scale = m == 0u ? 1.0f : __fdiv_rn(__uint_as_float(m), static_cast<float>(qmax));
        magnitudes[i] = __float_as_uint(scale);
    }
    __syncthreads();
    const float *k_scale = reinterpret_cast<const float *>(k_mag), *v_scale = reinterpret_cast<const float *>(v_mag);
    const uint32_t per_word = 32u / bits;
    uint8_t *block = job.block[page];
    uint32_t *kw = reinterpret_cast<uint32_t *>(block + lay.k_words), *vw = reinterpret_cast<uint32_t *>(block + lay.v_words);
    // lrint(x / scale), clamped. x * (1 / scale) is within 1.5 * 2^-23 * |q| of the quotient, so where it is further than 2^-14
    // from every half-integer both round alike, and only the few values closer than that take the division.
    auto symbol = [&](float x, float scale, float rcp) {
        float y = x * rcp, n = rintf(y);
        if (!(fabsf(fabsf(y - n) - 0.5f) >= 6.103515625e-05f) || rcp > 1e37f) n = rintf(__fdiv_rn(x, scale));
        return static_cast<uint32_t>(max(-(qmax + 1), min(qmax, __float2int_rn(n))) + zero);
    };
    if (quads && dim % per_word == 0) {   // a word is four or eight channels of one token
        const uint32_t row_words = dim / per_word;
        for (uint32_t w = threadIdx.x; w < lay.word_count; w += blockDim.x) {
            const uint32_t t = w / row_words, d0 = (w % row_words) * per_word;
            const float *k = k_row(t) + d0, *v = v_row(t) + d0;
            const float vs = v_scale[t], vr = __frcp_rn(vs);
            uint32_t kword = 0, vword = 0;
            for (uint32_t j = 0; j < per_word; j += 4u) {
                const float4 a = *reinterpret_cast<const float4 *>(k + j), b = *reinterpret_cast<const float4 *>(v + j);
                const float *ks = k_scale + d0 + j;
                const uint32_t ks4[4] = {symbol(a.x, ks[0], __frcp_rn(ks[0])), symbol(a.y, ks[1], __frcp_rn(ks[1])),
                                         symbol(a.z, ks[2], __frcp_rn(ks[2])), symbol(a.w, ks[3], __frcp_rn(ks[3]))};
                const uint32_t vs4[4] = {symbol(b.x, vs, vr), symbol(b.y, vs, vr), symbol(b.z, vs, vr), symbol(b.w, vs, vr)};
#pragma unroll
                for (int c = 0; c < 4; ++c) kword = kword << bits | ks4[c], vword = vword << bits | vs4[c];
            }
            kw[w] = kword;
            vw[w] = vword;
        }
    } else {
        const uint64_t symbols = static_cast<uint64_t>(tokens) * dim;
        for (uint32_t w = threadIdx.x; w < lay.word_count; w += blockDim.x) {
            uint32_t kword = 0, vword = 0;
            for (uint32_t j = 0; j < per_word; ++j) {
                const uint64_t i = static_cast<uint64_t>(w) * per_word + j;
                if (i >= symbols) break;
                const uint32_t t = static_cast<uint32_t>(i / dim), d = static_cast<uint32_t>(i % dim);
                const uint32_t shift = (32u - bits) - j * bits;
                kword |= symbol(k_row(t)[d], k_scale[d], __frcp_rn(k_scale[d])) << shift;
                vword |= symbol(v_row(t)[d], v_scale[t], __frcp_rn(v_scale[t])) << shift;
            }
            kw[w] = kword;
            vw[w] = vword;
        }
    }
    for (uint32_t d = threadIdx.x; d < dim; d += blockDim.x) reinterpret_cast<float *>(block + lay.k_scales)[d] = k_scale[d];
    for (uint32_t t = threadIdx.x; t < tokens; t += blockDim.x) reinterpret_cast<float *>(block + lay.v_scales)[t] = v_scale[t];
    for (uint32_t b = threadIdx.x; b < lay.block_count; b += blockDim.x) {
        reinterpret_cast<int32_t *>(block + lay.k_offsets)[b] = static_cast<int32_t>(b * 64u * bits);
        reinterpret_cast<int32_t *>(block + lay.v_offsets)[b] = static_cast<int32_t>(b * 64u * bits);
    }
    if (threadIdx.x == 0) {
        cf_kv_device_page d = job.page;
        d.k_words = kw;
        d.v_words = vw;
        d.k_scales = reinterpret_cast<const float *>(block + lay.k_scales);
        d.v_scales = reinterpret_cast<const float *>(block + lay.v_scales);
        d.k_block_offsets = reinterpret_cast<const int32_t *>(block + lay.k_offsets);
        d.v_block_offsets = reinterpret_cast<const int32_t *>(block + lay.v_offsets);
        d.token_begin += page * tokens;
        job.pages_out[page] = d;
    }
    if (page != 0) return;
    __syncthreads();   // the tail's old rows have been read: the rows after the last page take their place
    const uint32_t from = job.pages * tokens - job.tail_rows;
    for (uint32_t i = threadIdx.x; i < job.rest_rows * dim; i += blockDim.x) {
        const size_t at = static_cast<size_t>(i / dim) * job.row_stride + i % dim;
        job.tail_k[at] = job.stage_k[static_cast<size_t>(from) * dim + i];
        job.tail_v[at] = job.stage_v[static_cast<size_t>(from) * dim + i];
    }
}

// *first_bad = the smallest of itself and the numbers (from `first` on) of the rows that hold NaN or Inf. A warp per row.
__global__ void __launch_bounds__(256) first_bad_row_kernel(const float *k, const float *v, size_t row_stride, uint32_t dim, uint32_t rows, uint32_t first,
                                                            uint32_t *first_bad) {
    const uint32_t row = blockIdx.x * (blockDim.x / 32u) + threadIdx.x / 32u;
    if (row >= rows) return;
    bool bad = false;
    for (uint32_t d = threadIdx.x % 32u; d < dim; d += 32u) bad = bad || !isfinite(k[row * row_stride + d]) || !isfinite(v[row * row_stride + d]);
    if (__any_sync(0xffffffffu, bad) && threadIdx.x % 32u == 0) atomicMin(first_bad, first + row);
}

// Whether a copy reads this memory in stream order (pinned, managed and device memory): what it holds when the call is
// made need not be what the stream's earlier work will have put there, and the host may not be able to look at it.
bool in_stream_order(const void *ptr) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, ptr) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}

// Copies `rows` rows of `dim` floats and returns the first that holds NaN or Inf, or `rows`.
uint32_t copy_rows_checked(cfb::CopyHelpers &helpers, float *dst, const float *src, uint32_t rows, uint32_t dim) {
    if (helpers.copy(dst, src, static_cast<size_t>(rows) * dim) < 0x7f800000u) return rows;   // inf and NaN lie above every finite magnitude
    uint32_t r = 0;
    while (chromofold_copy_max_magnitude(dst + static_cast<size_t>(r) * dim, src + static_cast<size_t>(r) * dim, dim) < 0x7f800000u) ++r;
    return r;
}

uint32_t first_bad_row(const float *src, uint32_t rows, uint32_t dim) {
    uint32_t r = 0;
    while (r < rows && chromofold_max_magnitude(src + static_cast<size_t>(r) * dim, dim) < 0x7f800000u) ++r;
    return r;
}

// The stream of a call. Streams go by their id, which unlike the handle is never used again.
struct CallStream {
    cudaStream_t handle;
    unsigned long long id = 0;
    bool capturing = false;
    explicit CallStream(cudaStream_t s) : handle(s) {
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        cuda_check(cudaStreamIsCapturing(s, &status), "cudaStreamIsCapturing");
        capturing = status != cudaStreamCaptureStatusNone;
        if (!capturing) cuda_check(cudaStreamGetId(s, &id), "cudaStreamGetId");   // (ends a capture)
    }
};

// Work on the GPU that later calls on other streams have to come after: an event per stream, recorded anew by every call on it. The
// event of a stream whose work has ended serves the next stream.
class StreamMarks {
    struct Mark {
        unsigned long long stream_id;
        cudaEvent_t event;
        bool pending;
    };
    std::vector<Mark> marks;

public:
    StreamMarks() = default;
    StreamMarks(const StreamMarks &) = delete;
    StreamMarks &operator=(const StreamMarks &) = delete;
    ~StreamMarks() {
        for (const Mark &m : marks) cudaEventDestroy(m.event);
    }
    void mark(const CallStream &s) {   // everything issued on s so far (what a graph will run later is the graph's caller's to order)
        if (s.capturing) return;
        Mark *mine = nullptr;
        for (Mark &m : marks)
            if (m.stream_id == s.id) mine = &m;
        for (size_t i = 0; !mine && i < marks.size(); ++i)
            if (!marks[i].pending || cudaEventQuery(marks[i].event) == cudaSuccess) mine = &marks[i];
        if (!mine) {
            Mark fresh{s.id, nullptr, false};
            cuda_check(cudaEventCreateWithFlags(&fresh.event, cudaEventDisableTiming), "create adapter event");
            marks.push_back(fresh);
            mine = &marks.back();
        }
        mine->stream_id = s.id;
        cuda_check(cudaEventRecord(mine->event, s.handle), "record adapter event");
        mine->pending = true;
    }
    void join(const CallStream &s) {   // what is issued on s from now on comes after all that was marked
        if (s.capturing) {   // a graph cannot wait for what is outside of it: it ends before the call goes on
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // and only so may a capturing thread wait
            cuda_check(cudaThreadExchangeStreamCaptureMode(&mode), "cudaThreadExchangeStreamCaptureMode");
            const cudaError_t e = wait();
            cuda_check(cudaThreadExchangeStreamCaptureMode(&mode), "cudaThreadExchangeStreamCaptureMode");
            cuda_check(e, "wait for another stream's work");
            return;
        }
        for (Mark &m : marks) {
            if (!m.pending || m.stream_id == s.id) continue;
            if (cudaEventQuery(m.event) == cudaSuccess) m.pending = false;
            else cuda_check(cudaStreamWaitEvent(s.handle, m.event, 0), "wait for another stream's work");
        }
    }
    cudaError_t wait() const {   // on the host
        for (const Mark &m : marks) {
            const cudaError_t e = m.pending ? cudaEventSynchronize(m.event) : cudaSuccess;
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
};

struct HeadState {   // per (layer, kv head), in tokens
    uint64_t appended = 0;      // everything ever appended
    uint32_t sealed = 0;        // tokens in sealed tiles
    uint32_t tail = 0;          // tokens in the device tail
    uint32_t next_token = 0;    // position the next append must start at
    uint32_t bad_row = 0xffffffffu;   // first row of the tail that holds NaN or Inf, as far as it has been looked at
    bool unchecked = false;           // rows of the tail came in stream order: the GPU looks at them when they become a page
    bool started = false;
    bool flushed_partial = false;
};

struct LayerState {
    bool calibrated = false;
    std::vector<uint32_t> page_ids;   // tile index -> page id
    uint32_t device_sealed = 0xffffffffu, device_tail = 0xffffffffu;  // what the device scalars hold
};

}  // namespace

struct cf_llama_kv_adapter {
    cf_llama_kv_options opt{};
    uint32_t tile_tokens = 0;     // T: tokens per record, T * head_dim <= 4096, T divides page_size
    uint32_t coder = CF_B200_CODER_RANS;
    std::string last_error;
    std::vector<HeadState> heads;
    std::vector<LayerState> layers;
    uint32_t next_page_id = 1;
    uint64_t sealed_tiles = 0;

    DeviceBuffer<uint8_t> arena;
    DeviceBuffer<uint64_t> page_dir;
    DeviceBuffer<uint32_t> page_table;      // [layer][stride]
    uint32_t stride = 0;
    DeviceBuffer<uint32_t> scalars;          // [0,L): sealed tokens per layer; [L,2L): tail tokens per layer
    DeviceBuffer<float> tail_k, tail_v;      // [layer][kv_head][T][head_dim]
    DeviceBuffer<cf_b200_codebook_tables> tables;  // [layer][2]
    DeviceBuffer<uint32_t> slots;            // [layer][max_queries]: the layer index repeated
    DeviceBuffer<uint32_t> positions;        // iota
    DeviceBuffer<uint32_t> jobs;             // scratch for seal jobs: slot, page, tokens, head
    DeviceBuffer<unsigned long long> cursor; // [0] arena cursor, [1..512] histograms
    DeviceBuffer<uint32_t> status;
    DeviceBuffer<uint8_t> workspace;
    static constexpr uint32_t kMaxQueries = 4096;

    // Reference-exact mode (the default): pages as the reference's own fixed-width descriptors, made by
    // kivi_quantise_kernel, attended by cf_kv_paged_attention_async. CHROMOFOLD_B200_CODER switches to format v1.
    bool kivi = true;
    uint32_t kivi_bits = 4;
    static constexpr size_t kKiviChunk = 32u << 20;
    std::vector<uint8_t *> kivi_chunks;      // page blocks never move: descriptors hold their addresses
    size_t kivi_chunk_index = 0, kivi_chunk_used = 0;
    uint32_t kivi_chunk_limit = 0xffffffffu; // test hook: no further chunk is to be had
    DeviceBuffer<float> kivi_tail_k, kivi_tail_v;   // [layer][page_size][kv_head][head_dim]: the layout the attention reads
    DeviceBuffer<int32_t> kivi_lut;
    std::vector<std::unique_ptr<DeviceBuffer<cf_kv_device_page>>> kivi_descs;   // per layer, device
    std::vector<std::vector<cf_kv_device_page>> kivi_host_descs;                // per layer, the same on the host
    uint64_t kivi_resident_bytes = 0;
    DeviceBuffer<uint32_t> kivi_first_bad;   // result of first_bad_row_kernel
    DeviceBuffer<float> kivi_stage;          // rows of an append that fills pages: [K rows | V rows]
    float *kivi_pinned = nullptr;            // the same on their way from the caller's pageable memory, twice: appends take turns
    size_t kivi_stage_floats = 0;            // of one of the two streams
    cudaEvent_t kivi_done[2] = {};           // the append that used pinned half i has ended
    uint32_t kivi_turn = 0;                  // pinned half of the next append
    StreamMarks kivi_written, kivi_read;     // appends and flushes, attention calls
    cfb::CopyHelpers kivi_helpers;                // threads that share the copies there (a prompt's: a token's rows are too few)
    static constexpr size_t kKiviStageBytes = 1u << 20;   // of one stream, staged at a time (at least one page): the next turn copies meanwhile

    ~cf_llama_kv_adapter() {
        for (uint8_t *c : kivi_chunks) cudaFree(c);
        for (cudaEvent_t e : kivi_done)
            if (e) {
                cudaEventSynchronize(e);
                cudaEventDestroy(e);
            }
        if (kivi_pinned) cudaFreeHost(kivi_pinned);
    }
    // A call that writes pages or tails on stream s: after all earlier writes and attention calls, whatever streams they were on; its
    // own work is marked on every way out.
    struct WriteCall {
        cf_llama_kv_adapter &adapter;
        const CallStream s;
        WriteCall(cf_llama_kv_adapter &a, cudaStream_t stream) : adapter(a), s(stream) {
            adapter.kivi_written.join(s);
            adapter.kivi_read.join(s);
        }
        ~WriteCall() {
            try {
                adapter.kivi_written.mark(s);
            } catch (...) {   // no event to be had: the work ends before the call does
                cudaStreamSynchronize(s.handle);
            }
        }
    };
    size_t kivi_row_floats() const { return static_cast<size_t>(opt.kv_head_count) * opt.head_dim; }
    float *kivi_tail(DeviceBuffer<float> &buffer, uint32_t layer) const {
        return buffer.ptr + static_cast<size_t>(layer) * opt.page_size * kivi_row_floats();
    }
    uint8_t *kivi_take(size_t bytes) {
        if (bytes > kKiviChunk) throw std::runtime_error("page is larger than an adapter memory chunk");
        if (kivi_chunk_index < kivi_chunks.size() && kivi_chunk_used + bytes > kKiviChunk) {
            ++kivi_chunk_index;
            kivi_chunk_used = 0;
        }
        if (kivi_chunk_index >= kivi_chunks.size()) {
            uint8_t *fresh = nullptr;
            cuda_check(kivi_chunks.size() < kivi_chunk_limit ? cudaMalloc(reinterpret_cast<void **>(&fresh), kKiviChunk) : cudaErrorMemoryAllocation, "cudaMalloc");
            kivi_chunks.push_back(fresh);
            kivi_chunk_used = 0;
        }
        uint8_t *at = kivi_chunks[kivi_chunk_index] + kivi_chunk_used;
        kivi_chunk_used += (bytes + 255u) / 256u * 256u;
        return at;
    }
    void kivi_create() {
        cudaStream_t s = nullptr;
        const size_t tail = static_cast<size_t>(opt.layer_count) * opt.page_size * kivi_row_floats();
        kivi_tail_k.ensure(tail, s);
        kivi_tail_v.ensure(tail, s);
        const uint32_t levels = 1u << kivi_bits;
        std::vector<int32_t> lut(levels);
        for (uint32_t v = 0; v < levels; ++v) lut[v] = static_cast<int32_t>(v | (kivi_bits << 8));
        kivi_lut.ensure(levels, s);
        cuda_check(cudaMemcpy(kivi_lut.ptr, lut.data(), levels * 4, cudaMemcpyHostToDevice), "upload lut");
        for (cudaEvent_t &e : kivi_done) cuda_check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "create append event");
        kivi_descs.clear();
        for (uint32_t l = 0; l < opt.layer_count; ++l) {
            kivi_descs.push_back(std::make_unique<DeviceBuffer<cf_kv_device_page>>());
            kivi_descs.back()->ensure(64, s);
        }
        kivi_host_descs.assign(opt.layer_count, {});
        if (const char *reserve = std::getenv("CHROMOFOLD_B200_RESERVE_TOKENS")) {   // page memory and descriptors up front
            const unsigned long long tokens = std::strtoull(reserve, nullptr, 10);
            const size_t pages = static_cast<size_t>((tokens + opt.page_size - 1) / opt.page_size);   // per layer and kv head
            const size_t page_bytes = (kivi_layout(opt.page_size, opt.head_dim, kivi_bits).total + 255u) / 256u * 256u;
            const size_t per_chunk = kKiviChunk / page_bytes;
            const size_t chunks = per_chunk ? (pages * opt.layer_count * opt.kv_head_count + per_chunk - 1) / per_chunk : 0;
            for (size_t i = kivi_chunks.size(); i < chunks; ++i) {
                uint8_t *fresh = nullptr;
                cuda_check(cudaMalloc(reinterpret_cast<void **>(&fresh), kKiviChunk), "cudaMalloc");
                kivi_chunks.push_back(fresh);
            }
            for (uint32_t l = 0; l < opt.layer_count; ++l) kivi_descs[l]->ensure(std::max<size_t>(64, pages * opt.kv_head_count), s);
        }
        cuda_check(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
    }
    void kivi_reset() {
        kivi_chunk_index = 0;
        kivi_chunk_used = 0;
        kivi_resident_bytes = 0;
        for (auto &d : kivi_host_descs) d.clear();
    }
    cudaError_t kivi_mark(cudaStream_t s) {   // the copies out of a pinned half have been issued on s
        const cudaError_t e = cudaEventRecord(kivi_done[kivi_turn], s);
        if (e == cudaSuccess) kivi_turn ^= 1u;
        return e;
    }
    // Quantise `pages` pages of `tokens` rows of (layer, kv_head): the rows of the tail, then the staged ones; `rest` staged rows
    // after them become the tail. One launch, which also publishes the descriptors. The rows are known to be finite: they were
    // checked while they were copied, so that a refusal is thrown at once (the reference quantises on the host and does the
    // same) and no append waits for the GPU: one of 512 x 128 rows took 85 us, of which 40 are the copy.
    void kivi_seal(uint32_t layer, uint32_t kv_head, uint32_t pages, uint32_t tokens, uint32_t rest, cudaStream_t s) {
        HeadState &h = head(layer, kv_head);
        const uint32_t D = opt.head_dim;
        const KiviLayout lay = kivi_layout(tokens, D, kivi_bits);
        KiviJob job{};
        job.stage_k = kivi_stage.ptr;
        job.stage_v = kivi_stage.ptr + kivi_stage_floats;
        job.tail_k = kivi_tail(kivi_tail_k, layer) + static_cast<size_t>(kv_head) * D;
        job.tail_v = kivi_tail(kivi_tail_v, layer) + static_cast<size_t>(kv_head) * D;
        job.row_stride = static_cast<uint32_t>(kivi_row_floats());
        job.tail_rows = h.tail;
        job.tokens = tokens;
        job.dim = D;
        job.bits = kivi_bits;
        job.pages = pages;
        job.rest_rows = rest;
        cf_kv_device_page &common = job.page;
        common.k_lut = common.v_lut = kivi_lut.ptr;
        common.token_begin = h.next_token - h.tail;
        common.token_count = tokens;
        common.head_dim = D;
        common.block_size = 64;
        common.k_max_code_length = common.v_max_code_length = common.fixed_code_length = kivi_bits;
        common.zero_point = 1u << (kivi_bits - 1);
        common.kv_head = kv_head;
        // Everything that can fail comes first: the host's list names no page that the launch below does not write.
        std::vector<cf_kv_device_page> &host = kivi_host_descs[layer];
        const size_t first = host.size(), chunk_index = kivi_chunk_index, chunk_used = kivi_chunk_used;
        try {
            if (host.capacity() < first + pages) host.reserve(2 * first + pages);
            for (uint32_t p = 0; p < pages; ++p) job.block[p] = kivi_take(lay.total);
            DeviceBuffer<cf_kv_device_page> &dev = *kivi_descs[layer];
            dev.ensure(first + pages, s);
            job.pages_out = dev.ptr + first;
            kivi_quantise_kernel<<<pages, 1024, (static_cast<size_t>(D) + tokens) * sizeof(float), s>>>(job, lay);
            cuda_check(cudaGetLastError(), "page quantise launch");
        } catch (...) {
            kivi_chunk_index = chunk_index;
            kivi_chunk_used = chunk_used;
            throw;
        }
        for (uint32_t p = 0; p < pages; ++p) {
            const uint8_t *block = job.block[p];
            cf_kv_device_page page = common;
            page.k_words = reinterpret_cast<const uint32_t *>(block + lay.k_words);
            page.v_words = reinterpret_cast<const uint32_t *>(block + lay.v_words);
            page.k_scales = reinterpret_cast<const float *>(block + lay.k_scales);
            page.v_scales = reinterpret_cast<const float *>(block + lay.v_scales);
            page.k_block_offsets = reinterpret_cast<const int32_t *>(block + lay.k_offsets);
            page.v_block_offsets = reinterpret_cast<const int32_t *>(block + lay.v_offsets);
            page.token_begin += p * tokens;
            host.push_back(page);
        }
        // EncodedKvPage::resident_bytes: words, offsets, both LUTs, scales
        kivi_resident_bytes += pages * (8ull * lay.word_count + 8ull * lay.block_count + 8ull * (1u << kivi_bits) + 4ull * (D + tokens));
        if (tokens < opt.page_size) h.flushed_partial = true;
        h.sealed += pages * tokens;
        sealed_tiles += pages;
    }
    // The first row with NaN or Inf among the tail's rows that have not been looked at, and `staged` rows behind them.
    uint32_t kivi_look(uint32_t layer, uint32_t kv_head, uint32_t staged, cudaStream_t s) {
        HeadState &h = head(layer, kv_head);
        const uint32_t D = opt.head_dim;
        uint32_t first = 0xffffffffu;
        kivi_first_bad.ensure(1, s);
        cuda_check(cudaMemsetAsync(kivi_first_bad.ptr, 0xff, 4, s), "clear row check");
        if (h.unchecked)
            first_bad_row_kernel<<<(h.tail + 7u) / 8u, 256, 0, s>>>(kivi_tail(kivi_tail_k, layer) + static_cast<size_t>(kv_head) * D,
                                                                   kivi_tail(kivi_tail_v, layer) + static_cast<size_t>(kv_head) * D, kivi_row_floats(), D,
                                                                   h.tail, 0u, kivi_first_bad.ptr);
        if (staged)
            first_bad_row_kernel<<<(staged + 7u) / 8u, 256, 0, s>>>(kivi_stage.ptr, kivi_stage.ptr + kivi_stage_floats, D, D, staged, h.tail, kivi_first_bad.ptr);
        cuda_check(cudaGetLastError(), "row check launch");
        cuda_check(cudaMemcpyAsync(&first, kivi_first_bad.ptr, 4, cudaMemcpyDeviceToHost, s), "read row check");
        cuda_check(cudaStreamSynchronize(s), "cudaStreamSynchronize");   // a page is refused by the call that brings it
        if (first < h.tail) h.bad_row = std::min(h.bad_row, first);
        h.unchecked = false;
        return first;
    }
    void kivi_flush(uint32_t layer, uint32_t kv_head, cudaStream_t s) {
        HeadState &h = head(layer, kv_head);
        if (h.tail == 0) return;
        if (h.unchecked) kivi_look(layer, kv_head, 0, s);
        if (h.bad_row < h.tail) throw std::invalid_argument("invalid quantization input");   // kv_gpu_fixture.cpp:13
        kivi_seal(layer, kv_head, 1, h.tail, 0, s);
        h.tail = 0;
    }
    // `take` host rows into the tail ([token][kv head][dim]: the layout the attention reads).
    void kivi_rows_to_tail(uint32_t layer, uint32_t kv_head, const float *keys, const float *values, uint32_t take, bool ordered, cudaStream_t s) {
        if (take == 0) return;
        HeadState &h = head(layer, kv_head);
        if (ordered) {
            h.unchecked = true;
        } else if (h.bad_row >= h.tail) {
            const uint32_t bad = std::min(first_bad_row(keys, take, opt.head_dim), first_bad_row(values, take, opt.head_dim));
            h.bad_row = bad < take ? h.tail + bad : 0xffffffffu;
        }
        const size_t row = kivi_row_floats(), D = opt.head_dim, at = static_cast<size_t>(h.tail) * row + static_cast<size_t>(kv_head) * D;
        cuda_check(cudaMemcpy2DAsync(kivi_tail(kivi_tail_k, layer) + at, row * 4, keys, D * 4, D * 4, take, cudaMemcpyHostToDevice, s), "append keys");
        cuda_check(cudaMemcpy2DAsync(kivi_tail(kivi_tail_v, layer) + at, row * 4, values, D * 4, D * 4, take, cudaMemcpyHostToDevice, s), "append values");
        h.tail += take;
        h.next_token += take;
    }
    // Host rows of (layer, kv_head): those that only lengthen the tail are copied there; those that complete pages are staged,
    // as many pages at a time as the stage holds, and quantised by one launch.
    void kivi_append(uint32_t layer, uint32_t kv_head, const float *keys, const float *values, uint32_t token_count, cudaStream_t s) {
        HeadState &h = head(layer, kv_head);
        const uint32_t T = tile_tokens, D = opt.head_dim;
        const bool ordered = in_stream_order(keys) || in_stream_order(values);
        uint32_t done = 0;
        while (done < token_count) {
            const uint32_t left = token_count - done;
            if (h.tail + left < T) {
                kivi_rows_to_tail(layer, kv_head, keys + static_cast<size_t>(done) * D, values + static_cast<size_t>(done) * D, left, ordered, s);
                return;
            }
            const uint32_t room = std::max<uint32_t>(1u, std::min<uint32_t>(kKiviPagesPerLaunch, static_cast<uint32_t>(kKiviStageBytes / (4ull * T * D))));
            const uint32_t pages = std::min<uint32_t>(room, (h.tail + left) / T);
            const bool last = pages == (h.tail + left) / T;
            const uint32_t rows = last ? left : pages * T - h.tail, rest = last ? h.tail + left - pages * T : 0u;
            const size_t floats = static_cast<size_t>(rows) * D;
            if (floats > kivi_stage_floats) {
                const size_t wanted = std::max(floats, kivi_stage_floats * 2);
                for (cudaEvent_t e : kivi_done) cuda_check(cudaEventSynchronize(e), "wait for earlier appends");
                if (kivi_pinned) cudaFreeHost(kivi_pinned);
                kivi_pinned = nullptr;
                kivi_stage_floats = 0;
                cuda_check(cudaHostAlloc(reinterpret_cast<void **>(&kivi_pinned), 4 * wanted * sizeof(float), cudaHostAllocDefault), "cudaHostAlloc");
                kivi_stage.ensure(2 * wanted, s);
                kivi_stage_floats = wanted;
            }
            cuda_check(cudaEventSynchronize(kivi_done[kivi_turn]), "wait for an earlier append");   // its half of the pinned memory
            const float *source[2] = {keys + static_cast<size_t>(done) * D, values + static_cast<size_t>(done) * D};
            uint32_t bad = rows, sealed = 0;   // first staged row with NaN or Inf; pages in front of it
            try {
                for (int stream = 0; stream < 2; ++stream) {   // the copy of K crosses the bus while V is gathered
                    const float *half = source[stream];
                    if (!ordered) {
                        float *pinned = kivi_pinned + (2u * kivi_turn + stream) * kivi_stage_floats;
                        bad = std::min(bad, copy_rows_checked(kivi_helpers, pinned, half, rows, D));
                        half = pinned;
                    }
                    cuda_check(cudaMemcpyAsync(kivi_stage.ptr + stream * kivi_stage_floats, half, floats * sizeof(float), cudaMemcpyHostToDevice, s), "stage rows");
                }
                if (ordered || h.unchecked) {
                    const uint32_t first = kivi_look(layer, kv_head, ordered ? rows : 0u, s);
                    if (first >= h.tail) bad = std::min(bad, first - h.tail);
                }
                sealed = h.bad_row < h.tail ? 0u : std::min(pages, (h.tail + bad) / T);
                if (sealed) kivi_seal(layer, kv_head, sealed, T, sealed == pages ? rest : 0u, s);
            } catch (...) {   // the pinned half may still be on its way
                kivi_mark(s);
                throw;
            }
            cuda_check(kivi_mark(s), "record append event");
            if (sealed < pages) {   // pages before the refused one stay; its rows become the (full) tail, as if appended page by page
                const uint32_t skip = sealed ? sealed * T - h.tail : 0u, keep = sealed ? 0u : h.tail;
                if (sealed) {
                    h.next_token += skip;
                    h.bad_row = 0xffffffffu;
                }
                h.tail = keep;
                kivi_rows_to_tail(layer, kv_head, source[0] + static_cast<size_t>(skip) * D, source[1] + static_cast<size_t>(skip) * D, T - keep, ordered, s);
                cuda_check(cudaStreamSynchronize(s), "cudaStreamSynchronize");
                throw std::invalid_argument("invalid quantization input");
            }
            h.bad_row = bad < rows ? h.tail + bad - pages * T : 0xffffffffu;   // in the rest
            h.tail = rest;
            h.next_token += rows;
            done += rows;
        }
    }

    HeadState &head(uint32_t layer, uint32_t h) { return heads[static_cast<size_t>(layer) * opt.kv_head_count + h]; }
    size_t tile_values() const { return static_cast<size_t>(tile_tokens) * opt.head_dim; }
    size_t max_record_bytes() const { return 16 + 2 * ((tile_values() + 15) / 16 * 16); }

    void reset(cudaStream_t s) {
        heads.assign(static_cast<size_t>(opt.layer_count) * opt.kv_head_count, HeadState{});
        layers.assign(opt.layer_count, LayerState{});
        next_page_id = 1;
        sealed_tiles = 0;
        kivi_reset();
        if (cursor.ptr) cuda_check(cudaMemsetAsync(cursor.ptr, 0, sizeof(unsigned long long), s), "memset cursor");
        if (page_dir.ptr) cuda_check(cudaMemsetAsync(page_dir.ptr, 0, page_dir.count * sizeof(uint64_t), s), "memset dir");
        if (status.ptr) cuda_check(cudaMemsetAsync(status.ptr, 0, sizeof(uint32_t), s), "memset status");
    }

    void create_buffers() {
        cudaStream_t s = nullptr;
        const uint32_t L = opt.layer_count, H = opt.kv_head_count;
        stride = 4096;
        page_table.ensure(static_cast<size_t>(L) * stride, s);
        scalars.ensure(2 * L, s);
        tail_k.ensure(static_cast<size_t>(L) * H * tile_values(), s);
        tail_v.ensure(static_cast<size_t>(L) * H * tile_values(), s);
        tables.ensure(2 * L, s);
        cursor.ensure(1 + 512, s);
        status.ensure(1, s);
        jobs.ensure(4 * 64, s);
        arena.ensure(64u << 20, s);
        page_dir.ensure(static_cast<size_t>(65536) * H, s);
        std::vector<uint32_t> host(static_cast<size_t>(L) * kMaxQueries);
        for (uint32_t l = 0; l < L; ++l) std::fill_n(host.begin() + static_cast<size_t>(l) * kMaxQueries, kMaxQueries, l);
        slots.ensure(host.size(), s);
        cuda_check(cudaMemcpy(slots.ptr, host.data(), host.size() * 4, cudaMemcpyHostToDevice), "upload slots");
        grow_positions(1u << 16, s);
        // workspace: one chunk per query row is the floor; give 16-tile chunks room for 1M tokens
        cf_b200_sealed_attention_desc d{};
        d.kv_head_count = H;
        d.query_head_count = opt.query_head_count;
        d.head_dim = opt.head_dim;
        d.seq_count = kMaxQueries;
        uint64_t bytes = 0;
        cf_b200_sealed_attention_workspace_bytes(&d, 65536, &bytes);
        workspace.ensure(bytes + 256, s);
        cuda_check(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
    }

    void grow_positions(size_t wanted, cudaStream_t s) {
        if (wanted <= positions.count) return;
        const size_t old = positions.count;
        positions.ensure(wanted, s);
        std::vector<uint32_t> host(positions.count - old);
        for (size_t i = 0; i < host.size(); ++i) host[i] = static_cast<uint32_t>(old + i);
        cuda_check(cudaMemcpyAsync(positions.ptr + old, host.data(), host.size() * 4, cudaMemcpyHostToDevice, s), "upload positions");
        cuda_check(cudaStreamSynchronize(s), "cudaStreamSynchronize");
    }

    // Make sure `tiles` more tiles fit: arena by the worst-case record size, directory and page table by count.
    void reserve(uint32_t layer, uint32_t tile_index, cudaStream_t s) {
        arena.ensure((sealed_tiles + 1) * max_record_bytes() + 4096, s);
        page_dir.ensure(static_cast<size_t>(next_page_id + 2) * opt.kv_head_count, s);
        if (tile_index >= stride) {  // widen every row of the page table
            const uint32_t wider = stride * 2;
            DeviceBuffer<uint32_t> fresh;
            fresh.ensure(static_cast<size_t>(opt.layer_count) * wider, s);
            cuda_check(cudaMemcpy2DAsync(fresh.ptr, wider * 4, page_table.ptr, stride * 4, stride * 4, opt.layer_count,
                                         cudaMemcpyDeviceToDevice, s), "widen page table");
            cuda_check(cudaStreamSynchronize(s), "cudaStreamSynchronize");
            std::swap(fresh.ptr, page_table.ptr);
            std::swap(fresh.count, page_table.count);
            stride = wider;
        }
        (void)layer;
    }

    cf_b200_seal_desc seal_desc(uint32_t layer) const {
        cf_b200_seal_desc d{};
        d.struct_size = sizeof d;
        d.abi_version = CF_B200_ABI_VERSION;
        d.kv_head_count = opt.kv_head_count;
        d.head_dim = opt.head_dim;
        d.page_tokens = tile_tokens;
        d.block_size = 64;
        d.coder = coder;
        d.codebook_id = layer;
        d.k_tables = tables.ptr + 2 * layer;
        d.v_tables = tables.ptr + 2 * layer + 1;
        d.tail_k = tail_k.ptr;
        d.tail_v = tail_v.ptr;
        d.tail_type = CF_B200_F32;
        d.arena = arena.ptr;
        d.arena_units = arena.count / 16;
        d.arena_cursor_units = cursor.ptr;
        d.page_dir = page_dir.ptr;
        d.status = status.ptr;
        return d;
    }

    void upload_job(uint32_t slot, uint32_t page, uint32_t tokens, uint32_t kv_head, cudaStream_t s) {
        const uint32_t host[4] = {slot, page, tokens, kv_head};
        cuda_check(cudaMemcpyAsync(jobs.ptr, &host[0], 4, cudaMemcpyHostToDevice, s), "job");
        cuda_check(cudaMemcpyAsync(jobs.ptr + 64, &host[1], 4, cudaMemcpyHostToDevice, s), "job");
        cuda_check(cudaMemcpyAsync(jobs.ptr + 128, &host[2], 4, cudaMemcpyHostToDevice, s), "job");
        cuda_check(cudaMemcpyAsync(jobs.ptr + 192, &host[3], 4, cudaMemcpyHostToDevice, s), "job");
    }

    // First tile of a layer: histogram its quantised symbols on the GPU, build the layer's codebooks.
    void calibrate(uint32_t layer, uint32_t kv_head, uint32_t tokens, cudaStream_t s) {
        cf_b200_seal_desc d = seal_desc(layer);
        upload_job(layer, 0, tokens, kv_head, s);
        d.job_slots = jobs.ptr;
        d.job_tokens = jobs.ptr + 128;
        d.job_heads = jobs.ptr + 192;
        d.job_count = 1;
        cuda_check(cudaMemsetAsync(cursor.ptr + 1, 0, 512 * sizeof(unsigned long long), s), "memset hist");
        if (cf_b200_histogram_async(&d, cursor.ptr + 1, cursor.ptr + 257, s) != CF_OK)
            throw std::runtime_error("ChromoFold histogram launch rejected");
        unsigned long long hist[512];
        cuda_check(cudaMemcpyAsync(hist, cursor.ptr + 1, sizeof hist, cudaMemcpyDeviceToHost, s), "download hist");
        cuda_check(cudaStreamSynchronize(s), "cudaStreamSynchronize");
        std::vector<cf_b200_codebook_tables> host(2);
        uint64_t hk[256], hv[256];
        for (int i = 0; i < 256; ++i) { hk[i] = hist[i]; hv[i] = hist[256 + i]; }
        if (cf_b200_codebook_build(hk, &host[0]) != CF_OK || cf_b200_codebook_build(hv, &host[1]) != CF_OK)
            throw std::runtime_error("ChromoFold codebook build failed");
        cuda_check(cudaMemcpyAsync(tables.ptr + 2 * layer, host.data(), 2 * sizeof(cf_b200_codebook_tables),
                                   cudaMemcpyHostToDevice, s), "upload codebooks");
        cuda_check(cudaStreamSynchronize(s), "cudaStreamSynchronize");
        layers[layer].calibrated = true;
    }

    // Seal the tail of (layer, kv_head): `tokens` rows become tile number sealed / T.
    void seal_tail(uint32_t layer, uint32_t kv_head, cudaStream_t s) {
        HeadState &h = head(layer, kv_head);
        if (h.tail == 0) return;
        LayerState &ls = layers[layer];
        const uint32_t tile_index = h.sealed / tile_tokens;
        reserve(layer, tile_index, s);
        if (!ls.calibrated) calibrate(layer, kv_head, h.tail, s);
        if (tile_index >= ls.page_ids.size()) {  // first head to reach this tile names the page
            ls.page_ids.push_back(next_page_id);
            cuda_check(cudaMemcpyAsync(page_table.ptr + static_cast<size_t>(layer) * stride + tile_index, &next_page_id, 4,
                                       cudaMemcpyHostToDevice, s), "publish page id");
            ++next_page_id;
        }
        cf_b200_seal_desc d = seal_desc(layer);
        upload_job(layer, ls.page_ids[tile_index], h.tail, kv_head, s);
        d.job_slots = jobs.ptr;
        d.job_pages = jobs.ptr + 64;
        d.job_tokens = jobs.ptr + 128;
        d.job_heads = jobs.ptr + 192;
        d.job_count = 1;
        if (cf_b200_seal_pages_async(&d, s) != CF_OK) throw std::runtime_error("ChromoFold seal launch rejected");
        if (h.tail < tile_tokens) h.flushed_partial = true;
        h.sealed += h.tail;
        h.tail = 0;
        ++sealed_tiles;
    }
};

namespace {

template <class Operation>
int guarded(cf_llama_kv_adapter *adapter, Operation &&operation) {  // chromofold_kv_adapter.cpp:35-49
    if (adapter == nullptr) return -1;
    try {
        operation();
        adapter->last_error.clear();
        return 0;
    } catch (const std::exception &error) {
        adapter->last_error = error.what();
        return -1;
    } catch (...) {
        adapter->last_error = "unknown ChromoFold KV error";
        return -1;
    }
}

uint32_t choose_tile_tokens(uint32_t page_size, uint32_t head_dim) {
    // 16-token records at head_dim 128, 96, 64 and 32 are the geometries of the lane-per-block attention kernels
    if ((head_dim == 128 || head_dim == 96 || head_dim == 64 || head_dim == 32) && page_size % 16 == 0) return 16;
    const uint32_t limit = CF_B200_MAX_STREAM_SYMBOLS / head_dim;
    for (uint32_t t = std::min(page_size, limit); t >= 1; --t)
        if (page_size % t == 0) return t;
    return 1;
}

}  // namespace

extern "C" int cf_llama_kv_options_validate(const cf_llama_kv_options *options) {
    if (options == nullptr || options->struct_size != sizeof(cf_llama_kv_options)) return -1;
    if (options->backend == CF_LLAMA_KV_BACKEND_DENSE) return 0;
    if (options->backend != CF_LLAMA_KV_BACKEND_CHROMOFOLD || options->layer_count == 0 || options->kv_head_count == 0 ||
        options->query_head_count == 0 || options->head_dim == 0 || options->page_size == 0 ||
        options->gqa_group_size == 0 || options->query_head_count != options->kv_head_count * options->gqa_group_size)
        return -1;
    return 0;
}

extern "C" cf_llama_kv_adapter *cf_llama_kv_create(const cf_llama_kv_options *options) {
    if (cf_llama_kv_options_validate(options) != 0 || options->backend != CF_LLAMA_KV_BACKEND_CHROMOFOLD) return nullptr;
    if (options->head_dim > CF_KV_MAX_HEAD_DIM || options->gqa_group_size > 16) return nullptr;
    try {
        auto *a = new cf_llama_kv_adapter();
        a->opt = *options;
        a->tile_tokens = choose_tile_tokens(options->page_size, options->head_dim);
        a->kivi_bits = options->kv_bits == 8 ? 8u : 4u;   // chromofold_kv_adapter.cpp:30-31: 8 selects int8, anything else int4
        if (const char *env = std::getenv("CHROMOFOLD_B200_CODER")) {   // opt in to entropy-coded format-v1 pages
            a->kivi = false;
            if (std::strcmp(env, "huffman") == 0) a->coder = CF_B200_CODER_HUFFMAN;
            else if (std::strcmp(env, "fixed8") == 0) a->coder = CF_B200_CODER_FIXED8;
            else if (std::strcmp(env, "rans4") == 0) a->coder = CF_B200_CODER_RANS_SPLIT4;
            else if (std::strcmp(env, "huffman4") == 0) a->coder = CF_B200_CODER_HUFFMAN_SPLIT4;
            else if (std::strcmp(env, "rans") != 0) a->kivi = true;   // not a coder name: the default stands
        }
        if (a->kivi) a->tile_tokens = options->page_size;
        try {
            if (a->kivi) a->kivi_create();
            else a->create_buffers();
            a->reset(nullptr);
        } catch (...) {
            delete a;
            return nullptr;  // no usable CUDA device: there is no host fallback
        }
        return a;
    } catch (...) {
        return nullptr;
    }
}

extern "C" void cf_llama_kv_destroy(cf_llama_kv_adapter *adapter) { delete adapter; }

extern "C" int cf_llama_kv_append(cf_llama_kv_adapter *adapter, uint32_t layer, uint32_t kv_head, uint32_t token_begin,
                                  const float *keys, const float *values, uint32_t token_count, void *stream) {
    return guarded(adapter, [&] {
        if (keys == nullptr || values == nullptr || token_count == 0) throw std::invalid_argument("invalid KV append");
        if (layer >= adapter->opt.layer_count || kv_head >= adapter->opt.kv_head_count)
            throw std::out_of_range("KV layer or head out of range");
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        HeadState &h = adapter->head(layer, kv_head);
        if (h.started && token_begin != h.next_token) throw std::invalid_argument("KV append must be logically contiguous");
        if (h.flushed_partial && !adapter->kivi)
            throw std::runtime_error("append after a partial flush is not supported by the sealed format");
        if (!h.started) {
            h.started = true;
            h.next_token = token_begin;
        }
        const uint32_t D = adapter->opt.head_dim, T = adapter->tile_tokens;
        if (adapter->kivi) {
            const cf_llama_kv_adapter::WriteCall call(*adapter, s);
            adapter->kivi_append(layer, kv_head, keys, values, token_count, s);
            h.appended += token_count;
            return;
        }
        const size_t tile = (static_cast<size_t>(layer) * adapter->opt.kv_head_count + kv_head) * adapter->tile_values();
        uint32_t done = 0;
        while (done < token_count) {
            const uint32_t take = std::min(token_count - done, T - h.tail);
            const size_t dst = tile + static_cast<size_t>(h.tail) * D;
            cuda_check(cudaMemcpyAsync(adapter->tail_k.ptr + dst, keys + static_cast<size_t>(done) * D, sizeof(float) * take * D,
                                       cudaMemcpyHostToDevice, s), "append keys");
            cuda_check(cudaMemcpyAsync(adapter->tail_v.ptr + dst, values + static_cast<size_t>(done) * D,
                                       sizeof(float) * take * D, cudaMemcpyHostToDevice, s), "append values");
            h.tail += take;
            done += take;
            if (h.tail == T) adapter->seal_tail(layer, kv_head, s);
        }
        h.appended += token_count;
        h.next_token += token_count;
    });
}

extern "C" int cf_llama_kv_attention(cf_llama_kv_adapter *adapter, uint32_t layer, const float *queries_device,
                                     float *output_device, uint32_t query_count, uint32_t query_head_count,
                                     uint32_t gqa_group_size, uint32_t query_token_begin, float softmax_scale,
                                     uint32_t causal_window, void *stream) {
    return guarded(adapter, [&] {
        if (queries_device == nullptr || output_device == nullptr || gqa_group_size == 0 || query_head_count == 0 ||
            query_head_count % gqa_group_size != 0)
            throw std::invalid_argument("invalid ChromoFold attention request");
        if (layer >= adapter->opt.layer_count) throw std::out_of_range("KV layer out of range");
        if (query_head_count != adapter->opt.query_head_count || gqa_group_size != adapter->opt.gqa_group_size ||
            query_count == 0 || query_count > cf_llama_kv_adapter::kMaxQueries)
            throw std::invalid_argument("invalid ChromoFold attention request");
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        const HeadState &h0 = adapter->head(layer, 0);
        for (uint32_t k = 1; k < adapter->opt.kv_head_count; ++k) {
            const HeadState &h = adapter->head(layer, k);
            if (h.sealed != h0.sealed || h.tail != h0.tail) throw std::runtime_error("KV active tails are not aligned across heads");
        }
        if (adapter->kivi) {   // the reference's own call over the reference's own page descriptors (its adapter, :107-131)
            const CallStream call(s);
            adapter->kivi_written.join(call);
            cf_kv_paged_attention_desc desc{};
            desc.struct_size = sizeof desc;
            desc.abi_version = CF_KV_CUDA_ABI_VERSION;
            desc.pages = adapter->kivi_descs[layer]->ptr;
            desc.page_count = static_cast<uint32_t>(adapter->kivi_host_descs[layer].size());
            desc.kv_head_count = adapter->opt.kv_head_count;
            desc.query_head_count = query_head_count;
            desc.gqa_group_size = gqa_group_size;
            desc.active_k = h0.tail ? adapter->kivi_tail(adapter->kivi_tail_k, layer) : nullptr;
            desc.active_v = h0.tail ? adapter->kivi_tail(adapter->kivi_tail_v, layer) : nullptr;
            desc.active_token_begin = h0.next_token - h0.tail;
            desc.active_token_count = h0.tail;
            desc.queries = queries_device;
            desc.output = output_device;
            desc.query_token_begin = query_token_begin;
            desc.query_count = query_count;
            desc.head_dim = adapter->opt.head_dim;
            desc.causal_window = causal_window;
            desc.softmax_scale = softmax_scale;
            if (cf_kv_paged_attention_async(&desc, s) != CF_OK) throw std::runtime_error("ChromoFold paged attention launch rejected");
            adapter->kivi_read.mark(call);
            return;
        }
        LayerState &ls = adapter->layers[layer];
        const uint32_t L = adapter->opt.layer_count;
        if (ls.device_sealed != h0.sealed || ls.device_tail != h0.tail) {
            cuda_check(cudaMemcpyAsync(adapter->scalars.ptr + layer, &h0.sealed, 4, cudaMemcpyHostToDevice, s), "sealed count");
            cuda_check(cudaMemcpyAsync(adapter->scalars.ptr + L + layer, &h0.tail, 4, cudaMemcpyHostToDevice, s), "tail count");
            ls.device_sealed = h0.sealed;
            ls.device_tail = h0.tail;
        }
        adapter->grow_positions(static_cast<size_t>(query_token_begin) + query_count + 1, s);

        cf_b200_sealed_attention_desc d{};
        d.struct_size = sizeof d;
        d.abi_version = CF_B200_ABI_VERSION;
        d.kv_head_count = adapter->opt.kv_head_count;
        d.query_head_count = query_head_count;
        d.head_dim = adapter->opt.head_dim;
        d.page_tokens = adapter->tile_tokens;
        d.block_size = 64;
        d.codebook_id = layer;
        d.arena = adapter->arena.ptr;
        d.page_dir = adapter->page_dir.ptr;
        d.page_table = adapter->page_table.ptr;
        d.seq_sealed_tokens = adapter->scalars.ptr;
        d.seq_slots = adapter->slots.ptr + static_cast<size_t>(layer) * cf_llama_kv_adapter::kMaxQueries;
        d.page_table_stride = adapter->stride;
        d.seq_count = query_count;
        d.k_tables = adapter->tables.ptr + 2 * layer;
        d.v_tables = adapter->tables.ptr + 2 * layer + 1;
        d.tail_k = adapter->tail_k.ptr;
        d.tail_v = adapter->tail_v.ptr;
        d.tail_tokens = adapter->scalars.ptr + L;
        d.tail_type = CF_B200_F32;
        d.query_positions = adapter->positions.ptr + query_token_begin;
        d.queries = queries_device;
        d.output = output_device;
        d.query_type = CF_B200_F32;
        d.output_type = CF_B200_F32;
        d.softmax_scale = softmax_scale;
        d.causal_window = causal_window;
        // Prefill (llama.cpp evaluates a prompt in batches of query tokens): they share the layer's sealed records, which the
        // shared-prefix kernel then decodes once per 256 query rows instead of once per query token, masking what the
        // earlier tokens must not see. Given where it pays and the workspace has or can get the room.
        if (query_count >= 4 && causal_window == 0) {
            const uint32_t tiles = std::min(h0.sealed / adapter->tile_tokens, (query_token_begin + query_count - 1u) / adapter->tile_tokens + 1u);
            if (tiles >= 8 && tiles <= adapter->stride) {
                cf_b200_sealed_attention_desc room = d;   // the workspace grows for the extra partials, up to 1 GiB
                room.shared_prefix_pages = 1;
                uint64_t bytes = 0;
                if (cf_b200_sealed_attention_workspace_bytes(&room, 65536, &bytes) == CF_OK && bytes + 256 <= (1ull << 30)) {
                    adapter->workspace.ensure(bytes + 256, s);
                    d.shared_prefix_pages = tiles;
                }
            }
        }
        const uintptr_t ws = reinterpret_cast<uintptr_t>(adapter->workspace.ptr);
        const uintptr_t aligned = (ws + 255) / 256 * 256;
        d.workspace = reinterpret_cast<void *>(aligned);
        d.workspace_bytes = adapter->workspace.count - (aligned - ws);
        d.status = adapter->status.ptr;
        constexpr uint32_t kAll = CF_B200_STAGE_PLAN | CF_B200_STAGE_ATTENTION | CF_B200_STAGE_COMBINE;
        if (cfb::sealed_attention_stages(&d, kAll, s, false, true) != CF_OK) throw std::runtime_error("ChromoFold paged attention launch rejected");
    });
}

extern "C" int cf_llama_kv_attention_host(cf_llama_kv_adapter *adapter, uint32_t layer, const float *queries_host,
                                          float *output_host, uint32_t query_count, uint32_t query_head_count,
                                          uint32_t gqa_group_size, uint32_t query_token_begin, float softmax_scale,
                                          uint32_t causal_window, void *stream) {
    return guarded(adapter, [&] {
        if (queries_host == nullptr || output_host == nullptr) throw std::invalid_argument("null host attention buffer");
        const size_t bytes = static_cast<size_t>(query_count) * query_head_count * adapter->opt.head_dim * sizeof(float);
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        float *dq = nullptr, *dout = nullptr;
        if (cudaMalloc(reinterpret_cast<void **>(&dq), bytes) != cudaSuccess ||
            cudaMalloc(reinterpret_cast<void **>(&dout), bytes) != cudaSuccess) {
            if (dq) cudaFree(dq);
            throw std::runtime_error("failed to allocate attention scratch");
        }
        cudaMemcpyAsync(dq, queries_host, bytes, cudaMemcpyHostToDevice, s);
        const int rc = cf_llama_kv_attention(adapter, layer, dq, dout, query_count, query_head_count, gqa_group_size,
                                             query_token_begin, softmax_scale, causal_window, stream);
        const std::string inner = adapter->last_error;
        if (rc == 0) {
            cudaMemcpyAsync(output_host, dout, bytes, cudaMemcpyDeviceToHost, s);
            cudaStreamSynchronize(s);
        }
        cudaFree(dq);
        cudaFree(dout);
        if (rc != 0) throw std::runtime_error(inner.empty() ? "attention failed" : inner);
    });
}

extern "C" int cf_llama_kv_flush(cf_llama_kv_adapter *adapter, void *stream) {
    return guarded(adapter, [&] {
        std::unique_ptr<cf_llama_kv_adapter::WriteCall> call;
        if (adapter->kivi) call = std::make_unique<cf_llama_kv_adapter::WriteCall>(*adapter, static_cast<cudaStream_t>(stream));
        for (uint32_t layer = 0; layer < adapter->opt.layer_count; ++layer)
            for (uint32_t h = 0; h < adapter->opt.kv_head_count; ++h) {
                if (adapter->kivi) adapter->kivi_flush(layer, h, static_cast<cudaStream_t>(stream));
                else adapter->seal_tail(layer, h, static_cast<cudaStream_t>(stream));
            }
    });
}

extern "C" int cf_llama_kv_seq_rm(cf_llama_kv_adapter *adapter, uint64_t sequence_id) {
    return guarded(adapter, [&] {  // compressed_kv_cache.cu:180-183
        if (sequence_id != 0) throw std::invalid_argument("current ChromoFold cache supports sequence 0 only");
        cuda_check(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
        adapter->reset(nullptr);
    });
}

extern "C" int cf_llama_kv_seq_cp(cf_llama_kv_adapter *adapter, uint64_t source_id, uint64_t destination_id) {
    return guarded(adapter, [&] {  // compressed_kv_cache.cu:185-188
        if (source_id == destination_id) return;
        throw std::runtime_error("sequence copy requires the forthcoming shared-page table");
    });
}

extern "C" int cf_llama_kv_seq_shift(cf_llama_kv_adapter *adapter, uint64_t sequence_id, int32_t delta) {
    return guarded(adapter, [&] {  // compressed_kv_cache.cu:190-192
        if (sequence_id != 0 || delta != 0) throw std::runtime_error("non-zero context shift is not implemented");
    });
}

extern "C" int cf_llama_kv_clear(cf_llama_kv_adapter *adapter) {
    return guarded(adapter, [&] {
        cuda_check(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
        adapter->reset(nullptr);
    });
}

// Statistics in the reference's units (compressed_kv_cache.cu:198-210): a page is page_size tokens of one kv head.
extern "C" int cf_llama_kv_get_stats(const cf_llama_kv_adapter *adapter, cf_llama_kv_stats *stats) {
    if (adapter == nullptr || stats == nullptr) return -1;
    cf_llama_kv_stats out{};
    const uint32_t page = adapter->opt.page_size;
    for (const HeadState &h : adapter->heads) {
        out.appended_tokens += h.appended;
        const uint64_t whole = h.flushed_partial ? (h.sealed + page - 1) / page : h.sealed / page;
        const uint64_t sealed_tokens = h.flushed_partial ? h.sealed : whole * page;
        out.sealed_pages += whole;
        out.sealed_tokens += sealed_tokens;
        out.active_tokens += h.sealed + h.tail - sealed_tokens;
    }
    out.dense_active_bytes = out.active_tokens * adapter->opt.head_dim * 2 * sizeof(float);
    if (adapter->kivi) {
        out.compressed_bytes = adapter->kivi_resident_bytes;
        for (const auto &layer : adapter->kivi_host_descs) out.descriptor_bytes += layer.size() * sizeof(cf_kv_device_page);
    } else {
        unsigned long long units = 0;
        if (adapter->cursor.ptr) cudaMemcpy(&units, adapter->cursor.ptr, sizeof units, cudaMemcpyDeviceToHost);
        out.compressed_bytes = units * 16ull;
        out.descriptor_bytes = static_cast<uint64_t>(adapter->next_page_id) * adapter->opt.kv_head_count * sizeof(uint64_t);
    }
    *stats = out;
    return 0;
}

extern "C" const char *cf_llama_kv_last_error(const cf_llama_kv_adapter *adapter) {
    return adapter == nullptr ? "invalid ChromoFold KV adapter" : adapter->last_error.c_str();
}


// Additive: the device descriptor of a page of reference-exact mode (the reference's cf_kv_device_page: fixed-width words,
// K per-channel and V per-token fp32 scales), so that a test or a tool can read back exactly what was stored.
// page_index counts the pages of `layer` in the order they were sealed, over all kv heads. Returns -1 in format-v1 mode.
extern "C" uint64_t cf_b200_llama_kv_reserved_bytes(const cf_llama_kv_adapter *adapter) {
    return adapter ? static_cast<uint64_t>(adapter->kivi_chunks.size()) * cf_llama_kv_adapter::kKiviChunk : 0;
}

extern "C" int cf_b200_test_llama_kv_chunk_limit(cf_llama_kv_adapter *adapter, uint32_t chunks) {
    if (adapter == nullptr) return -1;
    adapter->kivi_chunk_limit = chunks;
    return 0;
}

extern "C" int cf_b200_llama_kv_reference_page(const cf_llama_kv_adapter *adapter, uint32_t layer, uint32_t page_index,
                                               cf_kv_device_page *out_page) {
    if (adapter == nullptr || out_page == nullptr || !adapter->kivi || layer >= adapter->kivi_host_descs.size() ||
        page_index >= adapter->kivi_host_descs[layer].size())
        return -1;
    adapter->kivi_written.wait();   // the caller reads the page by ways of its own
    *out_page = adapter->kivi_host_descs[layer][page_index];
    return 0;
}
