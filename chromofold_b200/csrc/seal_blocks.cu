// seal_blocks.cu — the sealer for 16-token pages of 64-symbol blocks (head_dim 128, 96, 80, 64, 32): the geometries the
// lane-per-block attention kernels read. It writes the same records as seal_pages_kernel (seal.cu), byte for byte.
//
// One WARP owns a (page, kv head) and a lane owns whole blocks, from the values to the coded bytes, so there is no barrier
// anywhere (two warps, a stream each, where that ends sooner: see kPair): a K block is 64 consecutive values of a token row (or of two), a V block is four channels of all sixteen tokens.
//   * head_dim 128: 32 blocks per stream, lane l codes K block l and V block l, interleaved (two independent chains);
//     head_dim 64 and 32: at most 16 per stream, lanes 0..15 code K and lanes 16..31 code V.
//   * values are loaded coalesced and quantised where they land, with a multiplication and the 1.5 * 2^23 rounding trick; the few whose quotient lies so close to
//     a half-integer that the product could round the other way take the IEEE division (see quantise_quad); the packed symbols go to the
//     slot of the block they belong to.
//   * the symbols wait in the block's slot of shared memory, the coded bytes grow down from the slot's end: a symbol codes into
//     at most 12 bits, so after 4 k symbols the bytes reach down to 100 - 6 k and the remaining symbols up to 64 - 4 k.
//   * block lengths become offsets with a warp scan, a lane moves its bytes into the part word by word (the words it shares
//     with a neighbour by atomicOr), the part leaves for the arena with 16-byte stores.
// Bound: the latency of a warp's own chain (table look-ups, one page's loads and stores) with 20 warps per SM to hide it: 3500
// warp instructions per page-head, issue slots 45 % busy (one warp per page-head). 2048 pages x 8 kv heads of binary16 tiles per
// launch, a 128-thread CTA per page-head, two of its warps coding and two waiting -> one warp -> two: nibble-split rANS 178 ->
// 133 -> 113 us, nibble-split Huffman 180 -> 140 -> 115, rANS 279 -> 176 -> 158, Huffman 253 -> 190 -> 168, fixed 8-bit 127 ->
// 90 -> 66.

#include <type_traits>

#include "seal_params.cuh"

namespace cfb {
namespace {

constexpr int kWarps = 10, kThreads = kWarps * 32;   // two CTAs per SM
constexpr uint32_t kSlot = 100;                      // bytes: 64 symbols; 64 * 12 bits + the bytes the start state sheds

template <int D>
struct Geo {
    static constexpr uint32_t kSyms = 16 * D, kBlocks = D / 4;
    static constexpr int kJobs = kBlocks > 16 ? 2 : 1;             // blocks per lane
    static constexpr uint32_t kPart = kSyms + 16;                  // a part never exceeds the fixed-width kSyms bytes
    static constexpr uint32_t kWarpBytes = kJobs * 32 * kSlot + 2 * kPart;
    static constexpr uint32_t kSmem = 2 * 256 * 16 + kWarps * kWarpBytes + 16;   // move_bytes reads a word past the last slot
};
static_assert(2 * Geo<128>::kSmem <= 232448 - 2 * 1024, "two CTAs per SM");

// A stream's quantiser (src/runtime/kv_gpu_fixture.cpp:12-16: round half to even of x / scale, clamped). With r = RN(1 / scale)
// the products x * r * (1 +- 2^-21) lie on either side of RN(x / scale), so where both round to the same integer that is the
// symbol; the few quads where they do not take the IEEE division. Adding 1.5 * 2^23 leaves the rounded value in the low
// mantissa bits: two FMAs per value. `exact`: the scale is so small (a binary16 denormal) or so large (capped) that the
// clamp matters; then every value is divided.
__device__ __noinline__ uint32_t divide_quad(float x0, float x1, float x2, float x3, float scale) {   // (once, not at every quad)
    return quantise_symbol(x0, scale) | quantise_symbol(x1, scale) << 8 | quantise_symbol(x2, scale) << 16 | quantise_symbol(x3, scale) << 24;
}
struct Quantiser {
    float scale, below, above;
    bool exact;
    __device__ __forceinline__ void set(uint16_t scale_bits, uint32_t magnitude) {
        scale = __half2float(__ushort_as_half(scale_bits));
        const float rcp = __frcp_rn(scale);
        below = rcp * (1.0f - 4.76837158203125e-07f);
        above = rcp * (1.0f + 4.76837158203125e-07f);
        exact = __uint_as_float(magnitude) * rcp > 127.4f;
    }
    // Four values -> four symbols, first in byte 0.
    __device__ __forceinline__ uint32_t quad(float x0, float x1, float x2, float x3) const {
        const float magic = 12582912.0f;
        auto pack = [&](float r) {
            const uint32_t t0 = __float_as_uint(__fmaf_rn(x0, r, magic)), t1 = __float_as_uint(__fmaf_rn(x1, r, magic));
            const uint32_t t2 = __float_as_uint(__fmaf_rn(x2, r, magic)), t3 = __float_as_uint(__fmaf_rn(x3, r, magic));
            return __byte_perm(__byte_perm(t0, t1, 0x0040), __byte_perm(t2, t3, 0x0040), 0x5410);
        };
        const uint32_t lo = pack(below), hi = pack(above);
        if (lo != hi || exact) return divide_quad(x0, x1, x2, x3, scale);
        return lo ^ 0x80808080u;
    }
};

__device__ __forceinline__ float2 half2_of(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2 *>(&v)); }
// Largest magnitude so far, as integers (inf and NaN lie above every finite value): one fp32, or two binary16 side by side.
template <bool kF32>
__device__ __forceinline__ uint32_t max_word(uint32_t m, uint32_t w) {
    if constexpr (kF32) return max(m, w & 0x7fffffffu);
    return __vmaxu2(m, w & 0x7fff7fffu);
}
template <bool kF32>
__device__ __forceinline__ uint32_t magnitude_of(uint32_t m) {   // as the bits of an fp32 value
    if constexpr (kF32) return m;
    return __float_as_uint(__half2float(__ushort_as_half(static_cast<unsigned short>(max(m & 0xffffu, m >> 16)))));
}

// The values of a tile as a warp reads them: 16-byte pieces of consecutive K values, four consecutive channels of each token
// for V, both coalesced. Rows past `rows` count as zeros.
template <int D, bool kF32>
struct KTile {
    static constexpr uint32_t kElem = kF32 ? 4 : 2, kPer = 16 / kElem;   // values of a piece
    static constexpr int kPieces = 16 * D / kPer / 32;
    uint4 piece[kPieces];
    __device__ __forceinline__ void load(const uint8_t *base, uint64_t row_bytes, uint32_t rows, uint32_t lane) {
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const uint32_t flat = (32u * i + lane) * kPer, t = flat / D, d = flat % D;
            piece[i] = t < rows ? *reinterpret_cast<const uint4 *>(base + t * row_bytes + d * kElem) : make_uint4(0u, 0u, 0u, 0u);
        }
    }
    __device__ __forceinline__ uint32_t absmax() const {
        uint32_t m = 0u;
#pragma unroll
        for (int i = 0; i < kPieces; ++i) m = max_word<kF32>(max_word<kF32>(max_word<kF32>(max_word<kF32>(m, piece[i].x), piece[i].y), piece[i].z), piece[i].w);
        return magnitude_of<kF32>(m);
    }
    // packed symbols to the slots of the blocks they belong to
    __device__ __forceinline__ void quantise(const Quantiser &q, uint8_t *slots, uint32_t lane) const {
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const uint32_t flat = (32u * i + lane) * kPer;
            uint32_t *to = reinterpret_cast<uint32_t *>(slots + (flat / 64u) * kSlot + flat % 64u);
            const uint4 x = piece[i];
            if constexpr (kF32) {
                to[0] = q.quad(__uint_as_float(x.x), __uint_as_float(x.y), __uint_as_float(x.z), __uint_as_float(x.w));
            } else {
                const float2 a = half2_of(x.x), b = half2_of(x.y), c = half2_of(x.z), d = half2_of(x.w);
                to[0] = q.quad(a.x, a.y, b.x, b.y);
                to[1] = q.quad(c.x, c.y, d.x, d.y);
            }
        }
    }
};
template <int D, bool kF32>
struct VTile {
    static constexpr uint32_t kElem = kF32 ? 4 : 2, kQuads = D / 4;                       // four-channel pieces of a token
    static constexpr uint32_t kLanes = kQuads > 16 ? 32 : kQuads > 8 ? 16 : 8;            // lanes that share a token
    static constexpr int kTokens = static_cast<int>(16 * kLanes / 32);                    // tokens of a lane: consecutive ones
    using Piece = typename std::conditional<kF32, float4, uint2>::type;
    Piece row[kTokens];
    __device__ __forceinline__ void load(const uint8_t *base, uint64_t row_bytes, uint32_t rows, uint32_t lane) {
        const uint32_t quad = lane % kLanes, first = lane / kLanes * kTokens;
#pragma unroll
        for (int t = 0; t < kTokens; ++t) {
            row[t] = Piece{};
            if (quad < kQuads && first + t < rows) row[t] = *reinterpret_cast<const Piece *>(base + (first + t) * row_bytes + 4u * quad * kElem);
        }
    }
    __device__ __forceinline__ float4 at(int t) const {
        if constexpr (kF32) return row[t];
        else {
            const float2 a = half2_of(row[t].x), b = half2_of(row[t].y);
            return make_float4(a.x, a.y, b.x, b.y);
        }
    }
    __device__ __forceinline__ uint32_t absmax() const {
        uint32_t m = 0u;
#pragma unroll
        for (int t = 0; t < kTokens; ++t) {
            if constexpr (kF32) {
                m = max_word<true>(max_word<true>(m, __float_as_uint(row[t].x)), __float_as_uint(row[t].y));
                m = max_word<true>(max_word<true>(m, __float_as_uint(row[t].z)), __float_as_uint(row[t].w));
            } else {
                m = max_word<false>(max_word<false>(m, row[t].x), row[t].y);
            }
        }
        return magnitude_of<kF32>(m);
    }
    __device__ __forceinline__ void quantise(const Quantiser &q, uint8_t *slots, uint32_t lane) const {
        const uint32_t quad = lane % kLanes, first = lane / kLanes * kTokens;
        if (quad >= kQuads) return;
        uint32_t *to = reinterpret_cast<uint32_t *>(slots + quad * kSlot) + first / 4u;   // [channel of the block][token quad]
#pragma unroll
        for (int tq = 0; tq < kTokens / 4; ++tq) {
            const float4 a = at(4 * tq), b = at(4 * tq + 1), c = at(4 * tq + 2), d = at(4 * tq + 3);
            to[tq] = q.quad(a.x, b.x, c.x, d.x);
            to[4 + tq] = q.quad(a.y, b.y, c.y, d.y);
            to[8 + tq] = q.quad(a.z, b.z, c.z, d.z);
            to[12 + tq] = q.quad(a.w, b.w, c.w, d.w);
        }
    }
};

// Coding table in shared memory, one 16-byte entry per symbol. rANS: {reciprocal, bound of the state, cum << 8 | shift, 4096 - f}
// (rans_enc of the codebook, taken apart once); Huffman: {length << 16 | code}.
__device__ __forceinline__ uint4 coder_entry(const cf_b200_codebook_tables *t, uint32_t sym, bool rans) {
    if (!rans) return make_uint4(t->huff_code[sym], 0u, 0u, 0u);
    const uint32_t rcp = t->rans_enc[sym][0], y = t->rans_enc[sym][1], cmpl = (y >> 13) & 0xfffu;   // cum | (4096 - f) << 13 | (shift - 1) << 25
    return make_uint4(rcp, (4096u - cmpl) << 19, (y & 0x1fffu) << 8 | (y >> 25), cmpl);
}

// While the state is not below its bound its low byte goes in front of the bytes written so far (predicated: as branches this
// diverged at every symbol).
__device__ __forceinline__ void shed_byte(uint32_t &x, uint32_t &p, uint32_t bound) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ge.u32 q, %0, %2;\n\t@q sub.u32 %1, %1, 1;\n\t@q st.shared.u8 [%1], %0;\n\t@q shr.u32 %0, %0, 8;\n\t}"
        : "+r"(x), "+r"(p)
        : "r"(bound)
        : "memory");
}

// kWords packed words of symbols at the bottom of each slot, pushed last to first; the bytes grow down from the slot's end.
// The update is src/cuda/rans.cu:20-22 run backwards: x + cum + floor(x / f) * (4096 - f), with the codebook's reciprocal.
template <int kJobs, int kWords>
__device__ __forceinline__ void rans_encode(uint8_t *const (&slot)[kJobs], const uint4 *const (&enc)[kJobs], uint32_t (&len)[kJobs], uint32_t (&state)[kJobs]) {
    uint32_t x[kJobs], p[kJobs], end[kJobs];   // p: shared-memory address of the last byte written
#pragma unroll
    for (int j = 0; j < kJobs; ++j) x[j] = kRansL, p[j] = end[j] = static_cast<uint32_t>(__cvta_generic_to_shared(slot[j] + kSlot));
#pragma unroll 1
    for (int w = kWords - 1; w >= 0; --w) {
        uint32_t word[kJobs];
#pragma unroll
        for (int j = 0; j < kJobs; ++j) word[j] = reinterpret_cast<const uint32_t *>(slot[j])[w];
#pragma unroll
        for (int k = 3; k >= 0; --k)
#pragma unroll
            for (int j = 0; j < kJobs; ++j) {
                const uint4 e = enc[j][(word[j] >> (8 * k)) & 0xffu];
                shed_byte(x[j], p[j], e.y);   // the state is below 2^31 and its bound at least 2^19: two bytes at most
                shed_byte(x[j], p[j], e.y);
                x[j] = __funnelshift_r(__umulhi(x[j], e.x), 0u, e.z) * e.w + (x[j] + (e.z >> 8));   // the shift takes e.z modulo 32
            }
    }
#pragma unroll
    for (int j = 0; j < kJobs; ++j) {
        state[j] = x[j];
        len[j] = end[j] - p[j];
    }
}

template <int kWords>
__device__ __forceinline__ uint32_t huffman_bits(const uint8_t *slot, const uint4 *enc) {
    uint32_t bits = 0;
#pragma unroll 4
    for (int w = 0; w < kWords; ++w) {
        const uint32_t word = reinterpret_cast<const uint32_t *>(slot)[w];
#pragma unroll
        for (int k = 0; k < 4; ++k) bits += enc[(word >> (8 * k)) & 0xffu].x >> 16;
    }
    return bits;
}
// MSB-first codes of the block at bit `bit` of the zeroed word array; the first and last word can be shared with a neighbour.
template <int kWords>
__device__ __forceinline__ void huffman_emit(const uint8_t *slot, const uint4 *enc, uint32_t *words, uint32_t bit) {
    uint32_t at = bit >> 5, filled = bit & 31u;
    unsigned long long acc = 0;
    bool first = true;
#pragma unroll 2
    for (int w = 0; w < kWords; ++w) {
        const uint32_t word = reinterpret_cast<const uint32_t *>(slot)[w];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t cl = enc[(word >> (8 * k)) & 0xffu].x, n = cl >> 16;
            acc |= static_cast<unsigned long long>(cl & 0xffffu) << (64u - filled - n);
            filled += n;
            if (filled >= 32u) {
                const uint32_t out = static_cast<uint32_t>(acc >> 32);
                if (first) atomicOr(&words[at], out);
                else words[at] = out;
                first = false;
                ++at;
                acc <<= 32;
                filled -= 32u;
            }
        }
    }
    if (filled) atomicOr(&words[at], static_cast<uint32_t>(acc >> 32));
}

// `len` bytes at `src` to `dst` in the zeroed part, a word at a time; the ends are shared with the neighbouring blocks.
__device__ __forceinline__ void move_bytes(const uint8_t *src, uint8_t *dst, uint32_t len) {
    if (len == 0) return;
    const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(dst)) & 3u;
    uint32_t *to = reinterpret_cast<uint32_t *>(dst - lead);
    const uint8_t *from = src - lead;   // stays inside the slot: bytes in front of it are other symbols or bytes, masked off
    const uint32_t skew = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(from)) & 3u, words = (lead + len + 3u) / 4u;
    const uint32_t *aligned = reinterpret_cast<const uint32_t *>(from - skew);
    const uint32_t tail = (lead + len) & 3u;
    uint32_t low = aligned[0], mask = 0xffffffffu << (8u * lead);
    for (uint32_t i = 0; i < words; ++i) {
        const uint32_t high = aligned[i + 1u];
        if (i + 1u == words && tail) mask &= 0xffffffffu >> (32u - 8u * tail);
        atomicOr(&to[i], __funnelshift_r(low, high, 8u * skew) & mask);
        low = high;
        mask = 0xffffffffu;
    }
}

struct CursorPlacement {};   // the public entry point: room from the arena cursor, page ids from job_pages

// What the two warps of a page-head tell each other (kPair).
struct StreamResult {
    uint32_t bytes, coder, scale_bits, magnitude;
};
__device__ __forceinline__ void pair_sync(uint32_t worker) { asm volatile("bar.sync %0, 64;" ::"r"(worker + 1u) : "memory"); }

// kPair: two warps share a page-head, one per stream. A launch with few page-heads lasts as long as one of them, and a warp that
// loads, quantises and codes both streams takes half as long again as two that take one each. Microseconds at head_dim 128 in
// nibble-split rANS, binary16 | fp32 (a 128-thread CTA per page-head took 14.3, 16.4, 18.4, 28.7, 43 | 14.4, 16.4, 20.4, 30.7, 45):
//                          8           512          1184         1600         2960 page-heads
//   one warp each     18.4 | 17.4  20.5 | 21.4  22.5 | 24.6       | 30.8  30.8 | 34.8
//   two warps each    12.3 | 12.3  12.3 | 14.3  16.4 | 18.4  22.5 |       28.7 | 36.9
template <int D, bool kF32, class Placement, bool kPair>
__global__ void __launch_bounds__(kThreads, 2) seal_blocks_kernel(const __grid_constant__ SealParams p, const __grid_constant__ Placement place) {
    using G = Geo<D>;
    static_assert(!kPair || G::kJobs == 2, "a warp per stream needs blocks for all of its lanes");
    constexpr int kJobs = kPair ? 1 : G::kJobs, kWorkers = kPair ? kWarps / 2 : kWarps;   // blocks per lane; page-heads at a time
    constexpr int kScan = G::kJobs == 2 ? 32 : 16;                                         // lanes that hold a stream's blocks
    constexpr bool kPlaced = std::is_same<Placement, SealPlacement>::value;
    __shared__ StreamResult s_result[kPair ? kWorkers : 1][2];
    __shared__ unsigned long long s_offset[kPair ? kWorkers : 1];
    extern __shared__ __align__(16) uint8_t smem[];
    uint4 *s_enc = reinterpret_cast<uint4 *>(smem);   // [K | V][256]
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t worker = kPair ? warp >> 1 : warp, role = kPair ? warp & 1u : 0u;   // role: the stream of a pair's warp
    uint8_t *parts = smem + 2 * 256 * 16 + worker * G::kWarpBytes, *slots = parts + 2 * G::kPart;
    const bool split = split_coder(p.coder), rans = rans_family(p.coder), fixed = p.coder == CF_B200_CODER_FIXED8;
    for (uint32_t i = tid; i < 512u; i += kThreads) {
        s_enc[i] = coder_entry(i < 256u ? p.k_tables : p.v_tables, i & 255u, rans);
    }
    if constexpr (kPlaced)
        if (blockIdx.x == 0 && tid == 0) place.used[p.job_count * p.kv_head_count] = *p.status;
    __syncthreads();
    const uint32_t head_bytes = rans ? align_up_u32(6u * G::kBlocks, 4u) : align_up_u32(2u * G::kBlocks, 4u);
    const uint32_t before = head_bytes + (split ? G::kSyms / 2u : 0u);   // block table, then the raw low-nibble plane, then the payload
    const uint32_t heads = p.job_heads ? 1u : p.kv_head_count;
    uint8_t *slot[kJobs];
    const uint4 *enc[kJobs];
    uint32_t stream[kJobs], block[kJobs];
    bool active[kJobs];
#pragma unroll
    for (int j = 0; j < kJobs; ++j) {
        stream[j] = kPair ? role : kJobs == 2 ? j : lane >> 4;
        block[j] = lane & (kScan - 1u);
        active[j] = block[j] < G::kBlocks;
        slot[j] = slots + ((kPair ? role : j) * 32u + lane) * kSlot;
        enc[j] = s_enc + 256u * stream[j];
    }

    // unit = job * heads + kv head; both move on by fixed steps
    const uint32_t stride = gridDim.x * kWorkers, stride_jobs = stride / heads, stride_heads = stride % heads;
    const uint32_t first = kPair ? worker * gridDim.x + blockIdx.x : blockIdx.x * kWorkers + worker;   // (few: spread over the SMs)
    uint32_t job = first / heads, head_at = first % heads;
    for (; job < p.job_count; job += stride_jobs, head_at += stride_heads, job += head_at >= heads, head_at -= head_at >= heads ? heads : 0u) {
        const uint32_t kv_head = p.job_heads ? p.job_heads[job] : head_at;
        const uint32_t rows = kPlaced ? 16u : p.job_tokens ? min(p.job_tokens[job], 16u) : 16u;
        const uint64_t row0 = kPlaced ? 16ull * job : p.job_rows ? p.job_rows[job] : 0u;
        const uint64_t at = (kPlaced ? 0ull : p.job_slots[job] * p.slot_stride) + kv_head * p.head_stride + row0 * p.row_stride;
        constexpr uint32_t kElem = kF32 ? 4u : 2u;
        const uint8_t *k_base = static_cast<const uint8_t *>(p.tail_k) + at * kElem, *v_base = static_cast<const uint8_t *>(p.tail_v) + at * kElem;
        const uint64_t row_bytes = p.row_stride * kElem;
        {   // the next page's rows into L2 while this one is coded: a 128-byte line per lane and pass
            uint32_t next_job = job + stride_jobs, next_head = head_at + stride_heads;
            if (next_head >= heads) next_head -= heads, ++next_job;
            if (next_job < p.job_count) {
                const uint64_t next = (kPlaced ? 0ull : p.job_slots[next_job] * p.slot_stride) + (p.job_heads ? p.job_heads[next_job] : next_head) * p.head_stride +
                                      (kPlaced ? 16ull * next_job : p.job_rows ? p.job_rows[next_job] : 0u) * p.row_stride;
                constexpr uint32_t kLines = (D * kElem + 127u) / 128u;   // of a row
                const uint32_t next_rows = kPlaced ? 16u : p.job_tokens ? min(p.job_tokens[next_job], 16u) : 16u;
#pragma unroll
                for (uint32_t i = lane; i < 16u * kLines; i += 32u)
                    if (i / kLines < next_rows) {
                        const uint64_t line = (next + (i / kLines) * p.row_stride) * kElem + (i % kLines) * 128u;
                        if (!kPair || role == 0u) asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const uint8_t *>(p.tail_k) + line));
                        if (!kPair || role == 1u) asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const uint8_t *>(p.tail_v) + line));
                    }
            }
        }
        __syncwarp();   // the previous page's slots and parts have been read
        uint32_t k_mag, v_mag;
        uint16_t k_bits, v_bits;
        if constexpr (kPair) {   // this warp's stream alone; what the other finds comes with its length
            Quantiser q;
            auto quantise = [&](auto &tile, const uint8_t *base, uint8_t *to) {
                tile.load(base, row_bytes, rows, lane);
                k_mag = v_mag = __reduce_max_sync(0xffffffffu, tile.absmax());
                k_bits = v_bits = scale_bits_from_absmax(__uint_as_float(k_mag));
                q.set(k_bits, k_mag);
                tile.quantise(q, to, lane);
            };
            if (role == 0u) {
                KTile<D, kF32> k;
                quantise(k, k_base, slots);
            } else {
                VTile<D, kF32> v;
                quantise(v, v_base, slots + 32u * kSlot);
            }
        } else {   // fp32 tiles one after the other: a lane holds 64 values of either
            KTile<D, kF32> k;
            VTile<D, kF32> v;
            k.load(k_base, row_bytes, rows, lane);
            if constexpr (!kF32) v.load(v_base, row_bytes, rows, lane);
            k_mag = __reduce_max_sync(0xffffffffu, k.absmax());
            k_bits = scale_bits_from_absmax(__uint_as_float(k_mag));
            Quantiser q;
            q.set(k_bits, k_mag);
            k.quantise(q, slots, lane);
            if constexpr (kF32) v.load(v_base, row_bytes, rows, lane);
            v_mag = __reduce_max_sync(0xffffffffu, v.absmax());
            v_bits = scale_bits_from_absmax(__uint_as_float(v_mag));
            q.set(v_bits, v_mag);
            v.quantise(q, slots + (kJobs == 2 ? 32u : 16u) * kSlot, lane);
        }
        if (rows == 0 || (!kPair && (k_mag >= 0x7f800000u || v_mag >= 0x7f800000u))) {   // finite validation failed: nothing is published
            if (lane == 0) {
                if (!kPlaced && p.status) atomicOr(p.status, CF_B200_DEVSTAT_NONFINITE);
                if constexpr (kPlaced) place.used[job * heads + head_at] = kSealRefused;
            }
            continue;
        }
        for (uint32_t i = lane; i < (kPair ? 1u : 2u) * G::kPart / 16u; i += 32u)
            reinterpret_cast<uint4 *>(parts + role * G::kPart)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
        uint32_t w[kJobs][16], len[kJobs], state[kJobs];
#pragma unroll
        for (int j = 0; j < kJobs; ++j) {
            len[j] = state[j] = 0u;
            uint32_t *in_slot = reinterpret_cast<uint32_t *>(slot[j]);
#pragma unroll
            for (int i = 0; i < 16; ++i) w[j][i] = in_slot[i];
            if (split) {
                // pair symbol = hi(s[2k]) << 4 | hi(s[2k+1]): with h = w & 0xf0f0f0f0, bytes 0 and 2 of h | h >> 12; plane
                // word = low nibbles of eight symbols, the first four in the low nibbles of the bytes
                uint32_t *plane = reinterpret_cast<uint32_t *>(parts + stream[j] * G::kPart + head_bytes) + block[j];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t h0 = w[j][2 * i] & 0xf0f0f0f0u, h1 = w[j][2 * i + 1] & 0xf0f0f0f0u;
                    in_slot[i] = __byte_perm(h0 | h0 >> 12, h1 | h1 >> 12, 0x6420);
                    if (active[j]) plane[i * G::kBlocks] = (w[j][2 * i] & 0x0f0f0f0fu) | (w[j][2 * i + 1] & 0x0f0f0f0fu) << 4;
                }
            }
        }
        if (rans) {
            if (split) rans_encode<kJobs, 8>(slot, enc, len, state);
            else rans_encode<kJobs, 16>(slot, enc, len, state);
        } else if (!fixed) {
#pragma unroll
            for (int j = 0; j < kJobs; ++j) len[j] = split ? huffman_bits<8>(slot[j], enc[j]) : huffman_bits<16>(slot[j], enc[j]);
        }
        // lengths to offsets, per stream
        uint32_t off[kJobs], run[2] = {0u, 0u};
#pragma unroll
        for (int j = 0; j < kJobs; ++j) {
            if (!active[j]) len[j] = 0u;
            uint32_t incl = len[j];
#pragma unroll
            for (int d = 1; d < kScan; d <<= 1) {
                const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d, kScan);
                if (block[j] >= static_cast<uint32_t>(d)) incl += up;
            }
            off[j] = incl - len[j];
            if constexpr (kScan == 32) {
                run[kPair ? role : j] = __shfl_sync(0xffffffffu, incl, 31);
            } else {
                run[0] = __shfl_sync(0xffffffffu, incl, 15);
                run[1] = __shfl_sync(0xffffffffu, incl, 31);
            }
        }
        uint32_t bytes[2], coder[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            bytes[s] = align_up_u32(before + (rans ? run[s] : 4u * ((run[s] + 31u) / 32u)), 16u);
            coder[s] = p.coder;
            if (fixed || bytes[s] > G::kSyms) bytes[s] = G::kSyms, coder[s] = CF_B200_CODER_FIXED8;   // would not shrink
        }
        if constexpr (kPair) {
            if (lane == 0) s_result[worker][role] = {role ? bytes[1] : bytes[0], role ? coder[1] : coder[0], k_bits, k_mag};
            pair_sync(worker);
            const StreamResult k = s_result[worker][0], v = s_result[worker][1];
            bytes[0] = k.bytes, bytes[1] = v.bytes, coder[0] = k.coder, coder[1] = v.coder;
            k_bits = static_cast<uint16_t>(k.scale_bits), v_bits = static_cast<uint16_t>(v.scale_bits);
            if (k.magnitude >= 0x7f800000u || v.magnitude >= 0x7f800000u) {
                if (role == 0u && lane == 0 && p.status) atomicOr(p.status, CF_B200_DEVSTAT_NONFINITE);
                pair_sync(worker);   // both have read the results
                continue;
            }
        }
        const uint32_t k_units = bytes[0] / 16u, units = 1u + k_units + bytes[1] / 16u;
        unsigned long long taken = 0;   // room in the arena: on its way while the parts are put together
        if (!kPlaced && role == 0u && lane == 0) taken = atomicAdd(p.cursor, static_cast<unsigned long long>(units));
        __syncwarp();   // (a split stream that falls back overwrites the plane its part already holds)
#pragma unroll
        for (int j = 0; j < kJobs; ++j) {
            if (!active[j]) continue;
            uint8_t *part = parts + stream[j] * G::kPart;
            if ((stream[j] ? coder[1] : coder[0]) == CF_B200_CODER_FIXED8) {   // fixed-width words, most significant byte first
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    reinterpret_cast<uint4 *>(part + 64u * block[j])[i] =
                        make_uint4(__byte_perm(w[j][4 * i], 0u, 0x0123), __byte_perm(w[j][4 * i + 1], 0u, 0x0123),
                                   __byte_perm(w[j][4 * i + 2], 0u, 0x0123), __byte_perm(w[j][4 * i + 3], 0u, 0x0123));
            } else if (rans) {
                reinterpret_cast<uint32_t *>(part)[block[j]] = state[j];
                reinterpret_cast<uint16_t *>(part + 4u * G::kBlocks)[block[j]] = static_cast<uint16_t>(off[j]);
                move_bytes(slot[j] + kSlot - len[j], part + before + off[j], len[j]);
            } else {
                reinterpret_cast<uint16_t *>(part)[block[j]] = static_cast<uint16_t>(off[j]);
                if (split) huffman_emit<8>(slot[j], enc[j], reinterpret_cast<uint32_t *>(part + before), off[j]);
                else huffman_emit<16>(slot[j], enc[j], reinterpret_cast<uint32_t *>(part + before), off[j]);
            }
        }
        uint64_t offset;
        uint32_t page;
        if constexpr (kPlaced) {
            const uint32_t page_slot = place.page_slot[job / place.tiles_per_page], tile = job % place.tiles_per_page;
            page = page_slot * place.tiles_per_page + 1u + tile;
            offset = 1ull + (static_cast<uint64_t>(page_slot) * place.tiles_per_page + tile) * heads * place.record_units + kv_head * place.record_units;
        } else {
            if constexpr (kPair) {
                if (role == 0u && lane == 0) s_offset[worker] = taken;
                pair_sync(worker);
                offset = s_offset[worker];
            } else {
                offset = __shfl_sync(0xffffffffu, taken, 0);
            }
            page = p.job_pages[job];
            if (offset + units > p.arena_units) {
                if (role == 0u && lane == 0 && p.status) atomicOr(p.status, CF_B200_DEVSTAT_ARENA_FULL);
                continue;
            }
        }
        __syncwarp();   // the parts are complete
        uint4 *dst = reinterpret_cast<uint4 *>(p.arena + 16ull * offset);
        if (role == 0u && lane == 0) {
            cf_b200_record_header h;
            h.k_part_units = static_cast<uint16_t>(k_units);
            h.v_part_units = static_cast<uint16_t>(bytes[1] / 16u);
            h.k_coder = static_cast<uint8_t>(coder[0]);
            h.v_coder = static_cast<uint8_t>(coder[1]);
            h.token_count = static_cast<uint16_t>(rows);
            h.k_scale_f16 = k_bits;
            h.v_scale_f16 = v_bits;
            h.codebook_id = static_cast<uint16_t>(p.codebook_id);
            h.flags = 0;
            h.version = CF_B200_FORMAT_VERSION;
            dst[0] = *reinterpret_cast<const uint4 *>(&h);
        }
        for (uint32_t i = lane + (kPair && role ? k_units : 0u); i + 1u < (kPair && !role ? 1u + k_units : units); i += 32u)
            dst[1u + i] = *reinterpret_cast<const uint4 *>(i < k_units ? parts + 16u * i : parts + G::kPart + 16u * (i - k_units));
        __threadfence();   // the record is in place before its directory entry is
        if constexpr (kPair) pair_sync(worker);
        else __syncwarp();
        if (role == 0u && lane == 0) {
            p.page_dir[static_cast<uint64_t>(page) * p.kv_head_count + kv_head] = CF_B200_DIR_ENTRY(offset, units);
            if constexpr (kPlaced) {
                place.used[job * heads + head_at] = units;
                if (kv_head == 0) place.table_row[job] = page;
            }
        }
    }
}

template <int D, bool kF32, bool kPair = false, class Placement>
cudaError_t launch_one(const SealParams &p, const Placement &place, cudaStream_t stream) {
    static LauncherState table[64];
    cudaError_t e;
    LauncherState *state = launcher_state(table, &e);
    if (!state) return e;
    if (!state->configured) {
        e = cudaFuncSetAttribute(seal_blocks_kernel<D, kF32, Placement, kPair>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Geo<D>::kSmem));
        if (e != cudaSuccess) return e;
        state->configured = true;
    }
    const uint64_t units = static_cast<uint64_t>(p.job_count) * (p.job_heads ? 1u : p.kv_head_count);
    const uint64_t wanted = kPair ? units : (units + kWarps - 1) / kWarps;
    const uint32_t grid = static_cast<uint32_t>(wanted < 2ull * state->sm_count ? wanted : 2ull * state->sm_count);
    seal_blocks_kernel<D, kF32, Placement, kPair><<<grid, kThreads, Geo<D>::kSmem, stream>>>(p, place);
    return cudaPeekAtLastError();
}

// Head_dim 128 through the public entry point, where launches of a page are usual: two warps per page-head for binary16 tiles; for fp32
// tiles, of which a lane holds twice as many registers, as long as all page-heads are resident at once (one warp each
// beyond that: 34.8 against 36.9 us for 2960, 64.4 against 62.3 for 5920).
template <bool kF32>
cudaError_t launch_128(const SealParams &p, const CursorPlacement &place, cudaStream_t stream) {
    if constexpr (!kF32) {
        return launch_one<128, false, true>(p, place, stream);
    } else {
        static LauncherState table[64];
        cudaError_t e;
        LauncherState *state = launcher_state(table, &e);
        if (!state) return e;
        const uint64_t units = static_cast<uint64_t>(p.job_count) * (p.job_heads ? 1u : p.kv_head_count);
        return units <= static_cast<uint64_t>(state->sm_count) * kWarps ? launch_one<128, true, true>(p, place, stream) : launch_one<128, true>(p, place, stream);
    }
}
template <bool kF32>
cudaError_t launch_128(const SealParams &p, const SealPlacement &place, cudaStream_t stream) {
    return launch_one<128, kF32>(p, place, stream);
}

template <class Placement>
cudaError_t launch_for(const SealParams &p, const Placement &place, cudaStream_t stream) {
    const bool f32 = p.tail_type == CF_B200_F32;
    switch (p.head_dim) {
        case 128: return f32 ? launch_128<true>(p, place, stream) : launch_128<false>(p, place, stream);
        case 96: return f32 ? launch_one<96, true>(p, place, stream) : launch_one<96, false>(p, place, stream);
        case 80: return f32 ? launch_one<80, true>(p, place, stream) : launch_one<80, false>(p, place, stream);
        case 64: return f32 ? launch_one<64, true>(p, place, stream) : launch_one<64, false>(p, place, stream);
        default: return f32 ? launch_one<32, true>(p, place, stream) : launch_one<32, false>(p, place, stream);
    }
}

}  // namespace

bool seal_blocks_supports(const SealParams &p) {
    const uint32_t d = p.head_dim, elem = p.tail_type == CF_B200_F32 ? 4u : 2u;
    return (d == 128 || d == 96 || d == 80 || d == 64 || d == 32) && p.page_tokens == 16 && p.block_size == 64 &&
           ((reinterpret_cast<uintptr_t>(p.tail_k) | reinterpret_cast<uintptr_t>(p.tail_v) | p.row_stride * elem | p.head_stride * elem |
             p.slot_stride * elem) & 15u) == 0;
}

cudaError_t launch_seal_blocks(const SealParams &p, cudaStream_t stream) { return launch_for(p, CursorPlacement{}, stream); }

cudaError_t launch_seal_placed(const SealParams &p, const SealPlacement &place, cudaStream_t stream) { return launch_for(p, place, stream); }

}  // namespace cfb
