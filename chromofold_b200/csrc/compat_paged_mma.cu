// compat_paged_mma.cu — cf_kv_paged_attention_async (src/cuda/paged_kv_attention.cu:41-176) at head_dim 128 and 64: attention
// over the reference's own page descriptors with the contractions on the tensor cores. Declared in compat_paged_mma.cuh.
//
// A row is one (query token, query head) of a kv head's group; a CTA owns 16 rows of one kv head (the m of
// mma.m16n8k16), its eight warps share out the 16-token groups of the head's visible pages and of the fp32 tail, and every
// warp keeps its own online softmax. The warps meet in shared memory, the CTAs of a split in `partials`.
//   * Fixed-width 4- and 8-bit words are loaded straight into mma fragments, in the layout they are stored in: the order of
//     the channels inside a contraction is free, so a lane takes 16 (V) or 32 (K) consecutive channels of a token instead
//     of the pairs the fragment names, and a token's row is read with one or two wide loads. Symbols become exact
//     binary16 codes (symbol - zero point) with a byte permute, a mask and one half2 operation per two symbols.
//   * A page's K scales are per channel: they go onto the queries, once per page and warp. q * scale is kept as binary16
//     value + binary16 residue after a power of two per row has been taken out, so that the product is good to 2^-22
//     whatever the magnitudes. V scales are per token: they go onto the softmax weights, in units of the largest scale met
//     so far (again a power of two), value + residue again.
//   * Variable-length pages, other code widths and unaligned words are decoded to bytes in the warp's shared memory, a
//     group at a time and one coded block per lane, and take the 8-bit path from there.
//   * The fp32 tail is contracted in 3 x tf32 (value and residue of both operands), good to fp32 as well.

#include <math_constants.h>

#include "cf_device_common.cuh"
#include "compat_paged_mma.cuh"

namespace cfb {
namespace {

constexpr int kMmaWarps = 8;
constexpr int kMmaThreads = kMmaWarps * 32;
constexpr float kLog2e = 1.4426950408889634f;
constexpr uint32_t kTailWeight = 3;
constexpr float kWeightScale = 32768.0f;   // weights are at most 1 (times a relative V scale of at most 1)

template <int D>
struct MmaLayout {
    static constexpr uint32_t kSteps = D / 16;                     // k16 steps of the score contraction
    static constexpr uint32_t kQueryBytes = 16 * D * 4;            // fp32 rows, fragment order
    static constexpr uint32_t kPlane = kSteps * 16 * 4 * 8;        // binary16 rows, fragment order: [step][row][lane & 3][4 channels]
    static constexpr uint32_t kWarpRows = 2 * kPlane;              // value plane, residue plane; reused for the warp's O at the end
    static constexpr uint32_t kSymbols = 16 * D;                   // one stream of one 16-token group
    static constexpr uint32_t kWarpBytes = kWarpRows + kSymbols;
    static constexpr uint32_t kOffWarps = kQueryBytes;
    static constexpr uint32_t kOffState = kOffWarps + kMmaWarps * kWarpBytes;   // (max, sum) per warp and row
    static constexpr uint32_t kOffTop = kOffState + kMmaWarps * 16 * 8;         // largest |q| of each row
    static constexpr uint32_t kOffScan = kOffTop + 16 * 4;
    static constexpr uint32_t kOffPages = kOffScan + 2 * kMmaWarps * 4 + 16;
    static_assert(16 * D * 4 <= kWarpRows, "a warp's O fits where its query planes were");
    static uint32_t bytes(uint32_t page_count) { return kOffPages + page_count * 6u + 16u; }
};

__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void tf32_split(float x, uint32_t &hi, uint32_t &lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
}
// The three products of (a_hi + a_lo) * (b_hi + b_lo) that matter, smallest first.
__device__ __forceinline__ void mma_3xtf32(float (&d)[4], const uint32_t (&ah)[4], const uint32_t (&al)[4], float b0, float b1) {
    uint32_t b0h, b0l, b1h, b1l;
    tf32_split(b0, b0h, b0l);
    tf32_split(b1, b1h, b1l);
    mma_tf32(d, al, b0h, b1h);
    mma_tf32(d, ah, b0l, b1l);
    mma_tf32(d, ah, b0h, b1h);
}
__device__ __forceinline__ uint32_t hfma2_u32(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t hsub2_u32(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ float2 unpack_half2(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2 *>(&v)); }

// Binary16 constants of a zero point: the code of symbol c is c - zp. 1024 + c has c in its mantissa, 1024 + 16 c a nibble
// that was left in the high half of its byte.
struct CodeBias {
    uint32_t minus, minus16, mixed_mul, mixed_add;   // (1024 + zp) x 2 | -(64 + zp) x 2 | (1/16, 1) | (-(64 + zp), -(1024 + zp))
    float rest;                                      // what of the zero point does not fit (above 1024): taken off afterwards
    __device__ __forceinline__ void set(uint32_t zp) {
        const float z = static_cast<float>(min(zp, 1024u));
        rest = static_cast<float>(zp - min(zp, 1024u));
        minus = pack_half2(1024.0f + z, 1024.0f + z);
        minus16 = pack_half2(-64.0f - z, -64.0f - z);
        mixed_mul = pack_half2(0.0625f, 1.0f);
        mixed_add = pack_half2(-64.0f - z, -1024.0f - z);
    }
};
constexpr uint32_t kMagic = 0x64006400u, kMagicBytes = 0x64646464u, kSixteenth = 0x2c002c00u;   // half2(1024), (1/16)

// Words of `kBytes` consecutive bytes, aligned to their size (at most 16).
template <int kBytes>
__device__ __forceinline__ void load_words(const uint8_t *src, uint32_t *dst) {
    if constexpr (kBytes >= 16) {
#pragma unroll
        for (int i = 0; i < kBytes / 16; ++i) {
            const uint4 v = reinterpret_cast<const uint4 *>(src)[i];
            dst[4 * i] = v.x, dst[4 * i + 1] = v.y, dst[4 * i + 2] = v.z, dst[4 * i + 3] = v.w;
        }
    } else if constexpr (kBytes == 8) {
        const uint2 v = *reinterpret_cast<const uint2 *>(src);
        dst[0] = v.x, dst[1] = v.y;
    } else {
        dst[0] = *reinterpret_cast<const uint32_t *>(src);
    }
}
__device__ __forceinline__ float4 load4(const float *p) {
    if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0) return *reinterpret_cast<const float4 *>(p);
    return make_float4(p[0], p[1], p[2], p[3]);
}

// Symbols [lo, hi) of a coded stream to bytes at (index - lo) ^ 3 (most significant byte first in a word, as the 8-bit pages
// are), a coded block per lane.
__device__ __noinline__ void decode_group(const uint32_t *words, const int32_t *offsets, const int32_t *lut, uint32_t maxlen, uint32_t fixed_bits,
                                          uint32_t block_size, uint32_t total, uint32_t lo, uint32_t hi, uint8_t *dst, uint32_t lane) {
    const uint32_t b_last = (hi - 1u) / block_size;
    for (uint32_t b = lo / block_size + lane; b <= b_last; b += 32u) {
        const uint32_t first = b * block_size, last = min(min(first + block_size, total), hi);
        if (fixed_bits) {
            const uint32_t mask = (1u << fixed_bits) - 1u;
            for (uint32_t i = max(first, lo); i < last; ++i) {
                const uint32_t bit = i * fixed_bits;
                dst[(i - lo) ^ 3u] = static_cast<uint8_t>((words[bit >> 5] >> ((32u - fixed_bits) - (bit & 31u))) & mask);
            }
        } else {
            uint32_t bit = static_cast<uint32_t>(offsets[b]);
            for (uint32_t i = first; i < last; ++i) {   // include/chromofold/detail/block_huffman_device.cuh:12-19
                const uint32_t w = bit >> 5, off = bit & 31u;
                uint32_t window = words[w] << off;
                if (off + maxlen > 32u) window |= words[w + 1] >> (32u - off);
                const uint32_t entry = static_cast<uint32_t>(lut[window >> (32u - maxlen)]);
                if (i >= lo) dst[(i - lo) ^ 3u] = static_cast<uint8_t>(entry & 0xffu);
                bit += entry >> 8;
            }
        }
    }
}

// The running state of one warp: rows g and g + 8 of the CTA's sixteen (g = lane / 4), tokens and channels by lane % 4. With
// NR = 1 the tile has at most eight rows (a decode step) and nothing is kept or computed for the upper half.
template <int D, int NR>
struct Rows {
    float acc[D / 8][4];   // n-tile j: channel g' * D / 8 + j of column g' = 2 (lane & 3) + {0, 1}, rows g | g + 8
    float m[NR], l[NR];    // l: this lane's tokens only
    float v_unit;          // O is kept in units of v_unit / kWeightScale; 0 = nothing accumulated yet

    // Online softmax over the 16 tokens whose scores (log2 units, -inf = not visible) are in s[tile][row pair]; the weights
    // replace the scores, times factor(tile, column) of their token.
    template <class Factor>
    __device__ __forceinline__ void softmax(float (&s)[2][4], float unit, Factor factor) {
        const float f = v_unit == unit ? 1.0f : __fdividef(v_unit, unit);   // powers of two
        v_unit = unit;
        float a[NR], z[NR];
        bool moved = false;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            float top = fmaxf(fmaxf(s[0][2 * r], s[0][2 * r + 1]), fmaxf(s[1][2 * r], s[1][2 * r + 1]));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float next = fmaxf(m[r], top);
            z[r] = next == -CUDART_INF_F ? 0.0f : next;
            a[r] = exp2f(m[r] - z[r]);
            m[r] = next;
            moved = moved || a[r] * f != 1.0f;
        }
        if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
            for (int j = 0; j < D / 8; ++j)
#pragma unroll
                for (int r = 0; r < NR; ++r) acc[j][2 * r] *= a[r] * f, acc[j][2 * r + 1] *= a[r] * f;
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            float sum = 0.0f;
#pragma unroll
            for (int tile = 0; tile < 2; ++tile)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float p = exp2f(s[tile][2 * r + c] - z[r]);
                    sum += p;
                    s[tile][2 * r + c] = p * factor(tile, c);
                }
            l[r] = l[r] * a[r] + sum;
        }
    }
};

// Smallest power of two that is not below v (v >= 0).
__device__ __forceinline__ float power_above(float v) {
    return __uint_as_float(min((min(__float_as_uint(v), 0x7f000000u) + 0x7fffffu) & 0x7f800000u, 0x7f000000u));
}

// One 16-token group of a page. kBits: width of the words at `k` / `v` (the page's own, or the decoded bytes of the group).
template <int D, int NR, int kBits, bool kDecoded>
__device__ __forceinline__ void page_group(Rows<D, NR> &st, const cf_kv_device_page &page, uint32_t t0, const uint8_t *planes, uint8_t *symbols,
                                           const float (&inv_scale)[NR], const float (&query_sum)[NR], const CodeBias &bias,
                                           const uint32_t (&qtok)[NR], const uint32_t (&first)[NR], uint32_t lane) {
    using L = MmaLayout<D>;
    constexpr int kKWords = D / 4 * kBits / 32, kVWords = D / 8 * kBits / 32;   // words of a lane's share of one token
    constexpr uint32_t kRowBytes = D * kBits / 8;
    const uint32_t g = lane >> 2, t = lane & 3u, count = page.token_count;
    const uint8_t *k_rows, *v_rows;
    if constexpr (kDecoded) {
        const uint32_t total = count * D, lo = t0 * D, hi = min(t0 + 16u, count) * D;
        __syncwarp();
        decode_group(page.k_words, page.k_block_offsets, page.k_lut, page.k_max_code_length, page.fixed_code_length, page.block_size,
                     total, lo, hi, symbols, lane);
        __syncwarp();
        k_rows = v_rows = symbols;
    } else {
        k_rows = reinterpret_cast<const uint8_t *>(page.k_words) + static_cast<size_t>(t0) * kRowBytes;
        v_rows = reinterpret_cast<const uint8_t *>(page.v_words) + static_cast<size_t>(t0) * kRowBytes;
    }
    uint32_t kw[2][kKWords], vw[4][kVWords];
#pragma unroll
    for (int tile = 0; tile < 2; ++tile) {
#pragma unroll
        for (int i = 0; i < kKWords; ++i) kw[tile][i] = 0u;
        if (t0 + 8u * tile + g < count) load_words<4 * kKWords>(k_rows + (8u * tile + g) * kRowBytes + t * (4 * kKWords), kw[tile]);
    }
    auto load_v = [&]() {
#pragma unroll
        for (int i = 0; i < 4; ++i) {   // tokens 2t, 2t + 1, 2t + 8, 2t + 9 of the group
            const uint32_t tok = 2u * t + (i & 1) + 8u * (i >> 1);
#pragma unroll
            for (int w = 0; w < kVWords; ++w) vw[i][w] = 0u;
            if (t0 + tok < count) load_words<4 * kVWords>(v_rows + tok * kRowBytes + g * (4 * kVWords), vw[i]);
        }
    };
    if constexpr (!kDecoded) load_v();
    float scale[2][2];   // V scales of the lane's four tokens
#pragma unroll
    for (int tile = 0; tile < 2; ++tile)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const uint32_t tok = t0 + 8u * tile + 2u * t + c;
            scale[tile][c] = tok < count ? page.v_scales[tok] : 0.0f;
        }

    // S = (q scaled) . codes, value and residue of the rows as two operands
    float s[2][4] = {};
#pragma unroll
    for (int step = 0; step < static_cast<int>(L::kSteps); ++step) {
        const uint2 h0 = *reinterpret_cast<const uint2 *>(planes + ((step * 16u + g) * 4u + t) * 8u);
        const uint2 l0 = *reinterpret_cast<const uint2 *>(planes + L::kPlane + ((step * 16u + g) * 4u + t) * 8u);
        uint2 h1 = make_uint2(0u, 0u), l1 = make_uint2(0u, 0u);
        if constexpr (NR == 2) {
            h1 = *reinterpret_cast<const uint2 *>(planes + ((step * 16u + g + 8u) * 4u + t) * 8u);
            l1 = *reinterpret_cast<const uint2 *>(planes + L::kPlane + ((step * 16u + g + 8u) * 4u + t) * 8u);
        }
#pragma unroll
        for (int tile = 0; tile < 2; ++tile) {
            uint32_t b0, b1;
            if constexpr (kBits == 4) {
                const uint32_t w = kw[tile][step >> 1];
                const uint32_t p0 = __byte_perm(w, 0u, (step & 1) ? 0x4141 : 0x4343), p1 = __byte_perm(w, 0u, (step & 1) ? 0x4040 : 0x4242);
                b0 = hfma2_u32((p0 & 0x000f00f0u) | kMagic, bias.mixed_mul, bias.mixed_add);
                b1 = hfma2_u32((p1 & 0x000f00f0u) | kMagic, bias.mixed_mul, bias.mixed_add);
            } else {
                const uint32_t w = kw[tile][step];
                b0 = hsub2_u32(__byte_perm(w, kMagicBytes, 0x4243), bias.minus);
                b1 = hsub2_u32(__byte_perm(w, kMagicBytes, 0x4041), bias.minus);
            }
            mma_f16(s[tile], h0.x, h1.x, h0.y, h1.y, b0, b1);
            mma_f16(s[tile], l0.x, l1.x, l0.y, l1.y, b0, b1);
        }
    }
    if constexpr (kDecoded) {
        __syncwarp();   // the K bytes have been read
        const uint32_t total = count * D, lo = t0 * D, hi = min(t0 + 16u, count) * D;
        decode_group(page.v_words, page.v_block_offsets, page.v_lut, page.v_max_code_length, page.fixed_code_length, page.block_size,
                     total, lo, hi, symbols, lane);
        __syncwarp();
        load_v();
    }
    float top = 1e-30f;
#pragma unroll
    for (int tile = 0; tile < 2; ++tile)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            top = fmaxf(top, fabsf(scale[tile][c]));
            const uint32_t in_page = t0 + 8u * tile + 2u * t + c, token = page.token_begin + in_page;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const float x = s[tile][2 * r + c] - bias.rest * query_sum[r];
                s[tile][2 * r + c] = in_page < count && token >= first[r] && token <= qtok[r] ? x * inv_scale[r] : -CUDART_INF_F;
            }
        }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    const float unit = top > st.v_unit ? power_above(top) : st.v_unit, to_unit = kWeightScale / unit;
    st.softmax(s, unit, [&](int tile, int c) { return scale[tile][c] * to_unit; });
    if (bias.rest != 0.0f) {   // sum_t w_t (c_t - zp) = sum_t w_t (c_t - 1024) - rest * sum_t w_t
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            float w = s[0][2 * r] + s[0][2 * r + 1] + s[1][2 * r] + s[1][2 * r + 1];
            w += __shfl_xor_sync(0xffffffffu, w, 1);
            w += __shfl_xor_sync(0xffffffffu, w, 2);
#pragma unroll
            for (int j = 0; j < D / 8; ++j) st.acc[j][2 * r] -= bias.rest * w, st.acc[j][2 * r + 1] -= bias.rest * w;
        }
    }
    // O += P V
    uint32_t ph[4], pl[4];   // A fragments: (row g, tile 0) (row g + 8, tile 0) (row g, tile 1) (row g + 8, tile 1)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        ph[i] = pl[i] = 0u;
        if (NR == 1 && (i & 1)) continue;
        const float w0 = s[i >> 1][2 * (i & 1)], w1 = s[i >> 1][2 * (i & 1) + 1];
        ph[i] = pack_half2(w0, w1);
        const float2 back = unpack_half2(ph[i]);
        pl[i] = pack_half2(w0 - back.x, w1 - back.y);
    }
#pragma unroll
    for (int w = 0; w < kVWords; ++w)
#pragma unroll
        for (int k = 0; k < 4; ++k) {   // bytes of the word, most significant first
            const uint32_t sel = (3u - k) * 0x11u + (7u - k) * 0x1100u;
            const uint32_t p0 = __byte_perm(vw[0][w], vw[1][w], sel), p1 = __byte_perm(vw[2][w], vw[3][w], sel);
            if constexpr (kBits == 4) {
                const int j = 8 * w + 2 * k;
                uint32_t b0 = hfma2_u32((p0 & 0x00f000f0u) | kMagic, kSixteenth, bias.minus16);
                uint32_t b1 = hfma2_u32((p1 & 0x00f000f0u) | kMagic, kSixteenth, bias.minus16);
                mma_f16(st.acc[j], ph[0], ph[1], ph[2], ph[3], b0, b1);
                mma_f16(st.acc[j], pl[0], pl[1], pl[2], pl[3], b0, b1);
                b0 = hsub2_u32((p0 & 0x000f000fu) | kMagic, bias.minus);
                b1 = hsub2_u32((p1 & 0x000f000fu) | kMagic, bias.minus);
                mma_f16(st.acc[j + 1], ph[0], ph[1], ph[2], ph[3], b0, b1);
                mma_f16(st.acc[j + 1], pl[0], pl[1], pl[2], pl[3], b0, b1);
            } else {
                const uint32_t b0 = hsub2_u32((p0 & 0x00ff00ffu) | kMagic, bias.minus), b1 = hsub2_u32((p1 & 0x00ff00ffu) | kMagic, bias.minus);
                mma_f16(st.acc[4 * w + k], ph[0], ph[1], ph[2], ph[3], b0, b1);
                mma_f16(st.acc[4 * w + k], pl[0], pl[1], pl[2], pl[3], b0, b1);
            }
        }
}

// Largest magnitude of four values and m; NaN wins.
__device__ __forceinline__ float top4(float m, const float4 &x) {
    asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(fabsf(x.x)), "f"(fabsf(x.y)));
    asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(fabsf(x.z)), "f"(fabsf(x.w)));
    return m;
}

// One 16-token group of the fp32 tail ([token][kv head][D]; paged_kv_attention.cu:154-166). Unlike a page's values the tail's are
// whatever the caller has, and products by value and residue spread NaN and infinities (0 * inf, inf - inf). A group with some among
// its K takes its scores one by one in fp32; so do four channels of V with some among them their products: they end where fp32
// arithmetic puts them, and a token that a row does not see adds nothing.
template <int D, int NR>
__device__ __forceinline__ void tail_group(Rows<D, NR> &st, const cf_kv_paged_attention_desc &desc, uint32_t kv_head, uint32_t t0, const float *q_rows,
                                           const uint32_t (&qtok)[NR], const uint32_t (&first)[NR], uint32_t lane) {
    const uint32_t g = lane >> 2, t = lane & 3u, count = desc.active_token_count;
    const size_t stride = static_cast<size_t>(desc.kv_head_count) * D;
    const float *k0 = desc.active_k + static_cast<size_t>(kv_head) * D, *v0 = desc.active_v + static_cast<size_t>(kv_head) * D;
    float s[2][4] = {};
#pragma unroll 2
    for (uint32_t step = 0; step < D / 16u; ++step) {   // 16 channels: two k8 steps
        const float4 qa = *reinterpret_cast<const float4 *>(q_rows + ((step * 16u + g) * 4u + t) * 4u);
        const float4 qb = NR == 2 ? *reinterpret_cast<const float4 *>(q_rows + ((step * 16u + g + 8u) * 4u + t) * 4u) : make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t ah[2][4], al[2][4];
        tf32_split(qa.x, ah[0][0], al[0][0]), tf32_split(qb.x, ah[0][1], al[0][1]);
        tf32_split(qa.y, ah[0][2], al[0][2]), tf32_split(qb.y, ah[0][3], al[0][3]);
        tf32_split(qa.z, ah[1][0], al[1][0]), tf32_split(qb.z, ah[1][1], al[1][1]);
        tf32_split(qa.w, ah[1][2], al[1][2]), tf32_split(qb.w, ah[1][3], al[1][3]);
#pragma unroll
        for (int tile = 0; tile < 2; ++tile) {
            const uint32_t tok = t0 + 8u * tile + g;
            const float4 k = tok < count ? load4(k0 + tok * stride + t * (D / 4) + 4u * step) : make_float4(0.f, 0.f, 0.f, 0.f);
            mma_3xtf32(s[tile], ah[0], al[0], k.x, k.y);
            mma_3xtf32(s[tile], ah[1], al[1], k.z, k.w);
        }
    }
    bool odd = false;   // an infinity's residue is NaN, so its token's scores are
#pragma unroll
    for (int tile = 0; tile < 2; ++tile)
#pragma unroll
        for (int i = 0; i < 2 * NR; ++i) odd = odd || isnan(s[tile][i]);
    if (__any_sync(0xffffffffu, odd)) {
#pragma unroll
        for (int tile = 0; tile < 2; ++tile)
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const uint32_t tok = t0 + 8u * tile + 2u * t + c;
                    float dot = 0.0f;
#pragma unroll 1
                    for (uint32_t i = 0; i < (tok < count ? D / 4u : 0u); ++i) {   // four channels: (step, lane & 3) of the row's order
                        const float4 q = *reinterpret_cast<const float4 *>(q_rows + (((i >> 2) * 16u + g + 8u * r) * 4u + (i & 3u)) * 4u);
                        const float4 k = load4(k0 + tok * stride + (i & 3u) * (D / 4) + 4u * (i >> 2));
                        dot += (q.x * k.x + q.y * k.y) + (q.z * k.z + q.w * k.w);
                    }
                    s[tile][2 * r + c] = dot;
                }
    }
#pragma unroll
    for (int tile = 0; tile < 2; ++tile)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const uint32_t in_tail = t0 + 8u * tile + 2u * t + c, token = desc.active_token_begin + in_tail;
#pragma unroll
            for (int r = 0; r < NR; ++r)
                if (!(in_tail < count && token >= first[r] && token <= qtok[r])) s[tile][2 * r + c] = -CUDART_INF_F;
        }
    // The tail comes after the pages and its weights stay in fp32: O goes over to plain units, in which nothing overflows that the
    // sums themselves do not (in units of pages with tiny scales an ordinary value would).
    const float unit = fmaxf(st.v_unit, kWeightScale), to_unit = kWeightScale / unit;
    st.softmax(s, unit, [&](int, int) { return to_unit; });
#pragma unroll 1
    for (int tile = 0; tile < 2; ++tile) {   // k index t = token 2t, t + 4 = token 2t + 1 of the tile
        const float w0 = tile ? s[1][0] : s[0][0], w1 = tile ? s[1][1] : s[0][1], w2 = NR == 1 ? 0.0f : tile ? s[1][2] : s[0][2], w3 = NR == 1 ? 0.0f : tile ? s[1][3] : s[0][3];
        uint32_t ah[4], al[4];
        tf32_split(w0, ah[0], al[0]), tf32_split(w2, ah[1], al[1]);
        tf32_split(w1, ah[2], al[2]), tf32_split(w3, ah[3], al[3]);
        const uint32_t tok = t0 + 8u * tile + 2u * t;
        const float *va = v0 + tok * stride + g * (D / 8), *vb = va + stride;
        odd = false;
#pragma unroll
        for (int j = 0; j < D / 8; j += 4) {
            float4 a = tok < count ? load4(va + j) : make_float4(0.f, 0.f, 0.f, 0.f);
            float4 b = tok + 1u < count ? load4(vb + j) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (!(top4(top4(0.0f, a), b) < CUDART_INF_F)) a = b = make_float4(0.f, 0.f, 0.f, 0.f), odd = true;
            mma_3xtf32(st.acc[j], ah, al, a.x, b.x);
            mma_3xtf32(st.acc[j + 1], ah, al, a.y, b.y);
            mma_3xtf32(st.acc[j + 2], ah, al, a.z, b.z);
            mma_3xtf32(st.acc[j + 3], ah, al, a.w, b.w);
        }
        if (!__any_sync(0xffffffffu, odd)) continue;
#pragma unroll 1
        for (uint32_t i = 0; i < 8u; ++i) {   // what was left out above (four channels of two tokens), for the rows and columns whose sums this lane holds
            const uint32_t at = t0 + 8u * tile + i, pair = at ^ 1u, from = (lane & 28u) | (i >> 1);
            const float wa = __shfl_sync(0xffffffffu, i & 1u ? w1 : w0, from), wb = __shfl_sync(0xffffffffu, i & 1u ? w3 : w2, from);
            if (at >= count) continue;
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int j = 0; j < D / 8; j += 4) {
                    const uint32_t channel = (2u * t + c) * (D / 8) + j;
                    const float4 v = load4(v0 + at * stride + channel);
                    const float4 other = pair < count ? load4(v0 + pair * stride + channel) : make_float4(0.f, 0.f, 0.f, 0.f);
                    if (top4(top4(0.0f, v), other) < CUDART_INF_F) continue;
                    if (wa != 0.0f) st.acc[j][c] += wa * v.x, st.acc[j + 1][c] += wa * v.y, st.acc[j + 2][c] += wa * v.z, st.acc[j + 3][c] += wa * v.w;
                    if (NR == 2 && wb != 0.0f)
                        st.acc[j][2 + c] += wb * v.x, st.acc[j + 1][2 + c] += wb * v.y, st.acc[j + 2][2 + c] += wb * v.z, st.acc[j + 3][2 + c] += wb * v.w;
                }
        }
    }
}

// Grid: (16-row tile, kv head, split). 128 registers: two CTAs per SM.
template <int D, int NR>
__global__ void __launch_bounds__(kMmaThreads, 2) paged_mma_kernel(cf_kv_paged_attention_desc desc, uint32_t splits, float *partials,
                                                                  uint32_t *arrived) {
    using L = MmaLayout<D>;
    extern __shared__ __align__(16) uint8_t smem[];
    float *q_rows = reinterpret_cast<float *>(smem);   // q * softmax_scale * log2(e)
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, g = lane >> 2, t = lane & 3u;
    uint8_t *planes = smem + L::kOffWarps + warp * L::kWarpBytes, *symbols = planes + L::kWarpRows;
    float2 *state = reinterpret_cast<float2 *>(smem + L::kOffState);
    uint32_t *q_top = reinterpret_cast<uint32_t *>(smem + L::kOffTop);
    uint32_t *scan = reinterpret_cast<uint32_t *>(smem + L::kOffScan);
    uint32_t *prefix = reinterpret_cast<uint32_t *>(smem + L::kOffPages);                       // groups before page m of the list
    uint16_t *match = reinterpret_cast<uint16_t *>(smem + L::kOffPages + 4u * desc.page_count);   // its descriptor
    __shared__ uint32_t s_last;
    const uint32_t G = desc.gqa_group_size, rows_total = desc.query_count * G;
    const uint32_t row0 = blockIdx.x * 16u, kv_head = blockIdx.y, split = blockIdx.z;
    const uint32_t last_row = min(row0 + 15u, rows_total - 1u);
    const uint32_t newest = desc.query_token_begin + last_row / G;                               // of the CTA's query tokens
    const uint32_t oldest_visible = window_begin(desc.query_token_begin + row0 / G, desc.causal_window);

    // The visible pages of this kv head in descriptor order, with the 16-token groups before each.
    const uint32_t run = (desc.page_count + kMmaThreads - 1) / kMmaThreads;   // at most 16
    const uint32_t run_begin = min(tid * run, desc.page_count), run_end = min(run_begin + run, desc.page_count);
    uint32_t mine = 0, my_pages = 0, my_groups = 0;
#pragma unroll 4
    for (uint32_t pi = run_begin; pi < run_end; ++pi) {
        const cf_kv_device_page *p = desc.pages + pi;
        const uint2 span = *reinterpret_cast<const uint2 *>(&p->token_begin);   // begin, count
        const uint32_t head = p->kv_head, dim = p->head_dim;
        const bool take = head == kv_head && dim == D && span.y != 0 && span.x <= newest && span.x + span.y > oldest_visible;
        mine |= static_cast<uint32_t>(take) << (pi - run_begin);
        my_pages += take;
        my_groups += take ? (span.y + 15u) / 16u : 0u;
    }
    if (tid < 16u) q_top[tid] = 0u;
    __syncthreads();
    for (uint32_t i = tid; i < 16u * (D / 4u); i += kMmaThreads) {   // (step, row, lane & 3) -> four channels
        const uint32_t tt = i & 3u, row = (i >> 2) & 15u, step = i >> 6;
        if (NR == 1 && row >= 8u) continue;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row0 + row < rows_total) {
            const uint32_t r = row0 + row;
            v = load4(desc.queries + (static_cast<size_t>(r / G) * desc.query_head_count + kv_head * G + r % G) * D + tt * (D / 4) + 4u * step);
            const float f = desc.softmax_scale * kLog2e;
            v.x *= f, v.y *= f, v.z *= f, v.w *= f;
            atomicMax(&q_top[row], __float_as_uint(fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)))));   // magnitudes order as integers
        }
        reinterpret_cast<float4 *>(q_rows)[i] = v;
    }
    uint32_t pages_incl = my_pages, groups_incl = my_groups;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, pages_incl, o), b = __shfl_up_sync(0xffffffffu, groups_incl, o);
        if (lane >= static_cast<uint32_t>(o)) pages_incl += a, groups_incl += b;
    }
    if (lane == 31u) scan[warp] = pages_incl, scan[kMmaWarps + warp] = groups_incl;
    __syncthreads();
    uint32_t matches = 0, page_groups = 0, at = pages_incl - my_pages, groups_before = groups_incl - my_groups;
#pragma unroll
    for (uint32_t w = 0; w < kMmaWarps; ++w) {
        if (w < warp) at += scan[w], groups_before += scan[kMmaWarps + w];
        matches += scan[w];
        page_groups += scan[kMmaWarps + w];
    }
    for (uint32_t pi = run_begin; pi < run_end; ++pi)
        if (mine >> (pi - run_begin) & 1u) {
            match[at] = static_cast<uint16_t>(pi);
            prefix[at++] = groups_before;
            groups_before += (desc.pages[pi].token_count + 15u) / 16u;
        }
    __syncthreads();

    Rows<D, NR> st;
#pragma unroll
    for (int j = 0; j < D / 8; ++j) st.acc[j][0] = st.acc[j][1] = st.acc[j][2] = st.acc[j][3] = 0.0f;
    st.v_unit = 0.0f;
    uint32_t qtok[NR], first[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        st.m[r] = -CUDART_INF_F;
        st.l[r] = 0.0f;
        qtok[r] = desc.query_token_begin + min(row0 + g + 8u * r, last_row) / G;
        first[r] = window_begin(qtok[r], desc.causal_window);
    }

    // This warp's share of the groups: pages first, then the tail, one of whose groups (fp32 loads, three products) weighs
    // as much as kTailWeight of the pages' and belongs to the warp its first unit falls to.
    const uint64_t total = static_cast<uint64_t>(page_groups) + kTailWeight * ((desc.active_token_count + 15u) / 16u);
    const uint32_t workers = splits * kMmaWarps, worker = split * kMmaWarps + warp;
    uint64_t at_group, end_group;
    if (total < (1u << 22)) {   // at most 512 workers: 32-bit divisions do
        at_group = static_cast<uint32_t>(total) * worker / workers;
        end_group = static_cast<uint32_t>(total) * (worker + 1u) / workers;
    } else {
        at_group = total * worker / workers;
        end_group = total * (worker + 1u) / workers;
    }
    uint32_t m_at = 0;
    if (at_group < end_group && at_group < page_groups) {   // the last page that starts at or before the first group
        uint32_t lo = 0, hi = matches;
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (prefix[mid] <= at_group) lo = mid; else hi = mid;
        }
        m_at = lo;
    }
    while (at_group < end_group && at_group < page_groups) {
        const cf_kv_device_page page = desc.pages[match[m_at]];
        const uint32_t g0 = static_cast<uint32_t>(at_group) - prefix[m_at];
        const uint32_t page_end = m_at + 1u < matches ? prefix[m_at + 1u] : page_groups;
        const uint32_t stop = static_cast<uint32_t>(min(end_group, static_cast<uint64_t>(page_end))) - prefix[m_at];
        if (page.fixed_code_length != 0u && lane < 24u) {   // the first two groups' bytes on their way while the rows are scaled
            const uint32_t row_bytes = D * page.fixed_code_length / 8u, bytes = min(32u, page.token_count - 16u * g0) * row_bytes;
            const uint32_t *words = lane & 1u ? page.v_words : page.k_words;
            if ((lane >> 1) * 512u < bytes) {
                const uint8_t *at = reinterpret_cast<const uint8_t *>(words) + 16u * g0 * row_bytes + (lane >> 1) * 512u;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
                if ((lane >> 1) * 512u + 128u < bytes) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + 128));
                if ((lane >> 1) * 512u + 256u < bytes) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + 256));
                if ((lane >> 1) * 512u + 384u < bytes) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + 384));
            }
        }
        // The page's K scales onto the rows. A power of two is taken out of every row: one above (largest |q|) * (largest scale),
        // which is at most a few binary orders above the largest term (the residue's range absorbs those).
        float inv_scale[NR], query_sum[NR], row_scale[NR], top = 0.0f;
#pragma unroll
        for (uint32_t c = 0; c < D / 32u; ++c) top = fmaxf(top, fabsf(page.k_scales[lane + 32u * c]));
        top = warp_max(top);
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const float bound = __uint_as_float(q_top[g + 8 * r]) * top;
            const uint32_t e = min(max(__float_as_uint(bound) >> 23, 30u), 225u);   // 2^(e - 127) <= bound < 2^(e - 126)
            row_scale[r] = __uint_as_float((267u - e) << 23);                       // 2^(140 - e): terms below 2^14
            inv_scale[r] = __uint_as_float((e - 13u) << 23);
            query_sum[r] = 0.0f;
        }
        __syncwarp();   // the previous page's readers of the planes are done
#pragma unroll 2
        for (int step = 0; step < static_cast<int>(L::kSteps); ++step) {
            const float4 ks = load4(page.k_scales + t * (D / 4) + 4 * step);
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const uint32_t at_row = (step * 16u + g + 8u * r) * 4u + t;
                const float4 q = *reinterpret_cast<const float4 *>(q_rows + at_row * 4u);
                const float x0 = q.x * ks.x * row_scale[r], x1 = q.y * ks.y * row_scale[r], x2 = q.z * ks.z * row_scale[r], x3 = q.w * ks.w * row_scale[r];
                query_sum[r] += (x0 + x1) + (x2 + x3);
                const uint2 hi = make_uint2(pack_half2(x0, x1), pack_half2(x2, x3));
                const float2 b0 = unpack_half2(hi.x), b1 = unpack_half2(hi.y);
                *reinterpret_cast<uint2 *>(planes + at_row * 8u) = hi;
                *reinterpret_cast<uint2 *>(planes + L::kPlane + at_row * 8u) = make_uint2(pack_half2(x0 - b0.x, x1 - b0.y), pack_half2(x2 - b1.x, x3 - b1.y));
            }
        }
#pragma unroll
        for (int r = 0; r < NR; ++r)
#pragma unroll
            for (int o = 1; o <= 2; o <<= 1) query_sum[r] += __shfl_xor_sync(0xffffffffu, query_sum[r], o);
        __syncwarp();
        CodeBias bias;
        bias.set(page.zero_point);
        const bool aligned = ((reinterpret_cast<uintptr_t>(page.k_words) | reinterpret_cast<uintptr_t>(page.v_words)) & 15u) == 0;
        for (uint32_t n = g0; n < stop; ++n) {
            const uint32_t t0 = 16u * n, begin = page.token_begin + t0;
            if (begin > newest || begin + 16u <= oldest_visible) continue;
            if (aligned && page.fixed_code_length == 4u)
                page_group<D, NR, 4, false>(st, page, t0, planes, symbols, inv_scale, query_sum, bias, qtok, first, lane);
            else if (aligned && page.fixed_code_length == 8u)
                page_group<D, NR, 8, false>(st, page, t0, planes, symbols, inv_scale, query_sum, bias, qtok, first, lane);
            else
                page_group<D, NR, 8, true>(st, page, t0, planes, symbols, inv_scale, query_sum, bias, qtok, first, lane);
        }
        at_group = static_cast<uint64_t>(prefix[m_at]) + stop;
        ++m_at;
    }
    for (; at_group < end_group; ++at_group) {
        const uint32_t unit = static_cast<uint32_t>(at_group - page_groups);
        if (unit % kTailWeight != 0u) continue;
        const uint32_t t0 = 16u * (unit / kTailWeight), begin = desc.active_token_begin + t0;
        if (begin > newest || begin + 16u <= oldest_visible) continue;
        tail_group<D, NR>(st, desc, kv_head, t0, q_rows, qtok, first, lane);
    }

    // ---- merge: the warps' (max, sum, O) in shared memory, then the CTA's rows to the output or to its split's partials ----
    const float o_unit = st.v_unit * (1.0f / kWeightScale);
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) st.l[r] += __shfl_xor_sync(0xffffffffu, st.l[r], o);
    if (t == 0) {
#pragma unroll
        for (int r = 0; r < NR; ++r) state[warp * 16u + g + 8u * r] = make_float2(st.m[r], st.l[r]);
    }
    __syncwarp();
    float *mine_o = reinterpret_cast<float *>(planes);   // [16][D]; channel c * (D / 8) + j of column c = 2t + {0, 1}
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        if (row0 + g + 8u * r >= rows_total) continue;
#pragma unroll
        for (int j = 0; j < D / 8; j += 4) {
            float *dst = mine_o + (g + 8u * r) * D + (2u * t) * (D / 8) + j;
            *reinterpret_cast<float4 *>(dst) = make_float4(st.acc[j][2 * r] * o_unit, st.acc[j + 1][2 * r] * o_unit, st.acc[j + 2][2 * r] * o_unit, st.acc[j + 3][2 * r] * o_unit);
            *reinterpret_cast<float4 *>(dst + D / 8) =
                make_float4(st.acc[j][2 * r + 1] * o_unit, st.acc[j + 1][2 * r + 1] * o_unit, st.acc[j + 2][2 * r + 1] * o_unit, st.acc[j + 3][2 * r + 1] * o_unit);
        }
    }
    __syncthreads();
    // partials: weighted sums [query row][split][D], then (max, sum) [query row][split]
    float2 *partial_ml = reinterpret_cast<float2 *>(partials + static_cast<size_t>(desc.query_count) * desc.query_head_count * splits * D);
    for (uint32_t i = tid; i < 16u * D; i += kMmaThreads) {
        const uint32_t row = i / D, d = i % D, r = row0 + row;
        if (r >= rows_total) break;
        float m = -CUDART_INF_F;
#pragma unroll
        for (int w = 0; w < kMmaWarps; ++w) m = fmaxf(m, state[w * 16u + row].x);
        float l = 0.0f, a = 0.0f;
        if (m != -CUDART_INF_F) {
#pragma unroll
            for (int w = 0; w < kMmaWarps; ++w) {
                const float2 ml = state[w * 16u + row];
                const float k = exp2f(ml.x - m);   // -inf gives 0
                l += ml.y * k;
                a += reinterpret_cast<const float *>(smem + L::kOffWarps + w * L::kWarpBytes)[i] * k;
            }
        }
        const size_t out_row = static_cast<size_t>(r / G) * desc.query_head_count + kv_head * G + r % G;
        if (splits > 1) {
            if (d == 0) partial_ml[out_row * splits + split] = make_float2(m, l);
            partials[(out_row * splits + split) * D + d] = a;
        } else {
            desc.output[out_row * D + d] = l > 0.0f ? a / l : 0.0f;   // no visible token: zeros (paged_kv_attention.cu:170-173)
        }
    }
    if (splits == 1) return;
    // ---- the last CTA of the row tile to arrive merges the splits (and leaves the counter at zero for the next call) ----
    __threadfence();
    __syncthreads();
    uint32_t *counter = arrived + blockIdx.y * gridDim.x + blockIdx.x;
    if (tid == 0) s_last = atomicAdd(counter, 1u) == splits - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    float *weight = reinterpret_cast<float *>(smem + L::kOffWarps);   // [row of the tile][split]
    const uint32_t tile_rows = min(16u, rows_total - row0);
    for (uint32_t row = warp; row < tile_rows; row += kMmaWarps) {   // at most 64 splits: two per lane
        const uint32_t r = row0 + row;
        const float2 *ml = partial_ml + (static_cast<size_t>(r / G) * desc.query_head_count + kv_head * G + r % G) * splits;
        const float2 ml0 = lane < splits ? __ldcg(ml + lane) : make_float2(-CUDART_INF_F, 0.0f);
        const float2 ml1 = lane + 32u < splits ? __ldcg(ml + lane + 32u) : make_float2(-CUDART_INF_F, 0.0f);
        const float m = warp_max(fmaxf(ml0.x, ml1.x));
        const float w0 = ml0.x == -CUDART_INF_F ? 0.0f : exp2f(ml0.x - m), w1 = ml1.x == -CUDART_INF_F ? 0.0f : exp2f(ml1.x - m);
        const float l = warp_sum(ml0.y * w0 + ml1.y * w1), inverse = l > 0.0f ? 1.0f / l : 0.0f;   // no visible token: zeros
        if (lane < splits) weight[row * splits + lane] = w0 * inverse;
        if (lane + 32u < splits) weight[row * splits + lane + 32u] = w1 * inverse;
    }
    __syncthreads();
    // D / 4 threads hold a row, four channels each; where the tile has few rows several such groups share a row's splits, so
    // that a decode step has (nearly) all of them in flight at once.
    constexpr uint32_t kRowThreads = D / 4u, kGroups = kMmaThreads / kRowThreads;
    const uint32_t group = tid / kRowThreads, quad = tid % kRowThreads, shares = max(1u, kGroups / tile_rows), share = group % shares;
    float4 *meet = reinterpret_cast<float4 *>(smem + L::kOffWarps + 16u * 64u * 4u);
    for (uint32_t row = group / shares; row < tile_rows; row += kGroups / shares) {
        const uint32_t r = row0 + row;
        const size_t out_row = static_cast<size_t>(r / G) * desc.query_head_count + kv_head * G + r % G;
        const float4 *src = reinterpret_cast<const float4 *>(partials + out_row * splits * D) + quad;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t k0 = share; k0 < splits; k0 += 8u * shares) {   // eight loads in flight whatever is left
            float4 x[8];
#pragma unroll
            for (uint32_t i = 0; i < 8u; ++i) {
                const uint32_t k = k0 + i * shares;
                x[i] = k < splits ? __ldcg(src + k * kRowThreads) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (uint32_t i = 0; i < 8u; ++i) {
                const float w = weight[row * splits + min(k0 + i * shares, splits - 1u)];
                a.x += x[i].x * w, a.y += x[i].y * w, a.z += x[i].z * w, a.w += x[i].w * w;
            }
        }
        if (shares == 1u) {
            float *out = desc.output + out_row * D + 4u * quad;
            out[0] = a.x, out[1] = a.y, out[2] = a.z, out[3] = a.w;
        } else {
            meet[tid] = a;
        }
    }
    if (shares > 1u) {   // one pass above: group / shares is the row
        __syncthreads();
        const uint32_t row = group / shares, r = row0 + row;
        if (share == 0 && row < tile_rows) {
            float4 a = meet[tid];
            for (uint32_t k = 1; k < shares; ++k) {
                const float4 x = meet[tid + k * kRowThreads];
                a.x += x.x, a.y += x.y, a.z += x.z, a.w += x.w;
            }
            float *out = desc.output + (static_cast<size_t>(r / G) * desc.query_head_count + kv_head * G + r % G) * D + 4u * quad;
            out[0] = a.x, out[1] = a.y, out[2] = a.z, out[3] = a.w;
        }
    }
    if (tid == 0) *counter = 0u;
}

}  // namespace

bool paged_mma_supports(const cf_kv_paged_attention_desc &d) { return d.head_dim == 128 || d.head_dim == 64; }

uint32_t paged_mma_splits(const cf_kv_paged_attention_desc &d, int sm_count) {
    // Two CTAs per SM; more splits than pages of a kv head would leave CTAs without work (a page is at least a group or two)
    const uint64_t tiles = (static_cast<uint64_t>(d.query_count) * d.gqa_group_size + 15u) / 16u * d.kv_head_count;
    const uint64_t wanted = (2ull * sm_count + tiles - 1u) / tiles;
    const uint64_t pages = (d.page_count + d.kv_head_count - 1u) / d.kv_head_count + (d.active_token_count + 127u) / 128u;
    return static_cast<uint32_t>(wanted < pages ? wanted : pages < 1u ? 1u : pages);
}

cudaError_t launch_paged_mma(const cf_kv_paged_attention_desc &d, uint32_t splits, float *partials, uint32_t *arrived, cudaStream_t stream) {
    static LauncherState table[64];
    cudaError_t e;
    LauncherState *state = launcher_state(table, &e);
    if (!state) return e;
    using Kernel = void (*)(cf_kv_paged_attention_desc, uint32_t, float *, uint32_t *);
    static constexpr Kernel kernels[2][2] = {{paged_mma_kernel<64, 1>, paged_mma_kernel<64, 2>}, {paged_mma_kernel<128, 1>, paged_mma_kernel<128, 2>}};
    if (!state->configured) {   // room for the largest descriptor list
        for (int wide = 0; wide < 2; ++wide)
            for (int rows = 0; rows < 2; ++rows) {
                e = cudaFuncSetAttribute(kernels[wide][rows], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(wide ? MmaLayout<128>::bytes(CF_KV_CUDA_MAX_PAGES_PER_LAUNCH)
                                                               : MmaLayout<64>::bytes(CF_KV_CUDA_MAX_PAGES_PER_LAUNCH)));
                if (e != cudaSuccess) return e;
            }
        state->configured = true;
    }
    const uint64_t rows = static_cast<uint64_t>(d.query_count) * d.gqa_group_size;
    const dim3 grid(static_cast<uint32_t>((rows + 15u) / 16u), d.kv_head_count, splits);
    const bool wide = d.head_dim == 128;
    kernels[wide][rows > 8u]<<<grid, kMmaThreads, wide ? MmaLayout<128>::bytes(d.page_count) : MmaLayout<64>::bytes(d.page_count), stream>>>(
        d, splits, partials, arrived);
    return cudaPeekAtLastError();
}

}  // namespace cfb
