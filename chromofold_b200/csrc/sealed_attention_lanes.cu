// sealed_attention_lanes.cu — the hot kernel: decode-step attention over sealed pages of 16 tokens. What follows describes head_dim
// 128 with blocks of 64 symbols (32 per stream); larger blocks, and head_dim 96, 80, 64 and 32, run the same kernel behind a
// staging step, see stage_blocks below. One decode serves up to eight query heads of a kv head; a larger group takes
// several passes, each with a decode of its own.
//
// What it computes is what src/cuda/paged_kv_attention.cu:183-276 computes for one query token; how it runs is new:
//
//   * One WARP owns one (stretch of the page line, kv head) unit. A page record arrives in shared memory as ONE bulk async copy
//     (cp.async.bulk + mbarrier); a warp has one place for it, free again once the record is decoded. Coding tables (rANS slot table, Huffman LUT) are loaded
//     once per CTA. No thread ever reads page bytes from global memory directly.
//   * Lane l decodes block l of the K stream and block l of the V stream, interleaved so that the two independent
//     decoder chains overlap. Symbols never leave registers: four symbols are packed into one register, turned
//     into two fp16 pairs with byte permutes (bias 1024, exact), and fed straight into mma.sync fragments.
//       K block l = token l/2, channels 64*(l&1)..+63  -> B operand of S = Q * K^T   (16 mma per page)
//       V block l = channels 4l..4l+3, all 16 tokens   -> B operand of O^T = P' * V  (16 mma per page)
//     The query group is the other operand, laid out with zeros so that every lane's private slice of the
//     contraction lands in its own output column/row. Tensor cores do the whole contraction for the group;
//     a code is decoded once for all query heads (the reference re-decodes per query head,
//     paged_kv_attention.cu:205-207).
//   * Online softmax per page in fp32; partial (max, sum, weighted) per piece of a stretch goes to the split-KV workspace and is
//     merged by the combine kernel (cf_online_softmax_merge rule, src/runtime/kv_runtime.cpp:219-243).
//   * Every wait on a copy is bounded; on expiry the warp raises CF_B200_DEVSTAT_WAIT_EXPIRED and leaves.

#include <math_constants.h>

#include <atomic>

#include "lanes_decoders.cuh"

namespace cfb {
namespace {

using namespace lanes;

// NG = groups of four query rows that one decode serves: 1 or 2 for up to four or eight heads of binary16 queries; fp32 queries
// (kSplitQ) take two groups for four heads, value and residue, and four for eight. NS = groups that go through softmax and P V.
template <int NG, bool kSplitQ> constexpr int kHeadGroups = kSplitQ ? NG / 2 : NG;
// Warps per CTA, one CTA per SM: what registers (65536, no spill worth the name) and shared memory (227 KB) leave. The
// decoders want warps, but not at the price of spilled registers, and as many on each of the four schedulers: 64 sequences of
// nibble-split rANS, 32 heads, take 1381, 1530, 1470, 1351, 1459, 1445 us with 20, 21, 22, 24, 26, 28 warps; 8 x 131072 tokens, 64
// heads, 2269, 2441, 2149 with 12, 14, 16.
template <int NG, int NB, bool kSplitQ, int kDim>
constexpr int kWarpsOf = NB == 32                ? (kHeadGroups<NG, kSplitQ> == 1 ? 24 : 16)
                         : kDim <= 64            ? 20
                         : NG == 4               ? (kDim < 128 ? 14 : 12)
                         : NG == 2               ? 14
                                                 : 16;
template <int NG, int NB, bool kSplitQ, int kDim> constexpr int kThreadsOf = kWarpsOf<NG, NB, kSplitQ, kDim> * 32;
// Per-warp running state of one unit; NG = number of four-head query groups served by one decode pass.
// kDim = head_dim: a lane holds kDim / 8 quads of each stream (K: kDim / 2 channels of one token; V: kDim / 32 channels,
// every token).
template <int NG, int kDim = 128>
struct UnitState {
    static constexpr int kPairs = (NG + 1) / 2;   // of groups, one mma each
    float score[kPairs][4];  // S fragments of the current page: the even group of a pair in rows 0..7, the odd one in rows 8..15
    float acc[NG][(kDim + 31) / 32][4];   // O fragments: [group][channel of the lane's V block][fragment register]
    uint32_t vq[4 * ((kDim + 31) / 32)];   // V symbols of the current page, [channel*4 + token quad]
    float m[NG], l[NG];      // running max / the lane's part of the running sum, of its head of each group
    uint32_t *dump;          // kDump only: where this lane's quads of the current record go (K at +0, V at +512 words)
};

// What the kernel does with the symbols: attention; or (measurement) fold them into a checksum; or (test) store
// every quad the lane decoders yield to global memory, so that they can be compared symbol for symbol.
constexpr int kAttend = 0, kFold = 1, kDump = 2;
// The softmax weights go to the tensor cores as binary16 (value + rounding residue) scaled by this power of two.
constexpr float kWeightScale = 32768.0f;

// Where a lane finds its A fragments of S = Q * K^T (row = parity of the token * 4 + head, eight rows further for the odd group of
// a pair; zero where the lane's slice of the contraction belongs to the other token): the query rows of a pair of groups sit in
// the warp's shared memory as [head][half] rows of [quad of channels]{even: channels 0, 1 | odd: 0, 1 | even: 2, 3 | odd: 2, 3},
// one 16-byte load per quad and pair, 16 bytes of padding a row, which puts the rows that eight lanes touch into different banks; a
// lane whose row is not its own reads zeros, from the banks that the other lanes of its eight leave alone. (Four binary16 heads have
// no odd group: their rows hold channels only, eight bytes a load, which serves sixteen lanes at a time; there the zeros share two
// banks with rows of their own, and a load takes four wavefronts where two would do.)
// With the codes as B operand one mma serves a pair of groups, where K * Q^T took one for each of them and two zero registers.
struct QSmem {
    uint32_t addr, pair_stride;  // byte address of the lane's row for pair 0; distance to the row for pair 1 (0 on the zero row)
    template <int NG, int PAIR>
    __device__ __forceinline__ void get(int q, uint32_t (&a)[4]) const {
        if constexpr (NG == 1) {
            a[1] = a[3] = 0u;
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(a[0]), "=r"(a[2]) : "r"(addr + 8u * q));
        } else asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(addr + PAIR * pair_stride + 16u * q));
    }
};

template <int NG, int kDim, class QSrc>
__device__ __forceinline__ void score_quad(UnitState<NG, kDim> &u, const QSrc &qs, int q, uint32_t kq) {
    uint32_t lo, hi, a[4];
    quad_to_half2(kq, lo, hi);
    qs.template get<NG, 0>(q, a);
    mma_16816(u.score[0], a[0], a[1], a[2], a[3], lo, hi);
    if constexpr (NG == 4) {
        qs.template get<NG, 1>(q, a);
        mma_16816(u.score[1], a[0], a[1], a[2], a[3], lo, hi);
    }
}

// kFold: the symbols are only folded into a checksum (u.vq[0]) — the decode work of the kernel without its attention.
// kDump: lane l's quad q of a stream holds the symbols 64 l + 4 q .. + 3 of that stream, first symbol in byte 0.
// kPasses: a page in four passes of four quads, a quarter of the code, so that more of it stays in the instruction cache; the V
// quads shift down, so that quad q ends in element q. Taken by the eight-head kernel of binary16 queries, whose 16 warps hide
// less of the fetches: 64 sequences of rANS pages 1403 -> 1335 us, of Huffman pages 1098 -> 1022. Half as many steps, as
// nibble-split pages have, gain nothing by it, and neither the 24 warps of the four-head kernels nor eight heads of split
// queries have registers to spare for it (64 sequences, nibble-split rANS, 32 heads: 1351 us in one pass, 1413 in two, 1410 in four).
template <int kEach>
__device__ __forceinline__ void shift_quads(uint32_t (&vq)[16]) {
#pragma unroll
    for (int i = 0; i < 16 - kEach; ++i) vq[i] = vq[i + kEach];
}
template <int kMode, int NG, class QSrc>
__device__ __forceinline__ void take_quads(UnitState<NG> &u, const QSrc &qs, int q, int at, uint32_t kq, uint32_t vq) {
    if constexpr (kMode == kFold) {
        u.vq[0] ^= kq ^ vq;
    } else if constexpr (kMode == kDump) {
        u.dump[q] = kq;
        u.dump[512 + q] = vq;
    } else {
        u.vq[at] = vq;
        score_quad(u, qs, q, kq);
    }
}
// Both streams of fixed width: nothing to decode, and no passes: their words lie one after the other and sixteen lanes' words share a
// bank, so that it matters that four of them go in one load, as the compiler makes them here, but not in the loop below (16 sequences
// of 2048 to 6144 tokens, 32 fp32 heads: 69 us here, 114 there; 64 binary16 heads 81 and 125). With all sixteen of a stream asked
// for at once the fp32 kernel spilled more (32 server slots of 900 to 8200 tokens: 201.6 -> 202.4 us).
template <int kMode, int NG, class QSrc>
__device__ __forceinline__ void decode_fixed(FixedLane &k, FixedLane &v, UnitState<NG> &u, const QSrc &qs) {
#pragma unroll
    for (int q = 0; q < 16; q += 4) {
        uint32_t kq[4], vq[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) kq[j] = k.quad(q + j), vq[j] = v.quad(q + j);
#pragma unroll
        for (int j = 0; j < 4; ++j) take_quads<kMode>(u, qs, q + j, q + j, kq[j], vq[j]);
    }
}
// Both streams with the same other coder: two independent decoder chains, interleaved symbol by symbol.
template <int kMode, int kPasses, class Lane, int NG, class QSrc>
__device__ __forceinline__ void decode_fused(Lane &k, Lane &v, UnitState<NG> &u, const QSrc &qs) {
    constexpr int kEach = 16 / kPasses;   // quads of a pass
#pragma unroll 1
    for (int pass = 0; pass < kPasses; ++pass) {
        if constexpr (kPasses > 1) shift_quads<kEach>(u.vq);
        uint32_t kw = 0u, vw = 0u;
#pragma unroll
        for (int j = 0; j < kEach; ++j) {
            const int q = kEach * pass + j, at = 16 - kEach + j;
            if constexpr (requires { k.lo_word(0); }) {   // nibble-split: a quad from every two steps
                uint32_t ke[2], ve[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    ke[i] = k.symbol(i);
                    ve[i] = v.symbol(i);
                }
                k.advance();
                v.advance();
                kw = j & 1 ? kw >> 4 : k.lo_word(q >> 1);
                vw = j & 1 ? vw >> 4 : v.lo_word(q >> 1);
                take_quads<kMode>(u, qs, q, at, merge_split_quad<Lane>(ke[0], ke[1], kw), merge_split_quad<Lane>(ve[0], ve[1], vw));
            } else {
                uint32_t ke[4], ve[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    ke[i] = k.symbol(i & 1);
                    ve[i] = v.symbol(i & 1);
                    if (i & 1) {
                        k.advance();
                        v.advance();
                    }
                }
                take_quads<kMode>(u, qs, q, at, Lane::pack(ke[0], ke[1], ke[2], ke[3]), Lane::pack(ve[0], ve[1], ve[2], ve[3]));
            }
        }
    }
}

template <int kMode = kAttend, class KLane, int NG, class QSrc>
__device__ __forceinline__ void decode_k_only(KLane &k, UnitState<NG> &u, const QSrc &qs) {
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const uint32_t kq = k.quad(q);
        if constexpr (kMode == kFold) u.vq[0] ^= kq;
        else if constexpr (kMode == kDump) u.dump[q] = kq;
        else score_quad(u, qs, q, kq);
    }
}

template <int kMode = kAttend, class VLane, int NG>
__device__ __forceinline__ void decode_v_only(VLane &v, UnitState<NG> &u) {
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const uint32_t vq = v.quad(q);
        if constexpr (kMode == kFold) u.vq[0] ^= vq;
        else if constexpr (kMode == kDump) u.dump[512 + q] = vq;
        else u.vq[q] = vq;
    }
}

// ---- blocks of 128 / 256 symbols (NB = 16 / 8 blocks per stream) ------------------------------------------------
// The attention part of the kernel wants lane l to hold symbols 64 l .. 64 l + 63 of both streams. With larger blocks
// there are fewer blocks than lanes, so the decode is laid out differently and its result re-dealt through a
// per-warp tile in shared memory: lanes 0 .. NB-1 decode the K blocks while lanes 16 .. 16+NB-1 decode the V blocks
// (at NB = 16 every lane is busy and a page costs as many decoder steps per lane as with 64-symbol blocks; at NB = 8
// half the lanes idle), every four quads leave as one 16-byte store, and after a warp barrier each lane reads its
// sixteen K quads and sixteen V quads back with 16-byte loads. A tile row is one lane's 64 symbols plus 16 bytes
// of padding (row stride 80 bytes), which keeps both the stores and the loads off each other's banks; the V tile
// sits 16 bytes further for the same reason.
// The same staging serves head_dim 96, 64 and 32 (streams of 1536 / 1024 / 512 symbols): a lane's share is then
// kDim / 2 symbols of each stream (K: half of one token's channels; V: kDim / 32 channels, every token). At head_dim
// 96 with 64-symbol blocks there are 48 blocks for 32 lanes: every lane takes block `lane`, the first sixteen
// lanes also block `lane + 32`.
// one lane's kDim / 2 symbols + padding that keeps the row stride off multiples of 64 bytes
// Head_dim 80 (1280 symbols, 20 blocks): a lane's K share is 40 symbols, and three V channels, of which lanes 27..31 have none and
// lane 26 two; what they read instead goes to channels that are never stored. Its tile has no padding: rows of 40 and 48
// bytes are off each other's banks as they are.
template <int kDim> constexpr int kVChannelsOf = (kDim + 31) / 32;
template <int kDim> constexpr uint32_t kTileRowOf = kDim / 2u + ((kDim / 2u + 16u) % 64u == 0 ? 32u : 16u);
template <int kDim> constexpr uint32_t kTileStreamOf = kDim == 80 ? 1280u : 32u * kTileRowOf<kDim>;   // bytes of the K part
template <int kDim> constexpr uint32_t kTileBytesOf = kDim == 80 ? 1280u + 32u * 48u + 32u : 2u * kTileStreamOf<kDim> + 32u;

template <int NB, int kDim, class Lane>
__device__ __forceinline__ void stage_with(Lane &d, uint32_t block, uint8_t *tile) {
    constexpr int kQuads = 4 * kDim / NB;   // per block
    constexpr uint32_t kRowQuads = kDim / 8;
#pragma unroll 2
    for (int q = 0; q < kQuads; q += 4) {
        const uint32_t a = d.quad(q), b = d.quad(q + 1), c = d.quad(q + 2), e = d.quad(q + 3);
        const uint32_t at = block * kQuads + q;   // quad index in the stream: row = at / kRowQuads, column = at % kRowQuads
        const uint32_t to = kDim == 80 ? 4u * at : (at / kRowQuads) * kTileRowOf<kDim> + (at % kRowQuads) * 4u;
        *reinterpret_cast<uint4 *>(tile + to) = make_uint4(a, b, c, e);
    }
}

// One lane's share: block `block` of the part, whatever its coder.
template <int NB, int kDim>
__device__ __forceinline__ void stage_blocks(const uint8_t *part, uint32_t part_bytes, uint32_t coder, uint32_t block,
                                             const uint32_t *slot_table, const uint16_t *lut, uint8_t *tile) {
    constexpr int kSyms = 16 * kDim;
    if (coder == CF_B200_CODER_RANS_SPLIT4) {
        RansSplitLaneT<NB, kSyms> d;
        d.open(part, part_bytes, block, slot_table);
        stage_with<NB, kDim>(d, block, tile);
    } else if (coder == CF_B200_CODER_HUFFMAN_SPLIT4) {
        HuffSplitLaneT<NB, kSyms> d;
        d.open(part, part_bytes, block, lut);
        stage_with<NB, kDim>(d, block, tile);
    } else if (coder == CF_B200_CODER_RANS) {
        RansLaneT<NB> d;
        d.open(part, part_bytes, block, slot_table);
        stage_with<NB, kDim>(d, block, tile);
    } else if (coder == CF_B200_CODER_HUFFMAN) {
        HuffLaneT<NB> d;
        d.open(part, part_bytes, block, lut);
        stage_with<NB, kDim>(d, block, tile);
    } else {
        FixedLaneT<NB, kSyms> d;
        d.open(part, part_bytes, block);
        stage_with<NB, kDim>(d, block, tile);
    }
}

// Shared memory of one warp: one record, the softmax scratch, an mbarrier and the query rows. A record is decoded before anything
// else happens to its page, so its place is free for the next one while the scores and weights are worked out; a second place
// would cost eight warps per SM.
//   scratch: P rows fp16 high halves [4 NS][16] | low halves [4 NS][16], NS = kHeadGroups
template <int NG, int NB, bool kSplitQ, int kDim>
struct WarpLayout {
    static constexpr uint32_t kStage = kDim == 128 ? kStageBytes : 16u + 32u * kDim + 48u;   // header, two streams, read-ahead
    static constexpr uint32_t kPRows = kStage;
    static constexpr uint32_t kPBytes = 4 * kHeadGroups<NG, kSplitQ> * 16 * 2;
    static constexpr uint32_t kPLo = kPRows + kPBytes;
    static constexpr uint32_t kBar = kPLo + kPBytes;
    static constexpr uint32_t kQRows = kBar + 16;
    static constexpr uint32_t kQRowWords = NG == 1 ? kDim / 4 + (kDim == 80 ? 8 : 4) : kDim / 2 + 4;
    static constexpr uint32_t kQPairBytes = 8 * kQRowWords * 4;
    static constexpr uint32_t kTile = kQRows + (NG + 1) / 2 * kQPairBytes;   // NB != 32 only
    static constexpr uint32_t kBytes = kTile + (NB != 32 ? kTileBytesOf<kDim> : 0u);
    static constexpr uint32_t kZeroBytes = 2 * 128 + 128;   // the CTA's zero row, after the tables
    static constexpr uint32_t kSmem = kTableBytes + kZeroBytes + kWarpsOf<NG, NB, kSplitQ, kDim> * kBytes;
    static_assert(kBytes % 16 == 0 && kQRows % 16 == 0, "16-byte loads");
    static_assert(kSmem <= 232448, "a CTA has 227 KB of shared memory");
};

// kSplitQ: the queries are fp32. Their rows are split into binary16(q) and binary16(q - binary16(q)): with four heads the two groups
// of the one pair, which one mma serves, with eight a pair of values and a pair of residues, a second score mma. The two score
// fragments of a head are added, and one softmax / P V follows: the scores equal fp32-query scores to 2^-22 relative.
template <int NG, int kMode, bool kSplitQ, int NB, int kDim>
__global__ void __launch_bounds__(kThreadsOf<NG, NB, kSplitQ, kDim>, 1) lanes_attention_kernel(AttentionParams p, uint32_t after_prefix) {
    constexpr bool kProbe = kMode != kAttend;
    static_assert(!kSplitQ || NG != 1, "split queries take two groups for four heads");
    static_assert(NB == 32 || NB == 24 || NB == 20 || NB == 16 || NB == 12 || NB == 8 || NB == 4, "blocks per stream");
    static_assert(kDim == 128 || ((kDim == 96 || kDim == 80 || kDim == 64 || kDim == 32) && NB != 32), "other head_dims go through the staging tile");
    constexpr int kQ = kDim / 8, kVCh = kVChannelsOf<kDim>, kSyms = 16 * kDim;   // K quads per lane; V channels per lane
    constexpr uint32_t kRowWords = kDim / 4;   // words of half a query row (the channels one lane's K block covers)
    using L = WarpLayout<NG, NB, kSplitQ, kDim>;
    constexpr int NS = kHeadGroups<NG, kSplitQ>;
    constexpr uint32_t kPassHeads = 4u * NS;
    constexpr int kPasses = NS == 2 && !kSplitQ && kMode == kAttend ? 4 : 1;   // of decode_fused
    extern __shared__ __align__(128) uint8_t smem[];
    uint32_t *k_slot = reinterpret_cast<uint32_t *>(smem);
    uint32_t *v_slot = k_slot + 4096;
    uint16_t *k_lut = reinterpret_cast<uint16_t *>(v_slot + 4096);
    uint16_t *v_lut = k_lut + 4096;

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint8_t *warp_mem = smem + kTableBytes + L::kZeroBytes + warp * L::kBytes;
    __half *p_rows = reinterpret_cast<__half *>(warp_mem + L::kPRows);         // [4 NS][16] fp16(p)
    __half *p_rows_lo = reinterpret_cast<__half *>(warp_mem + L::kPLo);        // [4 NS][16] fp16(p - fp16(p))
    const __half *zero_row = reinterpret_cast<const __half *>(smem + kTableBytes);   // what inactive lanes read their fragments from
    uint64_t *bar = reinterpret_cast<uint64_t *>(warp_mem + L::kBar);
    uint32_t *q_rows = reinterpret_cast<uint32_t *>(warp_mem + L::kQRows);

    if (after_prefix && __ldcg(&plan_header(p)->line.stretches) == 0u) {   // the shared-prefix kernel has taken every page
        // Only now may the combine kernel start: placed while these CTAs still held the SMs until the prefix kernel's end, and left all at
        // once, it went onto those of one die that were free first, six or eight CTAs each (64 rows after 16384 tokens 134 -> 120 us,
        // 100 rows of 12 heads after 8192 tokens 93 -> 82).
        wait_for_previous_kernel();
        allow_dependent_launch();
        return;
    }
    load_tables<kThreadsOf<NG, NB, kSplitQ, kDim>>(smem, p, tid);   // coding tables: once per CTA
    if (tid < L::kZeroBytes / 4u) reinterpret_cast<uint32_t *>(smem + kTableBytes)[tid] = 0u;
    if (lane == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    // The plan kernel's results. A shared-prefix kernel in front of this one has waited for them before it let this kernel start, and
    // nothing here needs what it writes: this kernel takes over each SM as that one leaves it, and waits for its end at its own.
    if (!after_prefix) wait_for_previous_kernel();
    allow_dependent_launch();
    const uint32_t subgroups = (p.group + kPassHeads - 1u) / kPassHeads;   // 4 NG query heads per pass
    const uint32_t g = lane >> 2, t = lane & 3u;
    uint32_t phase = 0u;   // parity the next wait on the record's barrier expects

    // fixed lane roles
    const bool q_row_mine = (t >> 1) == (g >> 2);          // S rows: parity of the token * 4 + head
    const uint32_t my_token = 4u * t + (g >> 2);           // S fragment: this lane's tokens are this one and the second after it,
    const uint32_t o_head = g & 3u;                        // its head (of each group) this one, and that of all its O fragments
    const bool row_lo_mine = t == (g >> 2), row_hi_mine = t == (g >> 2) + 2u;   // P rows with lane tag t

    // A unit is a stretch of the page line for one kv head (and one pass over its query group). The library's own cut makes at most
    // as many units as there are warps: unit u goes to warp u / gridDim of CTA u % gridDim, so that fewer of them spread over the
    // SMs. More, when the caller fixes the pages per unit, are handed out as warps come free.
    // One turn of the loop covers a unit's positions inside one sequence and one piece. Between turns only `unit` and `x`, where the
    // unit goes on (0: at its start), are kept; the line is read again, so that the pages' loop has the registers to itself.
    uint32_t unit = warp * gridDim.x + blockIdx.x, x = 0u;
    for (;;) {
        uint32_t partial, page_begin, n_pages, slot, sealed, qpos, q_row, sub, head_local;
        {
            const PageLine line = plan_line(p);
            const uint32_t unit_lanes = p.kv_head_span * subgroups, unit_count = line.stretches * unit_lanes, warps = kWarpsOf<NG, NB, kSplitQ, kDim> * gridDim.x;
            uint32_t stretch = unit / unit_lanes;
            if (x != 0u && x == line.begin(stretch + 1u)) {   // the unit is done
                if (unit_count <= warps) break;
                if (lane == 0) unit = warps + atomicAdd(&plan_header(p)->next_unit, 1u);
                unit = __shfl_sync(0xffffffffu, unit, 0);
                stretch = unit / unit_lanes;
                x = 0u;
            }
            if (unit >= unit_count) break;
            if (x == 0u) x = line.begin(stretch);
            const uint32_t piece = line.piece_of(stretch, x);
            const LineRun run = run_at(p, x, line.piece_end(stretch, piece), line.grain, lane);
            partial = line.slot(stretch, piece, x, run.seq);
            page_begin = run.page;
            n_pages = run.page_end - run.page;
            slot = run.info.slot, sealed = run.info.sealed, qpos = run.info.qpos, q_row = run.info.row;
            x = run.x_end;
            sub = unit % subgroups;
            head_local = (unit / subgroups) % p.kv_head_span;
        }
        const uint32_t kv_head = p.kv_head_begin + head_local;
        const uint32_t G = min(kPassHeads, p.group - kPassHeads * sub);       // query heads served by this pass
        const uint32_t q_head_base = kv_head * p.group + kPassHeads * sub;    // first of them
        const uint32_t out_head_base = head_local * p.group + kPassHeads * sub;
        const uint32_t first_token = window_begin(qpos, p.causal_window);
        const uint32_t *table_row = p.page_table + static_cast<uint64_t>(slot) * p.page_table_stride;

        // bit 63 of an entry (reserved, 0 in the directory) marks the page of the wait-expiry test: armed, never fetched
        auto load_entry = [&](uint32_t page) -> uint64_t {
            const uint32_t page_id = table_row[page];
            const uint64_t entry = p.page_dir[static_cast<uint64_t>(page_id) * p.kv_head_count + kv_head];
            return page_id == p.skip_copy_page ? entry | (1ull << 63) : entry;
        };
        auto issue = [&](uint64_t entry) {
            const uint32_t units16 = static_cast<uint32_t>(CF_B200_DIR_LENGTH_UNITS(entry));
            if (lane == 0 && units16 != 0 && units16 * 16u <= L::kStage - 32u) {
                mbar_expect_tx(bar, units16 * 16u);
                if (!(entry >> 63)) bulk_load(warp_mem, p.arena + 16ull * CF_B200_DIR_OFFSET_UNITS(entry), units16 * 16u, bar);
            }
        };
        auto entry_ok = [&](uint64_t entry) {
            const uint32_t units16 = static_cast<uint32_t>(CF_B200_DIR_LENGTH_UNITS(entry));
            return units16 != 0 && units16 * 16u <= L::kStage - 32u;
        };

        // the first record is on its way while the queries are fetched
        uint64_t entry_cur = load_entry(page_begin);
        uint64_t entry_next = n_pages > 1 ? load_entry(page_begin + 1) : 0ull;
        __syncwarp();   // the previous run's readers of the record and of the query rows are done
        issue(entry_cur);

        QSmem qs;
        if constexpr (kSplitQ) {
            const float2 *qsrc = reinterpret_cast<const float2 *>(
                reinterpret_cast<const float *>(p.queries) + (static_cast<uint64_t>(q_row) * p.query_head_count + q_head_base) * kDim);
#pragma unroll
            for (int j = 0; j < NS * kDim / 16; ++j) {    // 4 NS heads x kDim / 2 channel pairs; row = head*2 + half
                const uint32_t i = lane + 32u * j, head = i / (2u * kRowWords);
                const float2 x = head < G ? qsrc[i] : make_float2(0.0f, 0.0f);
                const __half2 hi = __floats2half2_rn(x.x, x.y);
                const float2 back = __half22float2(hi);
                const __half2 lo = __floats2half2_rn(x.x - back.x, x.y - back.y);
                // four heads: value and residue are the groups of the one pair; eight: a pair of values, a pair of residues
                uint32_t *row = q_rows + (i / kRowWords % 8u) * L::kQRowWords + (i % kRowWords) * 2u;
                row[NS == 1 ? 0u : i / (8u * kRowWords)] = *reinterpret_cast<const uint32_t *>(&hi);
                row[NS == 1 ? 1u : i / (8u * kRowWords) + L::kQPairBytes / 4u] = *reinterpret_cast<const uint32_t *>(&lo);
            }
            __syncwarp();
        } else {
            const uint32_t *qsrc = reinterpret_cast<const uint32_t *>(
                reinterpret_cast<const __half *>(p.queries) + (static_cast<uint64_t>(q_row) * p.query_head_count + q_head_base) * kDim);
#pragma unroll
            for (int j = 0; j < NG * kDim / 16; ++j) {   // 4 NG heads x kDim / 2 words; row = head*2 + half
                const uint32_t i = lane + 32u * j, head = i / (2u * kRowWords);
                uint32_t *row = q_rows + (i / kRowWords % 8u) * L::kQRowWords + (i % kRowWords) * (NG == 1 ? 1u : 2u);
                row[i / (8u * kRowWords)] = head < G ? qsrc[i] : 0u;
            }
        }
        __syncwarp();
        const uint32_t own = smem_addr(q_rows + (o_head * 2u + (t & 1u)) * L::kQRowWords);
        // 16 banks of the rows of heads 0 and 1, which the lanes of eight that read zeros stay out of, or of heads 2 and 3
        qs.addr = q_row_mine ? own : smem_addr(zero_row) + ((smem_addr(q_rows) - smem_addr(zero_row) + ((o_head & 2u) ? 0u : 64u)) & 112u);
        qs.pair_stride = q_row_mine ? L::kQPairBytes : 0u;

        UnitState<NG, kDim> u;
        if constexpr (kProbe) u.vq[0] = 0u;
        u.dump = nullptr;
#pragma unroll
        for (int n = 0; n < NG; ++n) {
#pragma unroll
            for (int a = 0; a < kVCh; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) u.acc[n][a][b] = 0.0f;
            u.m[n] = -CUDART_INF_F;
            u.l[n] = 0.0f;
        }
        // O is kept in units of a power of two at or above every V scale met so far; a page's scale relative to it rides on the
        // weights, together with kWeightScale. v_gain = kWeightScale / unit.
        float v_unit = 0x1p-25f, v_gain = kWeightScale * 0x1p25f;

        bool alive = true;

        for (uint32_t i = 0; i < n_pages; ++i) {
            const uint64_t entry_after = i + 2 < n_pages ? load_entry(page_begin + i + 2) : 0ull;
            bool next_issued = false;
            if (!entry_ok(entry_cur)) {
                if (lane == 0) raise_status(p, CF_B200_DEVSTAT_BAD_RECORD);
            } else {
                if (!mbar_wait(bar, phase, p.wait_polls)) {
                    if (lane == 0) raise_status(p, CF_B200_DEVSTAT_WAIT_EXPIRED);
                    alive = false;
                    break;
                }
                phase ^= 1u;
                const uint8_t *rec = warp_mem;
                const uint4 hv = *reinterpret_cast<const uint4 *>(rec);
                const uint32_t k_bytes = 16u * (hv.x & 0xffffu), v_bytes = 16u * (hv.x >> 16);
                const uint32_t k_coder = hv.y & 0xffu, v_coder = (hv.y >> 8) & 0xffu, token_count = hv.y >> 16;
                const uint8_t *k_part = rec + 16;
                const uint8_t *v_part = k_part + k_bytes;
                bool offsets_ok;
                if constexpr (NB == 32) {
                    offsets_ok = part_offsets_ok(k_part, k_coder, k_bytes, lane) && part_offsets_ok(v_part, v_coder, v_bytes, lane);
                } else if constexpr (NB <= 16) {   // lanes 0..NB-1 hold the K blocks, lanes 16..16+NB-1 the V blocks
                    const bool mine = (lane & 15u) < static_cast<uint32_t>(NB);
                    offsets_ok = !mine || (lane < 16u ? part_offsets_ok<NB, kSyms>(k_part, k_coder, k_bytes, lane)
                                                      : part_offsets_ok<NB, kSyms>(v_part, v_coder, v_bytes, lane - 16u));
                } else {   // more blocks than lanes: block lane and block lane + 32 of the 2 NB (K blocks first)
                    offsets_ok = true;
#pragma unroll
                    for (uint32_t gb = lane; gb < 2u * NB; gb += 32u)
                        offsets_ok = offsets_ok && (gb < static_cast<uint32_t>(NB) ? part_offsets_ok<NB, kSyms>(k_part, k_coder, k_bytes, gb)
                                                                                 : part_offsets_ok<NB, kSyms>(v_part, v_coder, v_bytes, gb - NB));
                }
                const bool good = record_header_ok(hv, entry_cur, p.codebook_id) && __all_sync(0xffffffffu, offsets_ok);
                uint32_t dump_page = 0u;
                if constexpr (kMode == kDump) dump_page = table_row[page_begin + i];
                if (!good || dump_page >= p.dump_pages) {   // dump_pages is 1 outside the dump mode
                    if (lane == 0) raise_status(p, CF_B200_DEVSTAT_BAD_RECORD);
                } else {
                    if constexpr (kMode == kDump)   // [page id][kv head][K stream | V stream], one byte per symbol
                        u.dump = reinterpret_cast<uint32_t *>(p.output) +
                                 (static_cast<uint64_t>(dump_page) * p.kv_head_count + kv_head) * (kSyms / 2) + (kDim == 80 ? 0u : kQ * lane);
                    const float k_scale = __half2float(__ushort_as_half(static_cast<unsigned short>(hv.z & 0xffffu))) *
                                          (p.softmax_scale * kLog2e);
                    const float v_scale = __half2float(__ushort_as_half(static_cast<unsigned short>(hv.z >> 16)));
#pragma unroll
                    for (int n = 0; n < u.kPairs; ++n) u.score[n][0] = u.score[n][1] = u.score[n][2] = u.score[n][3] = 0.0f;

                    if constexpr (NB != 32) {
                        uint8_t *tile = warp_mem + L::kTile;
                        // One call site for both streams: the lanes that decode V blocks differ from those that decode K
                        // blocks only in the pointers they pass, so the warp runs the decoder once, not once per stream.
                        auto stage_one = [&](bool is_v, uint32_t block) {
                            stage_blocks<NB, kDim>(is_v ? v_part : k_part, is_v ? v_bytes : k_bytes, is_v ? v_coder : k_coder, block,
                                                   is_v ? v_slot : k_slot, is_v ? v_lut : k_lut,
                                                   tile + (is_v ? kTileStreamOf<kDim> + 16u : 0u));
                        };
                        if constexpr (NB <= 16) {
                            if ((lane & 15u) < static_cast<uint32_t>(NB)) stage_one(lane >= 16u, lane & 15u);
                        } else {   // two rounds: 2 NB blocks dealt over the 32 lanes, K blocks first
                            for (uint32_t gb = lane; gb < 2u * NB; gb += 32u)
                                stage_one(gb >= static_cast<uint32_t>(NB), gb >= static_cast<uint32_t>(NB) ? gb - NB : gb);
                        }
                        __syncwarp();
                        if (i + 1 < n_pages) issue(entry_next);   // the record is decoded: its place takes the next one
                        next_issued = true;
                        if constexpr (kDim == 80) {
                            const uint8_t *k_row = tile + 40u * lane, *v_row = tile + kTileStreamOf<kDim> + 16u + 48u * lane;
#pragma unroll
                            for (int c = 0; c < 3; ++c) {
                                const uint4 vv = *reinterpret_cast<const uint4 *>(v_row + 16u * c);
                                const uint32_t vq[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    const uint32_t at = 12u * lane + 4u * c + j;   // of the stream's 320 quads
                                    if constexpr (kMode == kFold) u.vq[0] ^= at < 320u ? vq[j] : 0u;
                                    else if constexpr (kMode == kAttend) u.vq[4 * c + j] = vq[j];
                                    else if (at < 320u) u.dump[320u + at] = vq[j];
                                }
                            }
#pragma unroll
                            for (int q = 0; q < kQ; q += 2) {
                                const uint2 kk = *reinterpret_cast<const uint2 *>(k_row + 4u * q);
                                if constexpr (kMode == kFold) {
                                    u.vq[0] ^= kk.x ^ kk.y;
                                } else if constexpr (kMode == kDump) {
                                    u.dump[kQ * lane + q] = kk.x;
                                    u.dump[kQ * lane + q + 1] = kk.y;
                                } else {
                                    score_quad(u, qs, q, kk.x);
                                    score_quad(u, qs, q + 1, kk.y);
                                }
                            }
                        } else {
#pragma unroll
                        for (int c = 0; c < kQ / 4; ++c) {
                            const uint4 kk = *reinterpret_cast<const uint4 *>(tile + lane * kTileRowOf<kDim> + 16u * c);
                            const uint4 vv = *reinterpret_cast<const uint4 *>(tile + kTileStreamOf<kDim> + 16u + lane * kTileRowOf<kDim> + 16u * c);
                            const uint32_t kq[4] = {kk.x, kk.y, kk.z, kk.w}, vq[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const int q = 4 * c + j;
                                if constexpr (kMode == kFold) {
                                    u.vq[0] ^= kq[j] ^ vq[j];
                                } else if constexpr (kMode == kDump) {
                                    u.dump[q] = kq[j];
                                    u.dump[kSyms / 4 + q] = vq[j];
                                } else {
                                    u.vq[q] = vq[j];
                                    score_quad(u, qs, q, kq[j]);
                                }
                            }
                        }
                        }
                        if constexpr (kProbe) __syncwarp();   // the tile is rewritten for the next page
                    } else if (k_coder == CF_B200_CODER_RANS_SPLIT4 && v_coder == CF_B200_CODER_RANS_SPLIT4) {
                        RansSplitLane k, v;
                        k.open(k_part, k_bytes, lane, k_slot);
                        v.open(v_part, v_bytes, lane, v_slot);
                        decode_fused<kMode, 1>(k, v, u, qs);
                    } else if (k_coder == CF_B200_CODER_HUFFMAN_SPLIT4 && v_coder == CF_B200_CODER_HUFFMAN_SPLIT4) {
                        HuffSplitLane k, v;
                        k.open(k_part, k_bytes, lane, k_lut);
                        v.open(v_part, v_bytes, lane, v_lut);
                        decode_fused<kMode, 1>(k, v, u, qs);
                    } else if (k_coder == CF_B200_CODER_RANS && v_coder == CF_B200_CODER_RANS) {
                        RansLane k, v;
                        k.open(k_part, k_bytes, lane, k_slot);
                        v.open(v_part, v_bytes, lane, v_slot);
                        decode_fused<kMode, kPasses>(k, v, u, qs);
                    } else if (k_coder == CF_B200_CODER_HUFFMAN && v_coder == CF_B200_CODER_HUFFMAN) {
                        HuffLane k, v;
                        k.open(k_part, k_bytes, lane, k_lut);
                        v.open(v_part, v_bytes, lane, v_lut);
                        decode_fused<kMode, kPasses>(k, v, u, qs);
                    } else if (k_coder == CF_B200_CODER_FIXED8 && v_coder == CF_B200_CODER_FIXED8) {
                        FixedLane k, v;
                        k.open(k_part, k_bytes, lane);
                        v.open(v_part, v_bytes, lane);
                        decode_fixed<kMode>(k, v, u, qs);
                    } else {  // mixed coders (one stream fell back to fixed width): one stream after the other
                        if (k_coder == CF_B200_CODER_RANS) { RansLane k; k.open(k_part, k_bytes, lane, k_slot); decode_k_only<kMode>(k, u, qs); }
                        else if (k_coder == CF_B200_CODER_HUFFMAN) { HuffLane k; k.open(k_part, k_bytes, lane, k_lut); decode_k_only<kMode>(k, u, qs); }
                        else if (k_coder == CF_B200_CODER_RANS_SPLIT4) { RansSplitLane k; k.open(k_part, k_bytes, lane, k_slot); decode_k_only<kMode>(k, u, qs); }
                        else if (k_coder == CF_B200_CODER_HUFFMAN_SPLIT4) { HuffSplitLane k; k.open(k_part, k_bytes, lane, k_lut); decode_k_only<kMode>(k, u, qs); }
                        else { FixedLane k; k.open(k_part, k_bytes, lane); decode_k_only<kMode>(k, u, qs); }
                        if (v_coder == CF_B200_CODER_RANS) { RansLane v; v.open(v_part, v_bytes, lane, v_slot); decode_v_only<kMode>(v, u); }
                        else if (v_coder == CF_B200_CODER_HUFFMAN) { HuffLane v; v.open(v_part, v_bytes, lane, v_lut); decode_v_only<kMode>(v, u); }
                        else if (v_coder == CF_B200_CODER_RANS_SPLIT4) { RansSplitLane v; v.open(v_part, v_bytes, lane, v_slot); decode_v_only<kMode>(v, u); }
                        else if (v_coder == CF_B200_CODER_HUFFMAN_SPLIT4) { HuffSplitLane v; v.open(v_part, v_bytes, lane, v_lut); decode_v_only<kMode>(v, u); }
                        else { FixedLane v; v.open(v_part, v_bytes, lane); decode_v_only<kMode>(v, u); }
                    }

                    if constexpr (NB == 32) {
                        __syncwarp();   // the record is decoded: its place takes the next one
                        if (i + 1 < n_pages) issue(entry_next);
                        next_issued = true;
                    }
                    if constexpr (!kProbe) {
                    // ---- online softmax for this page (fp32), per group of four heads ----
                    const uint32_t page_token = (page_begin + i) * 16u;
                    const uint32_t seen_end = min(qpos < sealed ? qpos + 1u : sealed, page_token + token_count);   // tokens [first_token, seen_end)
                    const bool visible0 = page_token + my_token >= first_token && page_token + my_token < seen_end;
                    const bool visible1 = page_token + my_token + 2u >= first_token && page_token + my_token + 2u < seen_end;
                    float s0[NS], s1[NS];
                    bool higher = false;
#pragma unroll
                    for (int n = 0; n < NS; ++n) {
                        s0[n] = u.score[0][2 * n], s1[n] = u.score[0][2 * n + 1];
                        if constexpr (kSplitQ) {   // q k = binary16(q) k + residue k
                            s0[n] += NS == 1 ? u.score[0][2] : u.score[u.kPairs - 1][2 * n];
                            s1[n] += NS == 1 ? u.score[0][3] : u.score[u.kPairs - 1][2 * n + 1];
                        }
                        s0[n] = visible0 ? s0[n] * k_scale : -CUDART_INF_F;
                        s1[n] = visible1 ? s1[n] * k_scale : -CUDART_INF_F;
                        higher = higher || s0[n] > u.m[n] || s1[n] > u.m[n];
                    }
                    // The maximum moves on few pages (about one in n after n pages of a head): only then is it worked out, and O rescaled.
                    if (__any_sync(0xffffffffu, higher)) {
#pragma unroll
                        for (int n = 0; n < NS; ++n) {
                            float top = fmaxf(s0[n], s1[n]);
                            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));   // over the lanes of the same head
                            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
                            const float raised = fmaxf(u.m[n], top), alpha = raised == -CUDART_INF_F ? 0.0f : exp2f(u.m[n] - raised);
                            u.l[n] *= alpha;
                            u.m[n] = raised;
#pragma unroll
                            for (int dd = 0; dd < kVCh; ++dd)
#pragma unroll
                                for (int c = 0; c < 4; ++c) u.acc[n][dd][c] *= alpha;
                        }
                    }
                    if (v_scale > v_unit) {   // the whole warp: O changes its unit
                        const float unit = __uint_as_float((__float_as_uint(v_scale) & 0x7f800000u) + 0x00800000u);   // next power of two
                        const float gain = __uint_as_float(((2u * 127u + 15u) << 23) - __float_as_uint(unit));        // 2^15 / unit
                        const float shrink = gain * v_unit * (1.0f / kWeightScale);
                        v_unit = unit;
                        v_gain = gain;
#pragma unroll
                        for (int n = 0; n < NS; ++n)
#pragma unroll
                            for (int dd = 0; dd < kVCh; ++dd)
#pragma unroll
                                for (int c = 0; c < 4; ++c) u.acc[n][dd][c] *= shrink;
                    }
                    const float weight_scale = v_scale * v_gain;
                    __syncwarp();  // the previous page's readers of the scratch are done
#pragma unroll
                    for (int n = 0; n < NS; ++n) {
                        const float p0 = visible0 ? exp2f(s0[n] - u.m[n]) : 0.0f, p1 = visible1 ? exp2f(s1[n] - u.m[n]) : 0.0f;
                        u.l[n] += p0 + p1;
                        // P goes to the tensor cores as fp16; the rounding residue is fed as a second operand so that
                        // P V is accurate to fp32 level whatever the magnitude of V
                        // The weights (at most 1) are scaled by 2^15 on the way, O by 2^-15 at the partial's end, both exact:
                        // binary16 then resolves weights down to 2^-40 of the row maximum instead of 2^-25.
                        const uint32_t at = (4u * n + o_head) * 16u + my_token;
                        const float w0 = p0 * weight_scale, w1 = p1 * weight_scale;
                        const __half p0h = __float2half_rn(w0), p1h = __float2half_rn(w1);
                        p_rows[at] = p0h;
                        p_rows[at + 2u] = p1h;
                        p_rows_lo[at] = __float2half_rn(w0 - __half2float(p0h));
                        p_rows_lo[at + 2u] = __float2half_rn(w1 - __half2float(p1h));
                    }
                    __syncwarp();
                    // P rows as A fragments. Rows g / g+8 of the fragment belong to lane tags g>>2 / (g>>2)+2; a lane
                    // feeds the row whose tag is its own t and zeros (read from the zero row) otherwise.
                    uint32_t ra[2][NS][8], rb[2][NS][8];   // [fp16(p) | its rounding residue][group][fragment words]
#pragma unroll
                    for (int part = 0; part < 2; ++part) {
#pragma unroll
                        for (int n = 0; n < NS; ++n) {
                            const __half *rows = (part ? p_rows_lo : p_rows) + (4u * n + o_head) * 16u;
                            const __half *row_a = row_lo_mine ? rows : zero_row;
                            const __half *row_b = row_hi_mine ? rows : zero_row;
                            const uint4 a_lo = *reinterpret_cast<const uint4 *>(row_a);
                            const uint4 a_hi = *reinterpret_cast<const uint4 *>(row_a + 8);
                            const uint4 b_lo = *reinterpret_cast<const uint4 *>(row_b);
                            const uint4 b_hi = *reinterpret_cast<const uint4 *>(row_b + 8);
                            ra[part][n][0] = a_lo.x; ra[part][n][1] = a_lo.y; ra[part][n][2] = a_lo.z; ra[part][n][3] = a_lo.w;
                            ra[part][n][4] = a_hi.x; ra[part][n][5] = a_hi.y; ra[part][n][6] = a_hi.z; ra[part][n][7] = a_hi.w;
                            rb[part][n][0] = b_lo.x; rb[part][n][1] = b_lo.y; rb[part][n][2] = b_lo.z; rb[part][n][3] = b_lo.w;
                            rb[part][n][4] = b_hi.x; rb[part][n][5] = b_hi.y; rb[part][n][6] = b_hi.z; rb[part][n][7] = b_hi.w;
                        }
                    }
#pragma unroll
                    for (int tq = 0; tq < 4; ++tq) {   // token quads outside: consecutive mma feed different accumulators
#pragma unroll
                        for (int dd = 0; dd < kVCh; ++dd) {
                            uint32_t lo, hi;
                            quad_to_half2(u.vq[dd * 4 + tq], lo, hi);   // converted once, used by both parts
#pragma unroll
                            for (int part = 0; part < 2; ++part)
#pragma unroll
                                for (int n = 0; n < NS; ++n)
                                    mma_16816(u.acc[n][dd], ra[part][n][2 * tq], rb[part][n][2 * tq], ra[part][n][2 * tq + 1],
                                              rb[part][n][2 * tq + 1], lo, hi);
                        }
                    }
                    }   // !kProbe
                }
            }
            if (!next_issued && i + 1 < n_pages) {   // page skipped: nobody reads the record any more
                __syncwarp();
                issue(entry_next);
            }
            entry_cur = entry_next;
            entry_next = entry_after;
        }
        if (!alive) {
            // give the copy still in flight a bounded chance to land before this warp's buffers go away
            mbar_wait(bar, phase, p.wait_polls);
            break;
        }

        if constexpr (kMode == kDump) {
        } else if constexpr (kMode == kFold) {   // the checksum of everything the partial covers, so that the work cannot be dropped
            uint32_t folded = u.vq[0];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) folded ^= __shfl_xor_sync(0xffffffffu, folded, o);
            if (lane == 0) partial_ptr(p, partial, out_head_base)[0] = __uint_as_float(folded);
        } else {
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            float sum = u.l[n];
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            sum += __shfl_xor_sync(0xffffffffu, sum, 16);
            if (t == 0 && g < 4u && 4u * n + g < G) {
                float *dst = partial_ptr(p, partial, out_head_base + 4u * n + g);
                dst[0] = u.m[n];
                dst[1] = sum;
            }
            if (4u * n + o_head < G) {
                float *dst = partial_ptr(p, partial, out_head_base + 4u * n + o_head) + 2;
#pragma unroll
                for (int dd = 0; dd < kVCh; ++dd) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t owner = 4u * (2u * t + (c & 1)) + (g >> 2) + 2u * (c >> 1);  // lane whose V block it is
                        if (kDim != 80 || kVCh * owner + dd < 80u) dst[kVCh * owner + dd] = u.acc[n][dd][c] * (v_unit * (1.0f / kWeightScale));
                    }
                }
            }
        }
        }   // !kProbe
        __syncwarp();
    }
    wait_for_previous_kernel();
}

}  // namespace

bool lanes_kernel_supports(const AttentionParams &p) {
    const bool geometry = p.page_tokens == 16 &&
                          ((p.head_dim == 128 && (p.block_size == 64 || p.block_size == 128 || p.block_size == 256)) ||
                           ((p.head_dim == 96 || p.head_dim == 64) && (p.block_size == 64 || p.block_size == 128)) ||
                           ((p.head_dim == 80 || p.head_dim == 32) && p.block_size == 64));
    // queries are read two channels at a time; others go to the any-geometry kernel, which reads them one by one
    const uint32_t query_bytes = p.query_type == CF_B200_F32 ? 8u : 4u;
    return geometry && p.group >= 1 && p.group <= 16 && reinterpret_cast<uintptr_t>(p.queries) % query_bytes == 0 &&
           (p.query_type == CF_B200_F16 || p.query_type == CF_B200_F32);
}

namespace {

// Calls f with the kernel's template arguments for a launch. Query groups of up to four heads per kv head run the four-head kernel;
// larger groups the eight-head one, which decodes a page once for eight query heads (a group of 16 in two passes). fp32
// queries (the reference's own ABIs pass nothing else) take the forms with split queries.
template <int NB, int kDim, class F>
cudaError_t with_heads(const AttentionParams &p, F f) {
    if (p.decode_probe == 2u) return f.template operator()<1, kDump, false, NB, kDim>();
    if (p.decode_probe) return f.template operator()<1, kFold, false, NB, kDim>();
    if (p.query_type == CF_B200_F32)
        return p.group <= 4 ? f.template operator()<2, kAttend, true, NB, kDim>() : f.template operator()<4, kAttend, true, NB, kDim>();
    return p.group <= 4 ? f.template operator()<1, kAttend, false, NB, kDim>() : f.template operator()<2, kAttend, false, NB, kDim>();
}
template <class F>
cudaError_t with_variant(const AttentionParams &p, F f) {
    // 16 x 64 pages have 16 (or 8) blocks per stream, 16 x 96 pages 24 (or 12), 16 x 80 pages 20, 16 x 32
    // pages 8: always staged
    if (p.head_dim == 64) return p.block_size == 64 ? with_heads<16, 64>(p, f) : with_heads<8, 64>(p, f);
    if (p.head_dim == 96) return p.block_size == 64 ? with_heads<24, 96>(p, f) : with_heads<12, 96>(p, f);
    if (p.head_dim == 80) return with_heads<20, 80>(p, f);
    if (p.head_dim == 32) return with_heads<8, 32>(p, f);
    if (p.block_size == 128) return with_heads<16, 128>(p, f);
    if (p.block_size == 256) return with_heads<8, 128>(p, f);
    return with_heads<32, 128>(p, f);
}

template <int NG, int kMode, bool kSplitQ, int NB, int kDim>
cudaError_t launch_one(const AttentionParams &p, int sm_count, cudaStream_t stream, bool dependent, bool after_prefix) {
    using L = WarpLayout<NG, NB, kSplitQ, kDim>;
    static std::atomic<uint64_t> configured{0};   // bit = device ordinal
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (device & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        e = cudaFuncSetAttribute(lanes_attention_kernel<NG, kMode, kSplitQ, NB, kDim>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(L::kSmem));
        if (e != cudaSuccess) return e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    return launch_kernel(lanes_attention_kernel<NG, kMode, kSplitQ, NB, kDim>, sm_count, kThreadsOf<NG, NB, kSplitQ, kDim>, L::kSmem,
                         stream, dependent, p, static_cast<uint32_t>(after_prefix));
}

}  // namespace

void lanes_plan_shape(const AttentionParams &p, uint32_t sm_count, uint32_t *warps, uint32_t *unit_lanes) {
    with_variant(p, [&]<int NG, int kMode, bool kSplitQ, int NB, int kDim>() {
        constexpr uint32_t kHeads = 4u * kHeadGroups<NG, kSplitQ>;
        *warps = sm_count * kWarpsOf<NG, NB, kSplitQ, kDim>;
        *unit_lanes = p.kv_head_span * ((p.group + kHeads - 1u) / kHeads);
        return cudaSuccess;
    });
}

cudaError_t launch_lanes_attention(const AttentionParams &p, cudaStream_t stream, bool dependent, bool after_prefix) {
    static LauncherState table[64];
    cudaError_t e;
    LauncherState *state = launcher_state(table, &e);
    if (!state) return e;
    const int sm_count = state->sm_count;
    return with_variant(p, [&]<int NG, int kMode, bool kSplitQ, int NB, int kDim>() {
        return launch_one<NG, kMode, kSplitQ, NB, kDim>(p, sm_count, stream, dependent, after_prefix);
    });
}

}  // namespace cfb
