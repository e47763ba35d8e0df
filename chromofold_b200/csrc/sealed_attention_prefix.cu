// sealed_attention_prefix.cu — attention over a SHARED sealed prefix: pages that every sequence of the batch
// references (one copy in the arena, the same page ids at the head of every page-table row; the reference's
// shared-page semantics, src/multisequence_cache.cpp:235-292), or that the query tokens of one sequence share, on the
// 5th-generation tensor cores (tcgen05.mma with accumulators and the A operands in tensor memory). Geometry: head_dim 128 or
// 64, page_tokens 16, block 64.
//
// The per-sequence kernel would decode such a page once per sequence. Here a page is decoded once per tile of 128
// query rows (rows = sequence x query head of the kv head's group) and contracted with all those rows at once.
//
// One CTA of 20 warps per SM. The work is cut evenly (SharedSplit): the rounds (8 pages = 128 tokens) of every
// (kv head, row tile) pair form one line and each CTA takes an equal stretch of it; the part of a stretch inside one
// pair is a unit, which ends in one partial per row. From two row tiles on, two CTAs (a cluster) take a stretch together, a row
// tile each: each decodes half of every round's pages and sends them to the other, so that a page is decoded once per 256 rows.
// The warps are specialised:
//   decoder warps 0..11  the page slots of the CTA's units form one sequence; warp w takes slots w, w + 12, ... It
//                        receives the record by one bulk async copy (mbarrier, bounded wait), decodes it with the
//                        lane-per-block decoders INTO REGISTERS (32 packed quads per lane), starts the copy of its next
//                        record, and only then waits for the tile pair of the slot's round to be free; the symbols
//                        are written as exact binary16 codes into one of TWO tile pairs in shared memory: K tile
//                        [token][channel] (B of S = Q K^T), V tile [channel][token] (B of O = P V); then the warp
//                        arrives on the pair's "full" barrier (8 arrivals = one round). A pair is free when the tensor
//                        core's commit for the round that read it has arrived on its "free" barrier.
//   softmax warps 12..19 a thread owns one row (= tensor-memory lane, in its warp's quarter) and half of the round's
//                        128 score columns: one tcgen05.ld of its 64 scores (kept in registers), page K scales and masks,
//                        the row's two threads share their maxima through shared memory, running max / sum updated,
//                        O rescaled in tensor memory (tcgen05.ld / .st) only when some row of the warp moved its max by 2^0.9,
//                        P and its residue written over the scores (tcgen05.st) as the next A operands.
//                        Thread 0 of the group (in a pair of CTAs: warp 11) issues the tensor-core work (M 128, K 16):
//                          S     Q from tensor memory x K tile -> one of two sets of 128 score columns
//                          O     16 tcgen05.mma: P (binary16, then its rounding residue) from tensor memory x V tile
//                        Unit start: the Q rows go from global memory straight to tensor memory. Unit end: O read back,
//                        scaled, written with (max, sum) to the shared-prefix partials; the combine kernel merges
//                        them with the per-sequence partials of the private pages and the tail.
// Registers: the kernel starts at 96 per thread; the decoders drop to 80 and the softmax warps rise to 120 (setmaxnreg).
// Tensor memory (512 columns): scores and weights of even rounds 0..127, of odd rounds 128..255 (P 64 columns of binary16 pairs, then
// its residue), O 256..383, Q 384..447, Q residue 448..511 (fp32 queries only: the row is split into binary16(q) and its
// rounding residue, S = Q K^T + Q residue K^T). Row = lane. B tiles use the no-swizzle K-major canonical layout: 8 rows x 16
// bytes core matrices, element (row r, 16-byte chunk c) at (r % 8) * 16 + (r / 8) * 2048 + c * 128 bytes in the K tile and at
// (r % 8) * 16 + (r / 8) * 128 + c * 2048 in the V tile: a page (16 rows of K, two chunks of V) is then 4096 bytes in a row in
// either, which a pair's CTA sends to the other one by bulk copies. (Against storing them there 16 bytes at a time: 500 rows after
// 16384 tokens 560 -> 544 us. A decoder warp itself gains nothing by it: of its 22000 clocks per page the stores to both CTAs took
// 4000, now stores, fence and copies take 2200 and 2400.)
// Head_dim 64 runs the same kernel on the left half of the K tile and the upper half of the V tile.
// The page's V scale relative to the largest one met so far in the unit rides on P (never above 1); O is kept in units of
// that scale and rescaled when a larger one arrives.
// Every mbarrier wait is bounded. A warp whose wait ran out raises CF_B200_DEVSTAT_WAIT_EXPIRED and skips all later
// waits and work, but a decoder warp whose record never came, which goes on with absent pages, and a softmax warp still takes
// part in the barrier with its partner, which OR-reduces the failure so that both leave their loops at the same point; the roles
// that wait for one that left run out of their own waits; the CTA then frees its tensor memory.

#include "lanes_decoders.cuh"

namespace cfb {
namespace {

using namespace lanes;

constexpr int kDecodeWarps = 12;     // warps 0..11 (three warpgroups)
// In a pair of CTAs warp 11 issues the tensor-core work: decoding half of the pages needs no twelfth warp. A CTA on its own
// decodes them all, and thread 0 of the softmax group issues.
template <int kCluster> constexpr int kDecoders = kCluster == 2 ? kDecodeWarps - 1 : kDecodeWarps;
constexpr int kSoftmaxWarps = 8;     // warps 12..19 (two warpgroups)
constexpr int kRoundPages = 8;
constexpr int kTcThreads = (kDecodeWarps + kSoftmaxWarps) * 32;
constexpr uint32_t kTileBytes = 128 * 128 * 2;   // one operand tile: 128 rows x 128 binary16
// A stage takes the largest record. The decoders look up to two words past a part's end: there the next stage begins, or the tiles,
// and what they find is not used.
constexpr uint32_t kRecordBytes = 16 + 2 * 2048;
constexpr uint32_t kOffStages = kTableBytes;
constexpr uint32_t kOffTiles = (kOffStages + kDecodeWarps * kRecordBytes + 127u) / 128u * 128u;   // K[0] V[0] K[1] V[1]
constexpr uint32_t kOffMeta = kOffTiles + 4 * kTileBytes;      // [pair][page of the round]: k scale, v scale, token count, -
constexpr uint32_t kOffRound = kOffMeta + 2 * kRoundPages * 16;    // [pair]: unit, flags, -, -
constexpr uint32_t kOffBars = kOffRound + 2 * 16;              // 12 copy barriers, full[2], free[4], S[2], O[2], P[2], Q
constexpr uint32_t kBarFull = kDecodeWarps, kBarFree = kBarFull + 2, kBarS = kBarFree + 4, kBarO = kBarS + 2, kBarP = kBarO + 2, kBarQ = kBarP + kWeightBarriers,
                   kBarCount = kBarQ + 1;
constexpr uint32_t kOffMisc = kOffBars + kBarCount * 8;        // [0] tmem base, [kMiscRounds], [kMiscGaveUp], [kMiscNext + warp]
constexpr uint32_t kMiscRounds = 1;   // pair of CTAs: rounds in which some decoder warp of either has arrived, known once all have left
constexpr uint32_t kMiscGaveUp = 2;   // ... an issuing thread of either has left before the last round
constexpr uint32_t kMiscNext = 4;     // ... the first of its slots that decoder warp has not arrived for
constexpr uint32_t kOffRowMax = kOffMisc + 64;                 // [round parity][2 column halves][128 rows]
constexpr uint32_t kTcSmem = kOffRowMax + 4 * 128 * 4;
static_assert(kTcSmem <= 232448, "the shared-prefix kernel must fit the 227 KB of one CTA");
constexpr uint32_t kTmemColumns = 512;
constexpr uint32_t kColS = 0, kColO = 256, kColQ = 384, kColQResidue = 448;
constexpr uint32_t kStopUnit = 0xffffffffu;
constexpr float kWeightScale = 32768.0f;   // power of two the binary16 weights are scaled by (O sheds it at a unit's end)
// The maximum that the weights are relative to follows the true one only when that has risen by this much in the exponent of two. A
// weight is then at most 2^0.9 = 1.8661, and 2^(1/16) more where the maximum itself was rounded (products of 2^20).
constexpr float kMaxLag = 0.9f, kLargestWeight = 1.8661f * 1.0443f;
static_assert(kMaxLag <= 0.9f && kWeightScale * kLargestWeight < 65504.0f, "binary16 has to hold the scaled weights");
constexpr uint32_t kFirstRound = 1u, kLastRound = 2u;   // round flags
// Register split (setmaxnreg). A CTA can only redistribute the registers it was launched with: kLaunchRegs per thread,
// the most that 640 threads can have. What the softmax warps ask for must not exceed what the decoders give back, or
// the request would wait forever; the launch function checks kLaunchRegs against the compiled kernel.
constexpr int kLaunchRegs = 96, kDecoderRegs = 80, kSoftmaxRegs = 120;
static_assert(kLaunchRegs * kTcThreads <= 65536 && kDecoderRegs % 8 == 0 && kSoftmaxRegs % 8 == 0 &&
                  kDecodeWarps * 32 * kDecoderRegs + kSoftmaxWarps * 32 * kSoftmaxRegs <= kLaunchRegs * kTcThreads,
              "the register split must fit the CTA's own registers");
// instruction descriptors: f32 accumulate, f16 x f16, both operands K-major, M = 128; N = 128 tokens (S) or kDim channels (O)
constexpr uint32_t kIdescS = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
template <int kDim> constexpr uint32_t kIdescO = (1u << 4) | ((static_cast<uint32_t>(kDim) >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint32_t k_tile_offset(uint32_t row, uint32_t chunk) { return (row & 7u) * 16u + (row >> 3) * 2048u + chunk * 128u; }
__device__ __forceinline__ uint32_t v_tile_offset(uint32_t row, uint32_t chunk) { return (row & 7u) * 16u + (row >> 3) * 128u + chunk * 2048u; }
// Row of the V tile (= column of O) that holds channel 4 * lane + c, the c-th channel of the block lane decodes: the 32
// lanes of one store spread over all 8 rows of a core matrix, so a 16-byte store per lane meets no bank conflict.
// Inverse: column n of O is channel 4 * ((n & 7) + 8 * (n >> 5)) + ((n >> 3) & 3).
__device__ __forceinline__ uint32_t v_tile_row(uint32_t lane, uint32_t c) {
    return (lane & 7u) + 8u * c + 32u * (lane >> 3);
}
// shared-memory matrix descriptor: start address, leading (K) offset, stride (row group) offset, version 1
__device__ __forceinline__ uint64_t tile_desc(uint32_t smem_address, uint32_t chunk_stride, uint32_t group_stride) {
    return static_cast<uint64_t>((smem_address >> 4) & 0x3fffu) | (static_cast<uint64_t>(chunk_stride >> 4) << 16) |
           (static_cast<uint64_t>(group_stride >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ uint64_t k_desc(uint32_t k_tile, uint32_t step) { return tile_desc(k_tile + 256u * step, 128u, 2048u); }     // 16 channels
__device__ __forceinline__ uint64_t v_desc(uint32_t v_tile, uint32_t step) { return tile_desc(v_tile + 4096u * step, 2048u, 128u); }   // 16 tokens
// D[tmem_d] (+)= A[tmem_a: 128 lanes x 8 columns of binary16 pairs] x B[shared-memory tile]^T, one K step of 16
__device__ __forceinline__ void umma(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t accumulate, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// A pair of CTAs (a cluster of two) shares the decoded pages: each decodes half of every round and sends it to the other.
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t peer_address(uint32_t smem_address, uint32_t rank) {   // the same place in CTA `rank` of the pair
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_address), "r"(rank));
    return r;
}
__device__ __forceinline__ void store_peer(uint32_t address, uint4 v) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(address), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void store_peer(uint32_t address, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(address), "r"(v) : "memory");
}
__device__ __forceinline__ void max_peer(uint32_t address, uint32_t v) {
    asm volatile("red.relaxed.cluster.shared::cluster.max.u32 [%0], %1;" ::"r"(address), "r"(v) : "memory");
}
__device__ __forceinline__ void mbar_arrive_peer(uint32_t address) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(address) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_peer(uint32_t address, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(address), "r"(bytes) : "memory");
}
// Shared memory of this CTA to the other one's, counted by a barrier there.
__device__ __forceinline__ void copy_to_peer(uint32_t to, uint32_t from, uint32_t bytes, uint32_t peer_bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to), "r"(from), "r"(bytes),
                 "r"(peer_bar)
                 : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Waits and polls that also see what the other CTA of the pair stored before it arrived.
__device__ __forceinline__ bool mbar_wait_pair(uint64_t *bar, uint32_t parity, uint32_t polls) {
    for (uint32_t i = 0; i < polls; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(smem_addr(bar)), "r"(parity), "r"(1000u)
                     : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ bool mbar_test_pair(uint64_t *bar, uint32_t parity) {   // one poll that does not wait
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// The same, for both CTAs of the pair.
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_addr(bar)),
                 "h"(static_cast<uint16_t>(3))
                 : "memory");
}
// Barrier over whole warps that also ORs a predicate: every thread of them gets the same answer.
template <uint32_t kThreads>
__device__ __forceinline__ bool group_any(uint32_t barrier_id, bool pred) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"(static_cast<uint32_t>(pred)), "r"(barrier_id), "r"(kThreads)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void tmem_load32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_store32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
        "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]),
        "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]),
        "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Two quads of symbols (8 codes) -> one 16-byte chunk of binary16 codes, exact.
__device__ __forceinline__ uint4 codes8(uint32_t qa, uint32_t qb) {
    uint4 r;
    quad_to_half2(qa, r.x, r.y);
    quad_to_half2(qb, r.z, r.w);
    return r;
}

// Decode one record into registers: quad q of a stream = symbols 4q..4q+3 of the block this lane decodes.
template <class KLane, class VLane>
__device__ __forceinline__ void decode_page(KLane &k, VLane &v, uint32_t (&kq)[16], uint32_t (&vq)[16]) {
    // Four passes of four quads per stream. The pass is a real loop (its body is a quarter of the unrolled code, which
    // the instruction cache shares with the softmax warps' code); the results shift down the register arrays, so that
    // after the fourth pass quad q sits in element q.
#pragma unroll 1
    for (int pass = 0; pass < 4; ++pass) {
#pragma unroll
        for (int i = 0; i < 12; ++i) {
            kq[i] = kq[i + 4];
            vq[i] = vq[i + 4];
        }
#pragma unroll
        for (int q = 12; q < 16; ++q) {
            if constexpr (requires { k.lo_word(0); v.lo_word(0); }) {   // both nibble-split: two steps per quad, the chains interleave
                uint32_t ke[2], ve[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    ke[i] = k.symbol(i);
                    ve[i] = v.symbol(i);
                }
                k.advance();
                v.advance();
                const int j = 2 * pass + ((q - 12) >> 1), shift = 4 * (q & 1);
                kq[q] = merge_split_quad<KLane>(ke[0], ke[1], k.lo_word(j) >> shift);
                vq[q] = merge_split_quad<VLane>(ve[0], ve[1], v.lo_word(j) >> shift);
            } else if constexpr (KLane::kWholeQuads || VLane::kWholeQuads) {   // fixed width: a quad per call
                kq[q] = k.quad(4 * pass + (q - 12));
                vq[q] = v.quad(4 * pass + (q - 12));
            } else {   // both entropy coded: the two chains interleave symbol by symbol
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
                kq[q] = KLane::pack(ke[0], ke[1], ke[2], ke[3]);
                vq[q] = VLane::pack(ve[0], ve[1], ve[2], ve[3]);
            }
        }
    }
}
template <class Lane>
__device__ __forceinline__ void decode_stream(Lane &s, uint32_t (&quads)[16]) {
#pragma unroll
    for (int q = 0; q < 16; ++q) quads[q] = s.quad(q);
}
// The decoded page goes into slot `slot` of the round's tiles as exact binary16 codes. K quad q of lane l = token l/2,
// channels 64(l&1)+4q..+3 -> K tile row 16*slot + l/2; V quad q of lane l = channel 4l + q/4, tokens 4(q%4)..+3 -> V tile
// row v_tile_row(l, q/4), token chunks 2*slot and 2*slot+1.
// A page that is absent (past the unit's end, or refused) leaves zeros in its slot of both tiles.
__device__ __forceinline__ void store_tiles(const uint32_t (&kq)[16], const uint32_t (&vq)[16], bool present, uint8_t *k_tile, uint8_t *v_tile,
                                            uint32_t slot, uint32_t lane) {
    const uint32_t k_row = 16u * slot + (lane >> 1);
    auto put = [&](uint8_t *at, uint32_t qa, uint32_t qb) { *reinterpret_cast<uint4 *>(at) = present ? codes8(qa, qb) : make_uint4(0u, 0u, 0u, 0u); };
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint32_t k_chunk = 8u * (lane & 1u) + 2u * c;
        put(k_tile + k_tile_offset(k_row, k_chunk), kq[4 * c], kq[4 * c + 1]);
        put(k_tile + k_tile_offset(k_row, k_chunk + 1u), kq[4 * c + 2], kq[4 * c + 3]);
        const uint32_t v_row = v_tile_row(lane, c);
        put(v_tile + v_tile_offset(v_row, 2u * slot), vq[4 * c], vq[4 * c + 1]);
        put(v_tile + v_tile_offset(v_row, 2u * slot + 1u), vq[4 * c + 2], vq[4 * c + 3]);
    }
}
// Head_dim 64: a stream has sixteen blocks, a lane decodes one block of one stream. K block l = token l, V block l = channels
// 4 l .. 4 l + 3 of every token.
__device__ __forceinline__ void decode_half(const uint8_t *part, uint32_t part_bytes, uint32_t coder, uint32_t block, const uint32_t *slot_table,
                                            const uint16_t *lut, uint32_t (&quads)[16]) {
    if (coder == CF_B200_CODER_RANS_SPLIT4) {
        RansSplitLaneT<16, 1024> d;
        d.open(part, part_bytes, block, slot_table);
        decode_stream(d, quads);
    } else if (coder == CF_B200_CODER_HUFFMAN_SPLIT4) {
        HuffSplitLaneT<16, 1024> d;
        d.open(part, part_bytes, block, lut);
        decode_stream(d, quads);
    } else if (coder == CF_B200_CODER_RANS) {
        RansLaneT<16> d;
        d.open(part, part_bytes, block, slot_table);
        decode_stream(d, quads);
    } else if (coder == CF_B200_CODER_HUFFMAN) {
        HuffLaneT<16> d;
        d.open(part, part_bytes, block, lut);
        decode_stream(d, quads);
    } else {
        FixedLaneT<16, 1024> d;
        d.open(part, part_bytes, block);
        decode_stream(d, quads);
    }
}
__device__ __forceinline__ void store_half(const uint32_t (&quads)[16], bool present, uint8_t *k_tile, uint8_t *v_tile, uint32_t slot, uint32_t lane) {
    const uint32_t l = lane & 15u;
#pragma unroll
    for (int c = 0; c < 8; ++c) {   // K: chunk c of token l's row; V: half c & 1 of channel 4 l + c / 2's sixteen tokens
        const uint4 codes = present ? codes8(quads[2 * c], quads[2 * c + 1]) : make_uint4(0u, 0u, 0u, 0u);
        uint8_t *at = lane < 16u ? k_tile + k_tile_offset(16u * slot + l, c) : v_tile + v_tile_offset(v_tile_row(l, c >> 1), 2u * slot + (c & 1));
        *reinterpret_cast<uint4 *>(at) = codes;
    }
}

__device__ __forceinline__ void tmem_store8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
// Two fp32 operations in one instruction, and the largest of three.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float max3(uint32_t a, uint32_t b, uint32_t c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(__uint_as_float(a)), "f"(__uint_as_float(b)), "f"(__uint_as_float(c)));
    return r;
}
// 2^x by the special-function unit (inputs below -126 give 0, -inf gives 0)
__device__ __forceinline__ float fast_exp2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// What both groups derive from a unit number: unit j of CTA b is the CTA's stretch of rounds inside the j-th head-tile it
// meets (SharedSplit). `valid` is false past the CTA's last unit.
struct UnitShape {
    uint32_t tile_index, head_local, chunk, kv_head, page_begin, page_end, valid;
};
__device__ __forceinline__ UnitShape unit_shape(const AttentionParams &p, const SharedSplit &split, uint32_t cta, uint32_t unit,
                                                uint32_t tile_groups, uint32_t shared_pages) {
    UnitShape u = {};
    const uint64_t lo = split.first_round(cta), hi = split.first_round(cta + 1u);
    const uint64_t head_tile = lo / split.rounds + unit, base = head_tile * split.rounds;
    u.valid = lo < hi && base < hi;
    if (!u.valid) return u;
    const uint32_t r0 = static_cast<uint32_t>((lo > base ? lo : base) - base);
    const uint32_t r1 = static_cast<uint32_t>((hi < base + split.rounds ? hi : base + split.rounds) - base);
    u.tile_index = static_cast<uint32_t>(head_tile % tile_groups);   // of groups of kCluster tiles
    u.head_local = static_cast<uint32_t>(head_tile / tile_groups);
    u.chunk = cta - split.cta_of(base);
    u.kv_head = p.kv_head_begin + u.head_local;
    u.page_begin = 8u * r0;
    u.page_end = min(8u * r1, shared_pages);
    return u;
}

// ---- decoder group: warps 0..11 -----------------------------------------------------------------------------------
// The page slots of the CTA's units (pages of a unit padded to whole rounds of eight) form one sequence; decoder warp w takes slots w, w + 12, w + 24, ... A slot is decoded into registers first;
// only then does the warp wait for the tile pair of the slot's round, so that decoding never waits for the tensor core.
struct SlotCursor {
    uint32_t unit, valid, first_slot, first_round, slots;   // of the unit that holds the slot
    UnitShape u;
};

template <int kDim, int kCluster>
__device__ __forceinline__ void decoder_role(const AttentionParams &p, uint8_t *smem, PlanHeader *hdr, uint32_t warp, uint32_t lane,
                                             uint32_t tile_groups, const SharedSplit &split) {
    const uint32_t worker = blockIdx.x / kCluster, rank = kCluster == 1 ? 0u : cluster_rank();
    const uint32_t peer_delta = kCluster == 1 ? 0u : peer_address(smem_addr(smem), rank ^ 1u) - smem_addr(smem);   // own place -> the peer's
    // this CTA's m-th slot: all of them, or its half of every round
    auto slot_number = [&](uint32_t m) { return kCluster == 1 ? m : pair_slot(m, rank); };
    const uint32_t *k_slot = reinterpret_cast<const uint32_t *>(smem);
    const uint32_t *v_slot = k_slot + 4096;
    const uint16_t *k_lut = reinterpret_cast<const uint16_t *>(v_slot + 4096);
    const uint16_t *v_lut = k_lut + 4096;
    uint8_t *stage = smem + kOffStages + warp * kRecordBytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kOffBars);
    uint64_t *bar = bars + warp, *bar_full = bars + kBarFull, *bar_free = bars + kBarFree;
    uint32_t *round_desc = reinterpret_cast<uint32_t *>(smem + kOffRound);
    const uint32_t shared_pages = hdr->shared_pages;
    const uint32_t *table_row = p.page_table + static_cast<uint64_t>(slot_of(p, 0)) * p.page_table_stride;

    auto load_unit = [&](SlotCursor &c) {
        c.u = unit_shape(p, split, worker, c.unit, tile_groups, shared_pages);
        c.valid = c.u.valid;
        if (c.valid) c.slots = (c.u.page_end - c.u.page_begin + 7u) / 8u * 8u;
    };
    auto seek = [&](SlotCursor &c, uint32_t n) {   // the unit that holds slot n (n only grows)
        while (c.valid && n >= c.first_slot + c.slots) {
            c.first_slot += c.slots;
            c.first_round += c.slots / 8u;
            c.unit += 1u;
            load_unit(c);
        }
    };
    // directory entry of slot n, 0 if the slot is padding or past the CTA's last unit
    auto slot_entry = [&](const SlotCursor &c, uint32_t n) -> uint64_t {
        if (!c.valid) return 0ull;
        const uint32_t page = c.u.page_begin + (n - c.first_slot);
        if (page >= c.u.page_end) return 0ull;
        const uint32_t page_id = table_row[page];   // bit 63 marks the page of the wait-expiry test: armed, never fetched
        const uint64_t e = p.page_dir[static_cast<uint64_t>(page_id) * p.kv_head_count + c.u.kv_head];
        return page_id == p.skip_copy_page ? e | (1ull << 63) : e;
    };
    auto entry_ok = [&](uint64_t entry) {
        const uint32_t units16 = static_cast<uint32_t>(CF_B200_DIR_LENGTH_UNITS(entry));
        return units16 != 0 && units16 * 16u <= kRecordBytes;
    };
    auto issue = [&](uint64_t entry) {
        if (lane == 0 && entry_ok(entry)) {
            const uint32_t bytes = static_cast<uint32_t>(CF_B200_DIR_LENGTH_UNITS(entry)) * 16u;
            mbar_expect_tx(bar, bytes);
            if (!(entry >> 63)) bulk_load(stage, p.arena + 16ull * CF_B200_DIR_OFFSET_UNITS(entry), bytes, bar);
        }
    };
    uint32_t copy_phase = 0;
    // Warp-uniform. kNoRecord: a record never came; the warp decodes nothing more, but goes on by the rules: its pages are absent, and
    // both CTAs' tiles get zeros for them (zero weights alone would not do: what lies there from before may be NaN).
    // kNoTiles: no tiles were freed; the warp leaves, and arrives for nothing more.
    constexpr uint32_t kNoRecord = 1u, kNoTiles = 2u;
    uint32_t failed = 0u;
    // The pair of round `it` is free once the tensor core (of both CTAs) has finished round it - 2, which the barrier of that round's
    // number modulo four tells. The parity wait is sound because a warp's slots are at most three rounds apart, so that it has
    // seen the end of a round later than it - 6, the barrier's previous one.
    auto wait_pair_free = [&](uint32_t it) {
        if (it >= 2u && !__all_sync(0xffffffffu, mbar_wait_pair(&bar_free[(it - 2u) & 3u], ((it - 2u) >> 2) & 1u, p.wait_polls))) {
            failed = kNoTiles;
            if (lane == 0) raise_status(p, CF_B200_DEVSTAT_WAIT_EXPIRED);
        }
    };
    auto arrive_full = [&](uint32_t pair) {
        mbar_arrive(&bar_full[pair]);
        if constexpr (kCluster == 2) mbar_arrive_peer(smem_addr(&bar_full[pair]) + peer_delta);
    };
    auto describe_round = [&](uint32_t pair, uint32_t unit, uint32_t flags) {
        round_desc[4 * pair] = unit;
        round_desc[4 * pair + 1] = flags;
        if constexpr (kCluster == 2) store_peer(smem_addr(round_desc + 4 * pair) + peer_delta, make_uint4(unit, flags, 0u, 0u));
    };

    SlotCursor cur;
    cur.unit = 0;
    cur.first_slot = 0;
    cur.first_round = 0;
    cur.slots = 0;
    load_unit(cur);
    uint32_t m = warp, n = slot_number(m);
    seek(cur, n);
    uint64_t entry = slot_entry(cur, n);
    issue(entry);

    for (;; m += kDecoders<kCluster>, n = slot_number(m)) {
        if (!cur.valid) {   // past the last unit: the eight slots after it make the round that tells the softmax group to stop
            if (n < cur.first_slot + 8u) {
                wait_pair_free(cur.first_round);
                if (lane == 0 && failed != kNoTiles) {
                    if (n == cur.first_slot) describe_round(cur.first_round & 1u, kStopUnit, 0u);
                    arrive_full(cur.first_round & 1u);
                }
                if (failed != kNoTiles) m += kDecoders<kCluster>;
            }
            break;
        }
        const uint32_t in_unit = n - cur.first_slot, slot = in_unit & 7u, it = cur.first_round + (in_unit >> 3), pair = it & 1u;
        // the warp's next slot: its directory entry is fetched now (dependent loads), needed only after this decode
        SlotCursor next = cur;
        const uint32_t next_n = slot_number(m + kDecoders<kCluster>);
        seek(next, next_n);
        const uint64_t next_entry = slot_entry(next, next_n);

        float k_scale = 0.0f, v_scale = 0.0f;
        uint32_t token_count = 0;
        uint32_t kq[16] = {}, vq[16] = {};
        if (cur.u.page_begin + in_unit < cur.u.page_end && !failed) {
            if (!entry_ok(entry)) {
                if (lane == 0) raise_status(p, CF_B200_DEVSTAT_BAD_RECORD);
            } else if (!__all_sync(0xffffffffu, mbar_wait(bar, copy_phase & 1u, p.wait_polls))) {
                failed = kNoRecord;
                if (lane == 0) raise_status(p, CF_B200_DEVSTAT_WAIT_EXPIRED);
            } else {
                copy_phase ^= 1u;
                const uint4 hv = *reinterpret_cast<const uint4 *>(stage);
                const uint32_t k_bytes = 16u * (hv.x & 0xffffu), v_bytes = 16u * (hv.x >> 16);
                const uint32_t k_coder = hv.y & 0xffu, v_coder = (hv.y >> 8) & 0xffu;
                const uint8_t *k_part = stage + 16, *v_part = k_part + k_bytes;
                bool tables_ok;
                if constexpr (kDim == 128) tables_ok = part_offsets_ok(k_part, k_coder, k_bytes, lane) && part_offsets_ok(v_part, v_coder, v_bytes, lane);
                else tables_ok = lane < 16u ? part_offsets_ok<16, 1024>(k_part, k_coder, k_bytes, lane) : part_offsets_ok<16, 1024>(v_part, v_coder, v_bytes, lane - 16u);
                if (!record_header_ok(hv, entry, p.codebook_id) || !__all_sync(0xffffffffu, tables_ok)) {
                    if (lane == 0) raise_status(p, CF_B200_DEVSTAT_BAD_RECORD);
                } else {
                    token_count = hv.y >> 16;
                    k_scale = __half2float(__ushort_as_half(static_cast<unsigned short>(hv.z & 0xffffu))) * (p.softmax_scale * kLog2e);
                    v_scale = __half2float(__ushort_as_half(static_cast<unsigned short>(hv.z >> 16)));
                    if constexpr (kDim == 64) {   // lanes 0..15: the K blocks, lanes 16..31: the V blocks
                        const bool is_v = lane >= 16u;
                        decode_half(is_v ? v_part : k_part, is_v ? v_bytes : k_bytes, is_v ? v_coder : k_coder, lane & 15u, is_v ? v_slot : k_slot,
                                    is_v ? v_lut : k_lut, kq);
                    } else if (k_coder == CF_B200_CODER_RANS && v_coder == CF_B200_CODER_RANS) {
                        RansLane k, v;
                        k.open(k_part, k_bytes, lane, k_slot);
                        v.open(v_part, v_bytes, lane, v_slot);
                        decode_page(k, v, kq, vq);
                    } else if (k_coder == CF_B200_CODER_HUFFMAN && v_coder == CF_B200_CODER_HUFFMAN) {
                        HuffLane k, v;
                        k.open(k_part, k_bytes, lane, k_lut);
                        v.open(v_part, v_bytes, lane, v_lut);
                        decode_page(k, v, kq, vq);
                    } else if (k_coder == CF_B200_CODER_FIXED8 && v_coder == CF_B200_CODER_FIXED8) {
                        FixedLane k, v;
                        k.open(k_part, k_bytes, lane);
                        v.open(v_part, v_bytes, lane);
                        decode_page(k, v, kq, vq);
                    } else if (k_coder == CF_B200_CODER_RANS_SPLIT4 && v_coder == CF_B200_CODER_RANS_SPLIT4) {
                        RansSplitLane k, v;
                        k.open(k_part, k_bytes, lane, k_slot);
                        v.open(v_part, v_bytes, lane, v_slot);
                        decode_page(k, v, kq, vq);
                    } else if (k_coder == CF_B200_CODER_HUFFMAN_SPLIT4 && v_coder == CF_B200_CODER_HUFFMAN_SPLIT4) {
                        HuffSplitLane k, v;
                        k.open(k_part, k_bytes, lane, k_lut);
                        v.open(v_part, v_bytes, lane, v_lut);
                        decode_page(k, v, kq, vq);
                    } else {
                        if (k_coder == CF_B200_CODER_RANS) { RansLane k; k.open(k_part, k_bytes, lane, k_slot); decode_stream(k, kq); }
                        else if (k_coder == CF_B200_CODER_HUFFMAN) { HuffLane k; k.open(k_part, k_bytes, lane, k_lut); decode_stream(k, kq); }
                        else if (k_coder == CF_B200_CODER_RANS_SPLIT4) { RansSplitLane k; k.open(k_part, k_bytes, lane, k_slot); decode_stream(k, kq); }
                        else if (k_coder == CF_B200_CODER_HUFFMAN_SPLIT4) { HuffSplitLane k; k.open(k_part, k_bytes, lane, k_lut); decode_stream(k, kq); }
                        else { FixedLane k; k.open(k_part, k_bytes, lane); decode_stream(k, kq); }
                        if (v_coder == CF_B200_CODER_RANS) { RansLane v; v.open(v_part, v_bytes, lane, v_slot); decode_stream(v, vq); }
                        else if (v_coder == CF_B200_CODER_HUFFMAN) { HuffLane v; v.open(v_part, v_bytes, lane, v_lut); decode_stream(v, vq); }
                        else if (v_coder == CF_B200_CODER_RANS_SPLIT4) { RansSplitLane v; v.open(v_part, v_bytes, lane, v_slot); decode_stream(v, vq); }
                        else if (v_coder == CF_B200_CODER_HUFFMAN_SPLIT4) { HuffSplitLane v; v.open(v_part, v_bytes, lane, v_lut); decode_stream(v, vq); }
                        else { FixedLane v; v.open(v_part, v_bytes, lane); decode_stream(v, vq); }
                    }
                    if (p.decode_probe == 2u) {   // test mode: the quads as decoded, [page id][kv head][K stream | V stream]
                        const uint32_t page_id = table_row[cur.u.page_begin + in_unit];
                        if (page_id < p.dump_pages) {
                            uint32_t *dump = reinterpret_cast<uint32_t *>(p.output) +
                                             (static_cast<uint64_t>(page_id) * p.kv_head_count + cur.u.kv_head) * (8u * kDim) + 16u * lane;
#pragma unroll
                            for (int q = 0; q < 16; ++q) {
                                dump[q] = kq[q];
                                if constexpr (kDim == 128) dump[512 + q] = vq[q];
                            }
                        }
                    }
                }
            }
        }
        __syncwarp();   // every lane is done with the stage: the next record may land in it
        if (!failed) issue(next_entry);

        wait_pair_free(it);
        if (failed == kNoTiles) break;
        uint8_t *k_tile = smem + kOffTiles + pair * 2u * kTileBytes, *v_tile = k_tile + kTileBytes;
        if constexpr (kDim == 128) store_tiles(kq, vq, token_count != 0u, k_tile, v_tile, slot, lane);
        else store_half(kq, token_count != 0u, k_tile, v_tile, slot, lane);
        if (lane == 0) {
            uint4 *meta = reinterpret_cast<uint4 *>(smem + kOffMeta) + pair * 8u + slot;   // token count 0: the page contributes nothing
            const uint4 about = make_uint4(__float_as_uint(k_scale), __float_as_uint(v_scale), token_count, 0u);
            *meta = about;
            if constexpr (kCluster == 2) store_peer(smem_addr(meta) + peer_delta, about);
            if (slot == 0) describe_round(pair, cur.unit, (in_unit < 8u ? kFirstRound : 0u) | (in_unit + 8u >= cur.slots ? kLastRound : 0u));
        }
        fence_async_smem();   // the tiles were written through the generic proxy; the tensor core and the copies read through the async one
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&bar_full[pair]);
            if constexpr (kCluster == 2) {
                // the page's rows to the other CTA, whose round is full once they are there; its tiles are free, too
                constexpr uint32_t kPart = kDim == 128 ? 2048u : 1024u;   // of 2048 bytes of a row group, or a chunk
                const uint32_t bar = smem_addr(&bar_full[pair]) + peer_delta;
                mbar_arrive_expect_peer(bar, 4u * kPart);
#pragma unroll
                for (uint32_t part = 0; part < 2u; ++part) {
                    const uint32_t k_at = smem_addr(k_tile) + 4096u * slot + 2048u * part, v_at = smem_addr(v_tile) + 4096u * slot + 2048u * part;
                    copy_to_peer(k_at + peer_delta, k_at, kPart, bar);
                    copy_to_peer(v_at + peer_delta, v_at, kPart, bar);
                }
            }
        }
        cur = next;
        entry = next_entry;
    }
    // a copy whose wait ran out gets one more bounded chance to land before the CTA's shared memory is given back
    if (failed) mbar_wait(bar, copy_phase & 1u, p.wait_polls);
    if (kCluster == 2 && lane == 0) {   // for leave_pair
        uint32_t *misc = reinterpret_cast<uint32_t *>(smem + kOffMisc);
        const uint32_t rounds = pair_rounds_arrived(m, kDecoders<2>);
        misc[kMiscNext + warp] = m;
        atomicMax(misc + kMiscRounds, rounds);
        max_peer(smem_addr(misc + kMiscRounds) + peer_delta, rounds);
    }
}

// ---- tensor-core work, issued by one thread ----------------------------------------------------------------------------------
// S of round r, whose tiles are there.
template <int kDim, bool kSplitQ>
__device__ __forceinline__ void issue_scores(uint8_t *smem, uint32_t tmem, uint64_t *bars, uint32_t r) {
    fence_async_smem();
    tc_fence_after();
    const uint32_t k_tile = smem_addr(smem + kOffTiles + (r & 1u) * 2u * kTileBytes), s_to = tmem + kColS + 128u * (r & 1u);
#pragma unroll
    for (uint32_t s = 0; s < kDim / 16; ++s) umma(s_to, tmem + kColQ + 8u * s, k_desc(k_tile, s), s, kIdescS);
    if constexpr (kSplitQ) {
#pragma unroll
        for (uint32_t s = 0; s < kDim / 16; ++s) umma(s_to, tmem + kColQResidue + 8u * s, k_desc(k_tile, s), 1u, kIdescS);
    }
    umma_commit(bars + kBarS + (r & 1u));
}
// O (+)= P V of round r, whose weights are stored.
template <int kDim, int kCluster>
__device__ __forceinline__ void issue_output(uint8_t *smem, uint32_t tmem, uint64_t *bars, uint32_t r, bool first) {
    tc_fence_after();
    const uint32_t v_tile = smem_addr(smem + kOffTiles + (r & 1u) * 2u * kTileBytes + kTileBytes), p_from = tmem + kColS + 128u * (r & 1u);
#pragma unroll
    for (uint32_t s = 0; s < 8; ++s) umma(tmem + kColO, p_from + 8u * s, v_desc(v_tile, s), first && !s ? 0u : 1u, kIdescO<kDim>);
#pragma unroll
    for (uint32_t s = 0; s < 8; ++s) umma(tmem + kColO, p_from + 64u + 8u * s, v_desc(v_tile, s), 1u, kIdescO<kDim>);
    if constexpr (kCluster == 1) umma_commit(bars + kBarFree + (r & 3u));   // the decoders may refill this pair of tiles
    else umma_commit_pair(bars + kBarFree + (r & 3u));
    umma_commit(bars + kBarO + (r & 1u));
}
// The issuing thread of a pair's CTA (warp 11). Issuing a product takes some 70 clocks whatever its size, 24 to 32 of them a round
// (1700 to 2200 clocks): in the softmax group they are part of its serial chain, here they run beside it. Whichever comes first,
// the tiles of the next round or the weights of the last: O frees its tiles for the decoders, S is what the softmax warps wait
// for. S of a round two ahead would land on weights that are still to be read.
template <int kDim, bool kSplitQ, int kCluster>
__device__ __forceinline__ void issuer_role(const AttentionParams &p, uint8_t *smem, uint32_t tmem) {
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kOffBars);
    const uint32_t *round_desc = reinterpret_cast<const uint32_t *>(smem + kOffRound);
    bool ok = true, stop = false;
    uint32_t units = 0, s_round = 0, o_round = 0;   // units begun; the next round whose S, whose O, is due
    uint32_t fresh = 0;                             // bit: the round (by parity) is its unit's first
    for (uint32_t polls = 0; ok && !(stop && o_round == s_round);) {
        if (!stop && s_round < o_round + 2u && mbar_test_pair(bars + kBarFull + (s_round & 1u), (s_round >> 1) & 1u)) {
            const uint32_t pair = s_round & 1u;
            polls = 0;
            if (round_desc[4 * pair] == kStopUnit) {
                stop = true;
                mbar_arrive(bars + kBarS + pair);   // the softmax warps read the stop mark
                continue;
            }
            const bool first = (round_desc[4 * pair + 1] & kFirstRound) != 0u;
            fresh = first ? fresh | 1u << pair : fresh & ~(1u << pair);
            if (first) ok = mbar_wait(bars + kBarQ, units++ & 1u, p.wait_polls);   // the unit's queries are in tensor memory
            if (ok) issue_scores<kDim, kSplitQ>(smem, tmem, bars, s_round++);
        } else if (o_round < s_round && mbar_test_pair(bars + kBarP + weights_barrier(o_round).index, weights_barrier(o_round).parity)) {
            polls = 0;
            issue_output<kDim, kCluster>(smem, tmem, bars, o_round, (fresh >> (o_round & 1u) & 1u) != 0u);
            ++o_round;
        } else if (++polls / 16u >= p.wait_polls) {   // these polls do not suspend the thread
            ok = false;
        }
    }
    if (!ok) {
        raise_status(p, CF_B200_DEVSTAT_WAIT_EXPIRED);
        uint32_t *gave_up = reinterpret_cast<uint32_t *>(smem + kOffMisc) + kMiscGaveUp;
        *gave_up = 1u;
        store_peer(peer_address(smem_addr(gave_up), cluster_rank() ^ 1u), 1u);
    }
    // What the other CTA of the pair still signals here has to land before this one leaves; leaving early, the last product of
    // this one as well. Bounded, whatever happened.
    for (uint32_t r = o_round < 2u ? 0u : o_round - 2u; ok && r < o_round; ++r) mbar_wait_pair(bars + kBarFree + (r & 3u), (r >> 2) & 1u, p.wait_polls);
    if (!ok && o_round) mbar_wait(bars + kBarO + ((o_round - 1u) & 1u), ((o_round - 1u) >> 1) & 1u, p.wait_polls);
}

// ---- softmax group: warps 12..19; in a CTA on its own its thread 0 also issues the tensor-core work -------------------------------------------------------------------------------------------
// kSplitQ: the queries are fp32; a row goes to tensor memory as binary16(q) and as binary16(q - binary16(q)), and S is the
// sum of two products, which equals the fp32-query product to 2^-22 relative.
//
// S of the next round goes out in the middle of a round, if its tiles are there, into the other half of the score columns: its
// result is then ready when the round's weights have been stored. (Issued when the round's turn came, the chain S -> softmax -> O
// was serial and alone took 80 % of the kernel: 492 of 618 us with the page decoders switched off.) Products issued by
// one thread run in order, so S may overwrite the weights of the round before once their O has been issued.
template <int kDim, bool kSplitQ, int kCluster>
__device__ __forceinline__ void softmax_role(const AttentionParams &p, uint8_t *smem, PlanHeader *hdr, uint32_t tmem, uint32_t warp,
                                             uint32_t lane, uint32_t tile_groups, const SharedSplit &split) {
    constexpr uint32_t kHalfDim = kDim / 2;   // channels of a thread
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kOffBars);
    uint64_t *bar_full = bars + kBarFull, *bar_s = bars + kBarS, *bar_o = bars + kBarO;
    const uint32_t worker = blockIdx.x / kCluster, rank = kCluster == 1 ? 0u : cluster_rank();
    const uint32_t *round_desc = reinterpret_cast<const uint32_t *>(smem + kOffRound);
    const uint32_t shared_pages = hdr->shared_pages;
    const uint32_t G = p.group, rows_total = p.seq_count * G;
    // Thread (warp w, lane) owns row 32 (w & 3) + lane — its warp's quarter of the tensor-memory lanes — and the 64 score
    // columns (4 pages) of half (w - 12) >> 2; the two threads of a row meet through row_max[], their warps at a barrier of
    // their own.
    const uint32_t half = (warp - kDecodeWarps) >> 2, row_in_tile = (warp & 3u) * 32u + lane, pair_barrier = 2u + (warp & 3u);
    const uint32_t tmem_row = tmem + (((warp & 3u) * 32u) << 16);
    constexpr bool kIssuerWarp = kCluster == 2;
    const bool issuer = !kIssuerWarp && warp == kDecodeWarps && lane == 0;

    bool failed = false;   // warp-uniform
    auto wait = [&](uint64_t *bar, uint32_t parity) {
        if (!failed && !__all_sync(0xffffffffu, mbar_wait(bar, parity, p.wait_polls))) {
            failed = true;
            if (lane == 0) raise_status(p, CF_B200_DEVSTAT_WAIT_EXPIRED);
        }
    };
    // Q rows of a unit: global memory -> tensor memory (binary16 pairs)
    auto load_queries = [&](const UnitShape &u) {
        const uint32_t row = (u.tile_index * kCluster + rank) * 128u + row_in_tile, r = min(row, rows_total - 1u);
        const uint64_t first = (static_cast<uint64_t>(r / G) * p.query_head_count + u.kv_head * G + r % G) * kDim + kHalfDim * half;
        const uint32_t column = kHalfDim / 2u * half;
        if constexpr (kSplitQ) {
            const float4 *src = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(p.queries) + first);
#pragma unroll
            for (uint32_t c = 0; c < kHalfDim / 16; ++c) {   // 16 channels = 8 columns of pairs at a time
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float4 x = src[4 * c + j];
                    if (row >= rows_total) x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    const __half2 h0 = __floats2half2_rn(x.x, x.y), h1 = __floats2half2_rn(x.z, x.w);
                    const float2 b0 = __half22float2(h0), b1 = __half22float2(h1);
                    const __half2 l0 = __floats2half2_rn(x.x - b0.x, x.y - b0.y), l1 = __floats2half2_rn(x.z - b1.x, x.w - b1.y);
                    hi[2 * j] = *reinterpret_cast<const uint32_t *>(&h0);
                    hi[2 * j + 1] = *reinterpret_cast<const uint32_t *>(&h1);
                    lo[2 * j] = *reinterpret_cast<const uint32_t *>(&l0);
                    lo[2 * j + 1] = *reinterpret_cast<const uint32_t *>(&l1);
                }
                tmem_store8(tmem_row + kColQ + column + 8u * c, hi);
                tmem_store8(tmem_row + kColQResidue + column + 8u * c, lo);
            }
        } else {
            const uint4 *src = reinterpret_cast<const uint4 *>(reinterpret_cast<const __half *>(p.queries) + first);
#pragma unroll
            for (uint32_t c = 0; c < kHalfDim / 16; ++c) {
                uint4 a = src[2 * c], b = src[2 * c + 1];
                if (row >= rows_total) a = b = make_uint4(0u, 0u, 0u, 0u);
                const uint32_t q_raw[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                tmem_store8(tmem_row + kColQ + column + 8u * c, q_raw);
            }
        }
        tmem_store_wait();
        tc_fence_before();
        if constexpr (kIssuerWarp) {
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + kBarQ);
        }
    };
    auto issue_s = [&](uint32_t r) { issue_scores<kDim, kSplitQ>(smem, tmem, bars, r); };   // issuer only
    uint32_t rounds = 0;    // whose O has been issued
    uint32_t s_round = 0;   // issuer: the next round whose S is due
    // Issuer only: S of round r ahead of its turn, unless its tiles are not there yet or its queries are another unit's.
    auto issue_s_early = [&](uint32_t r) {
        if (s_round != r || !mbar_test_pair(&bar_full[r & 1u], (r >> 1) & 1u)) return;
        if (round_desc[4 * (r & 1u)] == kStopUnit || (round_desc[4 * (r & 1u) + 1] & kFirstRound)) return;
        issue_s(r);
        s_round = r + 1u;
    };

    UnitShape u = unit_shape(p, split, worker, 0u, tile_groups, shared_pages);
    if (u.valid) load_queries(u);
    if constexpr (!kIssuerWarp) group_any<kSoftmaxWarps * 32>(1u, false);
    float m_run = -CUDART_INF_F, l_run = 0.0f;   // the row's running maximum; this thread's half of its running sum
    float v_unit = 0.0f;                          // largest V scale met so far in the unit: the unit of O
    int32_t seen = 0;   // tokens from the round's first on that the row's query token sees (16 per page and more: all of it)
    auto seen_of = [&](uint32_t pg, uint32_t count) {   // of page pg of the round, which holds `count`
        const int32_t left = seen - 16 * static_cast<int32_t>(pg);
        return left >= 16 ? count : min(count, static_cast<uint32_t>(max(left, 0)));
    };
    const bool descending = p.softmax_scale < 0.0f;   // the largest score then comes from the smallest product

    for (uint32_t it = 0;; ++it) {
        const uint32_t pair = it & 1u;
        const float *meta = reinterpret_cast<const float *>(smem + kOffMeta) + pair * 4u * kRoundPages;
        float *row_max = reinterpret_cast<float *>(smem + kOffRowMax) + 256u * pair;
        const uint32_t s_cols = tmem_row + kColS + 128u * pair;   // scores, then weights [0, 64) and their residues [64, 128)
        if constexpr (!kIssuerWarp) {
            if (issuer && s_round == it) {   // one thread polls, the others sleep at the barrier
                if (!failed && !mbar_wait_pair(&bar_full[pair], (it >> 1) & 1u, p.wait_polls)) {
                    failed = true;
                    raise_status(p, CF_B200_DEVSTAT_WAIT_EXPIRED);
                }
                if (!failed && round_desc[4 * pair] != kStopUnit) issue_s(it);
                s_round = it + 1u;
            }
            failed = __any_sync(0xffffffffu, failed);
            if (group_any<kSoftmaxWarps * 32>(1u, failed) || round_desc[4 * pair] == kStopUnit) break;
        }
        wait(&bar_s[pair], (it >> 1) & 1u);
        tc_fence_after();
        const uint32_t unit = round_desc[4 * pair], flags = round_desc[4 * pair + 1];
        const bool stop = failed || unit == kStopUnit;
        uint32_t s_raw[2][32];
        if (!stop) {
            tmem_load32(s_cols + 64u * half, s_raw[0]);
            tmem_load32(s_cols + 64u * half + 32u, s_raw[1]);
            if (flags & kFirstRound) {
                m_run = -CUDART_INF_F;
                l_run = 0.0f;
                v_unit = 0.0f;
                // entries of one sequence see its pages up to their own position; entries of several see every shared page
                const uint32_t row = min((u.tile_index * kCluster + rank) * 128u + row_in_tile, rows_total - 1u);
                // (a position may be anything up to 2^32 - 1; pages end below 2^30 tokens)
                seen = p.one_slot ? static_cast<int32_t>(min(__ldcg(&seq_info(p)[row / G].qpos), 0x3fffffffu)) + 1 - static_cast<int32_t>(16u * u.page_begin)
                                  : 0x40000000;
            }
            tmem_load_wait();
            // maximum of the scaled, masked scores of this thread's 4 pages; the raw scores stay in the registers
            float part_max = -CUDART_INF_F;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t pg = 4u * half + q;
                const uint32_t count = seen_of(pg, __float_as_uint(meta[4 * pg + 2]));
                const float ks = meta[4 * pg];
                if (count == 16u && !descending) {   // a full page (the usual case): the scale is applied to the extreme, not to every score
                    const uint32_t *sc = &s_raw[q >> 1][16 * (q & 1)];
                    float a = max3(sc[0], sc[1], sc[2]), b = max3(sc[3], sc[4], sc[5]);
#pragma unroll
                    for (int j = 6; j < 14; j += 4) {
                        a = max3(__float_as_uint(a), sc[j], sc[j + 1]);
                        b = max3(__float_as_uint(b), sc[j + 2], sc[j + 3]);
                    }
                    a = max3(__float_as_uint(a), sc[14], sc[15]);
                    part_max = fmaxf(part_max, fmaxf(a, b) * ks);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (static_cast<uint32_t>(j) < count)
                            part_max = fmaxf(part_max, __uint_as_float(s_raw[q >> 1][16 * (q & 1) + j]) * ks);
                }
            }
            row_max[half * 128u + row_in_tile] = part_max;
        }
        tc_fence_before();   // both threads of a row have read their scores: the weights may overwrite them
        if (group_any<64>(pair_barrier, kIssuerWarp && failed) || (kIssuerWarp && stop)) break;
        tc_fence_after();
        if (issuer && !failed) issue_s_early(it + 1u);

        float round_scale = 0.0f;   // largest V scale among the round's present pages
#pragma unroll
        for (uint32_t pg = 0; pg < kRoundPages; ++pg)
            if (__float_as_uint(meta[4 * pg + 2]) != 0u) round_scale = fmaxf(round_scale, meta[4 * pg + 1]);
        // With the lag O is rescaled on few rounds (every second one of the first hundred met a higher maximum in one of a warp's 32
        // rows: 582 -> 560 us for 500 rows after 16384 tokens). The result is as close to double precision as without it (the error
        // over 351 stores and queries is 0.9994 +- 0.0009 of what it was); a maximum kept whole, for exact rescaling, was 0.6 % worse.
        float m_new = fmaxf(m_run, fmaxf(row_max[row_in_tile], row_max[128u + row_in_tile]));
        if (m_new - m_run < kMaxLag) m_new = m_run;
        const float z = m_new == -CUDART_INF_F ? 0.0f : m_new;
        const float alpha = fast_exp2(m_run - z);   // m_run = -inf gives 0
        m_run = m_new;
        // The unit of O is the largest V scale met so far in the unit, so that a page's scale relative to it (which
        // rides on the binary16 weights) never exceeds 1; when a round brings a larger one, O changes unit with it.
        float o_scale = alpha;
        if (round_scale > v_unit) {
            o_scale *= v_unit / round_scale;   // v_unit = 0: nothing accumulated yet
            v_unit = round_scale;
        }
        // weights as binary16 plus their rounding residue (two A operands), so that P V is accurate to fp32 level
        // whatever the spread of the V scales
        float2 sums = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t pg = 4u * half + q;
            const uint32_t count = seen_of(pg, __float_as_uint(meta[4 * pg + 2]));
            const float ks = meta[4 * pg];
            // the weights (at most 2^kMaxLag) also carry 2^15, exactly, which O sheds at the unit's end: binary16 then resolves
            // weights down to 2^-40 of the row maximum instead of 2^-25
            const float ratio = count ? __fdividef(meta[4 * pg + 1], v_unit) * kWeightScale : 0.0f;
            uint32_t hi[8], lo[8];
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
                const float2 x = fma2(make_float2(__uint_as_float(s_raw[q >> 1][16 * (q & 1) + j]), __uint_as_float(s_raw[q >> 1][16 * (q & 1) + j + 1])),
                                      make_float2(ks, ks), make_float2(-z, -z));
                float2 w = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                if (count != 16u) {   // tokens past the page's count, or past the row's position, weigh nothing
                    w.x = static_cast<uint32_t>(j) < count ? w.x : 0.0f;
                    w.y = static_cast<uint32_t>(j + 1) < count ? w.y : 0.0f;
                }
                sums = add2(sums, w);
                const float2 scaled = mul2(w, make_float2(ratio, ratio));
                const __half2 h = __floats2half2_rn(scaled.x, scaled.y);
                const float2 rest = fma2(__half22float2(h), make_float2(-1.0f, -1.0f), scaled);   // exact
                const __half2 l = __floats2half2_rn(rest.x, rest.y);
                hi[j >> 1] = *reinterpret_cast<const uint32_t *>(&h);
                lo[j >> 1] = *reinterpret_cast<const uint32_t *>(&l);
            }
            tmem_store8(s_cols + 8u * pg, hi);          // 16 tokens = 8 columns of pairs
            tmem_store8(s_cols + 64u + 8u * pg, lo);
        }
        l_run = l_run * alpha + (sums.x + sums.y);   // this thread's half of the row's sum; the halves are added at the unit's end
        // O in tensor memory follows the new maximum and unit (this thread's channels), once the previous round's product has
        // reached it; skipped when no row of the warp moved
        if (!(flags & kFirstRound) && !__all_sync(0xffffffffu, o_scale == 1.0f)) {
            wait(&bar_o[pair ^ 1u], ((it - 1u) >> 1) & 1u);
            tc_fence_after();
            if (!failed) {
#pragma unroll 1
                for (uint32_t c0 = 0; c0 < kHalfDim; c0 += 32u) {
                    uint32_t o_raw[32];
                    tmem_load32(tmem_row + kColO + kHalfDim * half + c0, o_raw);
                    tmem_load_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) o_raw[j] = __float_as_uint(__uint_as_float(o_raw[j]) * o_scale);
                    tmem_store32(tmem_row + kColO + kHalfDim * half + c0, o_raw);
                }
            }
        }
        tmem_store_wait();
        tc_fence_before();
        if constexpr (kIssuerWarp) {
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + kBarP + weights_barrier(it).index);
        } else {
            if (group_any<kSoftmaxWarps * 32>(1u, failed)) break;
            if (issuer) {
                issue_output<kDim, kCluster>(smem, tmem, bars, it, (flags & kFirstRound) != 0u);
                issue_s_early(it + 1u);
            }
            __syncwarp();
        }
        rounds = it + 1u;
        if (p.one_slot) seen -= 16 * static_cast<int32_t>(kRoundPages);

        // ---- last round of the unit: one (max, sum, weighted[kDim]) per row; each thread writes its channels ----
        if (flags & kLastRound) {
            const UnitShape done = u;
            u = unit_shape(p, split, worker, unit + 1u, tile_groups, shared_pages);
            if (u.valid) load_queries(u);   // this unit's last scores have been read: its queries may go
            wait(&bar_o[pair], (it >> 1) & 1u);
            tc_fence_after();
            // the two halves of the row's sum take the places of the maxima: O of this round is complete, so every warp has stored
            // its weights, and read the maxima before
            row_max[half * 128u + row_in_tile] = l_run;
            // for a CTA on its own the next unit's queries are stored, too
            if (kIssuerWarp ? group_any<64>(pair_barrier, failed) : group_any<kSoftmaxWarps * 32>(1u, failed)) break;
            const uint32_t row = (done.tile_index * kCluster + rank) * 128u + row_in_tile;
            const bool live = row < rows_total;   // whole warps go on: the tensor-memory loads are warp-wide
            float *dst = live ? shared_partial_ptr(p, done.chunk, row / G, done.head_local * G + row % G) : nullptr;
            const float o_unit = v_unit * (1.0f / kWeightScale);
            if (live && half == 0) {
                dst[0] = m_run;
                dst[1] = row_max[row_in_tile] + row_max[128u + row_in_tile];
            }
#pragma unroll 1
            for (uint32_t c0 = 0; c0 < kHalfDim; c0 += 32u) {
                uint32_t o_raw[32];
                tmem_load32(tmem_row + kColO + kHalfDim * half + c0, o_raw);
                tmem_load_wait();
                if (live) {
#pragma unroll
                    for (int t = 0; t < 8; ++t) {   // columns t, t + 8, t + 16, t + 24 of the 32 are 4 consecutive channels
                        float *out = dst + 2 + kHalfDim * half + c0 + 4 * t;
                        *reinterpret_cast<float2 *>(out) =
                            make_float2(__uint_as_float(o_raw[t]) * o_unit, __uint_as_float(o_raw[t + 8]) * o_unit);
                        *reinterpret_cast<float2 *>(out + 2) =
                            make_float2(__uint_as_float(o_raw[t + 16]) * o_unit, __uint_as_float(o_raw[t + 24]) * o_unit);
                    }
                }
            }
            tc_fence_before();
        }
    }
    // leaving early: give the tensor core's last commit a bounded chance to arrive before tensor memory is freed
    if (issuer && rounds && failed) mbar_wait(&bar_o[(rounds - 1u) & 1u], ((rounds - 1u) >> 1) & 1u, p.wait_polls);
}

// A CTA of a pair may leave once nothing is on its way into its shared memory or, to the other one, out of it. If both issuing threads have
// taken every round, they have seen all of it arrive. If one has not, the full barriers of the last two rounds that any decoder warp has
// arrived for tell (of the ones before, the tiles were freed): the warps that left before make up the arrivals that
// these lack, and then they complete when the pages that were sent are there.
__device__ __forceinline__ void leave_pair(const AttentionParams &p, uint8_t *smem, uint32_t warp, uint32_t lane) {
    constexpr uint32_t kWarps = kDecoders<2>;
    uint64_t *bar_full = reinterpret_cast<uint64_t *>(smem + kOffBars) + kBarFull;
    uint32_t *misc = reinterpret_cast<uint32_t *>(smem + kOffMisc);
    __syncwarp();
    cluster_sync();   // every role of both CTAs is done
    if (misc[kMiscGaveUp] == 0u) return;
    const uint32_t rounds = misc[kMiscRounds];
    if (warp < kWarps && lane == 0) {
        const uint32_t peer_delta = peer_address(smem_addr(smem), cluster_rank() ^ 1u) - smem_addr(smem);
        for (uint32_t next_slot = misc[kMiscNext + warp]; pair_round(next_slot) < rounds; next_slot += kWarps) {
            mbar_arrive(&bar_full[pair_round(next_slot) & 1u]);
            mbar_arrive_peer(smem_addr(&bar_full[pair_round(next_slot) & 1u]) + peer_delta);
        }
    } else if (warp == kWarps && lane == 0) {
        for (uint32_t r = rounds < 2u ? 0u : rounds - 2u; r < rounds; ++r) mbar_wait_pair(&bar_full[r & 1u], (r >> 1) & 1u, p.wait_polls);
    }
    __syncwarp();
    cluster_sync();
}

template <int kDim, bool kSplitQ, int kCluster>
__global__ void __launch_bounds__(kTcThreads, 1) prefix_attention_kernel(AttentionParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kOffBars);
    uint32_t *misc = reinterpret_cast<uint32_t *>(smem + kOffMisc);

    load_tables<kTcThreads>(smem, p, tid);   // the caller's: needs nothing of the plan kernel
    wait_for_previous_kernel();
    // From here on the plan is complete, so the per-sequence kernel may take over every SM this kernel leaves.
    allow_dependent_launch();
    PlanHeader *hdr = plan_header(p);
    // uniform: nothing shared, the plan refused the hint, or the split leaves this CTA without a share
    if (hdr->shared_pages == 0 || blockIdx.x / kCluster >= hdr->shared_ctas) return;   // both CTAs of a pair alike

    if (tid == 0) {
        misc[kMiscRounds] = misc[kMiscGaveUp] = 0u;
        for (uint32_t w = 0; w < kDecodeWarps; ++w) mbar_init(bars + w, 1);   // copies
        mbar_init(bars + kBarFull, kRoundPages);                    // full[0], full[1]: one arrival per page slot of the round
        mbar_init(bars + kBarFull + 1, kRoundPages);
        for (uint32_t i = 0; i < 4u; ++i) mbar_init(bars + kBarFree + i, kCluster);   // tensor-core commits, of both CTAs
        for (uint32_t i = kBarS; i < kBarP; ++i) mbar_init(bars + i, 1);          // tensor-core commits
        for (uint32_t i = kBarP; i < kBarCount; ++i) mbar_init(bars + i, kSoftmaxWarps);   // weights stored, queries stored (where a warp of its own issues)
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {   // one whole warp allocates the CTA's tensor memory and frees it at the end
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&misc[0])), "r"(kTmemColumns));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = misc[0];

    if constexpr (kCluster == 2) cluster_sync();   // the peer's barriers are set up

    const uint32_t tile_groups = shared_tile_groups(p.seq_count * p.group);
    const SharedSplit split = {hdr->shared_rounds, p.kv_head_span * tile_groups, hdr->shared_ctas};

    if (warp < kDecodeWarps) {   // whole warpgroups on either side: the register split is per warpgroup
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kDecoderRegs));
        if (warp < kDecoders<kCluster>) {
            decoder_role<kDim, kCluster>(p, smem, hdr, warp, lane, tile_groups, split);
        } else {
            if (lane == 0) issuer_role<kDim, kSplitQ, kCluster>(p, smem, tmem);
            __syncwarp();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
        softmax_role<kDim, kSplitQ, kCluster>(p, smem, hdr, tmem, warp, lane, tile_groups, split);
    }

    if constexpr (kCluster == 2) leave_pair(p, smem, warp, lane);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns));
}

}  // namespace

cudaError_t launch_prefix_attention(const AttentionParams &p, cudaStream_t stream, bool dependent) {
    static LauncherState table[64];
    cudaError_t e;
    LauncherState *state = launcher_state(table, &e);
    if (!state) return e;
    using Kernel = void (*)(AttentionParams);
    const Kernel kernels[2][2][2] = {   // [pair of CTAs][head_dim 64][fp32 queries]
        {{prefix_attention_kernel<128, false, 1>, prefix_attention_kernel<128, true, 1>},
         {prefix_attention_kernel<64, false, 1>, prefix_attention_kernel<64, true, 1>}},
        {{prefix_attention_kernel<128, false, 2>, prefix_attention_kernel<128, true, 2>},
         {prefix_attention_kernel<64, false, 2>, prefix_attention_kernel<64, true, 2>}}};
    if (!state->configured) {
        for (int i = 0; i < 8; ++i) {
            const Kernel kernel = kernels[i >> 2][i >> 1 & 1][i & 1];
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTcSmem));
            if (e != cudaSuccess) return e;
            cudaFuncAttributes attr;
            e = cudaFuncGetAttributes(&attr, kernel);
            if (e != cudaSuccess) return e;
            if ((attr.numRegs + 7) / 8 * 8 != kLaunchRegs) return cudaErrorLaunchOutOfResources;   // the register split assumes this count
        }
        state->configured = true;
    }
    const uint32_t cluster = shared_cluster(p.seq_count * p.group);
    return launch_in_clusters(cluster, kernels[cluster - 1u][p.head_dim == 64 ? 1 : 0][p.query_type == CF_B200_F32 ? 1 : 0],
                              static_cast<uint32_t>(state->sm_count) / cluster * cluster, kTcThreads, kTcSmem, stream, dependent, p);
}

}  // namespace cfb
