// sealed_attention.cu — decode-step attention over sealed pages: planning, the any-geometry kernel, the split-KV
// combine, the decode probe, and the C entry points.
//
// The arithmetic follows the reference's paged attention (src/cuda/paged_kv_attention.cu:41-176): dequantise inside
// the dot product, one online softmax over every page and the tail, output = weighted / sum. What differs is the
// execution: sequences are cut into chunks of pages, each (chunk, kv head) unit is processed independently for all
// query heads of the group at once (a K/V code is decoded once, not once per query head), and the partial
// (max, sum, weighted) triples are merged with the rule of cf_online_softmax_merge (src/runtime/kv_runtime.cpp:219-243).

#include <atomic>
#include <cstddef>
#include <math_constants.h>

#include "attention_params.cuh"

static std::atomic<unsigned long long> g_shared_prefix_launches{0};

namespace cfb {

namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kPlanThreads = 1024;
constexpr int kGenericThreads = 128;
constexpr uint32_t kGenericMaxGroup = 16;

// ---------------------------------------------------------------------------------------------------------------
// Plan: every entry's record, the line of pages and its cut (PageLine). One block.
//
// Bound by the chain of dependent loads slot -> counts -> record, once per entry, and a block scan; the kernels behind it set
// themselves up meanwhile (see launch_kernel). It used to write a record per unit of pages as well and to try 32 unit sizes:
// 5.2 us for one sequence and 9.4 us for 64, against 3.5 and 4.3 us now.
// ---------------------------------------------------------------------------------------------------------------

// Shared-prefix hint, part one: block s compares the first `shared_prefix_pages` ids of entry s's page-table row with the
// first entry's and leaves the result (1 = differs) in the entry's cell of the line-prefix array, which the plan kernel
// reads before it overwrites the array with the real prefix sums.
__global__ void __launch_bounds__(256) verify_prefix_kernel(AttentionParams p) {
    allow_dependent_launch();
    const uint32_t s = blockIdx.x;
    const uint32_t *row0 = p.page_table + static_cast<uint64_t>(slot_of(p, 0)) * p.page_table_stride;
    const uint32_t *row = p.page_table + static_cast<uint64_t>(slot_of(p, s)) * p.page_table_stride;
    int bad = 0;
    for (uint32_t pg = threadIdx.x; pg < p.shared_prefix_pages; pg += blockDim.x) bad |= row[pg] != row0[pg];
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) line_prefix(p)[s] = bad ? 1u : 0u;
}

// Inclusive sum over the block (whole warps, at most 32 of them); *total gets the block's sum.
__device__ __forceinline__ uint32_t block_scan(uint32_t value, uint32_t *warp_totals, uint32_t *total) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, warps = blockDim.x >> 5;
    uint32_t incl = value;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= static_cast<uint32_t>(o)) incl += up;
    }
    __syncthreads();   // the previous use of warp_totals is over
    if (lane == 31u) warp_totals[warp] = incl;
    __syncthreads();
    uint32_t v = lane < warps ? warp_totals[lane] : 0u;   // every warp sums the totals for itself
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= static_cast<uint32_t>(o)) v += up;
    }
    *total = __shfl_sync(0xffffffffu, v, 31);
    const uint32_t before = __shfl_sync(0xffffffffu, v, warp ? warp - 1u : 0u);
    return incl + (warp ? before : 0u);
}

__global__ void __launch_bounds__(kPlanThreads) plan_kernel(AttentionParams p) {
    __shared__ uint32_t warp_totals[kPlanThreads / 32];
    allow_dependent_launch();
    const uint32_t tid = threadIdx.x;
    const uint32_t per_thread = (p.seq_count + blockDim.x - 1) / blockDim.x;
    const uint32_t begin = min(tid * per_thread, p.seq_count);
    const uint32_t end = min(begin + per_thread, p.seq_count);
    PlanHeader *hdr = plan_header(p);
    uint32_t *prefix = line_prefix(p);
    SeqInfo *info = seq_info(p);

    // Shared prefix: taken only if every listed sequence has the pages sealed and its page-table row starts with the
    // same ids as the first sequence's (compared by verify_prefix_kernel, result per entry in prefix[]). The pages are
    // then left to the shared-prefix kernel and taken off the line.
    uint32_t shared = p.shared_prefix_pages;
    if (shared) {
        int bad = 0;
        wait_for_previous_kernel();
        for (uint32_t s = begin; s < end; ++s) {   // the pages must be sealed and wholly visible to the entry's query token
            const uint32_t slot = slot_of(p, s), sealed = p.seq_sealed_tokens[slot];
            const uint32_t qpos = query_position(p, s, sealed, p.tail_tokens ? p.tail_tokens[slot] : 0u);
            if (sealed / p.page_tokens < shared || qpos + 1u < shared * p.page_tokens || __ldcg(prefix + s) != 0u) bad = 1;
        }
        if (__syncthreads_or(bad)) {
            shared = 0;
            if (tid == 0) raise_status(p, CF_B200_DEVSTAT_PREFIX_MISMATCH);
        }
    }
    uint32_t shared_ctas = 0, shared_rounds = 0;
    if (shared) {   // an even split of the prefix's rounds over the CTAs of the shared-prefix kernel (SharedSplit)
        const uint32_t row_tiles = (p.seq_count * p.group + 127u) / 128u;
        shared_rounds = (shared + 7u) / 8u;
        shared_ctas = shared_split_ctas(shared_rounds, p.kv_head_span * row_tiles, p.sm_count, CF_B200_SHARED_CHUNKS_MAX);
        if (shared_ctas == 0u) shared = 0;   // no CTA to take it: the pages stay on the line
    }

    uint32_t local = 0;   // pages of this thread's sequences
    for (uint32_t s = begin; s < end; ++s) {
        const uint32_t slot = slot_of(p, s), row = row_of(p, s);
        const uint32_t sealed = p.seq_sealed_tokens[slot], tail = p.tail_tokens ? p.tail_tokens[slot] : 0u;
        const uint32_t qpos = query_position(p, s, sealed, tail);
        const uint32_t pages = min((sealed + p.page_tokens - 1u) / p.page_tokens, qpos / p.page_tokens + 1u);
        const uint32_t first = min(max(window_begin(qpos, p.causal_window) / p.page_tokens, shared), pages);
        reinterpret_cast<uint4 *>(info + s)[0] = make_uint4(slot, sealed, qpos, tail);
        reinterpret_cast<uint4 *>(info + s)[1] = make_uint4(first, pages, row, 0u);
        local += pages - first;
    }
    PageLine line = {};
    line.grain = 1;
    line.by_position = p.min_pages_per_unit != 0u;
    uint32_t incl, total;
    const uint32_t capacity = static_cast<uint32_t>(min(p.layout.chunk_capacity, static_cast<uint64_t>(0x7fffffffu)));
    if (!line.by_position) {
        // One stretch per resident warp for the units of a stretch (kv heads x passes), where there is a page for each and a
        // partial slot: the last slot is stretches * pieces + seq_count - 2. The capacity is at least seq_count.
        incl = block_scan(local, warp_totals, &total);
        const uint32_t room = capacity - (p.seq_count - 1u);
        line.stretches = min(min(max(p.plan_warps / p.unit_lanes, 1u), total), room);
        if (line.stretches) {
            line.base = total / line.stretches;
            line.longer = total % line.stretches;
            const uint32_t longest = line.base + (line.longer ? 1u : 0u);
            line.pieces = min(max(min((longest + kPiecePages - 1u) / kPiecePages, room / line.stretches), 1u), line.base);
        }
    } else {
        line.grain = p.min_pages_per_unit;
        for (;;) {   // units grow until every one has a slot; from one unit per sequence on they do
            local = 0;
            for (uint32_t s = begin; s < end; ++s) {
                const uint4 pages = reinterpret_cast<const uint4 *>(info + s)[1];   // this thread's own record
                local += (pages.y - pages.x + line.grain - 1u) / line.grain;
            }
            incl = block_scan(local, warp_totals, &total);
            if (total <= capacity || line.grain >= (1u << 30)) break;
            line.grain <<= 1;
        }
        line.stretches = total;
        line.base = line.pieces = 1;
    }
    line.positions = total;
    uint32_t running = incl - local;
    for (uint32_t s = begin; s < end; ++s) {
        const uint4 pages = reinterpret_cast<const uint4 *>(info + s)[1];
        prefix[s] = running;
        info[s].line_begin = running;
        running += line.grain == 1u ? pages.y - pages.x : (pages.y - pages.x + line.grain - 1u) / line.grain;
    }
    if (tid == 0) {
        prefix[p.seq_count] = total;
        hdr->line = line;
        hdr->next_unit = 0;
        hdr->shared_pages = shared;
        hdr->shared_ctas = shared_ctas;
        hdr->shared_rounds = shared_rounds;
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Query load helper.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float load_query(const AttentionParams &p, uint32_t seq, uint32_t q_head, uint32_t d) {
    const uint64_t i = (static_cast<uint64_t>(seq) * p.query_head_count + q_head) * p.head_dim + d;
    return p.query_type == CF_B200_F16 ? __half2float(reinterpret_cast<const __half *>(p.queries)[i])
                                       : reinterpret_cast<const float *>(p.queries)[i];
}

// ---------------------------------------------------------------------------------------------------------------
// Any-geometry attention kernel: one CTA per (stretch, kv head) unit. Each page record is copied to shared memory,
// both streams are decoded to symbols there (one thread per block), then scores and the online-softmax update
// are computed from shared memory. Built for coverage of every legal geometry, not for speed.
// ---------------------------------------------------------------------------------------------------------------
struct GenericSmem {
    uint32_t record_bytes, sym_bytes;
    uint32_t off_record, off_ksym, off_vsym, off_q, off_acc, off_scores, off_ml, total;
};

__host__ __device__ inline GenericSmem generic_smem(uint32_t symbols, uint32_t group, uint32_t head_dim,
                                                    uint32_t page_tokens) {
    GenericSmem s;
    s.record_bytes = 16u + 2u * align_up_u32(symbols, 16u) + 32u;
    s.sym_bytes = align_up_u32(symbols, 16u);
    s.off_record = 0;
    s.off_ksym = s.off_record + s.record_bytes;
    s.off_vsym = s.off_ksym + s.sym_bytes;
    s.off_q = s.off_vsym + s.sym_bytes;
    s.off_acc = s.off_q + group * head_dim * 4u;
    s.off_scores = s.off_acc + group * head_dim * 4u;
    s.off_ml = s.off_scores + group * page_tokens * 4u;
    s.total = s.off_ml + group * 8u + 16u;
    return s;
}

__global__ void __launch_bounds__(kGenericThreads) generic_attention_kernel(AttentionParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint32_t s_unit;
    const GenericSmem lay = generic_smem(p.symbols, p.group, p.head_dim, p.page_tokens);
    uint8_t *record = smem + lay.off_record;
    uint8_t *ksym = smem + lay.off_ksym;
    uint8_t *vsym = smem + lay.off_vsym;
    float *q = reinterpret_cast<float *>(smem + lay.off_q);
    float *acc = reinterpret_cast<float *>(smem + lay.off_acc);
    float *scores = reinterpret_cast<float *>(smem + lay.off_scores);
    float *ml = reinterpret_cast<float *>(smem + lay.off_ml);  // [group][2]: running max, running sum

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t D = p.head_dim, T = p.page_tokens, G = p.group;
    PlanHeader *hdr = plan_header(p);
    const PageLine line = plan_line(p);
    const uint32_t unit_count = line.stretches * p.kv_head_span;
    const uint32_t max_part_units = align_up_u32(p.symbols, 16u) / 16u;

    for (;;) {
        __syncthreads();
        if (tid == 0) s_unit = atomicAdd(&hdr->next_unit, 1u);
        __syncthreads();
        const uint32_t unit = s_unit;
        if (unit >= unit_count) break;
        const uint32_t stretch = unit / p.kv_head_span;
        const uint32_t head_local = unit % p.kv_head_span;
        const uint32_t kv_head = p.kv_head_begin + head_local;
        for (uint32_t x = line.begin(stretch), x_end = line.begin(stretch + 1u); x < x_end;) {
        const uint32_t piece = line.piece_of(stretch, x);
        const LineRun run = run_at(p, x, min(line.piece_end(stretch, piece), x_end), line.grain, lane);
        const uint32_t seq = run.seq, slot = run.info.slot, sealed = run.info.sealed, qpos = run.info.qpos;
        const uint32_t first_token = window_begin(qpos, p.causal_window);
        const uint32_t page_begin = run.page, page_end = run.page_end;
        x = run.x_end;
        __syncthreads();   // the previous run's results are written

        for (uint32_t i = tid; i < G * D; i += kGenericThreads) {
            q[i] = load_query(p, run.info.row, kv_head * G + i / D, i % D) * (p.softmax_scale * kLog2e);
            acc[i] = 0.0f;
        }
        if (tid < G) {
            ml[2 * tid] = -CUDART_INF_F;
            ml[2 * tid + 1] = 0.0f;
        }

        for (uint32_t page = page_begin; page < page_end; ++page) {
            __syncthreads();
            const uint32_t page_id = p.page_table[static_cast<uint64_t>(slot) * p.page_table_stride + page];
            const uint64_t entry = p.page_dir[static_cast<uint64_t>(page_id) * p.kv_head_count + kv_head];
            const uint32_t units = static_cast<uint32_t>(CF_B200_DIR_LENGTH_UNITS(entry));
            if (units == 0 || units > 1u + 2u * max_part_units) {
                if (tid == 0) raise_status(p, CF_B200_DEVSTAT_BAD_RECORD);
                continue;
            }
            const uint4 *src = reinterpret_cast<const uint4 *>(p.arena + 16ull * CF_B200_DIR_OFFSET_UNITS(entry));
            for (uint32_t i = tid; i < units; i += kGenericThreads) reinterpret_cast<uint4 *>(record)[i] = src[i];
            __syncthreads();
            const cf_b200_record_header h = *reinterpret_cast<const cf_b200_record_header *>(record);
            if (h.version != CF_B200_FORMAT_VERSION || h.codebook_id != p.codebook_id ||
                1u + h.k_part_units + h.v_part_units != units || h.k_part_units > max_part_units ||
                h.v_part_units > max_part_units || h.token_count == 0 || h.token_count > T || h.k_coder > CF_B200_CODER_MAX ||
                h.v_coder > CF_B200_CODER_MAX) {
                if (tid == 0) raise_status(p, CF_B200_DEVSTAT_BAD_RECORD);
                continue;
            }
            const uint8_t *k_part = record + 16;
            const uint8_t *v_part = record + 16 + 16u * h.k_part_units;
            const uint32_t k_bytes = 16u * h.k_part_units, v_bytes = 16u * h.v_part_units;
            int bad_table = 0;
            for (uint32_t b = tid; b < 2u * p.nblocks; b += kGenericThreads)
                bad_table |= b < p.nblocks ? !part_block_start_ok(k_part, k_bytes, h.k_coder, p.nblocks, b, p.symbols)
                                           : !part_block_start_ok(v_part, v_bytes, h.v_coder, p.nblocks, b - p.nblocks, p.symbols);
            if (__syncthreads_or(bad_table)) {   // a block starts outside its part
                if (tid == 0) raise_status(p, CF_B200_DEVSTAT_BAD_RECORD);
                continue;
            }
            for (uint32_t b = tid; b < 2u * p.nblocks; b += kGenericThreads) {
                if (b < p.nblocks) {
                    uint8_t *dst = ksym + b * p.block_size;
                    decode_part_block(k_part, k_bytes, h.k_coder, p.nblocks, b, p.block_size, p.symbols, p.k_tables,
                                      [&](int j, uint32_t s) { dst[j] = static_cast<uint8_t>(s); });
                } else {
                    const uint32_t vb = b - p.nblocks;
                    uint8_t *dst = vsym + vb * p.block_size;
                    decode_part_block(v_part, v_bytes, h.v_coder, p.nblocks, vb, p.block_size, p.symbols, p.v_tables,
                                      [&](int j, uint32_t s) { dst[j] = static_cast<uint8_t>(s); });
                }
            }
            __syncthreads();
            const float k_scale = __half2float(__ushort_as_half(h.k_scale_f16));
            const float v_scale = __half2float(__ushort_as_half(h.v_scale_f16));
            // scores[g][t], one warp per (g, t)
            for (uint32_t pair = warp; pair < G * T; pair += kGenericThreads / 32) {
                const uint32_t g = pair / T, t = pair % T;
                const uint32_t token = page * T + t;
                float s = -CUDART_INF_F;
                if (t < h.token_count && token >= first_token && token < sealed && token <= qpos) {
                    float dot = 0.0f;
                    for (uint32_t d = lane; d < D; d += 32)
                        dot += q[g * D + d] * static_cast<float>(static_cast<int>(ksym[t * D + d]) - kZero);
                    s = warp_sum(dot) * k_scale;
                }
                if (lane == 0) scores[g * T + t] = s;
            }
            __syncthreads();
            // online softmax update: thread d owns channel d of every group member
            float new_m[kGenericMaxGroup], new_l[kGenericMaxGroup];
            for (uint32_t g = 0; g < G; ++g) {
                const float m_old = ml[2 * g], l_old = ml[2 * g + 1];
                float pm = -CUDART_INF_F;
                for (uint32_t t = 0; t < T; ++t) pm = fmaxf(pm, scores[g * T + t]);
                const float m_new = fmaxf(m_old, pm);
                new_m[g] = m_new;
                new_l[g] = l_old;
                if (m_new == -CUDART_INF_F) continue;
                const float alpha = m_old == -CUDART_INF_F ? 0.0f : exp2f(m_old - m_new);
                float lsum = 0.0f, a = 0.0f;
                for (uint32_t t = 0; t < T; ++t) {
                    const float s = scores[g * T + t];
                    const float w = s == -CUDART_INF_F ? 0.0f : exp2f(s - m_new);
                    lsum += w;
                    if (tid < D) a += w * static_cast<float>(static_cast<int>(vsym[tid * T + t]) - kZero);
                }
                new_l[g] = l_old * alpha + lsum;
                if (tid < D) acc[g * D + tid] = acc[g * D + tid] * alpha + a * v_scale;
            }
            __syncthreads();
            if (tid == 0) {
                for (uint32_t g = 0; g < G; ++g) {
                    ml[2 * g] = new_m[g];
                    ml[2 * g + 1] = new_l[g];
                }
            }
        }
        __syncthreads();
        for (uint32_t i = tid; i < G * D; i += kGenericThreads) {
            const uint32_t g = i / D, d = i % D;
            float *dst = partial_ptr(p, line.slot(stretch, piece, run.x, seq), head_local * G + g);
            dst[2 + d] = acc[i];
            if (d == 0) {
                dst[0] = ml[2 * g];
                dst[1] = ml[2 * g + 1];
            }
        }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Combine: merge the partials of every (entry, query head) row with the unsealed tail and write the output.
//
// A CTA serves R rows: the query heads of one kv head, for one entry or, in multi-query calls, for several entries of one
// slot. The tail's K and V rows are then read once per CTA instead of once per row (at 500 rows over a tail of up to 127
// tokens those reads were all of the 274 us this stage took). A launch with too few rows for that, one or a few
// sequences, gives each row a CTA of its own (R = 1), whose warps share out the row's partials.
//
// Every sum has an order of its own that the shape of the CTA does not change, so that a row's result depends on nothing
// but the row: partials are added up in 32 consecutive strands and the strands in order, tail tokens in eight interleaved
// strands.
// ---------------------------------------------------------------------------------------------------------------
constexpr uint32_t kStrands = 32;

// Sums of V values over the warp, V a power of two up to 32: lane l gets the sum of value l / (32 / V).
template <int V>
__device__ __forceinline__ float sum_many(float (&v)[V], uint32_t lane) {
    int o = 16;
#pragma unroll
    for (int h = V / 2; h >= 1; h /= 2) {
        const bool upper = (lane & static_cast<uint32_t>(o)) != 0u;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float sent = upper ? v[i] : v[i + h], kept = upper ? v[i + h] : v[i];
            v[i] = kept + __shfl_xor_sync(0xffffffffu, sent, o);
        }
        o >>= 1;
    }
#pragma unroll
    for (int rest = V; rest < 32; rest *= 2) {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        o >>= 1;
    }
    return v[0];
}

template <int R, int kThreads>
struct CombineSmem {   // offsets in floats
    static constexpr int kGroups = kThreads / 128;          // thread groups of one thread per channel
    static constexpr int kRowStride = R == 1 ? 1 : R + 4;   // of a tail token's weights: 16-byte aligned, banks spread
    static constexpr int kQ = 0;                            // [R][128]
    static constexpr int kTail = kQ + R * 128;              // [groups (2 for one group)][R][128] sums of weighted V rows
    static constexpr int kTailGroups = kGroups < 2 ? 2 : kGroups;
    static constexpr int kStrand = kTail + kTailGroups * R * 128;   // R = 1: [strand][128]
    static constexpr int kWeights = kStrand + (R == 1 ? static_cast<int>(kStrands) * 128 : 0);   // [tail_capacity][kRowStride]
    static size_t bytes(uint32_t tail_capacity) { return (kWeights + static_cast<size_t>(tail_capacity) * kRowStride) * 4u; }
};

template <int R, int kThreads>
__global__ void __launch_bounds__(kThreads) combine_kernel(AttentionParams p, uint32_t cta_entries, uint32_t cta_heads) {
    using S = CombineSmem<R, kThreads>;
    constexpr int kWarps = kThreads / 32, kGroups = S::kGroups, kGroupStrands = 8 / kGroups;
    extern __shared__ __align__(16) float smem_f[];
    float *q = smem_f + S::kQ, *tail_acc = smem_f + S::kTail, *weights = smem_f + S::kWeights;
    __shared__ uint32_t e_slot[R], e_sealed[R], e_qpos[R], e_tail[R], e_row[R];
    __shared__ float tail_m[R], tail_l[R];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t G = p.group, D = p.head_dim, C = p.tail_capacity;   // C: rows per (slot, kv head) in the tails
    const uint32_t entry0 = blockIdx.x * cta_entries, entries = min(cta_entries, p.seq_count - entry0);
    const uint32_t head0 = blockIdx.y * cta_heads, rows = entries * cta_heads;   // local query heads; row = entry * heads + head
    const uint32_t kv_head = p.kv_head_begin + head0 / G;
    auto q_head_of = [&](uint32_t r) { return p.kv_head_begin * G + head0 + r % cta_heads; };

    if (tid < entries) {
        const uint32_t seq = entry0 + tid, slot = slot_of(p, seq), row = row_of(p, seq);
        const uint32_t sealed = p.seq_sealed_tokens[slot], tail = p.tail_tokens ? p.tail_tokens[slot] : 0u;
        e_slot[tid] = slot;
        e_sealed[tid] = sealed;
        e_qpos[tid] = query_position(p, seq, sealed, tail);
        e_tail[tid] = min(tail, C);
        e_row[tid] = row;
    }
    __syncthreads();
    uint32_t any_tail = 0;
    for (uint32_t e = 0; e < entries; ++e) any_tail |= e_tail[e];

    if (any_tail) {
        for (uint32_t i = tid; i < R * 128u; i += kThreads) {
            const uint32_t r = i >> 7, d = i & 127u;
            q[i] = r < rows && d < D ? load_query(p, e_row[r / cta_heads], q_head_of(r), d) : 0.0f;
        }
        __syncthreads();
        // Scores. Consecutive entries of one slot share the pass over its rows: two tokens per warp at a time, four channels
        // per lane, the sums of all rows reduced together.
        for (uint32_t e0 = 0, e1; e0 < entries; e0 = e1) {
            for (e1 = e0 + 1u; e1 < entries && e_slot[e1] == e_slot[e0]; ++e1) {}
            const uint32_t tail = e_tail[e0], sealed = e_sealed[e0];
            const uint64_t base = (static_cast<uint64_t>(e_slot[e0]) * p.kv_head_count + kv_head) * C;
            for (uint32_t t0 = 2u * warp; t0 < tail; t0 += 2u * kWarps) {
                float k0[4], k1[4], sums[2 * R];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint32_t d = lane + 32u * j;
                    k0[j] = d < D ? load_tail(p.tail_k, p.tail_type, (base + t0) * D + d) : 0.0f;
                    k1[j] = d < D && t0 + 1u < tail ? load_tail(p.tail_k, p.tail_type, (base + t0 + 1u) * D + d) : 0.0f;
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    float a = 0.0f, b = 0.0f;
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        const float qv = q[r * 128 + lane + 32u * j];
                        a = fmaf(qv, k0[j], a);
                        b = fmaf(qv, k1[j], b);
                    }
                    sums[r] = a;
                    sums[R + r] = b;
                }
                const float sum = sum_many<2 * R>(sums, lane);
                const uint32_t value = lane / (16u / R), r = value % R, t = t0 + value / R;
                if (lane % (16u / R) == 0u && t < tail && r < rows && r / cta_heads >= e0 && r / cta_heads < e1) {
                    const uint32_t qpos = e_qpos[r / cta_heads], token = sealed + t;
                    const bool visible = token >= window_begin(qpos, p.causal_window) && token <= qpos;
                    weights[t * S::kRowStride + r] = visible ? sum * p.softmax_scale * kLog2e : -CUDART_INF_F;
                }
            }
        }
        __syncthreads();
        // softmax of every row over its tail: scores become weights relative to the row's largest
        for (uint32_t r = warp; r < R; r += kWarps) {
            const uint32_t tail = r < rows ? e_tail[r / cta_heads] : 0u;
            float m = -CUDART_INF_F, l = 0.0f;
            for (uint32_t t = lane; t < tail; t += 32u) m = fmaxf(m, weights[t * S::kRowStride + r]);
            m = warp_max(m);
            for (uint32_t t = lane; t < tail; t += 32u) {
                const float s = weights[t * S::kRowStride + r], w = s == -CUDART_INF_F ? 0.0f : exp2f(s - m);
                weights[t * S::kRowStride + r] = w;
                l += w;
            }
            l = warp_sum(l);
            if (lane == 0) {
                tail_m[r] = m;
                tail_l[r] = l;
            }
        }
        __syncthreads();
        // weighted V rows: a thread per channel, thread group g takes the token strands g, g + groups, ... of eight
        const uint32_t d = tid & 127u, grp = tid >> 7;
        float acc[kGroupStrands][R];
#pragma unroll
        for (int k = 0; k < kGroupStrands; ++k)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[k][r] = 0.0f;
        for (uint32_t e0 = 0, e1; e0 < entries; e0 = e1) {
            for (e1 = e0 + 1u; e1 < entries && e_slot[e1] == e_slot[e0]; ++e1) {}
            const uint32_t tail = e_tail[e0];
            const bool whole = e0 == 0u && e1 == entries;   // one slot: every row takes every token
            const uint64_t base = (static_cast<uint64_t>(e_slot[e0]) * p.kv_head_count + kv_head) * C;
            for (uint32_t t0 = 0; t0 < tail; t0 += 8u) {
                float v[kGroupStrands];
#pragma unroll
                for (int k = 0; k < kGroupStrands; ++k) {
                    const uint32_t t = t0 + grp + static_cast<uint32_t>(k * kGroups);
                    v[k] = t < tail && d < D ? load_tail(p.tail_v, p.tail_type, (base + t) * D + d) : 0.0f;
                }
#pragma unroll
                for (int k = 0; k < kGroupStrands; ++k) {
                    const uint32_t t = t0 + grp + static_cast<uint32_t>(k * kGroups);
                    if (t >= tail) continue;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float w = whole || (r / cta_heads >= e0 && r / cta_heads < e1) ? weights[t * S::kRowStride + r] : 0.0f;
                        if (w != 0.0f) acc[k][r] = fmaf(w, v[k], acc[k][r]);   // a token the row does not see may hold anything
                    }
                }
            }
        }
        // ((s0 + s2) + (s4 + s6)) and ((s1 + s3) + (s5 + s7)), added below
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if constexpr (kGroups == 1) {
                tail_acc[r * 128 + d] = (acc[0][r] + acc[2][r]) + (acc[4][r] + acc[6][r]);
                tail_acc[(R + r) * 128 + d] = (acc[1][r] + acc[3][r]) + (acc[5][r] + acc[7][r]);
            } else if constexpr (kGroups == 2) {
                tail_acc[(grp * R + r) * 128 + d] = (acc[0][r] + acc[1][r]) + (acc[2][r] + acc[3][r]);
            } else {
                tail_acc[(grp * R + r) * 128 + d] = acc[0][r];
            }
        }
    } else if (tid < R) {
        tail_m[tid] = -CUDART_INF_F;
        tail_l[tid] = 0.0f;
    }
    __syncthreads();
    auto tail_sum = [&](uint32_t r, uint32_t d) {
        if (!any_tail) return 0.0f;
        float h[2];
        for (int i = 0; i < 2; ++i) {
            if constexpr (S::kTailGroups == 2) h[i] = tail_acc[(i * R + r) * 128 + d];
            else h[i] = (tail_acc[i * 128 + d] + tail_acc[(i + 2) * 128 + d]) + (tail_acc[(i + 4) * 128 + d] + tail_acc[(i + 6) * 128 + d]);
        }
        return h[0] + h[1];
    };
    auto store = [&](uint32_t r, uint32_t d, float value) {
        const uint64_t i = (static_cast<uint64_t>(e_row[r / cta_heads]) * p.query_head_count + q_head_of(r)) * D + d;
        if (p.output_type == CF_B200_F16) reinterpret_cast<__half *>(p.output)[i] = __float2half_rn(value);
        else reinterpret_cast<float *>(p.output)[i] = value;
    };

    // ---- the partials: what the attention kernels wrote ----
    wait_for_previous_kernel();
    const PageLine line = plan_line(p);
    const uint4 more = __ldcg(reinterpret_cast<const uint4 *>(p.workspace) + 2);   // shared_pages.. of the header, see below
    static_assert(sizeof(PageLine) == 28 && offsetof(PlanHeader, shared_pages) == 32 && offsetof(PlanHeader, shared_rounds) == 40, "");
    struct RowPartials { uint32_t first, regular, count, seq, local_q; };
    auto row_partials = [&](uint32_t r) {
        RowPartials rp = {};
        rp.seq = entry0 + r / cta_heads;
        rp.local_q = head0 + r % cta_heads;
        const uint32_t a = __ldcg(line_prefix(p) + rp.seq), b = __ldcg(line_prefix(p) + rp.seq + 1u);
        if (b > a) {
            const uint32_t j0 = line.stretch_of(a), j1 = line.stretch_of(b - 1u);
            rp.first = line.slot(j0, line.piece_of(j0, a), a, rp.seq);
            rp.regular = line.slot(j1, line.piece_of(j1, b - 1u), b - 1u, rp.seq) + 1u - rp.first;
        }
        rp.count = rp.regular;
        if (more.x != 0u && more.y != 0u) {   // the shared prefix's: one per CTA of the shared-prefix kernel that met the row's head-tile
            const uint32_t row_tiles = (p.seq_count * G + 127u) / 128u;
            const SharedSplit split = {more.z, p.kv_head_span * row_tiles, more.y};
            const uint64_t first = static_cast<uint64_t>((rp.local_q / G) * row_tiles + (rp.seq * G + rp.local_q % G) / 128u) * split.rounds;
            rp.count += min(split.cta_of(first + split.rounds - 1u) - split.cta_of(first) + 1u, CF_B200_SHARED_CHUNKS_MAX);
        }
        return rp;
    };
    auto partial_of = [&](const RowPartials &rp, uint32_t c) {
        return c < rp.regular ? partial_ptr(p, rp.first + c, rp.local_q) : shared_partial_ptr(p, c - rp.regular, rp.seq, rp.local_q);
    };
    // Adds up the partials [begin, end) of a row, a whole number of strands of `strand` each; `emit` gets every strand's sums
    // (of l, and of this lane's channels lane + 32 j). Eight partials' loads are in flight at a time.
    auto add_strands = [&](const RowPartials &rp, uint32_t begin, uint32_t end, uint32_t strand, float m, auto emit) {
        float part[4] = {0.0f, 0.0f, 0.0f, 0.0f}, part_l = 0.0f;
        uint32_t left = strand;
        for (uint32_t c0 = begin; c0 < end; c0 += 32u) {
            float w = 0.0f, wl = 0.0f;   // lane i: weight of partial c0 + i, and its l
            if (c0 + lane < end) {
                const float *src = partial_of(rp, c0 + lane);
                const float pm = __ldcg(src);
                wl = __ldcg(src + 1);
                w = pm == -CUDART_INF_F ? 0.0f : exp2f(pm - m);
            }
            const uint32_t n = min(32u, end - c0);
            for (uint32_t i0 = 0; i0 < n; i0 += 8u) {
                float x[8][4];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float *src = i0 + i < n ? partial_of(rp, c0 + i0 + i) + 2 : nullptr;
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) x[i][j] = src && lane + 32u * j < D ? __ldcg(src + lane + 32u * j) : 0.0f;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (i0 + i >= n) break;
                    const float wi = __shfl_sync(0xffffffffu, w, i0 + i), li = __shfl_sync(0xffffffffu, wl, i0 + i);
                    if (wi != 0.0f) {   // a partial without a visible token says nothing
                        part_l = fmaf(li, wi, part_l);
#pragma unroll
                        for (int j = 0; j < 4; ++j) part[j] = fmaf(x[i][j], wi, part[j]);
                    }
                    if (--left == 0u) {
                        emit(part_l, part);
                        left = strand;
                        part_l = part[0] = part[1] = part[2] = part[3] = 0.0f;
                    }
                }
            }
        }
        if (left != strand) emit(part_l, part);
    };
    if constexpr (R > 1) {   // a warp per row
        for (uint32_t r = warp; r < rows; r += kWarps) {
            const RowPartials rp = row_partials(r);
            float m = -CUDART_INF_F;
            for (uint32_t c = lane; c < rp.count; c += 32u) m = fmaxf(m, __ldcg(partial_of(rp, c)));
            m = warp_max(m);
            float l = 0.0f, a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            add_strands(rp, 0u, rp.count, (rp.count + kStrands - 1u) / kStrands, m, [&](float pl, const float (&pa)[4]) {
                l += pl;
#pragma unroll
                for (int j = 0; j < 4; ++j) a[j] += pa[j];
            });
            const float top = fmaxf(m, tail_m[r]);
            const float sp = m == -CUDART_INF_F ? 0.0f : exp2f(m - top), st = tail_m[r] == -CUDART_INF_F ? 0.0f : exp2f(tail_m[r] - top);
            const float total = l * sp + tail_l[r] * st;
            const float inv = total > 0.0f ? 1.0f / total : 0.0f;   // no visible token: zeros (paged_kv_attention.cu:170-173)
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t d = lane + 32u * j;
                if (d < D) store(r, d, (a[j] * sp + tail_sum(r, d) * st) * inv);
            }
        }
    } else {   // the CTA's warps share one row's strands
        constexpr uint32_t kOwn = kStrands / kWarps;
        __shared__ float warp_m[kWarps], strand_l[kStrands];
        float *strands = smem_f + S::kStrand;
        const RowPartials rp = row_partials(0u);
        const uint32_t strand = (rp.count + kStrands - 1u) / kStrands;
        const uint32_t begin = min(warp * kOwn * strand, rp.count), end = min(begin + kOwn * strand, rp.count);
        float m = -CUDART_INF_F;
        for (uint32_t c = begin + lane; c < end; c += 32u) m = fmaxf(m, __ldcg(partial_of(rp, c)));
        m = warp_max(m);
        if (lane == 0) warp_m[warp] = m;
        __syncthreads();
        m = warp_max(lane < kWarps ? warp_m[lane] : -CUDART_INF_F);
        uint32_t k = warp * kOwn;
        add_strands(rp, begin, end, strand, m, [&](float pl, const float (&pa)[4]) {
            if (lane == 0) strand_l[k] = pl;
#pragma unroll
            for (int j = 0; j < 4; ++j) strands[k * 128u + lane + 32u * j] = pa[j];
            ++k;
        });
        __syncthreads();
        const uint32_t used = strand ? (rp.count + strand - 1u) / strand : 0u;
        if (tid < D) {
            float l = 0.0f, a = 0.0f;
            for (uint32_t i = 0; i < used; ++i) {
                l += strand_l[i];
                a += strands[i * 128u + tid];
            }
            const float top = fmaxf(m, tail_m[0]);
            const float sp = m == -CUDART_INF_F ? 0.0f : exp2f(m - top), st = tail_m[0] == -CUDART_INF_F ? 0.0f : exp2f(tail_m[0] - top);
            const float total = l * sp + tail_l[0] * st;
            const float inv = total > 0.0f ? 1.0f / total : 0.0f;
            store(0u, tid, (a * sp + tail_sum(0u, tid) * st) * inv);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Decode probe: write the symbols of whole records to global memory.
// ---------------------------------------------------------------------------------------------------------------
__global__ void decode_pages_kernel(AttentionParams p, const uint32_t *page_ids, uint8_t *k_out, uint8_t *v_out) {
    const uint32_t page = blockIdx.x, kv_head = blockIdx.y;
    const uint64_t entry = p.page_dir[static_cast<uint64_t>(page_ids[page]) * p.kv_head_count + kv_head];
    if (CF_B200_DIR_LENGTH_UNITS(entry) == 0) {
        if (threadIdx.x == 0) raise_status(p, CF_B200_DEVSTAT_BAD_RECORD);
        return;
    }
    const uint8_t *record = p.arena + 16ull * CF_B200_DIR_OFFSET_UNITS(entry);
    const cf_b200_record_header h = *reinterpret_cast<const cf_b200_record_header *>(record);
    if (h.version != CF_B200_FORMAT_VERSION || h.k_coder > CF_B200_CODER_MAX || h.v_coder > CF_B200_CODER_MAX) {
        if (threadIdx.x == 0) raise_status(p, CF_B200_DEVSTAT_BAD_RECORD);
        return;
    }
    const uint8_t *k_part = record + 16;
    const uint8_t *v_part = record + 16 + 16u * h.k_part_units;
    const uint64_t base = (static_cast<uint64_t>(page) * p.kv_head_count + kv_head) * p.symbols;
    for (uint32_t b = threadIdx.x; b < 2u * p.nblocks; b += blockDim.x) {
        if (b < p.nblocks) {
            uint8_t *dst = k_out + base + b * p.block_size;
            decode_part_block(k_part, 16u * h.k_part_units, h.k_coder, p.nblocks, b, p.block_size, p.symbols, p.k_tables,
                              [&](int j, uint32_t s) { dst[j] = static_cast<uint8_t>(s); });
        } else {
            const uint32_t vb = b - p.nblocks;
            uint8_t *dst = v_out + base + vb * p.block_size;
            decode_part_block(v_part, 16u * h.v_part_units, h.v_coder, p.nblocks, vb, p.block_size, p.symbols, p.v_tables,
                              [&](int j, uint32_t s) { dst[j] = static_cast<uint8_t>(s); });
        }
    }
}

bool finite_float(float v) { return v == v && v - v == 0.0f; }

// Test hooks (cf_b200_test_wait_expiry): a lowered wait bound and one page whose copy is armed but never issued.
std::atomic<uint32_t> g_test_wait_polls{0}, g_test_skip_copy_page{0};

bool fill_params(const cf_b200_sealed_attention_desc *d, AttentionParams *p) {
    p->kv_head_count = d->kv_head_count;
    p->query_head_count = d->query_head_count;
    p->head_dim = d->head_dim;
    p->page_tokens = d->page_tokens;
    p->block_size = d->block_size;
    p->kv_head_begin = d->kv_head_begin;
    p->kv_head_span = d->kv_head_span ? d->kv_head_span : d->kv_head_count - d->kv_head_begin;
    p->group = d->query_head_count / d->kv_head_count;
    p->symbols = d->head_dim * d->page_tokens;
    p->nblocks = (p->symbols + d->block_size - 1) / d->block_size;
    p->codebook_id = d->codebook_id;
    p->arena = d->arena;
    p->page_dir = d->page_dir;
    p->page_table = d->page_table;
    p->seq_sealed_tokens = d->seq_sealed_tokens;
    p->seq_slots = d->seq_slots;
    p->page_table_stride = d->page_table_stride;
    p->seq_count = d->seq_count;
    p->k_tables = d->k_tables;
    p->v_tables = d->v_tables;
    p->tail_k = d->tail_k;
    p->tail_v = d->tail_v;
    p->tail_tokens = d->tail_tokens;
    p->tail_type = d->tail_type == CF_B200_F32 ? CF_B200_F32 : CF_B200_F16;
    p->query_positions = d->query_positions;
    p->row_map = d->row_map;
    p->tail_capacity = d->tail_capacity ? d->tail_capacity : d->page_tokens;
    p->queries = d->queries;
    p->output = d->output;
    p->query_type = d->query_type;
    p->output_type = d->output_type;
    p->softmax_scale = d->softmax_scale;
    p->causal_window = d->causal_window;
    p->workspace = static_cast<uint8_t *>(d->workspace);
    p->layout = workspace_layout(d->seq_count, p->kv_head_span * p->group, d->head_dim, d->workspace_bytes,
                                 d->shared_prefix_pages != 0);
    p->min_pages_per_unit = d->min_pages_per_unit;
    p->shared_prefix_pages = 0;   // the launch code sets it when the lanes kernels serve the call
    p->sm_count = 0;
    p->decode_probe = d->kernel == CF_B200_KERNEL_DECODE_PROBE ? 1u : d->kernel == CF_B200_KERNEL_DECODE_DUMP ? 2u : 0u;
    p->dump_pages = p->decode_probe == 2u ? d->reserved0 : 1u;
    const uint32_t polls = g_test_wait_polls.load(std::memory_order_relaxed);
    p->wait_polls = polls ? polls : kDefaultWaitPolls;
    p->skip_copy_page = g_test_skip_copy_page.load(std::memory_order_relaxed);
    p->status = d->status;
    p->pool_k = nullptr;
    p->pool_v = nullptr;
    return true;
}

}  // namespace

cudaError_t launch_plan(const AttentionParams &p, cudaStream_t stream) {
    if (p.shared_prefix_pages) verify_prefix_kernel<<<p.seq_count, 256, 0, stream>>>(p);
    const uint32_t threads = p.seq_count <= 128u ? 128u : kPlanThreads;   // small batches: fewer warps to start and to meet
    return launch_kernel(plan_kernel, 1, threads, 0, stream, p.shared_prefix_pages != 0u, p);
}

namespace {

template <int R, int kThreads>
cudaError_t launch_combine_as(const AttentionParams &p, cudaStream_t stream, bool dependent, uint32_t entries, uint32_t heads) {
    const dim3 grid((p.seq_count + entries - 1u) / entries, p.kv_head_span * p.group / heads);
    const size_t smem = CombineSmem<R, kThreads>::bytes(p.tail_capacity);
    if (smem > 47u * 1024u) {   // tails of thousands of tokens
        const cudaError_t e = cudaFuncSetAttribute(combine_kernel<R, kThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
    }
    return launch_kernel(combine_kernel<R, kThreads>, grid, kThreads, smem, stream, dependent, p, entries, heads);
}

}  // namespace

// Rows per CTA of the combine kernel: a kv head's whole query group where that still makes about a CTA per SM, and in
// multi-query calls as many entries beside it as make sixteen rows, if their tails are long enough to be worth sharing.
// Otherwise a CTA per row: of 1024 threads while all of them are resident at once, of 256 beyond that. The tail's weights must
// fit the 48 KB of shared memory that need no opt-in.
cudaError_t launch_combine(const AttentionParams &p, cudaStream_t stream, bool dependent) {
    constexpr uint32_t kEnoughCtas = 120, kSharedBytes = 48 * 1024 - 1024;
    const uint32_t groups = p.seq_count * p.kv_head_span, G = p.group, C = p.tail_capacity;
    if (groups >= kEnoughCtas) {
        const uint32_t entries = p.query_positions && p.seq_slots && C > 16u ? 16u / G : 1u;
        if (entries > 1u && (groups + entries - 1u) / entries >= kEnoughCtas && CombineSmem<16, 256>::bytes(C) <= kSharedBytes)
            return launch_combine_as<16, 256>(p, stream, dependent, entries, G);
        if (G <= 4u && CombineSmem<4, 128>::bytes(C) <= kSharedBytes) return launch_combine_as<4, 128>(p, stream, dependent, 1u, G);
        if (G <= 8u && CombineSmem<8, 256>::bytes(C) <= kSharedBytes) return launch_combine_as<8, 256>(p, stream, dependent, 1u, G);
        if (CombineSmem<16, 256>::bytes(C) <= kSharedBytes) return launch_combine_as<16, 256>(p, stream, dependent, 1u, G);
    }
    if (groups * G <= 2u * 148u && CombineSmem<1, 1024>::bytes(C) <= kSharedBytes) return launch_combine_as<1, 1024>(p, stream, dependent, 1u, 1u);
    return launch_combine_as<1, 256>(p, stream, dependent, 1u, 1u);
}

cudaError_t launch_generic_attention(const AttentionParams &p, cudaStream_t stream) {
    static LauncherState table[64];
    cudaError_t e;
    LauncherState *state = launcher_state(table, &e);
    if (!state) return e;
    const int sm_count = state->sm_count;
    const GenericSmem lay = generic_smem(p.symbols, p.group, p.head_dim, p.page_tokens);
    e = cudaFuncSetAttribute(generic_attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(lay.total));
    if (e != cudaSuccess) return e;
    generic_attention_kernel<<<sm_count * kGenericCtasPerSm, kGenericThreads, lay.total, stream>>>(p);
    return cudaPeekAtLastError();
}

}  // namespace cfb

using cfb::AttentionParams;

extern "C" cf_status cf_b200_sealed_attention_validate(const cf_b200_sealed_attention_desc *d) {
    if (d == nullptr || d->struct_size != sizeof(cf_b200_sealed_attention_desc) || d->abi_version != CF_B200_ABI_VERSION)
        return CF_ERR_INVALID_ARGUMENT;
    if (d->kv_head_count == 0 || d->query_head_count == 0 || d->head_dim == 0 || d->page_tokens == 0 ||
        d->block_size == 0 || d->query_head_count % d->kv_head_count != 0 || !cfb::finite_float(d->softmax_scale))
        return CF_ERR_INVALID_ARGUMENT;
    if (d->kv_head_begin >= d->kv_head_count || d->kv_head_span > d->kv_head_count - d->kv_head_begin)
        return CF_ERR_INVALID_ARGUMENT;
    if (d->queries == nullptr || d->output == nullptr || d->workspace == nullptr || d->seq_sealed_tokens == nullptr ||
        d->k_tables == nullptr || d->v_tables == nullptr)
        return CF_ERR_INVALID_ARGUMENT;
    if (d->seq_count == 0) return CF_ERR_INVALID_ARGUMENT;
    if (d->page_table_stride != 0 && (d->page_table == nullptr || d->page_dir == nullptr || d->arena == nullptr))
        return CF_ERR_INVALID_ARGUMENT;
    if (d->tail_tokens != nullptr && (d->tail_k == nullptr || d->tail_v == nullptr)) return CF_ERR_INVALID_ARGUMENT;
    if ((d->query_type != CF_B200_F16 && d->query_type != CF_B200_F32) ||
        (d->output_type != CF_B200_F16 && d->output_type != CF_B200_F32) || d->kernel > CF_B200_KERNEL_DECODE_DUMP ||
        (d->tail_type != 0 && d->tail_type != CF_B200_F16 && d->tail_type != CF_B200_F32))
        return CF_ERR_INVALID_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(d->arena) & 15u) != 0 || (reinterpret_cast<uintptr_t>(d->workspace) & 255u) != 0)
        return CF_ERR_INVALID_ARGUMENT;
    // format limits
    if (d->head_dim > CF_KV_MAX_HEAD_DIM || d->head_dim * d->page_tokens > CF_B200_MAX_STREAM_SYMBOLS ||
        d->block_size < 16 || d->block_size > 1024 || d->query_head_count / d->kv_head_count > cfb::kGenericMaxGroup)
        return CF_ERR_UNSUPPORTED;
    const uint32_t span = d->kv_head_span ? d->kv_head_span : d->kv_head_count - d->kv_head_begin;
    const cfb::WorkspaceLayout w = cfb::workspace_layout(d->seq_count, span * (d->query_head_count / d->kv_head_count),
                                                         d->head_dim, d->workspace_bytes, d->shared_prefix_pages != 0);
    if (w.chunk_capacity < d->seq_count) return CF_ERR_INVALID_ARGUMENT;  // at least one partial per sequence
    if (d->shared_prefix_pages > d->page_table_stride) return CF_ERR_INVALID_ARGUMENT;
    // reserved0 has one use: the number of page ids the dump buffer of CF_B200_KERNEL_DECODE_DUMP covers
    if ((d->kernel == CF_B200_KERNEL_DECODE_DUMP) != (d->reserved0 != 0)) return CF_ERR_INVALID_ARGUMENT;
    return CF_OK;
}

extern "C" cf_status cf_b200_sealed_attention_workspace_bytes(const cf_b200_sealed_attention_desc *d,
                                                              uint64_t total_pages, uint64_t *out_bytes) {
    if (d == nullptr || out_bytes == nullptr || d->kv_head_count == 0 || d->query_head_count == 0 ||
        d->query_head_count % d->kv_head_count != 0 || d->head_dim == 0)
        return CF_ERR_INVALID_ARGUMENT;
    const uint32_t span = d->kv_head_span ? d->kv_head_span : d->kv_head_count - d->kv_head_begin;
    const uint32_t local_q = span * (d->query_head_count / d->kv_head_count);
    const uint64_t slots = cfb::partial_slots_for(total_pages, d->seq_count, span, d->min_pages_per_unit);
    const cfb::WorkspaceLayout w = cfb::workspace_layout(d->seq_count, local_q, d->head_dim, 0, d->shared_prefix_pages != 0);
    *out_bytes = w.partials_offset + slots * (w.partial_stride_floats * 4ull * local_q) + 64ull;
    return CF_OK;
}

extern "C" cf_status cf_b200_sealed_attention_stages_async(const cf_b200_sealed_attention_desc *d, uint32_t stages,
                                                           void *stream) {
    return cfb::sealed_attention_stages(d, stages, stream, false);
}

// output_on_peer: the one exception to "every pointer is the current device's" — the multi-GPU scheduler lets the
// combine kernel store its output rows straight into the root GPU's tensor (plain coalesced stores over a peer mapping
// the scheduler has enabled and checked). Everything that is READ stays local.
cf_status cfb::sealed_attention_stages(const cf_b200_sealed_attention_desc *d, uint32_t stages, void *stream, bool output_on_peer) {
    const cf_status valid = cf_b200_sealed_attention_validate(d);
    if (valid != CF_OK) return valid;
    if (stages == 0 || stages > 7u) return CF_ERR_INVALID_ARGUMENT;
    if (!cfb::on_current_device(d->arena) || !cfb::on_current_device(d->workspace) || !cfb::on_current_device(d->queries) ||
        !cfb::on_current_device(d->row_map) || (!output_on_peer && !cfb::on_current_device(d->output)))
        return CF_ERR_INVALID_ARGUMENT;   // memory of another GPU: the call must be made with that GPU current
    AttentionParams p;
    cfb::fill_params(d, &p);
    const bool lanes_ok = cfb::lanes_kernel_supports(p);
    const bool probe = d->kernel == CF_B200_KERNEL_DECODE_PROBE || d->kernel == CF_B200_KERNEL_DECODE_DUMP;
    if ((d->kernel == CF_B200_KERNEL_LANES || probe) && !lanes_ok) return CF_ERR_UNSUPPORTED;
    if (d->kernel == CF_B200_KERNEL_DECODE_DUMP && (stages & CF_B200_STAGE_COMBINE)) return CF_ERR_INVALID_ARGUMENT;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool use_lanes = d->kernel == CF_B200_KERNEL_LANES || probe ||
                           (d->kernel == CF_B200_KERNEL_AUTO && lanes_ok);
    static cfb::LauncherState table[64];
    cudaError_t e;
    const cfb::LauncherState *state = cfb::launcher_state(table, &e);
    if (!state) return CF_ERR_CUDA;
    p.sm_count = static_cast<uint32_t>(state->sm_count);
    if (use_lanes) {
        cfb::lanes_plan_shape(p, p.sm_count, &p.plan_warps, &p.unit_lanes);
    } else {
        p.plan_warps = p.sm_count * cfb::kGenericCtasPerSm;
        p.unit_lanes = p.kv_head_span;
    }
    // the shared-prefix kernel works on rows of 128 = whole query groups and on pages every query token sees in full
    if (use_lanes && p.block_size == 64 && p.head_dim == 128 && d->row_map == nullptr && p.decode_probe != 1u && d->shared_prefix_pages && d->causal_window == 0 && 128u % p.group == 0)
        p.shared_prefix_pages = d->shared_prefix_pages;
    const bool plan = (stages & CF_B200_STAGE_PLAN) != 0, attention = (stages & CF_B200_STAGE_ATTENTION) != 0;
    if (plan && cfb::launch_plan(p, s) != cudaSuccess) return CF_ERR_CUDA;
    if (attention) {
        const bool prefix = p.shared_prefix_pages != 0u;
        if (prefix) {
            if (cfb::launch_prefix_attention(p, s, plan) != cudaSuccess) return CF_ERR_CUDA;
            g_shared_prefix_launches.fetch_add(1, std::memory_order_relaxed);
        }
        e = use_lanes ? cfb::launch_lanes_attention(p, s, plan || prefix, prefix) : cfb::launch_generic_attention(p, s);
        if (e != cudaSuccess) return CF_ERR_CUDA;
    }
    if ((stages & CF_B200_STAGE_COMBINE) && cfb::launch_combine(p, s, attention && use_lanes) != cudaSuccess) return CF_ERR_CUDA;
    return CF_OK;
}

extern "C" cf_status cf_b200_test_wait_expiry(uint32_t skip_copy_page_id, uint32_t wait_polls) {
    cfb::g_test_skip_copy_page.store(skip_copy_page_id, std::memory_order_relaxed);
    cfb::g_test_wait_polls.store(wait_polls, std::memory_order_relaxed);
    return CF_OK;
}

extern "C" unsigned long long cf_b200_shared_prefix_launches(void) {
    return g_shared_prefix_launches.load(std::memory_order_relaxed);
}

extern "C" cf_status cf_b200_sealed_attention_async(const cf_b200_sealed_attention_desc *d, void *stream) {
    return cf_b200_sealed_attention_stages_async(
        d, CF_B200_STAGE_PLAN | CF_B200_STAGE_ATTENTION | CF_B200_STAGE_COMBINE, stream);
}

extern "C" cf_status cf_b200_decode_pages_async(const cf_b200_sealed_attention_desc *d, const uint32_t *page_ids,
                                                uint32_t page_count, uint8_t *k_symbols, uint8_t *v_symbols,
                                                void *stream) {
    if (d == nullptr || d->struct_size != sizeof(cf_b200_sealed_attention_desc) ||
        d->abi_version != CF_B200_ABI_VERSION || page_ids == nullptr || k_symbols == nullptr || v_symbols == nullptr ||
        d->arena == nullptr || d->page_dir == nullptr || d->k_tables == nullptr || d->v_tables == nullptr ||
        d->kv_head_count == 0 || d->head_dim == 0 || d->page_tokens == 0 || d->block_size == 0)
        return CF_ERR_INVALID_ARGUMENT;
    if (d->head_dim * d->page_tokens > CF_B200_MAX_STREAM_SYMBOLS || d->block_size < 16 || d->block_size > 1024)
        return CF_ERR_UNSUPPORTED;
    if (page_count == 0) return CF_OK;
    AttentionParams p{};
    p.kv_head_count = d->kv_head_count;
    p.head_dim = d->head_dim;
    p.page_tokens = d->page_tokens;
    p.block_size = d->block_size;
    p.symbols = d->head_dim * d->page_tokens;
    p.nblocks = (p.symbols + d->block_size - 1) / d->block_size;
    p.arena = d->arena;
    p.page_dir = d->page_dir;
    p.k_tables = d->k_tables;
    p.v_tables = d->v_tables;
    p.status = d->status;
    cfb::decode_pages_kernel<<<dim3(page_count, d->kv_head_count), 128, 0, static_cast<cudaStream_t>(stream)>>>(
        p, page_ids, k_symbols, v_symbols);
    return cudaPeekAtLastError() == cudaSuccess ? CF_OK : CF_ERR_CUDA;
}
