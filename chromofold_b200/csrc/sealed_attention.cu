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
// 5.2 us for one sequence and 9.4 us for 64, against 3.5 and 3.4 us now (alone on the GPU, start-up included).
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

// A workspace with `room` stretches for more warps than that: an even cut leaves warps idle, because a stretch may need a slot in
// every sequence it meets. Units of a fixed size inside their sequence need one slot each. Returns their size in pages where they end
// sooner, 0 where the even cut does: in the built-in workspace (8 MiB) 250 sequences of 1024 tokens on 64 query heads take 485 us in
// units, 34.5 ms in the three stretches there is room for. Whole block; begin and end are this thread's entries.
__device__ uint32_t pages_per_unit_in_small_workspace(const SeqInfo *info, uint32_t begin, uint32_t end, uint32_t pages, uint32_t room, uint32_t capacity,
                                                      uint32_t warps, uint32_t *warp_totals) {
    uint32_t grain = max((pages + capacity - 1u) / capacity, 1u);
    for (;; grain += (grain + 3u) / 4u) {   // from one unit per sequence on they fit
        uint32_t mine = 0, units;
        for (uint32_t s = begin; s < end; ++s) mine += (info[s].page_end - info[s].first_page + grain - 1u) / grain;
        block_scan(mine, warp_totals, &units);
        if (units > capacity) continue;
        return static_cast<uint64_t>((units + warps - 1u) / warps) * grain < (pages + room - 1u) / room ? grain : 0u;
    }
}

// kSmall: the workspace may leave warps without a stretch. (A kernel of its own: the plan is one block whose instructions come from
// memory, and the few for this case cost a step of one sequence 0.3 us.)
template <bool kSmall>
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
    if (p.one_slot) {   // query tokens of one sequence: its pages are shared whatever the positions (the shared-prefix kernel masks)
        shared = min(shared, p.seq_sealed_tokens[slot_of(p, 0)] / p.page_tokens);
    } else if (shared) {
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
        const uint32_t rows = p.seq_count * p.group;
        shared_rounds = (shared + 7u) / 8u;
        shared_ctas = shared_split_ctas(shared_rounds, p.kv_head_span * shared_tile_groups(rows), p.sm_count / shared_cluster(rows), CF_B200_SHARED_CHUNKS_MAX);
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
    uint32_t incl, total, pages_per_unit = p.min_pages_per_unit;
    const uint32_t capacity = static_cast<uint32_t>(min(p.layout.chunk_capacity, static_cast<uint64_t>(0x7fffffffu)));
    if (pages_per_unit == 0u) {
        // One stretch per resident warp for the units of a stretch (kv heads x passes), where there is a page for each and a
        // partial slot: the last slot is stretches * pieces + seq_count - 2. The capacity is at least seq_count.
        incl = block_scan(local, warp_totals, &total);
        const uint32_t room = capacity - (p.seq_count - 1u), warps = max(p.plan_warps / p.unit_lanes, 1u);
        line.stretches = min(min(warps, total), room);
        if (kSmall && room < min(warps, total)) pages_per_unit = pages_per_unit_in_small_workspace(info, begin, end, total, room, capacity, warps, warp_totals);
        if (line.stretches) {
            line.base = total / line.stretches;
            line.longer = total % line.stretches;
            const uint32_t longest = line.base + (line.longer ? 1u : 0u);
            line.pieces = min(max(min((longest + kPiecePages - 1u) / kPiecePages, room / line.stretches), 1u), line.base);
        }
    }
    if (pages_per_unit != 0u) {
        line.by_position = 1u;
        line.longer = 0u;
        line.grain = pages_per_unit;
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
// Bound by the length of its chain of loads, not by what they carry (a few MB): record -> tail rows -> weights -> partials.
// So every stage has all of its loads in flight at once, the first V rows are fetched before the scores are worked out, and the
// tail is done before this kernel waits for the attention kernel. Everything the plan kernel wrote may be read before that wait:
// the attention kernel lets this one start only after it has seen the plan's end itself.
//
// Every sum of combine_kernel has an order of its own that the shape of the CTA does not change, so that its forms agree to the bit for
// given partials: they are added up in 32 consecutive strands, each relative to its own maximum, and the strands in order; tail
// tokens in eight interleaved strands. Which pages a partial covers follows the batch (an even cut of its whole line; a caller's
// min_pages_per_unit keeps the cut to the sequence), and combine_tile_kernel, which large prompts take, adds in another
// order: the last bits of a row can differ with the batch it is in.
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

__device__ __forceinline__ SeqInfo load_seq_info(const AttentionParams &p, uint32_t seq) {
    const uint4 *src = reinterpret_cast<const uint4 *>(seq_info(p) + seq);
    const uint4 a = __ldcg(src), b = __ldcg(src + 1);
    SeqInfo info;
    info.slot = a.x, info.sealed = a.y, info.qpos = a.z, info.tail = a.w;
    info.first_page = b.x, info.page_end = b.y, info.row = b.z, info.line_begin = b.w;
    return info;
}

// The partials of a row: slots [first, first + regular), then the shared prefix's cells.
struct RowPartials {
    uint32_t first, regular, cells;
};
__device__ __forceinline__ RowPartials row_partials(const AttentionParams &p, const PageLine &line, const SeqInfo &info, uint32_t seq,
                                                    uint32_t local_q) {
    RowPartials rp = {};
    const uint32_t pages = info.page_end - info.first_page;
    if (pages) {
        const uint32_t a = info.line_begin, b = a + (line.grain == 1u ? pages : (pages + line.grain - 1u) / line.grain) - 1u;
        const uint32_t j0 = line.stretch_of(a), j1 = line.stretch_of(b);
        rp.first = line.slot(j0, line.piece_of(j0, a), a, seq);
        rp.regular = line.slot(j1, line.piece_of(j1, b), b, seq) + 1u - rp.first;
    }
    // one per CTA of the shared-prefix kernel that met the row's head-tile
    static_assert(sizeof(PageLine) == 28 && offsetof(PlanHeader, shared_pages) == 32 && offsetof(PlanHeader, shared_rounds) == 40, "");
    const uint4 shared = __ldcg(reinterpret_cast<const uint4 *>(p.workspace) + 2);
    if (shared.x != 0u && shared.y != 0u) {
        const uint32_t rows = p.seq_count * p.group, groups = shared_tile_groups(rows);
        const SharedSplit split = {shared.z, p.kv_head_span * groups, shared.y};
        const uint64_t first =
            static_cast<uint64_t>((local_q / p.group) * groups + (seq * p.group + local_q % p.group) / (128u * shared_cluster(rows))) * split.rounds;
        rp.cells = min(split.cta_of(first + split.rounds - 1u) - split.cta_of(first) + 1u, CF_B200_SHARED_CHUNKS_MAX);
    }
    return rp;
}
__device__ __forceinline__ const float *partial_of(const AttentionParams &p, const RowPartials &rp, uint32_t c, uint32_t seq, uint32_t local_q) {
    return c < rp.regular ? partial_ptr(p, rp.first + c, local_q) : shared_partial_ptr(p, c - rp.regular, seq, local_q);
}
__device__ __forceinline__ void store_output(const AttentionParams &p, uint64_t i, float value) {
    if (p.output_type == CF_B200_F16) reinterpret_cast<__half *>(p.output)[i] = __float2half_rn(value);
    else reinterpret_cast<float *>(p.output)[i] = value;
}

// A CTA serves R query heads of one kv head for one entry; kThreads / 32 / R warps share a row's partials. R = 4 reads a tail's rows
// once for four heads: on 512 threads while all CTAs are resident at once, on 128 beyond that, where a warp per row
// needs no strands in shared memory and issues a quarter of the instructions (256 sequences: 23 against 68 us). R = 1 on 1024
// threads spreads a launch with few rows.
template <int R, int kThreads>
struct CombineSmem {   // offsets in floats
    static constexpr int kGroups = kThreads / 128;                     // thread groups of one thread per channel
    static constexpr int kTail = 0;                                    // [group][R][128] sums of weighted V rows
    static constexpr int kStrand = kTail + kGroups * R * 128;          // [R][strand][128], where several warps share a row
    static constexpr int kWeights = kStrand + (kThreads == 32 * R ? 0 : R * static_cast<int>(kStrands) * 128);   // [tail_capacity][R]
    static size_t bytes(uint32_t tail_capacity) { return (kWeights + static_cast<size_t>(tail_capacity) * R) * 4u; }
};

template <int R, int kThreads>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads > 8 ? 8 : 1024 / kThreads) combine_kernel(AttentionParams p) {
    using S = CombineSmem<R, kThreads>;
    constexpr int kWarps = kThreads / 32, kGroups = S::kGroups, kBatch = 8;
    constexpr uint32_t kRowWarps = kWarps / R, kOwn = kStrands / kRowWarps;
    extern __shared__ __align__(16) float smem_f[];
    float *tail_acc = smem_f + S::kTail, *strands = smem_f + S::kStrand, *weights = smem_f + S::kWeights;
    __shared__ float tail_m[R], tail_l[R], strand_m[R][kStrands], strand_l[R][kStrands];
    __shared__ RowPartials r_partials[R];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, d = tid & 127u, grp = tid >> 7;
    const uint32_t G = p.group, D = p.head_dim, C = p.tail_capacity;   // C: rows per (slot, kv head) in the tails
    const uint32_t seq = blockIdx.x, subs = (G + R - 1u) / R;
    const uint32_t head_local = blockIdx.y / subs, in_group = blockIdx.y % subs * R, rows = min(static_cast<uint32_t>(R), G - in_group);
    const uint32_t kv_head = p.kv_head_begin + head_local, q_head = kv_head * G + in_group, local_q = head_local * G + in_group;
    const SeqInfo info = load_seq_info(p, seq);
    const PageLine line = plan_line(p);
    const uint32_t tail = min(info.tail, C);
    if (tid < R) r_partials[tid] = row_partials(p, line, info, seq, local_q + min(tid, rows - 1u));

    if (tail) {
        const uint64_t base = (static_cast<uint64_t>(info.slot) * p.kv_head_count + kv_head) * C;
        float v[kBatch];
        auto load_v = [&](uint32_t t0) {
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                const uint32_t t = t0 + grp + static_cast<uint32_t>(k * kGroups);
                v[k] = t < tail && d < D ? load_tail(p.tail_v, p.tail_type, (base + t) * D + d) : 0.0f;
            }
        };
        load_v(0u);
        float q[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                q[r][j] = r < rows && lane + 32u * j < D ? load_query(p, info.row, q_head + r, lane + 32u * j) : 0.0f;
        // scores: two tokens per warp at a time, four channels per lane, the sums of all rows reduced together
        for (uint32_t t0 = 2u * warp; t0 < tail; t0 += 2u * kWarps) {
            float k0[4], k1[4], sums[2 * R];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t c = lane + 32u * j;
                k0[j] = c < D ? load_tail(p.tail_k, p.tail_type, (base + t0) * D + c) : 0.0f;
                k1[j] = c < D && t0 + 1u < tail ? load_tail(p.tail_k, p.tail_type, (base + t0 + 1u) * D + c) : 0.0f;
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float a = 0.0f, b = 0.0f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    a = fmaf(q[r][j], k0[j], a);
                    b = fmaf(q[r][j], k1[j], b);
                }
                sums[r] = a;
                sums[R + r] = b;
            }
            const float sum = sum_many<2 * R>(sums, lane);
            const uint32_t value = lane / (16u / R), r = value % R, t = t0 + value / R, token = info.sealed + t;
            if (lane % (16u / R) == 0u && t < tail) {
                const bool visible = token >= window_begin(info.qpos, p.causal_window) && token <= info.qpos;
                weights[t * R + r] = visible ? sum * p.softmax_scale * kLog2e : -CUDART_INF_F;
            }
        }
        __syncthreads();
        // softmax of every row over its tail: scores become weights relative to the row's largest
        if (warp < R) {
            float m = -CUDART_INF_F, l = 0.0f;
            for (uint32_t t = lane; t < tail; t += 32u) m = fmaxf(m, weights[t * R + warp]);
            m = warp_max(m);
            for (uint32_t t = lane; t < tail; t += 32u) {
                const float s = weights[t * R + warp], w = s == -CUDART_INF_F ? 0.0f : exp2f(s - m);
                weights[t * R + warp] = w;
                l += w;
            }
            l = warp_sum(l);
            if (lane == 0) {
                tail_m[warp] = m;
                tail_l[warp] = l;
            }
        }
        __syncthreads();
        // weighted V rows: a thread per channel, thread group g takes the token strands g, g + groups, ... of eight
        constexpr int kOwnTokens = 8 / kGroups;
        float acc[kOwnTokens][R];
#pragma unroll
        for (int k = 0; k < kOwnTokens; ++k)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[k][r] = 0.0f;
        for (uint32_t t0 = 0;;) {
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                const uint32_t t = t0 + grp + static_cast<uint32_t>(k * kGroups);
                if (t >= tail) break;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float w = weights[t * R + r];
                    if (w != 0.0f) acc[k % kOwnTokens][r] = fmaf(w, v[k], acc[k % kOwnTokens][r]);   // a token the row does not see may hold anything
                }
            }
            t0 += kBatch * kGroups;
            if (t0 >= tail) break;
            load_v(t0);
        }
        static_assert(kGroups == 1 || kGroups == 4 || kGroups == 8, "strands g and g + 4 are added first, then 0 + 2 and 1 + 3");
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if constexpr (kGroups == 1)
                tail_acc[r * 128 + d] = ((acc[0][r] + acc[4][r]) + (acc[2][r] + acc[6][r])) + ((acc[1][r] + acc[5][r]) + (acc[3][r] + acc[7][r]));
            else
                tail_acc[(grp * R + r) * 128 + d] = kGroups == 4 ? acc[0][r] + acc[kOwnTokens - 1][r] : acc[0][r];
        }
    }
    __syncthreads();

    // ---- the partials: what the attention kernels wrote ----
    const uint32_t my_row = warp / kRowWarps;
    const RowPartials rp = r_partials[my_row];
    const uint32_t count = rp.regular + rp.cells, strand = (count + kStrands - 1u) / kStrands;
    wait_for_previous_kernel();
    if (my_row < rows) {
        const uint32_t lq = local_q + my_row;
        uint32_t j = (warp % kRowWarps) * kOwn;   // strand
        const uint32_t begin = min(j * strand, count), end = min(begin + kOwn * strand, count);
        const uint32_t whole = strand && strand <= 32u ? 32u / strand * strand : 0u;   // partials per turn: whole strands, or 32 of a long one
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f}, acc_l = 0.0f, mj = -CUDART_INF_F;
        uint32_t left = strand;
        float top = tail ? tail_m[my_row] : -CUDART_INF_F, row_acc[4] = {0.0f, 0.0f, 0.0f, 0.0f}, row_l = 0.0f;   // a warp per row only
        if constexpr (kRowWarps == 1u) {
            float m = -CUDART_INF_F;
            for (uint32_t c = lane; c < count; c += 32u) m = fmaxf(m, __ldcg(partial_of(p, rp, c, seq, lq)));
            top = fmaxf(warp_max(m), top);
        }
        for (uint32_t c0 = begin, n; c0 < end; c0 += n) {
            n = min(whole ? whole : min(32u, left), end - c0);
            float pm = -CUDART_INF_F, pl = 0.0f, x[8][4];
            if (lane < n) {
                const float *src = partial_of(p, rp, c0 + lane, seq, lq);
                pm = __ldcg(src);
                pl = __ldcg(src + 1);
            }
            auto load_batch = [&](uint32_t i0) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float *src = partial_of(p, rp, c0 + min(i0 + i, n - 1u), seq, lq) + 2;
#pragma unroll
                    for (uint32_t c = 0; c < 4; ++c) x[i][c] = i0 + i < n && lane + 32u * c < D ? __ldcg(src + lane + 32u * c) : 0.0f;
                }
            };
            load_batch(0u);   // on its way before its weights are known
            if (whole) {   // every strand's own maximum
                mj = pm;
                const uint32_t first = lane / strand * strand;
                for (uint32_t i = 0; strand > 1u && i < strand; ++i) mj = fmaxf(mj, __shfl_sync(0xffffffffu, pm, (first + i) & 31u));
            } else if (left == strand) {
                mj = -CUDART_INF_F;
                for (uint32_t c = c0 + lane; c < min(c0 + strand, end); c += 32u) mj = fmaxf(mj, __ldcg(partial_of(p, rp, c, seq, lq)));
                mj = warp_max(mj);
            }
            const float w = pm == -CUDART_INF_F ? 0.0f : exp2f(pm - mj);
            for (uint32_t i0 = 0; i0 < n; i0 += 8u) {
                if (i0) load_batch(i0);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (i0 + i >= n) break;
                    const float wi = __shfl_sync(0xffffffffu, w, i0 + i), li = __shfl_sync(0xffffffffu, pl, i0 + i);
                    const float mi = __shfl_sync(0xffffffffu, mj, i0 + i);
                    if (wi != 0.0f) {   // a partial without a visible token says nothing
                        acc_l = fmaf(li, wi, acc_l);
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[c] = fmaf(x[i][c], wi, acc[c]);
                    }
                    if (--left == 0u || c0 + i0 + i + 1u == end) {
                        if constexpr (kRowWarps == 1u) {
                            const float f = mi == -CUDART_INF_F ? 0.0f : exp2f(mi - top);
                            if (lane == j) row_l = acc_l * f;
#pragma unroll
                            for (int c = 0; c < 4; ++c) row_acc[c] = fmaf(acc[c], f, row_acc[c]);
                        } else {
                            if (lane == 0) {
                                strand_m[my_row][j] = mi;
                                strand_l[my_row][j] = acc_l;
                            }
#pragma unroll
                            for (int c = 0; c < 4; ++c) strands[(my_row * kStrands + j) * 128u + lane + 32u * c] = acc[c];
                        }
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[c] = 0.0f;
                        acc_l = 0.0f;
                        left = strand;
                        ++j;
                    }
                }
            }
        }
        if constexpr (kRowWarps == 1u) {
            const float tm = tail ? tail_m[my_row] : -CUDART_INF_F, ft = tm == -CUDART_INF_F ? 0.0f : exp2f(tm - top);
            float l = warp_sum(row_l);
            if (ft != 0.0f) l = fmaf(tail_l[my_row], ft, l);
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) {
                const uint32_t ch = lane + 32u * c;
                const float a = ft != 0.0f ? fmaf(tail_acc[my_row * 128u + ch], ft, row_acc[c]) : row_acc[c];
                if (ch < D) store_output(p, (static_cast<uint64_t>(info.row) * p.query_head_count + q_head + my_row) * D + ch, l > 0.0f ? a / l : 0.0f);
            }
        }
    }
    if constexpr (kRowWarps == 1u) return;
    __syncthreads();
    const uint32_t r = grp;   // a thread per row and channel
    if (r < rows) {
        const uint32_t n = r_partials[r].regular + r_partials[r].cells, per = (n + kStrands - 1u) / kStrands, used = n ? (n + per - 1u) / per : 0u;
        const float sm = lane < used ? strand_m[r][lane] : -CUDART_INF_F, tm = tail ? tail_m[r] : -CUDART_INF_F;
        const float top = fmaxf(warp_max(sm), tm);
        const float f = sm == -CUDART_INF_F ? 0.0f : exp2f(sm - top), ft = tm == -CUDART_INF_F ? 0.0f : exp2f(tm - top);
        float l = warp_sum(f != 0.0f ? strand_l[r][lane] * f : 0.0f), a = 0.0f;
#pragma unroll 4
        for (uint32_t i = 0; i < used; ++i) a = fmaf(strands[(r * kStrands + i) * 128u + d], __shfl_sync(0xffffffffu, f, i), a);
        if (tail && ft != 0.0f) {
            float h[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                h[i] = kGroups == 8 ? tail_acc[(i * R + r) * 128 + d] + tail_acc[((i + kGroups - 4) * R + r) * 128 + d] : tail_acc[(i * R + r) * 128 + d];
            a = fmaf((h[0] + h[2]) + (h[1] + h[3]), ft, a);
            l = fmaf(tail_l[r], ft, l);
        }
        if (d < D) store_output(p, (static_cast<uint64_t>(info.row) * p.query_head_count + q_head + r) * D + d, l > 0.0f ? a / l : 0.0f);
        // no visible token: zeros (paged_kv_attention.cu:170-173)
    }
}

// Two fp32 multiply-adds in one instruction.
__device__ __forceinline__ void fma_pair(float2 &acc, float2 a, float2 b) {
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%0, %1};\n\t"
        "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "+f"(acc.x), "+f"(acc.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
}

// Several query tokens of ONE sequence (prefill): a CTA serves 32 rows, the query heads of a kv head for 32 / group
// tokens. They all read the same tail of up to a page, so its two contractions are register-tiled: a thread forms 4 rows x 2
// tokens of the scores from shared memory, and 4 rows x 4 channels of the weighted V rows. (A warp per pair of tokens and a
// block per 16 rows took 366 us for 500 query tokens of 32 heads over 116 tail tokens, most of it index arithmetic and
// reductions; the products alone are 13 us of multiply-adds.)
constexpr uint32_t kTileRows = 32, kTileThreads = 256, kTileTokens = 64, kTileStride = 132, kTileWeights = 36;
inline size_t combine_tile_smem(uint32_t tail_capacity) {
    return (kTileRows * 128u + kTileTokens * kTileStride + static_cast<size_t>((tail_capacity + kTileTokens - 1u) / kTileTokens * kTileTokens) * kTileWeights) * 4u;
}
__global__ void __launch_bounds__(kTileThreads) combine_tile_kernel(AttentionParams p) {
    extern __shared__ __align__(16) float smem_f[];
    float *q = smem_f, *k_tile = q + kTileRows * 128u, *weights = k_tile + kTileTokens * kTileStride;   // weights: [token][36]
    __shared__ uint32_t e_qpos[kTileRows], e_row[kTileRows];
    __shared__ RowPartials r_partials[kTileRows];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t G = p.group, D = p.head_dim, C = p.tail_capacity, quads = D / 4u;
    const uint32_t cta_entries = kTileRows / G, entry0 = blockIdx.x * cta_entries, head_local = blockIdx.y;
    const uint32_t rows = min(cta_entries, p.seq_count - entry0) * G, kv_head = p.kv_head_begin + head_local;
    const SeqInfo info0 = load_seq_info(p, entry0);
    const PageLine line = plan_line(p);
    const uint32_t tail = min(info0.tail, C), sealed = info0.sealed;
    if (tid < kTileRows) {
        const uint32_t seq = entry0 + min(tid, rows - 1u) / G, lq = head_local * G + min(tid, rows - 1u) % G;
        const SeqInfo info = load_seq_info(p, seq);
        e_qpos[tid] = info.qpos;
        e_row[tid] = info.row;
        r_partials[tid] = row_partials(p, line, info, seq, lq);
    }
    __syncthreads();
    const uint64_t base = (static_cast<uint64_t>(info0.slot) * p.kv_head_count + kv_head) * C;
    const uint32_t row0 = 4u * warp;   // this warp's rows
    float m[4], l[4];
    float2 acc[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        m[r] = -CUDART_INF_F;
        l[r] = 0.0f;
        acc[r][0] = acc[r][1] = make_float2(0.0f, 0.0f);
    }
    if (tail) {
        for (uint32_t r = warp; r < kTileRows; r += kTileThreads / 32u)
            for (uint32_t d = lane; d < D; d += 32u) q[r * 128u + d] = r < rows ? load_query(p, e_row[r], kv_head * G + r % G, d) : 0.0f;
        for (uint32_t t0 = 0; t0 < tail; t0 += kTileTokens) {
            const float4 *src = reinterpret_cast<const float4 *>(static_cast<const float *>(p.tail_k) + (base + t0) * D);
            const uint32_t n = min(kTileTokens, tail - t0);
            if (lane < quads) {
#pragma unroll
                for (uint32_t t = warp; t < kTileTokens; t += kTileThreads / 32u)
                    if (t < n) *reinterpret_cast<float4 *>(k_tile + t * kTileStride + 4u * lane) = src[t * quads + lane];
            }
            __syncthreads();
            float2 s[4][2];
#pragma unroll
            for (int r = 0; r < 4; ++r) s[r][0] = s[r][1] = make_float2(0.0f, 0.0f);
#pragma unroll 4
            for (uint32_t c = 0; c < quads; ++c) {
                const float4 ka = *reinterpret_cast<const float4 *>(k_tile + lane * kTileStride + 4u * c);
                const float4 kb = *reinterpret_cast<const float4 *>(k_tile + (lane + 32u) * kTileStride + 4u * c);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float4 qv = *reinterpret_cast<const float4 *>(q + (row0 + r) * 128u + 4u * c);
                    fma_pair(s[r][0], make_float2(qv.x, qv.y), make_float2(ka.x, ka.y));
                    fma_pair(s[r][1], make_float2(qv.x, qv.y), make_float2(kb.x, kb.y));
                    fma_pair(s[r][0], make_float2(qv.z, qv.w), make_float2(ka.z, ka.w));
                    fma_pair(s[r][1], make_float2(qv.z, qv.w), make_float2(kb.z, kb.w));
                }
            }
            __syncthreads();   // the next tile of K rows may come
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t t = t0 + lane + 32u * i, token = sealed + t;
                float w[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const uint32_t qpos = e_qpos[row0 + r];
                    const bool visible = t < tail && token >= window_begin(qpos, p.causal_window) && token <= qpos;
                    w[r] = visible ? (s[r][i].x + s[r][i].y) * p.softmax_scale * kLog2e : -CUDART_INF_F;
                    m[r] = fmaxf(m[r], w[r]);
                }
                *reinterpret_cast<float4 *>(weights + t * kTileWeights + row0) = make_float4(w[0], w[1], w[2], w[3]);
            }
        }
        // this warp's columns of the weights are its own: no barrier from here on
#pragma unroll
        for (int r = 0; r < 4; ++r) m[r] = warp_max(m[r]);
        __syncwarp();
        for (uint32_t t = lane; t < tail; t += 32u) {
            float4 *at = reinterpret_cast<float4 *>(weights + t * kTileWeights + row0);
            const float4 s = *at;
            const float4 w = make_float4(s.x == -CUDART_INF_F ? 0.0f : exp2f(s.x - m[0]), s.y == -CUDART_INF_F ? 0.0f : exp2f(s.y - m[1]),
                                         s.z == -CUDART_INF_F ? 0.0f : exp2f(s.z - m[2]), s.w == -CUDART_INF_F ? 0.0f : exp2f(s.w - m[3]));
            *at = w;
            l[0] += w.x, l[1] += w.y, l[2] += w.z, l[3] += w.w;
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 4; ++r) l[r] = warp_sum(l[r]);
        const float4 *src = reinterpret_cast<const float4 *>(static_cast<const float *>(p.tail_v) + base * D) + lane;
        for (uint32_t t0 = 0; t0 < tail; t0 += 8u) {
            float4 v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = t0 + k < tail && lane < quads ? src[(t0 + k) * quads] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (t0 + k >= tail) break;
                const float4 w4 = *reinterpret_cast<const float4 *>(weights + (t0 + k) * kTileWeights + row0);
                const float w[4] = {w4.x, w4.y, w4.z, w4.w};
                const float2 va = make_float2(v[k].x, v[k].y), vb = make_float2(v[k].z, v[k].w);
                if (w[0] != 0.0f && w[1] != 0.0f && w[2] != 0.0f && w[3] != 0.0f) {
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        fma_pair(acc[r][0], make_float2(w[r], w[r]), va);
                        fma_pair(acc[r][1], make_float2(w[r], w[r]), vb);
                    }
                } else {   // a token the row does not see may hold anything
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (w[r] != 0.0f) {
                            fma_pair(acc[r][0], make_float2(w[r], w[r]), va);
                            fma_pair(acc[r][1], make_float2(w[r], w[r]), vb);
                        }
                }
            }
        }
    }
    wait_for_previous_kernel();
#pragma unroll 1
    for (int r = 0; r < 4; ++r) {
        if (row0 + r >= rows) break;
        const RowPartials rp = r_partials[row0 + r];
        const uint32_t seq = entry0 + (row0 + r) / G, lq = head_local * G + (row0 + r) % G, count = rp.regular + rp.cells;
        float mr = r == 0 ? m[0] : r == 1 ? m[1] : r == 2 ? m[2] : m[3], lr = r == 0 ? l[0] : r == 1 ? l[1] : r == 2 ? l[2] : l[3];
        const float2 a01 = r == 0 ? acc[0][0] : r == 1 ? acc[1][0] : r == 2 ? acc[2][0] : acc[3][0];
        const float2 a23 = r == 0 ? acc[0][1] : r == 1 ? acc[1][1] : r == 2 ? acc[2][1] : acc[3][1];
        float4 a = make_float4(a01.x, a01.y, a23.x, a23.y);
        for (uint32_t c0 = 0; c0 < count; c0 += 32u) {
            float pm = -CUDART_INF_F, pl = 0.0f;
            if (c0 + lane < count) {
                const float *src = partial_of(p, rp, c0 + lane, seq, lq);
                pm = __ldcg(src);
                pl = __ldcg(src + 1);
            }
            const float top = fmaxf(mr, warp_max(pm));
            if (top == -CUDART_INF_F) continue;
            const float keep = exp2f(mr - top), w = exp2f(pm - top);   // -inf gives 0
            mr = top;
            lr = lr * keep + warp_sum(pl * w);
            a.x *= keep, a.y *= keep, a.z *= keep, a.w *= keep;
            const uint32_t n = min(32u, count - c0);
            for (uint32_t i0 = 0; i0 < n; i0 += 4u) {
                float2 x[4][2];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 *src = reinterpret_cast<const float2 *>(partial_of(p, rp, c0 + min(i0 + i, n - 1u), seq, lq) + 2) + 2u * lane;
                    x[i][0] = lane < quads ? __ldcg(src) : make_float2(0.0f, 0.0f);
                    x[i][1] = lane < quads ? __ldcg(src + 1) : make_float2(0.0f, 0.0f);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float wi = __shfl_sync(0xffffffffu, w, (i0 + i) & 31u);
                    if (i0 + i < n && wi != 0.0f) {
                        a.x = fmaf(x[i][0].x, wi, a.x);
                        a.y = fmaf(x[i][0].y, wi, a.y);
                        a.z = fmaf(x[i][1].x, wi, a.z);
                        a.w = fmaf(x[i][1].y, wi, a.w);
                    }
                }
            }
        }
        const float inv = lr > 0.0f ? 1.0f / lr : 0.0f;
        const uint64_t at = (static_cast<uint64_t>(e_row[row0 + r]) * p.query_head_count + kv_head * G + (row0 + r) % G) * D + 4u * lane;
        if (lane < quads) {
            store_output(p, at, a.x * inv);
            store_output(p, at + 1u, a.y * inv);
            store_output(p, at + 2u, a.z * inv);
            store_output(p, at + 3u, a.w * inv);
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
    p->one_slot = 0;
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
    const bool verify = p.shared_prefix_pages != 0u && !p.one_slot;
    if (verify) verify_prefix_kernel<<<p.seq_count, 256, 0, stream>>>(p);
    const uint32_t threads = p.seq_count <= 128u ? 128u : kPlanThreads;   // small batches: fewer warps to start and to meet
    const bool small = p.min_pages_per_unit == 0u &&   // fewer stretches than warps and, as far as the host knows, pages
                       p.layout.chunk_capacity < p.seq_count - 1ull + min(static_cast<uint64_t>(max(p.plan_warps / p.unit_lanes, 1u)),
                                                                         static_cast<uint64_t>(p.seq_count) * p.page_table_stride);
    return launch_kernel(small ? plan_kernel<true> : plan_kernel<false>, 1, threads, 0, stream, verify, p);
}

namespace {

constexpr size_t kCombineSmemMax = 200u * 1024u;

template <class Kernel>
cudaError_t allow_shared_memory(Kernel kernel, std::atomic<uint64_t> &configured) {   // once per device
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (device & 63);
    if (configured.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kCombineSmemMax));
    if (e == cudaSuccess) configured.fetch_or(bit, std::memory_order_release);
    return e;
}

template <int R, int kThreads>
cudaError_t launch_combine_as(const AttentionParams &p, cudaStream_t stream, bool dependent) {
    static std::atomic<uint64_t> configured{0};
    const cudaError_t e = allow_shared_memory(combine_kernel<R, kThreads>, configured);
    if (e != cudaSuccess) return e;
    const dim3 grid(p.seq_count, p.kv_head_span * ((p.group + R - 1u) / R));
    return launch_kernel(combine_kernel<R, kThreads>, grid, kThreads, CombineSmem<R, kThreads>::bytes(p.tail_capacity), stream, dependent, p);
}

}  // namespace

// Four rows per CTA where that still makes about a CTA per SM, or where a CTA per row would not find room for all at once, else one; 32 where all entries are query tokens of one sequence
// (the caller says so), their tail is worth sharing and its rows can be read 16 bytes at a time.
cudaError_t launch_combine(const AttentionParams &p, cudaStream_t stream, bool dependent) {
    const uint32_t sms = p.sm_count, enough_ctas = sms * 13u / 16u;   // 120 of 148
    const uint32_t G = p.group, C = p.tail_capacity;
    const uint32_t tiles = (p.seq_count + kTileRows / G - 1u) / (kTileRows / G) * p.kv_head_span;
    const bool by_16 = p.tail_type == CF_B200_F32 && p.head_dim % 4u == 0u &&
                       ((reinterpret_cast<uintptr_t>(p.tail_k) | reinterpret_cast<uintptr_t>(p.tail_v)) & 15u) == 0u;
    if (p.one_slot && C > 16u && by_16 && tiles >= enough_ctas / 2u && combine_tile_smem(C) <= kCombineSmemMax) {
        static std::atomic<uint64_t> configured{0};
        const cudaError_t e = allow_shared_memory(combine_tile_kernel, configured);
        if (e != cudaSuccess) return e;
        return launch_kernel(combine_tile_kernel, dim3(tiles / p.kv_head_span, p.kv_head_span), kTileThreads, combine_tile_smem(C), stream, dependent, p);
    }
    const uint32_t fours = p.seq_count * p.kv_head_span * ((G + 3u) / 4u);
    if ((fours >= enough_ctas || p.seq_count * p.kv_head_span * G > 2u * sms) && CombineSmem<4, 512>::bytes(C) <= kCombineSmemMax / 2u)
        return fours <= 2u * sms ? launch_combine_as<4, 512>(p, stream, dependent) : launch_combine_as<4, 128>(p, stream, dependent);
    return launch_combine_as<1, 1024>(p, stream, dependent);
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
// one_slot: every entry is a query token of the same sequence (seq_slots repeats one slot). The shared-prefix hint may then name
// pages that the earlier tokens see in part or not at all.
cf_status cfb::sealed_attention_stages(const cf_b200_sealed_attention_desc *d, uint32_t stages, void *stream, bool output_on_peer, bool one_slot) {
    const cf_status valid = cf_b200_sealed_attention_validate(d);
    if (valid != CF_OK) return valid;
    if (stages == 0 || stages > 7u) return CF_ERR_INVALID_ARGUMENT;
    if (!cfb::on_current_device(d->arena) || !cfb::on_current_device(d->workspace) || !cfb::on_current_device(d->queries) ||
        !cfb::on_current_device(d->row_map) || (!output_on_peer && !cfb::on_current_device(d->output)))
        return CF_ERR_INVALID_ARGUMENT;   // memory of another GPU: the call must be made with that GPU current
    AttentionParams p;
    cfb::fill_params(d, &p);
    p.one_slot = one_slot ? 1u : 0u;
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
    // the shared-prefix kernel works on whole records of 16 x 128 or 16 x 64 symbols in blocks of 64, on pages without a window, and
    // reads query rows 16 bytes at a time
    if (use_lanes && p.block_size == 64 && (p.head_dim == 128 || p.head_dim == 64) && d->row_map == nullptr && p.decode_probe != 1u && d->shared_prefix_pages &&
        d->causal_window == 0 && reinterpret_cast<uintptr_t>(d->queries) % 16u == 0)
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
