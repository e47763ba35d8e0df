// attention_params.cuh — launch parameters shared by the plan, attention and combine kernels.
#ifndef CHROMOFOLD_B200_ATTENTION_PARAMS_CUH
#define CHROMOFOLD_B200_ATTENTION_PARAMS_CUH

#include "cf_device_common.cuh"

namespace cfb {

constexpr uint32_t kDefaultWaitPolls = 1u << 22;   // about a microsecond each at most: seconds before a wait gives up

struct AttentionParams {
    // geometry
    uint32_t kv_head_count, query_head_count, head_dim, page_tokens, block_size;
    uint32_t kv_head_begin, kv_head_span, group;  // group = query heads per kv head
    uint32_t symbols, nblocks, codebook_id;
    // sealed pages
    const uint8_t *arena;
    const uint64_t *page_dir;
    const uint32_t *page_table;
    const uint32_t *seq_sealed_tokens;
    const uint32_t *seq_slots;
    uint32_t page_table_stride, seq_count;
    const cf_b200_codebook_tables *k_tables, *v_tables;
    // tails
    const void *tail_k, *tail_v;
    const uint32_t *tail_tokens;
    uint32_t tail_type, tail_capacity;
    const uint32_t *query_positions;
    const uint32_t *row_map;        // optional: batch entry -> row of queries / output
    // io
    const void *queries;
    void *output;
    uint32_t query_type, output_type;
    float softmax_scale;
    uint32_t causal_window;
    // split-KV
    uint8_t *workspace;
    WorkspaceLayout layout;
    uint32_t min_pages_per_unit;    // 0 = the line of pages is cut evenly over plan_warps (PageLine)
    uint32_t plan_warps;            // warps (any-geometry kernel: CTAs) that are resident at once in the attention kernel
    uint32_t unit_lanes;            // units that share a stretch: kv heads x passes over a kv head's query group
    uint32_t shared_prefix_pages;   // the caller's hint, already zeroed when the launch cannot use it
    uint32_t one_slot;              // 1: every entry is a query token of the same sequence
    uint32_t sm_count;
    uint32_t decode_probe;          // 1 = measurement: decode every page, fold the symbols into a checksum, no attention;
                                    // 2 = test: store every decoded symbol to `output` ([page id][kv head][K | V stream])
    uint32_t dump_pages;            // page ids the dump buffer covers (1 when decode_probe != 2)
    uint32_t wait_polls;            // bound of every wait on a copy or a barrier, in polls
    uint32_t skip_copy_page;        // test hook: the record of this page id is never fetched (its wait must run out); 0 = off
    uint32_t *status;
    // uncompressed comparison pools (dense kernel only)
    const __half *pool_k, *pool_v;
};

#ifdef __CUDACC__
__device__ __forceinline__ PlanHeader *plan_header(const AttentionParams &p) {
    return reinterpret_cast<PlanHeader *>(p.workspace);
}
__device__ __forceinline__ uint32_t *line_prefix(const AttentionParams &p) {
    return reinterpret_cast<uint32_t *>(p.workspace + p.layout.prefix_offset);
}
__device__ __forceinline__ SeqInfo *seq_info(const AttentionParams &p) {
    return reinterpret_cast<SeqInfo *>(p.workspace + p.layout.info_offset);
}
__device__ __forceinline__ float *partial_ptr(const AttentionParams &p, uint32_t slot, uint32_t local_q_head) {
    return reinterpret_cast<float *>(p.workspace + p.layout.partials_offset) +
           (static_cast<uint64_t>(slot) * (p.kv_head_span * p.group) + local_q_head) * p.layout.partial_stride_floats;
}
// Shared-prefix partial of (cell, batch entry, local query head); cells as SharedSplit numbers them.
__device__ __forceinline__ float *shared_partial_ptr(const AttentionParams &p, uint32_t chunk, uint32_t seq, uint32_t local_q_head) {
    return reinterpret_cast<float *>(p.workspace + p.layout.shared_offset) +
           ((static_cast<uint64_t>(chunk) * p.seq_count + seq) * (p.kv_head_span * p.group) + local_q_head) *
               p.layout.partial_stride_floats;
}
// Row of the query and output tensors that batch entry `seq` stands for.
__device__ __forceinline__ uint32_t row_of(const AttentionParams &p, uint32_t seq) {
    return p.row_map ? p.row_map[seq] : seq;
}
__device__ __forceinline__ uint32_t slot_of(const AttentionParams &p, uint32_t seq) {
    return p.seq_slots ? p.seq_slots[seq] : seq;
}
// Position of the query token of batch entry `seq`: given, or right after everything cached (a decode step).
__device__ __forceinline__ uint32_t query_position(const AttentionParams &p, uint32_t seq, uint32_t sealed, uint32_t tail) {
    return p.query_positions ? p.query_positions[seq] : sealed + tail;
}
__device__ __forceinline__ float load_tail(const void *base, uint32_t type, uint64_t i) {
    return type == CF_B200_F32 ? static_cast<const float *>(base)[i] : __half2float(static_cast<const __half *>(base)[i]);
}
__device__ __forceinline__ void raise_status(const AttentionParams &p, uint32_t bits) {
    if (p.status) atomicOr(p.status, bits);
}
// The sequence that holds line position x: the last s with line_prefix[s] <= x. Whole warps, 32 probes at a time.
__device__ __forceinline__ uint32_t sequence_at(const uint32_t *prefix, uint32_t seq_count, uint32_t x, uint32_t lane) {
    uint32_t lo = 0, hi = seq_count;
    while (hi - lo > 1u) {
        const uint32_t step = (hi - lo + 31u) / 32u, at = lo + (lane + 1u) * step;
        const uint32_t below = __popc(__ballot_sync(0xffffffffu, at < hi && __ldcg(prefix + at) <= x));
        lo += below * step;
        hi = min(lo + step, hi);
    }
    return lo;
}
// The part of a stretch inside one sequence: positions [x, x_end) of the line, pages [page, page_end) of the entry.
struct LineRun {
    uint32_t x, x_end, seq, page, page_end;
    SeqInfo info;
};
// The run that starts at position x and ends at x_stop (the stretch's end) at the latest. Whole warps.
__device__ __forceinline__ LineRun run_at(const AttentionParams &p, uint32_t x, uint32_t x_stop, uint32_t grain, uint32_t lane) {
    LineRun run;
    run.x = x;
    run.seq = sequence_at(line_prefix(p), p.seq_count, x, lane);
    const uint4 *src = reinterpret_cast<const uint4 *>(seq_info(p) + run.seq);
    const uint4 a = __ldcg(src), b = __ldcg(src + 1);
    run.info.slot = a.x, run.info.sealed = a.y, run.info.qpos = a.z, run.info.tail = a.w;
    run.info.first_page = b.x, run.info.page_end = b.y, run.info.row = b.z, run.info.line_begin = b.w;
    const uint32_t length = b.y - b.x, positions = grain == 1u ? length : (length + grain - 1u) / grain;
    run.x_end = min(x_stop, b.w + positions);
    run.page = b.x + (x - b.w) * grain;
    run.page_end = min(b.x + (run.x_end - b.w) * grain, b.y);
    return run;
}
// The plan's line, past every level-1 cache: the kernels that read it may have started before the plan kernel ended.
__device__ __forceinline__ PageLine plan_line(const AttentionParams &p) {
    const uint4 *src = reinterpret_cast<const uint4 *>(p.workspace);
    const uint4 a = __ldcg(src), b = __ldcg(src + 1);
    PageLine line;
    line.positions = a.x, line.grain = a.y, line.stretches = a.z, line.base = a.w;
    line.longer = b.x, line.pieces = b.y, line.by_position = b.z;
    return line;
}
#endif

// Implemented in sealed_attention.cu
cf_status sealed_attention_stages(const cf_b200_sealed_attention_desc *d, uint32_t stages, void *stream, bool output_on_peer, bool one_slot = false);
// dependent: the kernel before it on the stream belongs to the same call and lets this one start early.
cudaError_t launch_plan(const AttentionParams &p, cudaStream_t stream);
cudaError_t launch_combine(const AttentionParams &p, cudaStream_t stream, bool dependent);
cudaError_t launch_generic_attention(const AttentionParams &p, cudaStream_t stream);
constexpr uint32_t kGenericCtasPerSm = 4;
// Implemented in sealed_attention_lanes.cu
bool lanes_kernel_supports(const AttentionParams &p);
void lanes_plan_shape(const AttentionParams &p, uint32_t sm_count, uint32_t *warps, uint32_t *unit_lanes);
cudaError_t launch_lanes_attention(const AttentionParams &p, cudaStream_t stream, bool dependent, bool after_prefix);
// Implemented in sealed_attention_prefix.cu
cudaError_t launch_prefix_attention(const AttentionParams &p, cudaStream_t stream, bool dependent);
// Implemented in dense_attention.cu
cudaError_t launch_dense_attention(const AttentionParams &p, cudaStream_t stream);

}  // namespace cfb

#endif
