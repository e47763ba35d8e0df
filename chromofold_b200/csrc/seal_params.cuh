// seal_params.cuh — what the page sealers (seal.cu, seal_blocks.cu) share: launch parameters, the stream scale and the
// quantiser, and the seam through which a sequence store seals many pages of a prompt in one launch.
#ifndef CHROMOFOLD_B200_SEAL_PARAMS_CUH
#define CHROMOFOLD_B200_SEAL_PARAMS_CUH

#include "cf_device_common.cuh"

namespace cfb {

__host__ __device__ inline bool split_coder(uint32_t coder) {
    return coder == CF_B200_CODER_RANS_SPLIT4 || coder == CF_B200_CODER_HUFFMAN_SPLIT4;
}
__host__ __device__ inline bool rans_family(uint32_t coder) { return coder == CF_B200_CODER_RANS || coder == CF_B200_CODER_RANS_SPLIT4; }

struct SealParams {
    uint32_t kv_head_count, head_dim, page_tokens, block_size, coder, codebook_id, symbols, nblocks;
    const cf_b200_codebook_tables *k_tables, *v_tables;
    const void *tail_k, *tail_v;
    uint32_t tail_type, tail_capacity;
    uint64_t slot_stride, head_stride, row_stride;   // of tail_k / tail_v, in elements
    const uint32_t *job_slots, *job_pages, *job_tokens, *job_heads, *job_rows;
    uint32_t job_count;
    uint8_t *arena;
    uint64_t arena_units;
    unsigned long long *cursor;
    uint64_t *page_dir;
    uint32_t *status;
};

// Many full pages of one sequence straight from its rows: tile j = rows 16 j .. 16 j + 15 of tail_k / tail_v, in page
// j / tiles_per_page of the list, whose arena slot is page_slot[]. Every record has a fixed place in its slot (the slots are
// sized for the largest records), so nothing is counted or read back to place it.
constexpr uint32_t kBulkPages = 512;   // pages per launch: the list travels with the launch
struct SealPlacement {
    uint32_t tiles_per_page, record_units;   // 16-byte units of the largest record
    uint32_t *table_row;                     // the sequence's page-table row at its first new tile
    uint32_t *used;                          // [tile][kv head]: record units, or kSealRefused for a non-finite tile; behind
                                             // them the status word as the launch found it
    uint32_t page_slot[kBulkPages];
};
constexpr uint32_t kSealRefused = 0xffffffffu;

#ifdef __CUDACC__
__device__ __forceinline__ uint16_t scale_bits_from_absmax(float maximum) {
    if (maximum == 0.0f) return 0x3c00u;  // all-zero stream: scale 1 (kv_gpu_fixture.cpp:70)
    uint16_t bits = __half_as_ushort(__float2half_rn(__fdiv_rn(maximum, 127.0f)));
    if (bits == 0) bits = 1;
    if ((bits & 0x7c00u) == 0x7c00u) bits = 0x7bffu;
    return bits;
}
__device__ __forceinline__ uint32_t quantise_symbol(float x, float scale) {
    int q = __float2int_rn(__fdiv_rn(x, scale));
    q = max(-128, min(127, q));
    return static_cast<uint32_t>(q + kZero);
}
#endif

// Implemented in seal_blocks.cu
bool seal_blocks_supports(const SealParams &p);   // 16-token pages, 64-symbol blocks, head_dim 128 / 96 / 80 / 64 / 32, aligned rows
cudaError_t launch_seal_blocks(const SealParams &p, cudaStream_t stream);
cudaError_t launch_seal_placed(const SealParams &p, const SealPlacement &place, cudaStream_t stream);

}  // namespace cfb

#endif
