// compat_paged_mma.cuh — the tensor-core form of cf_kv_paged_attention_async (compat_paged_mma.cu) as compat_kv.cu calls it.
#ifndef CHROMOFOLD_B200_COMPAT_PAGED_MMA_CUH
#define CHROMOFOLD_B200_COMPAT_PAGED_MMA_CUH

#include <cuda_runtime.h>

#include "chromofold_b200/compat_kv.h"

namespace cfb {

// head_dim 128 and 64: the fragment layout gives every lane 32 / 16 channels of K and 16 / 8 of V, i.e. whole words.
bool paged_mma_supports(const cf_kv_paged_attention_desc &d);
// Splits of the tokens that fill the GPU (before the caller bounds them by the room for partials).
uint32_t paged_mma_splits(const cf_kv_paged_attention_desc &d, int sm_count);
// With splits > 1 every (query token, query head) leaves (max, sum, weighted[head_dim]) per split in `partials`, and the last CTA
// of a 16-row tile merges them; `arrived` counts the CTAs of each tile (kPagedMmaCounters words, zero before and after).
constexpr uint32_t kPagedMmaCounters = 1024;   // splits > 1 only where the tiles alone do not give every SM two CTAs
cudaError_t launch_paged_mma(const cf_kv_paged_attention_desc &d, uint32_t splits, float *partials, uint32_t *arrived, cudaStream_t stream);

}  // namespace cfb

#endif
