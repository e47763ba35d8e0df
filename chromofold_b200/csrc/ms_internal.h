// ms_internal.h — what the host caches (ms_host_cache.cpp) use of the device sequence store (ms_resolver.cu) beyond its C ABI.
#ifndef CHROMOFOLD_B200_MS_INTERNAL_H
#define CHROMOFOLD_B200_MS_INTERNAL_H

#include "chromofold_b200/compat_ms.h"

namespace cfb_engine {

// cf_b200_ms_append_active_async and, whenever the active page is full, cf_b200_ms_seal_active_async, for any number of dense
// fp32 rows [token][kv head][dim] in device memory at once: pages the rows fill are sealed from where they lie, in one launch.
// The outcome is that of the two calls page by page, a refused page included: the pages before it stay sealed, its rows are
// the (full) active page.
int ms_append_rows(cf_ms_cuda_resolver *r, int64_t id, uint32_t layer, uint32_t token_begin, const float *keys, const float *values,
                   uint32_t token_count, void *stream);

}  // namespace cfb_engine

#endif
