// host_rows.cpp — the copy of an append's rows into pinned memory, which looks for NaN and Inf on the way: bound by the
// memory, so the look is free. Two versions, by what the processor has (eight values at a time, or four).
#include "host_rows.h"

#include <string.h>

namespace {

// 32 values a turn in independent accumulators, the shape that compilers turn into vector code.
template <bool kCopy>
inline __attribute__((always_inline)) uint32_t pass(float *dst, const float *src, size_t n) {
    uint32_t m[32] = {};
    size_t i = 0;
    for (; i + 32 <= n; i += 32) {
        uint32_t x[32];
        memcpy(x, src + i, sizeof x);
        if (kCopy) memcpy(dst + i, x, sizeof x);
        for (int j = 0; j < 32; ++j) {
            const uint32_t a = x[j] & 0x7fffffffu;
            m[j] = a > m[j] ? a : m[j];
        }
    }
    uint32_t top = 0;
    for (; i < n; ++i) {
        uint32_t x;
        memcpy(&x, src + i, sizeof x);
        if (kCopy) memcpy(dst + i, &x, sizeof x);
        x &= 0x7fffffffu;
        top = x > top ? x : top;
    }
    for (int j = 0; j < 32; ++j) top = m[j] > top ? m[j] : top;
    return top;
}

#if defined(__x86_64__) || defined(__i386__)
__attribute__((target("avx2"))) uint32_t copy_avx2(float *dst, const float *src, size_t n) { return pass<true>(dst, src, n); }
__attribute__((target("avx2"))) uint32_t look_avx2(float *dst, const float *src, size_t n) { return pass<false>(dst, src, n); }
bool has_avx2() {
    static const bool yes = __builtin_cpu_supports("avx2") != 0;
    return yes;
}
#else   // (a GPU beside Arm cores: what the compiler assumes everywhere there is four values wide already)
uint32_t copy_avx2(float *, const float *, size_t) { return 0; }
uint32_t look_avx2(float *, const float *, size_t) { return 0; }
constexpr bool has_avx2() { return false; }
#endif
uint32_t copy_any(float *dst, const float *src, size_t n) { return pass<true>(dst, src, n); }
uint32_t look_any(float *dst, const float *src, size_t n) { return pass<false>(dst, src, n); }

}  // namespace

uint32_t chromofold_copy_max_magnitude(float *dst, const float *src, size_t n) { return has_avx2() ? copy_avx2(dst, src, n) : copy_any(dst, src, n); }
uint32_t chromofold_max_magnitude(const float *src, size_t n) { return has_avx2() ? look_avx2(nullptr, src, n) : look_any(nullptr, src, n); }
