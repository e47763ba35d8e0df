// host_rows.h — passes over fp32 rows in host memory (host_rows.cpp).
#ifndef CHROMOFOLD_B200_HOST_ROWS_H
#define CHROMOFOLD_B200_HOST_ROWS_H

#include <stddef.h>
#include <stdint.h>

// Largest magnitude of n floats, as bits: above 0x7f7fffff if one of them is NaN or Inf. The first also copies them.
uint32_t chromofold_copy_max_magnitude(float *dst, const float *src, size_t n);
uint32_t chromofold_max_magnitude(const float *src, size_t n);

#endif
