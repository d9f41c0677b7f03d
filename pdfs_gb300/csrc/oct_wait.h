/* oct_wait.h -- which earlier sweep of a round a brick has to wait for (host and
 * device code: the CPU tests compile it by themselves). */
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define PDFS_HD __host__ __device__ __forceinline__
#else
#define PDFS_HD inline
#endif

namespace pdfs {

/* The latest sweep before sweep osw of a round that visits brick n, or -1.  Sweep j
 * runs ordering (first + j) % 8 and visits every brick when bit j of full is set,
 * else those whose bits in tbits (one byte per brick) name its ordering.  tbits is
 * read only where full does not answer: a round of one sweep, or of full sweeps
 * alone, has none and passes nullptr. */
PDFS_HD int oct_latest(int osw, int first, unsigned full, const uint8_t *tbits, int n) {
  if (osw <= 0) return -1;
  if ((full >> (osw - 1)) & 1u) return osw - 1;
#ifdef __CUDA_ARCH__
  const unsigned tb = __ldg(tbits + n);
#else
  const unsigned tb = tbits[n];
#endif
  for (int j = osw - 1; j >= 0; --j)
    if (((full >> j) & 1u) || ((tb >> ((first + j) % 8)) & 1u)) return j;
  return -1;
}

}  // namespace pdfs
