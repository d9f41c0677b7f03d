// tile3d_launch.cuh -- the launcher of one brick kernel instance (tile3d.cuh), and the
// choice among the instances.
#pragma once
#include <algorithm>

#include "internal.h"
#include "tile3d.cuh"

namespace pdfs {

template <class T, int BX, int BY, int BZ, int MODE, int ARITH, bool ISO, bool OCT, bool MAIL = true>
static cudaError_t launch_t3(const SweepArgs &a, const Layout &L, int sms, cudaStream_t st, int *grid_used) {
  using G = T3GeoOf<T, BX, BY, BZ, ARITH>;
  auto kern = t3_sweep_kernel<T, BX, BY, BZ, MODE, ARITH, ISO, OCT, MAIL>;
  CUtensorMap m;
  cudaError_t e = encode_field_map(&m, a.u, sizeof(T), L, a.nz + 2, G::W, G::RY, G::RZ);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::BYTES);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, G::NT, G::BYTES);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  // every CTA resident: a ticket waits only on smaller tickets
  const long long tickets = (OCT && a.nticket ? (long long)kOctMax : 1) * a.ntx * a.nty * a.ntz;
  const int grid = (int)std::max(1ll, std::min((long long)per_sm * sms, tickets));
  kern<<<grid, G::NT, G::BYTES, st>>>(m, a);
  if (grid_used) *grid_used = grid;
  return cudaGetLastError();
}

// The instances of the selectable bricks (by x bz) and of octant rounds: with mailboxes
// (tile3d.cu) and without (tile3d_flags.cu).
template <bool MAIL>
cudaError_t dispatch_bricks(int which, int by, int bz, int arith, bool iso, const SweepArgs &a, const Layout &L, int sms,
                            cudaStream_t st, int *g);
template <bool MAIL>
cudaError_t dispatch_octant(int which, int arith, bool iso, const SweepArgs &a, const Layout &L, int sms,
                            cudaStream_t st, int *g);

}  // namespace pdfs
