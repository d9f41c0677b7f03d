// tile3d_dispatch.cuh -- which instance of the brick kernel a sweep or round takes.
#pragma once
#include "tile3d_launch.cuh"

namespace pdfs {

template <bool MAIL, int BY, int BZ>
static cudaError_t dispatch_t3(int which, int arith, bool iso, const SweepArgs &a, const Layout &L, int sms,
                               cudaStream_t st, int *g) {
  if (which == 0)
    return iso ? launch_t3<float, 16, BY, BZ, MODE_MIN, ARITH_FAST, true, false, MAIL>(a, L, sms, st, g)
               : launch_t3<float, 16, BY, BZ, MODE_MIN, ARITH_FAST, false, false, MAIL>(a, L, sms, st, g);
  if (which == 1) {
    if (arith == ARITH_REF) return launch_t3<double, 16, BY, BZ, MODE_MIN, ARITH_REF, false, false, MAIL>(a, L, sms, st, g);
    if (arith == ARITH_FAST) return launch_t3<double, 16, BY, BZ, MODE_MIN, ARITH_FAST, false, false, MAIL>(a, L, sms, st, g);
    if (arith == ARITH_PAIR)
      return iso ? launch_t3<double, 16, BY, BZ, MODE_MIN, ARITH_PAIR, true, false, MAIL>(a, L, sms, st, g)
                 : launch_t3<double, 16, BY, BZ, MODE_MIN, ARITH_PAIR, false, false, MAIL>(a, L, sms, st, g);
    return iso ? launch_t3<double, 16, BY, BZ, MODE_MIN, ARITH_MIXED, true, false, MAIL>(a, L, sms, st, g)
               : launch_t3<double, 16, BY, BZ, MODE_MIN, ARITH_MIXED, false, false, MAIL>(a, L, sms, st, g);
  }
  if (arith == ARITH_REF) return launch_t3<double, 16, BY, BZ, MODE_REPLACE, ARITH_REF, false, false, MAIL>(a, L, sms, st, g);
  if (arith == ARITH_FAST) return launch_t3<double, 16, BY, BZ, MODE_REPLACE, ARITH_FAST, false, false, MAIL>(a, L, sms, st, g);
  if (arith == ARITH_PAIR)
    return iso ? launch_t3<double, 16, BY, BZ, MODE_REPLACE, ARITH_PAIR, true, false, MAIL>(a, L, sms, st, g)
               : launch_t3<double, 16, BY, BZ, MODE_REPLACE, ARITH_PAIR, false, false, MAIL>(a, L, sms, st, g);
  return iso ? launch_t3<double, 16, BY, BZ, MODE_REPLACE, ARITH_MIXED, true, false, MAIL>(a, L, sms, st, g)
             : launch_t3<double, 16, BY, BZ, MODE_REPLACE, ARITH_MIXED, false, false, MAIL>(a, L, sms, st, g);
}

template <bool MAIL>
cudaError_t dispatch_bricks(int which, int by, int bz, int arith, bool iso, const SweepArgs &a, const Layout &L, int sms,
                            cudaStream_t st, int *g) {
  if (by == 16 && bz == 16) return dispatch_t3<MAIL, 16, 16>(which, arith, iso, a, L, sms, st, g);
  if (by == 16 && bz == 32) return dispatch_t3<MAIL, 16, 32>(which, arith, iso, a, L, sms, st, g);
  if (by == 8 && bz == 32) return dispatch_t3<MAIL, 8, 32>(which, arith, iso, a, L, sms, st, g);
  if (by == 8 && bz == 48 && which == 0)  // FP32 only
    return iso ? launch_t3<float, 16, 8, 48, MODE_MIN, ARITH_FAST, true, false, MAIL>(a, L, sms, st, g)
               : launch_t3<float, 16, 8, 48, MODE_MIN, ARITH_FAST, false, false, MAIL>(a, L, sms, st, g);
  return cudaErrorInvalidValue;
}

template <bool MAIL, class T, int BZ, int MODE, int ARITH, bool ISO>
static cudaError_t launch_oct(const SweepArgs &a, const Layout &L, int sms, cudaStream_t st, int *grid_used) {
  return launch_t3<T, 16, 16, BZ, MODE, ARITH, ISO, true, MAIL>(a, L, sms, st, grid_used);
}

template <bool MAIL>
cudaError_t dispatch_octant(int which, int arith, bool iso, const SweepArgs &a, const Layout &L, int sms,
                            cudaStream_t st, int *g) {
  if (which == 0)
    return iso ? launch_oct<MAIL, float, 32, MODE_MIN, ARITH_FAST, true>(a, L, sms, st, g)
               : launch_oct<MAIL, float, 32, MODE_MIN, ARITH_FAST, false>(a, L, sms, st, g);
  switch (arith) {
    case ARITH_PAIR:
      return iso ? launch_oct<MAIL, double, 16, MODE_REPLACE, ARITH_PAIR, true>(a, L, sms, st, g)
                 : launch_oct<MAIL, double, 16, MODE_REPLACE, ARITH_PAIR, false>(a, L, sms, st, g);
    case ARITH_MIXED:
      return iso ? launch_oct<MAIL, double, 16, MODE_REPLACE, ARITH_MIXED, true>(a, L, sms, st, g)
                 : launch_oct<MAIL, double, 16, MODE_REPLACE, ARITH_MIXED, false>(a, L, sms, st, g);
    case ARITH_FAST:
      return launch_oct<MAIL, double, 16, MODE_REPLACE, ARITH_FAST, false>(a, L, sms, st, g);
    case ARITH_REF:
      return launch_oct<MAIL, double, 16, MODE_REPLACE, ARITH_REF, false>(a, L, sms, st, g);
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace pdfs
