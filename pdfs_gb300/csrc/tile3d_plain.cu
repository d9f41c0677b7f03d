// tile3d_plain.cu -- plain sweeps on bricks: every node, no block mask and no
// block-change output.  They run on the round kernel (tile3d.cuh, OCT) as a round
// of one sweep: it carries no block-change bookkeeping.
#include "tile3d_launch.cuh"

namespace pdfs {

// The ordering (1..8) that sweeps in these directions.
static int ordering_of(int sx, int sy, int sz) {
  for (int sn = 1; sn <= 8; ++sn) {
    int x, y, z;
    ordering_signs(sn, &x, &y, &z);
    if (x == sx && y == sy && z == sz) return sn;
  }
  return 1;
}

template <int MODE>
static cudaError_t plain64(int b, int bz, int arith, bool iso, const SweepArgs &a, const Layout &L, int sms,
                           cudaStream_t st, int *g) {
  if (b == 8 && bz == 16) {
    if (arith == ARITH_REF) return launch_t3<double, 8, 8, 16, MODE, ARITH_REF, false, true>(a, L, sms, st, g);
    if (arith == ARITH_FAST) return launch_t3<double, 8, 8, 16, MODE, ARITH_FAST, false, true>(a, L, sms, st, g);
  }
  if (b == 16 && bz == 32) {
    if (arith == ARITH_MIXED)
      return iso ? launch_t3<double, 16, 16, 32, MODE, ARITH_MIXED, true, true>(a, L, sms, st, g)
                 : launch_t3<double, 16, 16, 32, MODE, ARITH_MIXED, false, true>(a, L, sms, st, g);
    if (arith == ARITH_PAIR)
      return iso ? launch_t3<double, 16, 16, 32, MODE, ARITH_PAIR, true, true>(a, L, sms, st, g)
                 : launch_t3<double, 16, 16, 32, MODE, ARITH_PAIR, false, true>(a, L, sms, st, g);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_sweep_plain(int which, int b, int bz, int arith, bool iso, const SweepArgs &a0, const Layout &L,
                               int sms, cudaStream_t st, int *g) {
  if (!a0.pmail || !a0.torder || a0.ntx < 1 || a0.nty < 1 || a0.ntz < 1 || L.tx != 16 || L.ty != 16 || L.xo != 0 ||
      a0.blk_active || a0.blk_chg || a0.ntz != (a0.nz + bz - 1) / bz || (which == 2 && (!a0.bcap64 || !a0.bcap32)) ||
      (long long)a0.ntx * a0.nty * a0.ntz >= (1ll << 27))
    return cudaErrorInvalidValue;
  SweepArgs a = a0;
  a.oct_first = ordering_of(a.sx, a.sy, a.sz) - 1;
  a.oct_full = 1u;
  a.tflag = nullptr;  // no later sweep waits for its flags
  a.nticket = nullptr;
  a.tact = nullptr;
  if (which == 0 && b == 8 && bz == 32)
    return iso ? launch_t3<float, 8, 8, 32, MODE_MIN, ARITH_FAST, true, true>(a, L, sms, st, g)
               : launch_t3<float, 8, 8, 32, MODE_MIN, ARITH_FAST, false, true>(a, L, sms, st, g);
  if (which == 0 && b == 16 && bz == 32)
    return iso ? launch_t3<float, 16, 16, 32, MODE_MIN, ARITH_FAST, true, true>(a, L, sms, st, g)
               : launch_t3<float, 16, 16, 32, MODE_MIN, ARITH_FAST, false, true>(a, L, sms, st, g);
  if (which == 0) return cudaErrorInvalidValue;
  return which == 2 ? plain64<MODE_REPLACE>(b, bz, arith, iso, a, L, sms, st, g)
                    : plain64<MODE_MIN>(b, bz, arith, iso, a, L, sms, st, g);
}

}  // namespace pdfs
