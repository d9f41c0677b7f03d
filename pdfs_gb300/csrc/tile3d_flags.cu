// tile3d_flags.cu -- the brick sweeps and octant rounds without mailboxes: bricks wait
// for whole upwind bricks (tile3d.cuh, MAIL false).
#include "tile3d_dispatch.cuh"

namespace pdfs {

template cudaError_t dispatch_bricks<false>(int, int, int, int, bool, const SweepArgs &, const Layout &, int, cudaStream_t,
                                            int *);
template cudaError_t dispatch_octant<false>(int, int, bool, const SweepArgs &, const Layout &, int, cudaStream_t, int *);

}  // namespace pdfs
