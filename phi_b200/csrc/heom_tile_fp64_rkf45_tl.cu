// The tile kernel's FP64 instantiations: RKF45 stages of
// time-local runs.
#include "heom_tile_pipe.cuh"

namespace phi {
namespace tile_detail {
cudaError_t launch_tile_fp64_rkf45_tl(const TileParams &p, cudaStream_t stream, int *per_sm) {
  return launch_tile_dispatch<false, kTileRkf45, true>(p, stream, per_sm);
}
}  // namespace tile_detail
}  // namespace phi
