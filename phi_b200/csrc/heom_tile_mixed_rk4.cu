// The tile kernel's mixed-precision instantiations: apply and RK4 stages.
#include "heom_tile_pipe.cuh"

namespace phi {
namespace tile_detail {
cudaError_t launch_tile_mixed_rk4(const TileParams &p, cudaStream_t stream, int *per_sm) {
  return launch_tile_dispatch<true, kTileRk4, false>(p, stream, per_sm);
}
}  // namespace tile_detail
}  // namespace phi
