// The tile kernel for the general law without kinematic terms (Hill48).
#include "sbk_tile.cuh"

namespace sbk {

int launch_tile_general0(const Params& p, const TileArgs& a, const TileScratch& s, unsigned grid, cudaStream_t stream) {
  return launch_tile<0>(p, a, s, grid, stream);
}

}  // namespace sbk
