// The tile kernel for the general law with two kinematic terms.
#include "sbk_tile.cuh"

namespace sbk {

int launch_tile_general2(const Params& p, const TileArgs& a, const TileScratch& s, unsigned grid, cudaStream_t stream) {
  return launch_tile<2>(p, a, s, grid, stream);
}

}  // namespace sbk
