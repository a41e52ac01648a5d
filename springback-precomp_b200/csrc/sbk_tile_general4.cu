// The tile kernel for the general law with up to four kinematic terms.
#include "sbk_tile.cuh"

namespace sbk {

int launch_tile_general4(const Params& p, const TileArgs& a, const TileScratch& s, unsigned grid, cudaStream_t stream) {
  return launch_tile<4>(p, a, s, grid, stream);
}

}  // namespace sbk
