// The tile kernel for the general law with one kinematic term.
#include "sbk_tile.cuh"

namespace sbk {

int launch_tile_general1(const Params& p, const TileArgs& a, const TileScratch& s, unsigned grid, cudaStream_t stream) {
  return launch_tile<1>(p, a, s, grid, stream);
}

}  // namespace sbk
