// trail_tile_64.cu - the shared-memory trail tiles 64 columns wide.
#include "trail_tile.cuh"

namespace slime {
cudaError_t launch_tile_64x8(SLIME_TILE_ARGS) { return launch_tile<64, 8>(p, in, counts, marks, o, s, win); }
cudaError_t launch_tile_64x16(SLIME_TILE_ARGS) { return launch_tile<64, 16>(p, in, counts, marks, o, s, win); }
cudaError_t launch_tile_64x32(SLIME_TILE_ARGS) { return launch_tile<64, 32>(p, in, counts, marks, o, s, win); }
} // namespace slime
