// trail_tile_128.cu - the shared-memory trail tiles 128 columns wide.
#include "trail_tile.cuh"

namespace slime {
cudaError_t launch_tile_128x8(SLIME_TILE_ARGS) { return launch_tile<128, 8>(p, in, counts, marks, o, s, win); }
cudaError_t launch_tile_128x16(SLIME_TILE_ARGS) { return launch_tile<128, 16>(p, in, counts, marks, o, s, win); }
} // namespace slime
