// trail_tile_128t.cu - the shared-memory trail tiles 128 columns wide, 32 and
// 64 rows tall.
#include "trail_tile.cuh"

namespace slime {
cudaError_t launch_tile_128x32(SLIME_TILE_ARGS) { return launch_tile<128, 32>(p, in, counts, marks, o, s, win); }
cudaError_t launch_tile_128x64(SLIME_TILE_ARGS) { return launch_tile<128, 64>(p, in, counts, marks, o, s, win); }
} // namespace slime
