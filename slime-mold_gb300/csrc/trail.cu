// trail.cu - fused deposit-fold + decay + diffuse.
//
// The reference runs decay_trail (compute.wgsl:148-161) and diffuse_trail
// (compute.wgsl:164-195) as two full passes over the trail, the blur in place.
// Here one kernel reads the pre-step trail and the step's deposit record once,
// applies the sequential deposit fold and the decay, blurs, writes the new
// trail to the other buffer and zeroes the other step's record: rows streamed
// through registers (trail_stream.cuh), tiles staged in shared memory
// (trail_tile.cuh) or by tensor copies (trail_tma.cu).
// HBM traffic per cell: 4 B trail in + 4 B out, and 4 B read + 4 B zeroed of
// counts or 1 B + 1 B of marks; halo re-reads hit L2.
//
// Box mode sums the nine taps in the shader's order (dy outer, dx inner,
// starting from 0.0) and divides by 9.0, so it matches the shader's arithmetic
// bit for bit; Gaussian mode is separable (horizontal then vertical, fused
// multiply-adds over taps -R..R).
#include "kernels.h"
#include "trail_stream.cuh"
#include "trail_tile.cuh"

namespace slime {
namespace {

template <int R, bool kGauss, int ROWS, class D>
__global__ void __launch_bounds__(128) trail_stream_kernel(const __grid_constant__ DevParams p,
                                                           const float* __restrict__ in, const D* __restrict__ cin,
                                                           float* __restrict__ out, D* __restrict__ czero,
                                                           int warps_x) {
    const int gw = blockIdx.x * 4 + (threadIdx.x >> 5);
    // the deposit record this reads is the agent pass's output
    pdl_wait();
    pdl_trigger();
    process_strip<R, kGauss, ROWS, false, true, D>(p, in, cin, out, czero, gw % warps_x, gw / warps_x);
}

template <int R, bool kGauss, int ROWS, class D>
cudaError_t launch_stream(const DevParams& p, const float* in, const D* cin, float* out, D* cz, cudaStream_t s,
                          const cudaAccessPolicyWindow* win, bool pdl) {
    int warps_x = (p.W + 127) / 128;
    long long warps = (long long)warps_x * ((p.H + ROWS - 1) / ROWS);
    unsigned blocks = (unsigned)((warps + 3) / 4);
    return launch_kp(trail_stream_kernel<R, kGauss, ROWS, D>, dim3(blocks), dim3(128), 0, s, win, pdl, p, in, cin,
                     out, cz, warps_x);
}

template <int ROWS, class D>
cudaError_t launch_stream_rows(const DevParams& p, const float* in, const D* cin, float* out, D* cz, cudaStream_t s,
                               const cudaAccessPolicyWindow* win, bool pdl) {
    if (p.blur_mode != SLIME_BLUR_GAUSS) return launch_stream<1, false, ROWS, D>(p, in, cin, out, cz, s, win, pdl);
    if (p.R == 1) return launch_stream<1, true, ROWS, D>(p, in, cin, out, cz, s, win, pdl);
    return launch_stream<2, true, ROWS, D>(p, in, cin, out, cz, s, win, pdl);
}

// Sets *flag where a value is negative or NaN.
__global__ void trail_check_kernel(const float* __restrict__ t, uint64_t n, uint32_t* __restrict__ flag) {
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    bool bad = false;
#pragma unroll 4
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) bad |= !(__ldg(t + i) >= 0.0f);
    if (bad) *flag = 1;
}

const TrailTile kTiles[] = {{64, 8}, {64, 16}, {64, 32}, {128, 8}, {128, 16}, {128, 32}, {128, 64}};
constexpr int kNumTiles = (int)(sizeof(kTiles) / sizeof(kTiles[0]));

cudaError_t launch_tile_index(int tile, SLIME_TILE_ARGS) {
    switch (tile) {
    case 0: return launch_tile_64x8(p, in, counts, marks, o, s, win);
    case 1: return launch_tile_64x16(p, in, counts, marks, o, s, win);
    case 2: return launch_tile_64x32(p, in, counts, marks, o, s, win);
    case 3: return launch_tile_128x8(p, in, counts, marks, o, s, win);
    case 4: return launch_tile_128x16(p, in, counts, marks, o, s, win);
    case 5: return launch_tile_128x32(p, in, counts, marks, o, s, win);
    default: return launch_tile_128x64(p, in, counts, marks, o, s, win);
    }
}

} // namespace

// Tile table: entries 0..kNumTiles-1 are the shared-memory tiles, the next
// kNumStream entries the streaming kernel with 8, 16 and 32 rows per strip,
// the last one (kTrailTileTma) the tensor-copy tile of 128 x 32 cells.
constexpr int kNumStream = 3;
static_assert(kNumTiles + kNumStream == kTrailTileTma, "the tensor-copy tile follows the streaming ones");
int trail_tile_count() { return kNumTiles + kNumStream + 1; }
TrailTile trail_tile(int index) {
    if (index == kTrailTileTma) return TrailTile{128, 32};
    if (index >= kNumTiles && index < kNumTiles + kNumStream) return TrailTile{128, 8 << (index - kNumTiles)};
    return kTiles[(index >= 0 && index < kNumTiles) ? index : 0];
}
// Measured as whole steps of one agent (us; tile 4 = 128 x 16, 5 = 128 x 32,
// 7 = 8-row strips), each side of the lines drawn here:
//   box, tile 4 / 5 / 7: 512^2 4.0 / 4.5 / 4.8, 1600x900 5.6 / 5.7 / 6.2,
//     2048^2 11.3 / 9.7 / 9.8, 4096^2 42.7 / 37.5 / 32.7 (the strips walk
//     their rows one after another, which only a large grid hides);
//   Gaussian radius 1, marks, 4 / 7: 512^2 4.0 / 3.7, 2048^2 10.9 / 7.3;
//     counts (four times the registers a row): 512^2 4.4 / 6.1,
//     1600x900 6.4 / 6.5, 2048^2 12.5 / 9.9;
//   what strips cannot run, 4 / 5: radius 5 1600x900 7.5 / 7.3, 2048^2
//     15.5 / 13.1; radius 1 3001x2003 18.9 / 20.9, radius 2 19.9 / 17.9.
int trail_tile_default(const DevParams& p, bool marks, bool aligned) {
    const int64_t cells = (int64_t)p.W * p.H;
    const bool gauss = p.blur_mode == SLIME_BLUR_GAUSS;
    const int64_t strips_from = gauss ? (marks ? 0 : 2000000) : 6000000;
    if (aligned && cells >= strips_from && trail_tile_supported(p, kNumTiles)) return kNumTiles;
    return cells < 2000000 || (gauss && p.R == 1) ? 4 : 5;
}
int trail_tile_strips(const DevParams& p) { return trail_tile_supported(p, kNumTiles) ? kNumTiles : -1; }
bool trail_tile_supported(const DevParams& p, int tile) {
    if (tile == kTrailTileTma) return trail_tma_supported(p);
    if (tile < 0 || tile >= kNumTiles + kNumStream) return false;
    if (tile < kNumTiles) return true;
    // streaming kernel: whole float4 groups per row and radius <= 2, grid
    // wider than a halo
    int R = p.blur_mode == SLIME_BLUR_GAUSS ? p.R : 1;
    return (p.W % 4) == 0 && p.W >= 8 && R >= 1 && R <= 2 && p.H >= 1;
}

bool trail_tile_streams(const DevParams& p, int tile) { return tile >= kNumTiles && trail_tile_supported(p, tile); }

// Whether the values of an uploaded trail are looked at on the device, where
// they just arrived, or by the host (which deposit marks want finite and >= 0,
// or +inf).  An upload takes, host (a scalar loop; an OR
// over all values, which vectorises, takes 10 us less at 256^2) / device: 128^2
// 15.5 / 28.7 us, 256^2 40.9 / 30.3, 512^2 117 / 35, 1024^2 431 / 53, 4096^2
// 6689 / 423 (of which the copy takes all but 20).
bool device_check_pays(uint64_t cells) { return cells >= 65536; }
cudaError_t launch_trail_check(const float* t, uint64_t n, uint32_t* flag, cudaStream_t s) {
    const uint64_t blocks = (n + 1023) / 1024;
    trail_check_kernel<<<(unsigned)(blocks < 1216 ? blocks : 1216), 256, 0, s>>>(t, n, flag);
    return cudaGetLastError();
}

cudaError_t launch_trail_marks(const DevParams& p, int tile, const float* in, const uint8_t* marks_in, float* out,
                               uint8_t* marks_zero, cudaStream_t s, const cudaAccessPolicyWindow* win, bool pdl,
                               const TrailMaps* maps, int cur) {
    if (!trail_tile_supported(p, tile)) tile = trail_tile_default(p, true);
    // without tensor maps, the 8-row streaming tile (same requirements, same bits)
    if (tile == kTrailTileTma && !(maps && maps->ok)) tile = kNumTiles;
    switch (tile) {
    case 7: return launch_stream_rows<8>(p, in, marks_in, out, marks_zero, s, win, pdl);
    case 8: return launch_stream_rows<16>(p, in, marks_in, out, marks_zero, s, win, pdl);
    case 9: return launch_stream_rows<32>(p, in, marks_in, out, marks_zero, s, win, pdl);
    case kTrailTileTma: return launch_trail_tma_marks(p, *maps, cur, in, marks_in, out, marks_zero, s, win, pdl);
    default: return launch_tile_index(tile, p, in, nullptr, marks_in, TileOut{out, nullptr, marks_zero}, s, win);
    }
}

cudaError_t launch_trail(const DevParams& p, int tile, const float* in, const uint32_t* counts_in, float* out,
                         uint32_t* counts_zero, cudaStream_t s, const cudaAccessPolicyWindow* win, bool pdl,
                         const TrailMaps* maps, int cur) {
    if (!trail_tile_supported(p, tile)) tile = trail_tile_default(p, false);
    if (tile == kTrailTileTma && !(maps && maps->ok)) tile = kNumTiles;
    switch (tile) {
    case 7: return launch_stream_rows<8>(p, in, counts_in, out, counts_zero, s, win, pdl);
    case 8: return launch_stream_rows<16>(p, in, counts_in, out, counts_zero, s, win, pdl);
    case 9: return launch_stream_rows<32>(p, in, counts_in, out, counts_zero, s, win, pdl);
    case kTrailTileTma: return launch_trail_tma(p, *maps, cur, in, counts_in, out, counts_zero, s, win, pdl);
    default: return launch_tile_index(tile, p, in, counts_in, nullptr, TileOut{out, counts_zero, nullptr}, s, win);
    }
}

} // namespace slime
