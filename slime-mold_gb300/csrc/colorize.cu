// colorize.cu - headless display feed: the colourise pass of
// src/display.wgsl:44-86 (trail -> 256-entry LUT -> RGBA8 with aspect fit and
// black bars) written to a device buffer instead of a storage texture.
#include "kernels.h"

namespace slime {
namespace {

// A thread makes four pixels of a row, from a table of packed colours that the
// block builds once in shared memory: one lookup and a quarter of a 16-byte
// store a pixel.  Bound by the two divisions a pixel and launch latency: a
// 1600x900 image of a 4096^2 trail 4.6 us, a 1001x777 one of its own trail 3.2 (6.0
// and 4.3 with a pixel a thread, three byte loads and a 4-byte store each).
__global__ void __launch_bounds__(256) colorize_kernel(const float* __restrict__ trail, int W, int H,
                                                       const uint8_t* __restrict__ lut, int tw, int th, float scale,
                                                       float off_x, float off_y, uint32_t* __restrict__ rgba,
                                                       int quads_x, int vec) {
    __shared__ uint32_t colour[256];
    const int e = threadIdx.x;
    colour[e] = (uint32_t)lut[e] | (uint32_t)lut[e + 256] << 8 | (uint32_t)lut[e + 512] << 16 | 0xff000000u;
    __syncthreads();
    const int q = blockIdx.x * 256 + threadIdx.x;
    const int iy = q / quads_x, ix = (q - iy * quads_x) * 4;
    if (iy >= th) return;
    const float sim_w = slm_i2f(W), sim_h = slm_i2f(H);
    const float fy = slm_div(slm_sub(slm_i2f(iy), off_y), scale); // display.wgsl:72-73
    const bool row = fy >= 0.0f && fy < sim_h;
    const size_t base = (size_t)(row ? slm_f2i(fy) : 0) * W;
    float t[4];
    bool in[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float fx = slm_div(slm_sub(slm_i2f(ix + j), off_x), scale);
        in[j] = row && fx >= 0.0f && fx < sim_w; // :76
        t[j] = in[j] ? __ldg(trail + base + slm_f2i(fx)) : 0.0f;
    }
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) { // get_lut_color, :29-42
        const int idx = slm_f2i(slm_mul(slm_clamp(t[j], 0.0f, 1.0f), 255.0f));
        o[j] = in[j] ? colour[idx] : 0xff000000u;
    }
    uint32_t* out = rgba + (size_t)iy * tw + ix;
    if (vec) {
        *reinterpret_cast<uint4*>(out) = make_uint4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (ix + j < tw) out[j] = o[j];
    }
}

} // namespace

cudaError_t launch_colorize(const float* trail, uint32_t W, uint32_t H, const uint8_t* lut, uint32_t tw,
                            uint32_t th, uint8_t* rgba, cudaStream_t s) {
    // Aspect fit, display.wgsl:53-69, computed once on the host with the same
    // binary32 operations.
    float sim_w = (float)W, sim_h = (float)H, tex_w = (float)tw, tex_h = (float)th;
    float sim_aspect = slm_div(sim_w, sim_h), tex_aspect = slm_div(tex_w, tex_h);
    float scale, off_x = 0.0f, off_y = 0.0f;
    if (tex_aspect > sim_aspect) {
        scale = slm_div(tex_h, sim_h);
        off_x = slm_mul(slm_sub(tex_w, slm_mul(sim_w, scale)), 0.5f);
    } else {
        scale = slm_div(tex_w, sim_w);
        off_y = slm_mul(slm_sub(tex_h, slm_mul(sim_h, scale)), 0.5f);
    }
    const int quads_x = (int)((tw + 3) / 4);
    const uint64_t quads = (uint64_t)quads_x * th;
    const int vec = tw % 4 == 0 && ((uintptr_t)rgba & 15) == 0;
    colorize_kernel<<<(unsigned)((quads + 255) / 256), 256, 0, s>>>(trail, (int)W, (int)H, lut, (int)tw, (int)th, scale,
                                                                    off_x, off_y, (uint32_t*)rgba, quads_x, vec);
    return cudaGetLastError();
}

} // namespace slime
