// packed_products.cu - packed binary32x2 products whose lanes go into scalar
// sums and differences, the form in which the agent kernels use
// mul.rn.f32x2: each lane must be the scalar product rounded, then the scalar
// sum rounded, with no contraction of the two.
//
// The device evaluates each form for 2^20 random pairs, written with the
// kernels' own functions; the host evaluates it one rounded operation at a
// time and counts the lanes that differ:
//   0  sensor position: (x + d * c, y + d * s)
//   1  sin/cos reduction: x * (2/pi) + 1.5 * 2^23, for two arguments
//   2  bilinear interpolation: both rows and the column between them
//   3  jitter hash argument: i * a + x * b + y * c, for two agents
//   4  the fraction of a product, for two
// Prints one line per form: "form <k> <differing lanes> <lanes>".
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>
#include <cuda_runtime.h>

#include "slime_math.h"

__host__ __device__ static inline uint32_t mix32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}
// A random binary32, of magnitude 2^-20 to 2^20 or, with `unit`, in [0, 1).
__host__ __device__ static inline float operand(uint32_t i, uint32_t k, bool unit = false) {
    const uint32_t h = mix32(i * 16u + k + 0x9e3779b9u);
    if (unit) return (float)(h >> 8) * 0x1p-24f;
    const uint32_t u = (h & 0x80000000u) | ((127u - 20u + mix32(h) % 41u) << 23) | (h & 0x7fffffu);
    float f;
    memcpy(&f, &u, 4);
    return f;
}

constexpr uint32_t kPairs = 1u << 20;
constexpr int kForms = 5;

__global__ void packed(int form, float2* out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kPairs) return;
    float a[8];
    for (int k = 0; k < 8; k++) a[k] = operand(i, k);
    float2 r = make_float2(0.0f, 0.0f);
    if (form == 0) {
        const float2 m = __fmul2_rn(make_float2(a[0], a[0]), make_float2(a[1], a[2]));
        r = make_float2(slm_add(a[3], m.x), slm_add(a[4], m.y));
    } else if (form == 1) {
        const float2 m = __fmul2_rn(make_float2(4096.0f * operand(i, 0, true), -4096.0f * operand(i, 1, true)),
                                    make_float2(SLM_TWO_OVER_PI_F, SLM_TWO_OVER_PI_F));
        r = make_float2(slm_add(m.x, 12582912.0f), slm_add(m.y, 12582912.0f));
    } else if (form == 2) {
        const float dx = operand(i, 8, true), dy = operand(i, 9, true);
        const float ex = slm_sub(1.0f, dx), ey = slm_sub(1.0f, dy);
        const float2 p1 = __fmul2_rn(make_float2(a[0], a[1]), make_float2(ex, dx));
        const float v0 = slm_add(slm_mul(a[2], ex), slm_mul(a[3], dx));
        const float v1 = slm_add(p1.x, p1.y);
        const float2 p2 = __fmul2_rn(make_float2(v0, v1), make_float2(ey, dy));
        r = make_float2(slm_add(p2.x, p2.y), v1);
    } else if (form == 3) {
        const float2 mi = __fmul2_rn(make_float2(slm_i2f((int32_t)(mix32(i) >> 7)), slm_i2f((int32_t)(mix32(~i) >> 7))),
                                     make_float2(12.9898f, 12.9898f));
        const float2 mx = __fmul2_rn(make_float2(a[0], a[1]), make_float2(78.233f, 78.233f));
        const float2 my = __fmul2_rn(make_float2(a[2], a[3]), make_float2(37.719f, 37.719f));
        r = make_float2(slm_add(slm_add(mi.x, mx.x), my.x), slm_add(slm_add(mi.y, mx.y), my.y));
    } else {
        const float2 m = __fmul2_rn(make_float2(operand(i, 0, true), -operand(i, 1, true)),
                                    make_float2(43758.5453f, 43758.5453f));
        r = make_float2(slm_fract(m.x), slm_fract(m.y));
    }
    out[i] = r;
}

// One rounded binary32 operation each (no contraction across volatile objects).
static float mul(float a, float b) { volatile float r = a * b; return r; }
static float add(float a, float b) { volatile float r = a + b; return r; }
static float sub(float a, float b) { volatile float r = a - b; return r; }

static void scalar(int form, uint32_t i, float* r) {
    float a[8];
    for (int k = 0; k < 8; k++) a[k] = operand(i, k);
    if (form == 0) {
        r[0] = add(a[3], mul(a[0], a[1]));
        r[1] = add(a[4], mul(a[0], a[2]));
    } else if (form == 1) {
        r[0] = add(mul(4096.0f * operand(i, 0, true), SLM_TWO_OVER_PI_F), 12582912.0f);
        r[1] = add(mul(-4096.0f * operand(i, 1, true), SLM_TWO_OVER_PI_F), 12582912.0f);
    } else if (form == 2) {
        const float dx = operand(i, 8, true), dy = operand(i, 9, true);
        const float ex = sub(1.0f, dx), ey = sub(1.0f, dy);
        const float v0 = add(mul(a[2], ex), mul(a[3], dx));
        r[1] = add(mul(a[0], ex), mul(a[1], dx));
        r[0] = add(mul(v0, ey), mul(r[1], dy));
    } else if (form == 3) {
        const float i0 = (float)(int32_t)(mix32(i) >> 7), i1 = (float)(int32_t)(mix32(~i) >> 7);
        r[0] = add(add(mul(i0, 12.9898f), mul(a[0], 78.233f)), mul(a[2], 37.719f));
        r[1] = add(add(mul(i1, 12.9898f), mul(a[1], 78.233f)), mul(a[3], 37.719f));
    } else {
        const float m0 = mul(operand(i, 0, true), 43758.5453f), m1 = mul(-operand(i, 1, true), 43758.5453f);
        r[0] = sub(m0, floorf(m0));
        r[1] = sub(m1, floorf(m1));
    }
}

int main() {
    float2* d = nullptr;
    if (cudaMalloc(&d, kPairs * sizeof(float2)) != cudaSuccess) return 2;
    std::vector<float2> h(kPairs);
    for (int form = 0; form < kForms; form++) {
        packed<<<kPairs / 256, 256>>>(form, d);
        if (cudaMemcpy(h.data(), d, kPairs * sizeof(float2), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
        unsigned long long bad = 0;
        for (uint32_t i = 0; i < kPairs; i++) {
            float want[2] = {0.0f, 0.0f};
            scalar(form, i, want);
            bad += (memcmp(&h[i].x, &want[0], 4) != 0) + (memcmp(&h[i].y, &want[1], 4) != 0);
        }
        printf("form %d %llu %u\n", form, bad, 2u * kPairs);
    }
    cudaFree(d);
    return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
