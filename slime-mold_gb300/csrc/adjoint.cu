// adjoint.cu - checkpointed adjoint of the deposit -> decay -> diffuse chain.
//
// With the agent trajectories frozen (steering is piecewise constant in the
// trail, so its a.e. derivative is zero) the per-step deposit counts k_s are
// constants and one step is the map
//   T_{s+1} = (1 - r) u + r B(u),   u = Decay(f),   f = Fold(T_s, k_s)
// with B the toroidal blur (3x3 box or separable Gaussian; symmetric, so
// B^T = B).  Its adjoint, given g = dL/dT_{s+1}:
//   dL/dr      += sum g (B(u) - u)                       (if 0 < rate < 1)
//   g_u         = (1 - r) g + r B(g)
//   multiply:  dL/ddecay += sum g_u f,  g_f = decay g_u
//   subtract:  a = [f - decay*0.001 > 0], dL/ddecay += -0.001 sum a g_u, g_f = a g_u
//   fold:      c = [k == 0 or 0 < f < 1] (unclamped),
//              dL/ddep += sum c k g_f,  dL/dT_s = c g_f.
// The forward is recorded with a checkpoint of agents and trail every K steps;
// the backward replays each segment from its checkpoint (bit-identical to the
// recorded run), keeps T_s and k_s of the segment in HBM, and runs one fused
// stencil kernel per step backwards through it.  The last segment, the
// backward's first, is recorded straight into those buffers where memory
// allows, and not replayed.
#include <string.h>

#include "ctx.h"
#include "trail_tile.cuh"

using namespace slime;

namespace slime {
namespace {

// One backward step.  A block takes a tile of 128 x 16 cells, a thread four
// adjacent columns of every fourth row, and stages the window of u (T_s folded
// and decayed) and of g with 16-byte loads.  A block that reads T and k a second
// time for its own cells, blurs one cell per thread and adds its three sums up in
// every step (binary64 butterflies over all its threads, on a GPU with two
// binary64 operations per SM and cycle) is bound by those, so
//   * a thread sums each of its columns' four cells in binary32 and adds those
//     to its three sums over all steps, in binary64 and in memory; all threads'
//     are added up once per backward, in one order, so the gradients do not
//     depend on which block finishes first;
//   * a thread's own cells of T and k are read once (with a shared-memory
//     carve-out this large nothing stays in L1 for a second read), folded once
//     and kept in registers, as is its g;
//   * u is staged before the wait for the step it follows, which writes only g.
// The blur of g is separable; B(u) - u, small against u, is summed term by term
// from neighbour-minus-centre differences.  Cell for cell the arithmetic of a
// block that sums over all its threads in every step: 1024^2, radius 1, 22.6 us a
// step so and 11.0 here (16.8 MB of T, k and g: 2.5 us at the measured copy
// bandwidth).  2.3 of the 11.0 are the twelve binary64 additions and conversions
// a thread; sums kept as pairs of binary32 numbers did without, in 48 bits and
// binary32's range.  Conversions by integer operations measure the same.
constexpr int kTW = 128, kTH = 16;
constexpr int kSlots = 4;              // a thread's rows are its slot and every fourth after it
constexpr int kRows = kTH / kSlots;
constexpr int kThreads = kTW / 4 * kSlots;

// The first n of four cells from i.
__device__ __forceinline__ float4 row4(const float* __restrict__ a, size_t i, int n) {
    return make_float4(n > 0 ? __ldg(a + i) : 0.0f, n > 1 ? __ldg(a + i + 1) : 0.0f, n > 2 ? __ldg(a + i + 2) : 0.0f,
                       n > 3 ? __ldg(a + i + 3) : 0.0f);
}
__device__ __forceinline__ uint4 row4(const uint32_t* __restrict__ a, size_t i, int n) {
    return make_uint4(n > 0 ? __ldg(a + i) : 0u, n > 1 ? __ldg(a + i + 1) : 0u, n > 2 ? __ldg(a + i + 2) : 0u,
                      n > 3 ? __ldg(a + i + 3) : 0u);
}

// Columns 4c - LP .. 4c + 3 + LP of a window row (row points at column 4c - LP).
template <int LP>
__device__ __forceinline__ void window4(const float* row, float* e) {
#pragma unroll
    for (int i = 0; i < 1 + LP / 2; i++) {
        const float4 v = *reinterpret_cast<const float4*>(row + 4 * i);
        e[4 * i] = v.x, e[4 * i + 1] = v.y, e[4 * i + 2] = v.z, e[4 * i + 3] = v.w;
    }
}

// The 2R halo rows of a window, spread over the slots: window row of a slot's
// i-th one, or -1.
template <int R>
__device__ __forceinline__ int halo_row(int slot, int i) {
    const int h = slot + i * kSlots;
    return h >= 2 * R ? -1 : (h < R ? h : kTH + h);
}

__device__ __forceinline__ float4 decayed(const DevParams& p, const float4& f) {
    return make_float4(apply_decay(p, f.x), apply_decay(p, f.y), apply_decay(p, f.z), apply_decay(p, f.w));
}
__device__ __forceinline__ float4 folded(const DevParams& p, const float4& t, const uint4& k) {
    return make_float4(fold_deposits(t.x, k.x, p.dep), fold_deposits(t.y, k.y, p.dep), fold_deposits(t.z, k.z, p.dep),
                       fold_deposits(t.w, k.w, p.dep));
}

template <int R, bool kGauss>
__global__ void __launch_bounds__(kThreads) adjoint_kernel(const __grid_constant__ DevParams p,
                                                           const float* __restrict__ T, const uint32_t* __restrict__ K,
                                                           const float* gin, float* gout, double* acc,
                                                           uint32_t rate_active, int tiles_x, int vec) {
    typedef TileGeom<kTW, kTH, R> G; // window layout
    constexpr int NH = (2 * R + kSlots - 1) / kSlots; // halo rows per slot
    extern __shared__ __align__(16) float sm[];
    float* su = sm;
    float* sg = sm + G::window;
    float* hg = sg + G::window; // Gaussian only: the rows of g blurred
    const int W = p.W, H = p.H;
    const int by = blockIdx.x / tiles_x;
    const int x0 = (blockIdx.x - by * tiles_x) * kTW, y0 = by * kTH;
    const int c = threadIdx.x & 31, slot = threadIdx.x >> 5;
    const int gx = wrap_coord(x0 + 4 * c, W);
    constexpr int NC = (kTW + 2 * R + 31) / 32; // rows of any width: cells per lane and row, and their columns
    int cols[NC];
#pragma unroll
    for (int q = 0; q < NC; q++) cols[q] = wrap_coord(x0 - R + min(c + 32 * q, kTW + 2 * R - 1), W);
    float4 f4[kRows], g4[kRows];
    uint4 k4[kRows];
    constexpr int HN = G::SH * 2 * R; // halo columns: 2R cells of every window row
    if (vec) {
        float4 th[NH > 0 ? NH : 1];
        uint4 kh[NH > 0 ? NH : 1];
#pragma unroll
        for (int i = 0; i < kRows; i++) {
            const size_t at = (size_t)wrap_coord(y0 + slot + i * kSlots, H) * W + gx;
            f4[i] = __ldg(reinterpret_cast<const float4*>(T + at));
            k4[i] = __ldg(reinterpret_cast<const uint4*>(K + at));
        }
#pragma unroll
        for (int i = 0; i < NH; i++) {
            const int r = halo_row<R>(slot, i);
            if (r >= 0) {
                const size_t at = (size_t)wrap_coord(y0 - R + r, H) * W + gx;
                th[i] = __ldg(reinterpret_cast<const float4*>(T + at));
                kh[i] = __ldg(reinterpret_cast<const uint4*>(K + at));
            }
        }
        for (int i = threadIdx.x; i < HN; i += kThreads) {
            const int r = i / (2 * R > 0 ? 2 * R : 1), j = i - r * 2 * R;
            const int cc = j < R ? j - R : kTW + j - R;
            const size_t at = (size_t)wrap_coord(y0 - R + r, H) * W + wrap_coord(x0 + cc, W);
            su[r * G::stride + G::LP + cc] = apply_decay(p, fold_deposits(__ldg(T + at), __ldg(K + at), p.dep));
        }
#pragma unroll
        for (int i = 0; i < kRows; i++) {
            f4[i] = folded(p, f4[i], k4[i]);
            *reinterpret_cast<float4*>(su + (R + slot + i * kSlots) * G::stride + G::LP + 4 * c) = decayed(p, f4[i]);
        }
#pragma unroll
        for (int i = 0; i < NH; i++) {
            const int r = halo_row<R>(slot, i);
            if (r >= 0)
                *reinterpret_cast<float4*>(su + r * G::stride + G::LP + 4 * c) = decayed(p, folded(p, th[i], kh[i]));
        }
    } else {
#pragma unroll 2
        for (int r = slot; r < G::SH; r += kSlots) {
            const size_t row = (size_t)wrap_coord(y0 - R + r, H) * W;
            float t[NC];
            uint32_t k[NC];
#pragma unroll
            for (int q = 0; q < NC; q++) {
                t[q] = __ldg(T + row + cols[q]);
                k[q] = __ldg(K + row + cols[q]);
            }
#pragma unroll
            for (int q = 0; q < NC; q++)
                if (c + 32 * q < kTW + 2 * R)
                    su[r * G::stride + G::LP - R + c + 32 * q] = apply_decay(p, fold_deposits(t[q], k[q], p.dep));
        }
#pragma unroll
        for (int i = 0; i < kRows; i++) {
            const int gy = y0 + slot + i * kSlots, n = gy < H ? min(4, W - (x0 + 4 * c)) : 0;
            const size_t at = (size_t)gy * W + x0 + 4 * c;
            k4[i] = row4(K, at, n);
            f4[i] = folded(p, row4(T, at, n), k4[i]);
        }
    }
    // g and the sums are the output of the step this one follows
    pdl_wait();
    pdl_trigger();
    double* own_acc = acc + (size_t)blockIdx.x * (3 * kThreads) + threadIdx.x;
    double s[3] = {own_acc[0], own_acc[kThreads], own_acc[2 * kThreads]};
    if (vec) {
        float4 gh[NH > 0 ? NH : 1];
#pragma unroll
        for (int i = 0; i < kRows; i++)
            g4[i] = *reinterpret_cast<const float4*>(gin + (size_t)wrap_coord(y0 + slot + i * kSlots, H) * W + gx);
#pragma unroll
        for (int i = 0; i < NH; i++) {
            const int r = halo_row<R>(slot, i);
            if (r >= 0) gh[i] = *reinterpret_cast<const float4*>(gin + (size_t)wrap_coord(y0 - R + r, H) * W + gx);
        }
        for (int i = threadIdx.x; i < HN; i += kThreads) {
            const int r = i / (2 * R > 0 ? 2 * R : 1), j = i - r * 2 * R;
            const int cc = j < R ? j - R : kTW + j - R;
            sg[r * G::stride + G::LP + cc] = gin[(size_t)wrap_coord(y0 - R + r, H) * W + wrap_coord(x0 + cc, W)];
        }
#pragma unroll
        for (int i = 0; i < kRows; i++)
            *reinterpret_cast<float4*>(sg + (R + slot + i * kSlots) * G::stride + G::LP + 4 * c) = g4[i];
#pragma unroll
        for (int i = 0; i < NH; i++) {
            const int r = halo_row<R>(slot, i);
            if (r >= 0) *reinterpret_cast<float4*>(sg + r * G::stride + G::LP + 4 * c) = gh[i];
        }
        __syncthreads();
    } else {
#pragma unroll 2
        for (int r = slot; r < G::SH; r += kSlots) {
            const size_t row = (size_t)wrap_coord(y0 - R + r, H) * W;
            float t[NC];
#pragma unroll
            for (int q = 0; q < NC; q++) t[q] = gin[row + cols[q]];
#pragma unroll
            for (int q = 0; q < NC; q++)
                if (c + 32 * q < kTW + 2 * R) sg[r * G::stride + G::LP - R + c + 32 * q] = t[q];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kRows; i++)
            g4[i] = *reinterpret_cast<const float4*>(sg + (R + slot + i * kSlots) * G::stride + G::LP + 4 * c);
    }
    if (kGauss) {
        for (int r = slot; r < G::SH; r += kSlots) {
            float e[4 + 2 * G::LP], b[4];
            window4<G::LP>(sg + r * G::stride + 4 * c, e);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                b[j] = 0.0f;
#pragma unroll
                for (int t = 0; t <= 2 * R; t++) b[j] = slm_fma(p.w[t], e[G::LP - R + j + t], b[j]);
            }
            *reinterpret_cast<float4*>(hg + r * kTW + 4 * c) = make_float4(b[0], b[1], b[2], b[3]);
        }
        __syncthreads();
    }
    const float r = p.rate;
    float sd[4] = {}, sr[4] = {}, sp[4] = {}; // by column
#pragma unroll
    for (int i = 0; i < kRows; i++) {
        const int ry = slot + i * kSlots; // row of the tile
        const int gy = y0 + ry;
        const int n = gy < H ? min(4, W - (x0 + 4 * c)) : 0; // cells of this thread in the row
        if (n <= 0) continue;
        float bg[4], bmu[4]; // B(g), B(u) - u
        const float4 uc4 = *reinterpret_cast<const float4*>(su + (R + ry) * G::stride + G::LP + 4 * c);
        const float uc[4] = {uc4.x, uc4.y, uc4.z, uc4.w};
#pragma unroll
        for (int j = 0; j < 4; j++) bg[j] = bmu[j] = 0.0f;
        if (kGauss) {
#pragma unroll
            for (int t = 0; t <= 2 * R; t++) {
                const float4 a = *reinterpret_cast<const float4*>(hg + (ry + t) * kTW + 4 * c);
                bg[0] = slm_fma(p.w[t], a.x, bg[0]);
                bg[1] = slm_fma(p.w[t], a.y, bg[1]);
                bg[2] = slm_fma(p.w[t], a.z, bg[2]);
                bg[3] = slm_fma(p.w[t], a.w, bg[3]);
            }
            if (rate_active) {
                for (int t = 0; t <= 2 * R; t++) {
                    float e[4 + 2 * G::LP];
                    window4<G::LP>(su + (ry + t) * G::stride + 4 * c, e);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        float row = 0.0f;
#pragma unroll
                        for (int d = 0; d <= 2 * R; d++) row += p.w[d] * (e[G::LP - R + j + d] - uc[j]);
                        bmu[j] += p.w[t] * row;
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; j++) bmu[j] = bmu[j] + p.w2sum_m1 * uc[j];
            }
        } else {
#pragma unroll
            for (int dy = 0; dy < 3; dy++) {
                const float* rg = sg + (ry + dy) * G::stride + G::LP + 4 * c;
                const float* ru = su + (ry + dy) * G::stride + G::LP + 4 * c;
                const float4 vg = *reinterpret_cast<const float4*>(rg), vu = *reinterpret_cast<const float4*>(ru);
                const float eg[6] = {rg[-1], vg.x, vg.y, vg.z, vg.w, rg[4]};
                const float eu[6] = {ru[-1], vu.x, vu.y, vu.z, vu.w, ru[4]};
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int dx = 0; dx < 3; dx++) {
                        bg[j] += eg[j + dx];
                        bmu[j] += eu[j + dx] - uc[j];
                    }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                bg[j] = bg[j] * (1.0f / 9.0f);
                bmu[j] = bmu[j] * (1.0f / 9.0f);
            }
        }
        const float fv[4] = {f4[i].x, f4[i].y, f4[i].z, f4[i].w}, gv[4] = {g4[i].x, g4[i].y, g4[i].z, g4[i].w};
        const uint32_t kv[4] = {k4[i].x, k4[i].y, k4[i].z, k4[i].w};
        float o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float g = gv[j], f = fv[j];
            const uint32_t k = kv[j];
            const float g_u = (1.0f - r) * g + r * bg[j];
            float g_f, d_decay;
            if (p.decay_mode == SLIME_DECAY_MULTIPLY) {
                d_decay = g_u * f;
                g_f = p.decay * g_u;
            } else {
                const bool act = slm_sub(f, p.decay_k) > 0.0f;
                d_decay = act ? -0.001f * g_u : 0.0f;
                g_f = act ? g_u : 0.0f;
            }
            const bool unclamped = (k == 0u) || (f > 0.0f && f < 1.0f);
            if (j < n) {
                sd[j] += d_decay;
                if (rate_active) sr[j] += g * bmu[j];
                if (unclamped) sp[j] += g_f * (float)k;
            }
            o[j] = unclamped ? g_f : 0.0f;
        }
        const size_t at = (size_t)gy * W + x0 + 4 * c;
        if (vec) {
            *reinterpret_cast<float4*>(gout + at) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j < n) gout[at + j] = o[j];
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        s[0] += (double)sd[j];
        s[1] += (double)sr[j];
        s[2] += (double)sp[j];
    }
    own_acc[0] = s[0];
    own_acc[kThreads] = s[1];
    own_acc[2 * kThreads] = s[2];
}

constexpr uint32_t kSumBlocks = kThreads; // blocks of the first pass over the threads' sums

// The threads' sums, in two passes, each in a fixed order.
__device__ __forceinline__ double block_sum(double v) {
    __shared__ double s[kThreads];
    s[threadIdx.x] = v;
    __syncthreads();
    for (int o = kThreads / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    return s[0];
}
__global__ void __launch_bounds__(kThreads) sum_threads_kernel(const double* __restrict__ acc, uint32_t blocks,
                                                          double* __restrict__ part) {
    double v = 0.0;
    for (uint32_t b = blockIdx.x; b < blocks; b += kSumBlocks)
        v += acc[((size_t)b * 3 + blockIdx.y) * kThreads + threadIdx.x];
    v = block_sum(v);
    if (threadIdx.x == 0) part[blockIdx.y * kSumBlocks + blockIdx.x] = v;
}
__global__ void __launch_bounds__(kThreads) sum_parts_kernel(const double* __restrict__ part, double* __restrict__ out) {
    const double v = block_sum(part[blockIdx.x * kSumBlocks + threadIdx.x]);
    if (threadIdx.x == 0) out[blockIdx.x] = v;
}

uint32_t adjoint_blocks(uint32_t W, uint32_t H) {
    return ((W + kTW - 1) / kTW) * ((H + kTH - 1) / kTH);
}

template <int R, bool kGauss>
cudaError_t launch_adj(const DevParams& p, const float* T, const uint32_t* K, const float* gin, float* gout,
                       double* acc, uint32_t rate_active, cudaStream_t s, bool pdl) {
    typedef TileGeom<kTW, kTH, R> G;
    const size_t smem = sizeof(float) * (2 * G::window + (kGauss ? G::SH * kTW : 0));
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(adjoint_kernel<R, kGauss>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
    }
    const int vec = p.W % 4 == 0 && (((uintptr_t)T | (uintptr_t)K | (uintptr_t)gin | (uintptr_t)gout) & 15) == 0;
    return launch_kp(adjoint_kernel<R, kGauss>, dim3(adjoint_blocks((uint32_t)p.W, (uint32_t)p.H)), dim3(kThreads), smem, s,
                     nullptr, pdl, p, T, K, gin, gout, acc, rate_active, (p.W + kTW - 1) / kTW, vec);
}

} // namespace

cudaError_t launch_adjoint_step(const DevParams& p, const float* T, const uint32_t* K, const float* gin,
                                float* gout, double* acc, uint32_t rate_active, cudaStream_t s, bool pdl) {
    if (p.blur_mode != SLIME_BLUR_GAUSS) return launch_adj<1, false>(p, T, K, gin, gout, acc, rate_active, s, pdl);
    switch (p.R) {
    case 0: return launch_adj<0, true>(p, T, K, gin, gout, acc, rate_active, s, pdl);
    case 1: return launch_adj<1, true>(p, T, K, gin, gout, acc, rate_active, s, pdl);
    case 2: return launch_adj<2, true>(p, T, K, gin, gout, acc, rate_active, s, pdl);
    case 3: return launch_adj<3, true>(p, T, K, gin, gout, acc, rate_active, s, pdl);
    case 4: return launch_adj<4, true>(p, T, K, gin, gout, acc, rate_active, s, pdl);
    case 5: return launch_adj<5, true>(p, T, K, gin, gout, acc, rate_active, s, pdl);
    case 6: return launch_adj<6, true>(p, T, K, gin, gout, acc, rate_active, s, pdl);
    case 7: return launch_adj<7, true>(p, T, K, gin, gout, acc, rate_active, s, pdl);
    case 8: return launch_adj<8, true>(p, T, K, gin, gout, acc, rate_active, s, pdl);
    default: return cudaErrorInvalidValue;
    }
}

void drop_segment_graphs(slime_ctx* ctx) {
    for (auto& kv : ctx->adj.seg_graphs) cudaGraphExecDestroy(kv.second);
    ctx->adj.seg_graphs.clear();
}

// Gives back the buffers of the backward; the recording stays (every segment
// can be replayed from its checkpoint).
void release_segment(slime_ctx* ctx) {
    auto& a = ctx->adj;
    cudaStreamSynchronize(ctx->stream);
    drop_segment_graphs(ctx);
    for (auto it = ctx->graphs.begin(); it != ctx->graphs.end();) { // recorded segments write these buffers
        if (it->first.second & slime_ctx::kGraphRecord) {
            cudaGraphExecDestroy(it->second);
            it = ctx->graphs.erase(it);
        } else {
            ++it;
        }
    }
    for (cudaTextureObject_t t : a.seg_tex)
        if (t) cudaDestroyTextureObject(t);
    a.seg_tex.clear();
    a.seg_holds = -1;
    void** ptrs[] = {(void**)&a.seg_trail, (void**)&a.seg_counts, (void**)&a.g[0], (void**)&a.g[1],
                     (void**)&a.acc, (void**)&a.ids_tmp, (void**)&a.agents_tmp};
    for (void** q : ptrs) {
        if (*q) dev_free(*q);
        *q = nullptr;
    }
}

void free_adjoint(slime_ctx* ctx) {
    auto& a = ctx->adj;
    release_segment(ctx);
    void* ptrs[] = {a.ckpt_agents, a.ckpt_ids, a.ckpt_trail};
    for (void* q : ptrs)
        if (q) dev_free(q);
    a = slime_ctx::Adjoint();
}

} // namespace slime

#define CK(expr, what)                                                                                      \
    do {                                                                                                    \
        cudaError_t _e = (expr);                                                                            \
        if (_e != cudaSuccess) return cuda_error(ctx->err, _e, what);                                       \
    } while (0)

namespace {

// Cells from one step's trail (or counts) of a segment to the next one's: rows
// of every step 256-byte aligned, for 16-byte loads and gather textures.
size_t segment_stride(const slime_ctx* ctx) { return ((size_t)ctx->W * ctx->H + 63) & ~(size_t)63; }

size_t acc_bytes(const slime_ctx* ctx) {
    return (4 + 3 * kSumBlocks) * sizeof(double) +
           (size_t)adjoint_blocks(ctx->W, ctx->H) * 3 * kThreads * sizeof(double);
}

// The buffers of the backward, as the recording's sizes have them: all of them
// or, without memory, none.
cudaError_t alloc_segment(slime_ctx* ctx, cudaError_t (*alloc)(slime_ctx*, void**, size_t)) {
    auto& a = ctx->adj;
    const size_t cells = (size_t)ctx->W * ctx->H, stride = segment_stride(ctx);
    const uint32_t K = a.ckpt_every;
    // W + 2 zero floats past the last trail: the sampler's discarded taps
    const size_t trail_bytes = ((size_t)K * stride + ctx->W + 2) * sizeof(float);
    cudaError_t e;
    if ((e = alloc(ctx, (void**)&a.seg_trail, trail_bytes)) == cudaSuccess &&
        (e = cudaMemsetAsync(a.seg_trail, 0, trail_bytes, ctx->stream)) == cudaSuccess &&
        (e = alloc(ctx, (void**)&a.seg_counts, (size_t)K * stride * sizeof(uint32_t))) == cudaSuccess &&
        (e = alloc(ctx, (void**)&a.g[0], cells * sizeof(float))) == cudaSuccess &&
        (e = alloc(ctx, (void**)&a.g[1], cells * sizeof(float))) == cudaSuccess &&
        (e = alloc(ctx, (void**)&a.acc, acc_bytes(ctx))) == cudaSuccess &&
        (!a.with_ids || (e = alloc(ctx, (void**)&a.ids_tmp, a.n_pad * sizeof(uint32_t))) == cudaSuccess))
        e = alloc(ctx, (void**)&a.agents_tmp, 4 * a.n_pad * sizeof(float));
    if (e != cudaSuccess) {
        cudaGetLastError();
        release_segment(ctx);
        return e;
    }
    for (uint32_t i = 0; i < K && agent_shape_uses_texture(a.agent_shape); i++)
        a.seg_tex.push_back(make_trail_texture(a.seg_trail + i * stride, ctx->W, ctx->H));
    return cudaSuccess;
}

// m steps of `ag` from the trail in the segment's first slot, keeping T_s and
// k_s (counts cleared by the caller); the trail after the last one goes to
// `last`, or is not made.
cudaError_t enqueue_forward(slime_ctx* ctx, const AgentsSoA& ag, uint32_t m, float* last) {
    auto& a = ctx->adj;
    const size_t stride = segment_stride(ctx);
    const bool strips = trail_tile_streams(a.dev, a.tile);
    cudaError_t e = cudaSuccess;
    for (uint32_t i = 0; i < m && e == cudaSuccess; i++) {
        float* Ti = a.seg_trail + (size_t)i * stride;
        uint32_t* Ki = a.seg_counts + (size_t)i * stride;
        e = launch_agents(a.dev, ag, Ti, Ki, ctx->stream, a.agent_shape, nullptr,
                          i < a.seg_tex.size() ? a.seg_tex[i] : 0, nullptr, i > 0 && strips);
        float* to = i + 1 < m ? Ti + stride : last;
        if (e == cudaSuccess && to)
            e = launch_trail(a.dev, a.tile, Ti, Ki, to, nullptr, ctx->stream, nullptr, a.n > 0);
    }
    return e;
}

// Whether the last segment can be recorded into the backward's buffers: they
// are there, or are taken now from memory that is amply there (a quarter of
// what is free; the backward would take them in any case).
bool segment_ready(slime_ctx* ctx) {
    auto& a = ctx->adj;
    if (a.agents_tmp) return true;
    size_t free_b = 0, total_b = 0;
    const size_t bytes = ((size_t)a.ckpt_every * 2 * segment_stride(ctx) + 5 * a.n_pad) * sizeof(float);
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || bytes > free_b / 4) {
        cudaGetLastError();
        return false;
    }
    return alloc_segment(ctx, [](slime_ctx*, void** p, size_t b) { return dev_alloc(p, b); }) == cudaSuccess;
}

// The last m recorded steps, keeping T_s and k_s for the backward.  What they
// leave behind is what m steps leave: the trail in the buffer that is current
// then, the last step's counts, the agents.  The records that later steps write
// are not touched.  Measured on 1024^2 with 1 M agents, 200 steps, segments of
// 50: recording and backward 10.5 ms with every segment replayed, 9.5 so.
int record_last_segment(slime_ctx* ctx, uint32_t m) {
    auto& a = ctx->adj;
    const size_t cells = (size_t)ctx->W * ctx->H, stride = segment_stride(ctx);
    const int to = (m & 1) ? 1 - ctx->cur : ctx->cur;
    CK(cudaMemcpyAsync(a.seg_trail, ctx->trail[ctx->cur], cells * sizeof(float), cudaMemcpyDeviceToDevice,
                       ctx->stream), "keeping the trail");
    CK(cudaMemsetAsync(a.seg_counts, 0, (size_t)m * stride * sizeof(uint32_t), ctx->stream), "clearing counts");
    cudaGraphExec_t exec = nullptr;
    if (ctx->opt.use_graphs) {
        auto key = std::make_pair(m, ctx->cur | (ctx->in_sorted_run ? slime_ctx::kGraphSorted : 0) | slime_ctx::kGraphRecord);
        auto it = ctx->graphs.find(key);
        if (it == ctx->graphs.end()) {
            cudaError_t ce = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
            if (ce == cudaSuccess) ce = enqueue_forward(ctx, ctx->agents, m, ctx->trail[to]);
            cudaGraph_t graph = nullptr;
            cudaError_t ee = cudaStreamEndCapture(ctx->stream, &graph);
            if (ce == cudaSuccess && ee == cudaSuccess) ee = instantiate_graph(&exec, graph);
            if (graph) cudaGraphDestroy(graph);
            if (ce == cudaSuccess && ee == cudaSuccess) {
                ctx->graphs[key] = exec;
            } else {
                cudaGetLastError();
                exec = nullptr; // direct launches
            }
        } else {
            exec = it->second;
        }
    }
    if (exec)
        CK(cudaGraphLaunch(exec, ctx->stream), "launching recorded steps");
    else
        CK(enqueue_forward(ctx, ctx->agents, m, ctx->trail[to]), "launching recorded steps");
    CK(cudaMemcpyAsync(ctx->counts[1 - to], a.seg_counts + (size_t)(m - 1) * stride, cells * sizeof(uint32_t),
                       cudaMemcpyDeviceToDevice, ctx->stream), "keeping the last step's counts");
    ctx->launches += (uint64_t)m * (1 + agent_pass_kernels(a.dev, a.n, false));
    ctx->steps_done += m;
    ctx->cur = to;
    const bool dirty[4] = {ctx->counts_dirty[0], ctx->counts_dirty[1], ctx->marks_dirty[0], ctx->marks_dirty[1]};
    after_steps(ctx, false, m);
    for (int i = 0; i < 2; i++) {
        ctx->counts_dirty[i] = dirty[i] || i == 1 - to;
        ctx->marks_dirty[i] = dirty[2 + i];
    }
    return SLIME_OK;
}

// The recorded steps, on the context's agents as they are now (its own, or the
// sorted copy of begin_sorted_run).
int record_steps(slime_ctx* ctx, uint32_t n_steps, uint32_t ckpt_every) {
    auto& a = ctx->adj;
    const size_t cells = (size_t)ctx->W * ctx->H;
    const uint64_t n_pad = ctx->agents.n_pad;
    const uint32_t K = ckpt_every < n_steps ? ckpt_every : n_steps;
    const uint32_t n_ckpt = (n_steps + K - 1) / K;
    const bool with_ids = ctx->agents.ids != nullptr;
    // the last recording's buffers serve this one when it is of the same size
    if (a.ckpt_trail && (a.n_ckpt != n_ckpt || a.ckpt_every != K || a.n != ctx->agents.n || a.n_pad != n_pad ||
                         a.with_ids != with_ids))
        free_adjoint(ctx);
    if (memcmp(&a.dev, &ctx->dev, sizeof a.dev) != 0 || a.tile != ctx->tile || a.agent_shape != ctx->agent_shape)
        drop_segment_graphs(ctx);
    a.recorded = false;
    a.seg_holds = -1;
    a.n_steps = n_steps;
    a.ckpt_every = K;
    a.n_ckpt = n_ckpt;
    a.dev = ctx->dev;
    a.tile = ctx->tile;
    a.agent_shape = ctx->agent_shape;
    const uint32_t rate_active = (ctx->params.diffusion_rate > 0.0f && ctx->params.diffusion_rate < 1.0f) ? 1u : 0u;
    if (rate_active != a.rate_active) drop_segment_graphs(ctx);
    a.rate_active = rate_active;
    a.n = ctx->agents.n;
    a.n_pad = n_pad;
    a.with_ids = with_ids;
    cudaError_t e;
    if (!a.ckpt_trail &&
        ((e = ctx_alloc(ctx, (void**)&a.ckpt_agents, (size_t)a.n_ckpt * 4 * n_pad * sizeof(float))) != cudaSuccess ||
         (a.with_ids && (e = ctx_alloc(ctx, (void**)&a.ckpt_ids, (size_t)a.n_ckpt * n_pad * sizeof(uint32_t))) != cudaSuccess) ||
         (e = ctx_alloc(ctx, (void**)&a.ckpt_trail, (size_t)a.n_ckpt * cells * sizeof(float))) != cudaSuccess)) {
        free_adjoint(ctx);
        return cuda_error(ctx->err, e, "allocating checkpoints");
    }
    for (uint32_t j = 0; j < a.n_ckpt; j++) {
        uint32_t m = (n_steps - j * K) < K ? (n_steps - j * K) : K;
        int rc = resort_run(ctx, m);
        if (rc != SLIME_OK) return rc;
        CK(cudaMemcpyAsync(a.ckpt_agents + (size_t)j * 4 * n_pad, ctx->agents.x, 4 * n_pad * sizeof(float),
                           cudaMemcpyDeviceToDevice, ctx->stream), "checkpointing agents");
        if (a.with_ids)
            CK(cudaMemcpyAsync(a.ckpt_ids + (size_t)j * n_pad, ctx->agents.ids, n_pad * sizeof(uint32_t),
                               cudaMemcpyDeviceToDevice, ctx->stream), "checkpointing ids");
        CK(cudaMemcpyAsync(a.ckpt_trail + (size_t)j * cells, ctx->trail[ctx->cur], cells * sizeof(float),
                           cudaMemcpyDeviceToDevice, ctx->stream), "checkpointing trail");
        if (j + 1 == a.n_ckpt && segment_ready(ctx)) {
            if ((rc = record_last_segment(ctx, m)) != SLIME_OK) return rc;
            a.seg_holds = (int)j;
            break;
        }
        while (m > 0) {
            const bool marks = use_marks(ctx);
            if ((rc = prepare_deposits(ctx, marks)) != SLIME_OK) return rc;
            const uint32_t chunk = ctx->opt.graph_chunk ? ctx->opt.graph_chunk : 50;
            const uint32_t take = m < chunk ? m : chunk;
            // a graph that cannot be made must not end a recording that is under way
            cudaGraphExec_t exec = nullptr;
            const bool graph = ctx->opt.use_graphs && step_graph(ctx, take, marks, &exec) == SLIME_OK;
            if (!graph) {
                cudaGetLastError();
                ctx->err.clear();
            }
            rc = graph ? run_steps_graph(ctx, take, marks) : run_steps_direct(ctx, take, marks);
            if (rc != SLIME_OK) return rc;
            after_steps(ctx, marks, take);
            m -= take;
        }
    }
    return SLIME_OK;
}

} // namespace

extern "C" {

int slime_forward_record(slime_ctx* ctx, uint32_t n_steps, uint32_t ckpt_every) {
    if (!ctx) return SLIME_ERR_INVALID_ARGUMENT;
    if (n_steps == 0 || ckpt_every == 0)
        return set_error(ctx->err, SLIME_ERR_INVALID_ARGUMENT, "n_steps and ckpt_every must be >= 1");
    cudaSetDevice(ctx->device);
    CK(cudaStreamSynchronize(ctx->stream), "forward_record");
    int rc = ensure_dispatch_order(ctx);
    if (rc != SLIME_OK) return rc;
    if ((rc = begin_sorted_run(ctx, n_steps)) != SLIME_OK) return rc;
    ctx->keep_sorted = ctx->in_sorted_run;
    const uint64_t before = ctx->steps_done;
    rc = record_steps(ctx, n_steps, ckpt_every);
    ctx->keep_sorted = false;
    if (rc == SLIME_ERR_OUT_OF_MEMORY && ctx->in_sorted_run && ctx->steps_done == before) {
        // before the first step: on the context's own agents, without the copy
        if ((rc = end_sorted_run(ctx)) != SLIME_OK) return rc;
        release_sorted(ctx);
        ctx->sorted_refused = true;
        rc = record_steps(ctx, n_steps, ckpt_every);
    }
    if (rc != SLIME_OK) return rc;
    CK(cudaStreamSynchronize(ctx->stream), "forward_record");
    ctx->adj.recorded = true;
    return SLIME_OK;
}

int slime_backward(slime_ctx* ctx, const float* dl_dtrail_final, SlimeGrads* grads, float* d_trail0) {
    if (!ctx || !dl_dtrail_final || !grads) return SLIME_ERR_INVALID_ARGUMENT;
    auto& a = ctx->adj;
    if (!a.recorded) return set_error(ctx->err, SLIME_ERR_STATE, "no recorded forward run (slime_forward_record)");
    if (a.n != ctx->agents.n || a.n_pad != ctx->agents.n_pad)
        return set_error(ctx->err, SLIME_ERR_STATE, "the agent buffer changed since the recording");
    cudaSetDevice(ctx->device);
    const size_t cells = (size_t)ctx->W * ctx->H;
    const uint32_t K = a.ckpt_every;
    const size_t stride = segment_stride(ctx);
    const uint32_t blocks = adjoint_blocks(ctx->W, ctx->H);
    if (!a.agents_tmp) CK(alloc_segment(ctx, ctx_alloc), "allocating adjoint buffers");
    CK(cudaMemcpyAsync(a.g[0], dl_dtrail_final, cells * sizeof(float), cudaMemcpyHostToDevice, ctx->stream),
       "uploading dL/dT");
    CK(cudaMemsetAsync(a.acc, 0, acc_bytes(ctx), ctx->stream), "clearing gradients");
    double* parts = (double*)a.acc;                      // 3, then 3 x kSumBlocks, then every thread's
    double* thread_acc = parts + 4 + 3 * kSumBlocks;
    int cg = 0;
    AgentsSoA tmp;
    tmp.x = a.agents_tmp;
    tmp.y = a.agents_tmp + a.n_pad;
    tmp.th = a.agents_tmp + 2 * a.n_pad;
    tmp.v = a.agents_tmp + 3 * a.n_pad;
    tmp.ids = a.with_ids ? a.ids_tmp : nullptr;
    tmp.n = a.n;
    tmp.n_pad = a.n_pad;
    // One segment: after its restore the replay of its m steps from the
    // checkpoint (keeping T_s and k_s), unless they are held already, then its m
    // backward steps, starting from g[g0].  The same launches for every segment
    // of m steps: captured once per (m, g0, held) as a CUDA graph and replayed.
    auto enqueue_segment = [&](uint32_t m, int g0, bool held) -> cudaError_t {
        cudaError_t ce = held ? cudaSuccess : enqueue_forward(ctx, tmp, m, nullptr);
        int gi = g0;
        for (int64_t i = (int64_t)m - 1; i >= 0 && ce == cudaSuccess; i--) {
            // the first backward step follows the replay, the others each other
            ce = launch_adjoint_step(a.dev, a.seg_trail + (size_t)i * stride, a.seg_counts + (size_t)i * stride,
                                     a.g[gi], a.g[1 - gi], thread_acc, a.rate_active, ctx->stream, i + 1 < (int64_t)m);
            gi = 1 - gi;
        }
        return ce;
    };
    auto segment_graph = [&](uint32_t m, int g0, bool held) -> cudaGraphExec_t {
        auto key = std::make_pair(m, g0 | (held ? 2 : 0));
        auto it = a.seg_graphs.find(key);
        if (it != a.seg_graphs.end()) return it->second;
        cudaGraphExec_t exec = nullptr;
        cudaError_t ce = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
        if (ce == cudaSuccess) ce = enqueue_segment(m, g0, held);
        cudaGraph_t graph = nullptr;
        cudaError_t ee = cudaStreamEndCapture(ctx->stream, &graph);
        if (ce == cudaSuccess && ee == cudaSuccess) ee = instantiate_graph(&exec, graph);
        if (graph) cudaGraphDestroy(graph);
        if (ce != cudaSuccess || ee != cudaSuccess) {
            cudaGetLastError();
            return nullptr; // the segment runs as direct launches
        }
        a.seg_graphs[key] = exec;
        return exec;
    };
    for (int64_t j = (int64_t)a.n_ckpt - 1; j >= 0; j--) {
        const uint32_t s0 = (uint32_t)j * K;
        const uint32_t m = (a.n_steps - s0) < K ? (a.n_steps - s0) : K;
        const bool held = a.seg_holds == (int)j;
        if (!held) { // replay the segment from its checkpoint, keeping T_s and k_s
            a.seg_holds = -1; // until that is launched
            CK(cudaMemcpyAsync(a.agents_tmp, a.ckpt_agents + (size_t)j * 4 * a.n_pad, 4 * a.n_pad * sizeof(float),
                               cudaMemcpyDeviceToDevice, ctx->stream), "restoring agents");
            if (a.with_ids)
                CK(cudaMemcpyAsync(a.ids_tmp, a.ckpt_ids + (size_t)j * a.n_pad, a.n_pad * sizeof(uint32_t),
                                   cudaMemcpyDeviceToDevice, ctx->stream), "restoring ids");
            CK(cudaMemcpyAsync(a.seg_trail, a.ckpt_trail + (size_t)j * cells, cells * sizeof(float),
                               cudaMemcpyDeviceToDevice, ctx->stream), "restoring trail");
            CK(cudaMemsetAsync(a.seg_counts, 0, (size_t)m * stride * sizeof(uint32_t), ctx->stream), "clearing counts");
        }
        cudaGraphExec_t exec = segment_graph(m, cg, held);
        if (exec)
            CK(cudaGraphLaunch(exec, ctx->stream), "launching a backward segment");
        else
            CK(enqueue_segment(m, cg, held), "replaying a segment and its backward steps");
        a.seg_holds = (int)j;
        if (!held) ctx->launches += (uint64_t)m * agent_pass_kernels(a.dev, a.n, false) + (m - 1);
        ctx->launches += m;
        if (m & 1) cg = 1 - cg;
    }
    sum_threads_kernel<<<dim3(kSumBlocks, 3), kThreads, 0, ctx->stream>>>(thread_acc, blocks, parts + 4);
    sum_parts_kernel<<<3, kThreads, 0, ctx->stream>>>(parts + 4, parts);
    CK(cudaGetLastError(), "summing gradients");
    ctx->launches += 2;
    double acc[3];
    CK(cudaMemcpyAsync(acc, parts, 3 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream), "reading gradients");
    if (d_trail0)
        CK(cudaMemcpyAsync(d_trail0, a.g[cg], cells * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream),
           "reading dL/dT0");
    CK(cudaStreamSynchronize(ctx->stream), "backward");
    grads->d_decay_factor = acc[0];
    grads->d_diffusion_rate = acc[1];
    grads->d_deposition_amount = acc[2];
    grads->reserved = 0.0;
    return SLIME_OK;
}

} // extern "C"
