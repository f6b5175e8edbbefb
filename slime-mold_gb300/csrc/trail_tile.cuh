// trail_tile.cuh - the shared-memory form of the fused deposit-fold + decay +
// diffuse pass (decay_trail, compute.wgsl:148-161, and diffuse_trail,
// compute.wgsl:164-195): any trail width, any blur radius, deposit counts or
// byte marks.
//
// A block computes TW x TH output cells with TW / 4 x 8 threads.  It stages
// its window (the tile and a halo of R cells), folded and decayed, in shared
// memory, blurs the rows into a second buffer and the columns of that buffer
// into the output.  What bounds it is the staging's loads (10 or 16 bytes a
// cell plus the halo) and, for wide radii, shared-memory reads; so
//   * rows of W % 4 == 0 are staged 16 bytes at a time, a thread's loads all
//     issued before the first is used; other widths load one cell per lane,
//     consecutive lanes consecutive cells, and hand the outputs through shared
//     memory so that their stores are consecutive too;
//   * a thread blurs four adjacent columns: the row pass reads 16 bytes of its
//     window at a time, the column pass reads each row of the buffer once and
//     adds it to every output row it belongs to (each output still takes its
//     taps in order, one fused multiply-add a tap).
// The tiles are launched in order and not as programmatic dependents of the agent
// pass: a block that starts while that pass samples takes the SM's L1 for its
// shared memory (3 us more a step at 512^2).  Streaming strips have no such
// carve-out and overlap.
#pragma once

#include "kernels.h"
#include "trail_stream.cuh"

namespace slime {

constexpr int kTileRowSlots = 8; // a block's threads cover 8 rows of the tile at a time

template <int TW, int TH, int R>
struct TileGeom {
    static constexpr int G = TW / 4;                  // 4-column groups per row
    static constexpr int threads = G * kTileRowSlots;
    static constexpr int LP = (R + 3) / 4 * 4;        // columns left (and right) of the tile in shared memory
    static constexpr int stride = TW + 2 * LP;        // floats per window row, a multiple of 4
    static constexpr int SH = TH + 2 * R;             // window rows
    static constexpr int rows = TH / kTileRowSlots;   // output rows per thread
    static constexpr size_t window = (size_t)SH * stride;
};

// Stage the window: s[r * stride + LP + c] holds the folded and decayed cell
// (x0 + c, y0 - R + r) of the torus, for c in [-R, TW + R).
template <int TW, int TH, int R, bool kVec, class D>
__device__ __forceinline__ void stage_window(const DevParams& p, const float* __restrict__ in,
                                             const D* __restrict__ din, float* __restrict__ s, int x0, int y0) {
    typedef TileGeom<TW, TH, R> T;
    constexpr bool kMarks = sizeof(D) == 1;
    const int W = p.W, H = p.H;
    if (kVec) {
        const int g = threadIdx.x % T::G, slot = threadIdx.x / T::G;
        const int gx = wrap_coord(x0 + 4 * g, W);
        constexpr int N = (T::SH + kTileRowSlots - 1) / kTileRowSlots;
        float4 t[N];
        typename DepVec<D>::type k[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int r = slot + i * kTileRowSlots;
            if (r < T::SH) {
                const size_t at = (size_t)wrap_coord(y0 - R + r, H) * W + gx;
                t[i] = __ldg(reinterpret_cast<const float4*>(in + at));
                k[i] = load_dep4<false>(din + at);
            }
        }
        // the halo columns: 2R cells of every row, one per thread
        constexpr int HN = T::SH * 2 * R;
        for (int i = threadIdx.x; i < HN; i += T::threads) {
            const int r = i / (2 * R > 0 ? 2 * R : 1), j = i - r * 2 * R;
            const int c = j < R ? j - R : TW + j - R;
            const size_t at = (size_t)wrap_coord(y0 - R + r, H) * W + wrap_coord(x0 + c, W);
            s[r * T::stride + T::LP + c] = apply_decay(p, fold_dep<kMarks>(__ldg(in + at), load_dep<false>(din + at), p.dep));
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int r = slot + i * kTileRowSlots;
            if (r < T::SH) {
                float4 v;
                v.x = apply_decay(p, fold_dep<kMarks>(t[i].x, dep_at(k[i], 0), p.dep));
                v.y = apply_decay(p, fold_dep<kMarks>(t[i].y, dep_at(k[i], 1), p.dep));
                v.z = apply_decay(p, fold_dep<kMarks>(t[i].z, dep_at(k[i], 2), p.dep));
                v.w = apply_decay(p, fold_dep<kMarks>(t[i].w, dep_at(k[i], 3), p.dep));
                *reinterpret_cast<float4*>(s + r * T::stride + T::LP + 4 * g) = v;
            }
        }
    } else {
        // a warp per row, a lane per cell
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        constexpr int kWarps = T::threads / 32;
        constexpr int N = (TW + 2 * R + 31) / 32;
        int gx[N];
#pragma unroll
        for (int i = 0; i < N; i++) gx[i] = wrap_coord(x0 - R + min(lane + 32 * i, TW + 2 * R - 1), W);
#pragma unroll 2
        for (int r = warp; r < T::SH; r += kWarps) {
            const size_t row = (size_t)wrap_coord(y0 - R + r, H) * W;
            float t[N];
            uint32_t k[N];
#pragma unroll
            for (int i = 0; i < N; i++) {
                t[i] = __ldg(in + row + gx[i]);
                k[i] = load_dep<false>(din + row + gx[i]);
            }
#pragma unroll
            for (int i = 0; i < N; i++) {
                const int c = lane + 32 * i;
                if (c < TW + 2 * R) s[r * T::stride + T::LP - R + c] = apply_decay(p, fold_dep<kMarks>(t[i], k[i], p.dep));
            }
        }
    }
}

template <int TW, int TH, int R>
__device__ __forceinline__ void stage_any(const DevParams& p, const float* __restrict__ in,
                                          const uint32_t* __restrict__ counts, const uint8_t* __restrict__ marks,
                                          bool vec, float* __restrict__ s, int x0, int y0) {
    if (vec) {
        if (marks) stage_window<TW, TH, R, true, uint8_t>(p, in, marks, s, x0, y0);
        else stage_window<TW, TH, R, true, uint32_t>(p, in, counts, s, x0, y0);
    } else {
        if (marks) stage_window<TW, TH, R, false, uint8_t>(p, in, marks, s, x0, y0);
        else stage_window<TW, TH, R, false, uint32_t>(p, in, counts, s, x0, y0);
    }
}

// Where a pass's outputs go: the new trail and the deposit record it clears.
struct TileOut {
    float* __restrict__ out;
    uint32_t* __restrict__ counts_zero;
    uint8_t* __restrict__ marks_zero;
};

__device__ __forceinline__ void store4(const TileOut& o, size_t at, const float* v) {
    *reinterpret_cast<float4*>(o.out + at) = make_float4(v[0], v[1], v[2], v[3]);
    if (o.marks_zero) zero_dep4(o.marks_zero + at);
    else if (o.counts_zero) zero_dep4(o.counts_zero + at);
}

// Rows of any width: the warp's finished rows, in shared memory at
// s + row * stride, written one cell per lane.
template <int TW, int ROWS>
__device__ __forceinline__ void store_rows(const DevParams& p, const TileOut& o, const float* __restrict__ s, int stride,
                                           int x0, int y, int rows_per_slot_gap) {
    const int lane = threadIdx.x & 31;
    constexpr int kSlots = 128 / TW; // row slots of one warp
#pragma unroll
    for (int q = 0; q < kSlots; q++) {
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const int yy = y + q * rows_per_slot_gap + r;
            if (yy >= p.H) break;
            const float* row = s + (q * rows_per_slot_gap + r) * stride;
#pragma unroll
            for (int i = 0; i < TW / 32; i++) {
                const int c = lane + 32 * i;
                if (x0 + c < p.W) {
                    const size_t at = (size_t)yy * p.W + x0 + c;
                    o.out[at] = row[c];
                    if (o.marks_zero) o.marks_zero[at] = 0;
                    else if (o.counts_zero) o.counts_zero[at] = 0u;
                }
            }
        }
    }
}

template <int TW, int TH>
__global__ void __launch_bounds__(TileGeom<TW, TH, 1>::threads) trail_box3_kernel(
    const __grid_constant__ DevParams p, const float* __restrict__ in, const uint32_t* __restrict__ counts,
    const uint8_t* __restrict__ marks, const TileOut o, int tiles_x, int vec) {
    typedef TileGeom<TW, TH, 1> T;
    extern __shared__ __align__(16) float smem[];
    float* s = smem;
    const int by = blockIdx.x / tiles_x;
    const int x0 = (blockIdx.x - by * tiles_x) * TW, y0 = by * TH;
    stage_any<TW, TH, 1>(p, in, counts, marks, vec != 0, s, x0, y0);
    __syncthreads();
    const int g = threadIdx.x % T::G, slot = threadIdx.x / T::G;
    const int ry = slot * T::rows;
    float win[3][6]; // window rows, columns 4g-1 .. 4g+4
    float* own = smem + T::window; // rows of any width: the finished tile
#pragma unroll
    for (int q = 0; q < T::rows + 2; q++) {
#pragma unroll
        for (int j = 0; j < 6; j++) {
            win[0][j] = win[1][j];
            win[1][j] = win[2][j];
        }
        const float* row = s + (ry + q) * T::stride + T::LP + 4 * g;
        const float4 v = *reinterpret_cast<const float4*>(row);
        win[2][0] = row[-1];
        win[2][1] = v.x;
        win[2][2] = v.y;
        win[2][3] = v.z;
        win[2][4] = v.w;
        win[2][5] = row[4];
        if (q < 2) continue;
        const int y = y0 + ry + q - 2;
        float res[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float sum = 0.0f;
#pragma unroll
            for (int dy = 0; dy < 3; dy++)
#pragma unroll
                for (int dx = 0; dx < 3; dx++) sum = slm_add(sum, win[dy][j + dx]);
            res[j] = sum;
        }
        slm_div9x4(res);
#pragma unroll
        for (int j = 0; j < 4; j++) res[j] = slm_mix(win[1][1 + j], res[j], p.rate);
        if (vec) {
            if (y < p.H && x0 + 4 * g < p.W) store4(o, (size_t)y * p.W + x0 + 4 * g, res);
        } else {
            *reinterpret_cast<float4*>(own + (ry + q - 2) * TW + 4 * g) = make_float4(res[0], res[1], res[2], res[3]);
        }
    }
    if (!vec) {
        __syncwarp();
        const int ry0 = __shfl_sync(0xffffffffu, ry, 0); // the warp's first row
        store_rows<TW, T::rows>(p, o, own + ry0 * TW, TW, x0, y0 + ry0, T::rows);
    }
}

template <int TW, int TH, int R>
__global__ void __launch_bounds__(TileGeom<TW, TH, R>::threads) trail_gauss_kernel(
    const __grid_constant__ DevParams p, const float* __restrict__ in, const uint32_t* __restrict__ counts,
    const uint8_t* __restrict__ marks, const TileOut o, int tiles_x, int vec) {
    typedef TileGeom<TW, TH, R> T;
    extern __shared__ __align__(16) float smem[];
    float* s = smem;             // SH x stride: the window
    float* h = smem + T::window; // SH x TW: its rows blurred
    const int by = blockIdx.x / tiles_x;
    const int x0 = (blockIdx.x - by * tiles_x) * TW, y0 = by * TH;
    stage_any<TW, TH, R>(p, in, counts, marks, vec != 0, s, x0, y0);
    __syncthreads();
    const int g = threadIdx.x % T::G, slot = threadIdx.x / T::G;
    // row pass: a thread reads columns 4g - LP .. 4g + 3 + LP of a row
    for (int r = slot; r < T::SH; r += kTileRowSlots) {
        float e[4 + 2 * T::LP];
        const float* row = s + r * T::stride + 4 * g;
#pragma unroll
        for (int i = 0; i < 1 + T::LP / 2; i++) {
            const float4 v = *reinterpret_cast<const float4*>(row + 4 * i);
            e[4 * i] = v.x;
            e[4 * i + 1] = v.y;
            e[4 * i + 2] = v.z;
            e[4 * i + 3] = v.w;
        }
        float acc[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            acc[j] = 0.0f;
#pragma unroll
            for (int t = 0; t <= 2 * R; t++) acc[j] = slm_fma(p.w[t], e[T::LP - R + j + t], acc[j]);
        }
        *reinterpret_cast<float4*>(h + r * TW + 4 * g) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    }
    __syncthreads();
    // column pass: `rows` output rows per thread, each row of h read once
    const int ry = slot * T::rows;
    float acc[T::rows][4];
#pragma unroll
    for (int q = 0; q < T::rows; q++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[q][j] = 0.0f;
#pragma unroll
    for (int q = 0; q < T::rows + 2 * R; q++) {
        const float4 v = *reinterpret_cast<const float4*>(h + (ry + q) * TW + 4 * g);
#pragma unroll
        for (int y = 0; y < T::rows; y++) {
            const int t = q - y; // the tap this row is for output row y
            if (t >= 0 && t <= 2 * R) {
                acc[y][0] = slm_fma(p.w[t], v.x, acc[y][0]);
                acc[y][1] = slm_fma(p.w[t], v.y, acc[y][1]);
                acc[y][2] = slm_fma(p.w[t], v.z, acc[y][2]);
                acc[y][3] = slm_fma(p.w[t], v.w, acc[y][3]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < T::rows; q++) {
        float* own = s + (ry + q + R) * T::stride + T::LP + 4 * g;
        const float4 c = *reinterpret_cast<const float4*>(own);
        const float res[4] = {slm_mix(c.x, acc[q][0], p.rate), slm_mix(c.y, acc[q][1], p.rate),
                              slm_mix(c.z, acc[q][2], p.rate), slm_mix(c.w, acc[q][3], p.rate)};
        if (vec) {
            const int y = y0 + ry + q;
            if (y < p.H && x0 + 4 * g < p.W) store4(o, (size_t)y * p.W + x0 + 4 * g, res);
        } else {
            // the window's own cells are read by nobody else any more
            *reinterpret_cast<float4*>(own) = make_float4(res[0], res[1], res[2], res[3]);
        }
    }
    if (!vec) {
        __syncwarp();
        const int ry0 = __shfl_sync(0xffffffffu, ry, 0);
        store_rows<TW, T::rows>(p, o, s + (ry0 + R) * T::stride + T::LP, T::stride, x0, y0 + ry0, T::rows);
    }
}

// Whether the 16-byte path applies: whole groups of four columns in every
// row, and every buffer's rows 16-byte aligned (4-byte for marks).
inline bool tile_vec(const DevParams& p, const float* in, const uint32_t* counts, const uint8_t* marks,
                     const TileOut& o) {
    const uintptr_t a16 = (uintptr_t)in | (uintptr_t)o.out | (marks ? 0 : (uintptr_t)counts | (uintptr_t)o.counts_zero);
    const uintptr_t a4 = marks ? (uintptr_t)marks | (uintptr_t)o.marks_zero : 0;
    return p.W % 4 == 0 && (a16 & 15) == 0 && (a4 & 3) == 0;
}

template <typename K>
cudaError_t launch_tile_kernel(K k, const DevParams& p, int tw, int th, int threads, size_t smem, const float* in,
                               const uint32_t* counts, const uint8_t* marks, const TileOut& o, cudaStream_t s,
                               const cudaAccessPolicyWindow* win) {
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const int tiles_x = (p.W + tw - 1) / tw;
    const long long tiles = (long long)tiles_x * ((p.H + th - 1) / th);
    return launch_k(k, dim3((unsigned)tiles), dim3(threads), smem, s, win, p, in, counts, marks, o, tiles_x,
                    (int)tile_vec(p, in, counts, marks, o));
}

template <int TW, int TH, int R>
cudaError_t launch_gauss_tile(const DevParams& p, const float* in, const uint32_t* counts, const uint8_t* marks,
                              const TileOut& o, cudaStream_t s, const cudaAccessPolicyWindow* win) {
    typedef TileGeom<TW, TH, R> T;
    return launch_tile_kernel(trail_gauss_kernel<TW, TH, R>, p, TW, TH, T::threads,
                              sizeof(float) * (T::window + (size_t)T::SH * TW), in, counts, marks, o, s, win);
}

template <int TW, int TH>
cudaError_t launch_tile(const DevParams& p, const float* in, const uint32_t* counts, const uint8_t* marks,
                        const TileOut& o, cudaStream_t s, const cudaAccessPolicyWindow* win) {
    if (p.blur_mode != SLIME_BLUR_GAUSS) {
        typedef TileGeom<TW, TH, 1> T;
        return launch_tile_kernel(trail_box3_kernel<TW, TH>, p, TW, TH, T::threads,
                                  sizeof(float) * (T::window + (size_t)TH * TW), in, counts, marks, o, s, win);
    }
    switch (p.R) {
    case 0: return launch_gauss_tile<TW, TH, 0>(p, in, counts, marks, o, s, win); // the identity; weights are {1}
    case 1: return launch_gauss_tile<TW, TH, 1>(p, in, counts, marks, o, s, win);
    case 2: return launch_gauss_tile<TW, TH, 2>(p, in, counts, marks, o, s, win);
    case 3: return launch_gauss_tile<TW, TH, 3>(p, in, counts, marks, o, s, win);
    case 4: return launch_gauss_tile<TW, TH, 4>(p, in, counts, marks, o, s, win);
    case 5: return launch_gauss_tile<TW, TH, 5>(p, in, counts, marks, o, s, win);
    case 6: return launch_gauss_tile<TW, TH, 6>(p, in, counts, marks, o, s, win);
    case 7: return launch_gauss_tile<TW, TH, 7>(p, in, counts, marks, o, s, win);
    case 8: return launch_gauss_tile<TW, TH, 8>(p, in, counts, marks, o, s, win);
    default: return cudaErrorInvalidValue;
    }
}

// The instantiations (trail_tile_64.cu, trail_tile_128.cu, trail_tile_128t.cu).
#define SLIME_TILE_ARGS                                                                                      \
    const DevParams &p, const float *in, const uint32_t *counts, const uint8_t *marks, const TileOut &o,     \
        cudaStream_t s, const cudaAccessPolicyWindow *win
cudaError_t launch_tile_64x8(SLIME_TILE_ARGS);
cudaError_t launch_tile_64x16(SLIME_TILE_ARGS);
cudaError_t launch_tile_64x32(SLIME_TILE_ARGS);
cudaError_t launch_tile_128x8(SLIME_TILE_ARGS);
cudaError_t launch_tile_128x16(SLIME_TILE_ARGS);
cudaError_t launch_tile_128x32(SLIME_TILE_ARGS);
cudaError_t launch_tile_128x64(SLIME_TILE_ARGS);

} // namespace slime
