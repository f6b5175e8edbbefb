// reorder.cu - Morton reordering of agent slots.
//
// Agents that sit in nearby cells sense and deposit into nearby trail lines;
// placing them in neighbouring slots turns the agent pass's scattered 4-byte
// gathers into a few shared lines per warp.  The order of slots does not
// change any result: sensing reads the pre-step trail, deposits are counted,
// and every slot carries its original id (which seeds the jitter hash), so the
// reorder is a pure performance transform.
//
// Counting sort on the Morton code of the agent's (cell >> cell_log2):
// key + histogram, exclusive scan, scatter to scratch as one 16-byte record and
// an id per agent (a slot's five fields scattered each on its own would cost
// five memory sectors an agent when the agents come unsorted, 160 bytes against
// 64), and a pass that unpacks the records into the fields' arrays: the
// agents' own, or another set, which is then sorted while the first stays as
// it is.  A key has as many bits as the two sides need: where one side is longer
// its upper bits stand above the interleaved ones (the order of the codes of a
// square, whose unused bits are left out), so there are no more keys than four
// times the squares of cells, however long and thin the trail.  The order inside
// one key is whatever the scatter atomics produce.  Agents whose id is at or above `visited` (those the reference's dispatch never updates) get
// one key past every Morton code, so they end up in the last slots and the
// updated agents fill the first ones.
#include "kernels.h"

namespace slime {
namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t spread_bits(uint32_t v) {
    v &= 0xffffu;
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}

// Agents that are already nearly in order share keys with their warp
// neighbours (about 2^(2 cell_log2) per key at one agent per cell), so the
// histogram and the slot claims are aggregated per warp: the lanes holding
// one key elect a leader that adds the group's size with a single atomic.
__global__ void key_hist_kernel(const float* __restrict__ x, const float* __restrict__ y,
                                const uint32_t* __restrict__ ids, uint64_t visited, uint32_t frozen_key, uint64_t n,
                                int W, int H, int cl, int low, uint32_t* __restrict__ keys,
                                uint32_t* __restrict__ hist) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int cx = min(max(slm_f2i(x[i]), 0), W - 1) >> cl;
    int cy = min(max(slm_f2i(y[i]), 0), H - 1) >> cl;
    const uint32_t mask = (1u << low) - 1u; // `low` bits of either side are interleaved
    uint32_t k = spread_bits((uint32_t)cx & mask) | (spread_bits((uint32_t)cy & mask) << 1);
    if (low < 16) k |= (((uint32_t)cx | (uint32_t)cy) >> low) << (2 * low);
    if (visited < n && (ids ? ids[i] : (uint32_t)i) >= visited) k = frozen_key;
    keys[i] = k;
    const unsigned group = __match_any_sync(__activemask(), k);
    if ((int)(threadIdx.x & 31) == __ffs(group) - 1) atomicAdd(hist + k, (uint32_t)__popc(group));
}

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t ws = (lane < (int)(blockDim.x >> 5)) ? warp_sums[lane] : 0u;
        uint32_t wi = ws;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        warp_sums[lane] = wi - ws;
        if (lane == 31) *total = wi;
    }
    __syncthreads();
    uint32_t r = warp_sums[warp] + incl - v;
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const uint32_t* __restrict__ in, uint64_t n,
                                                                   uint32_t* __restrict__ block_sums) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t tot;
    uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t s = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; j++)
        if (base + j < n) s += in[base + j];
    block_exclusive_scan(s, ws, &tot);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = tot;
}

// Single block: exclusive scan of the block sums in place.
__global__ void __launch_bounds__(kScanThreads) scan_block_sums_kernel(uint32_t* __restrict__ sums, uint32_t nb) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t tot;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < nb; base += kScanThreads) {
        uint32_t i = base + threadIdx.x;
        uint32_t v = i < nb ? sums[i] : 0u;
        uint32_t ex = block_exclusive_scan(v, ws, &tot);
        if (i < nb) sums[i] = carry + ex;
        carry += tot;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(uint32_t* __restrict__ data, uint64_t n,
                                                                  const uint32_t* __restrict__ block_offsets) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t tot;
    uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        v[j] = (base + j < n) ? data[base + j] : 0u;
        s += v[j];
    }
    uint32_t ex = block_exclusive_scan(s, ws, &tot) + block_offsets[blockIdx.x];
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        if (base + j < n) data[base + j] = ex;
        ex += v[j];
    }
}

__global__ void scatter_kernel(const float* __restrict__ x, const float* __restrict__ y,
                               const float* __restrict__ th, const float* __restrict__ v,
                               const uint32_t* __restrict__ ids, const uint32_t* __restrict__ keys, uint64_t n,
                               uint32_t* __restrict__ offsets, float4* __restrict__ rec, uint32_t* __restrict__ rid) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t k = keys[i];
    const float4 a = make_float4(__ldcs(x + i), __ldcs(y + i), __ldcs(th + i), __ldcs(v + i));
    const uint32_t id = ids ? __ldcs(ids + i) : (uint32_t)i;
    const unsigned active = __activemask();
    const unsigned group = __match_any_sync(active, k);
    const int lane = (int)(threadIdx.x & 31);
    const int leader = __ffs(group) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(offsets + k, (uint32_t)__popc(group));
    base = __shfl_sync(active, base, leader);
    // slots of one key are claimed in lane order within the warp
    const uint32_t pos = base + (uint32_t)__popc(group & ((1u << lane) - 1u));
    rec[pos] = a;
    rid[pos] = id;
}

__global__ void unpack_kernel(const float4* __restrict__ rec, const uint32_t* __restrict__ rid, uint64_t n,
                              float* __restrict__ x, float* __restrict__ y, float* __restrict__ th,
                              float* __restrict__ v, uint32_t* __restrict__ ids) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = __ldcs(rec + i);
    x[i] = a.x;
    y[i] = a.y;
    th[i] = a.z;
    v[i] = a.w;
    ids[i] = __ldcs(rid + i);
}

__global__ void iota_kernel(uint32_t* __restrict__ ids, uint64_t n) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ids[i] = (uint32_t)i;
}

inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

} // namespace

cudaError_t launch_iota(uint32_t* ids, uint64_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    iota_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(ids, n);
    return cudaGetLastError();
}

namespace {

// Bits of the sort key along a side.
int key_bits(uint32_t side, int cell_log2) {
    const uint32_t d = (side + (1u << cell_log2) - 1) >> cell_log2;
    int L = 0;
    while ((1u << L) < d) L++;
    return L;
}

struct ReorderSizes {
    uint64_t keys, blocks; // histogram entries, and blocks that scan them
    size_t bytes;          // of scratch
};
ReorderSizes reorder_sizes(uint64_t n, uint32_t W, uint32_t H, int cell_log2, bool partition) {
    ReorderSizes r;
    r.keys = (1ull << (key_bits(W, cell_log2) + key_bits(H, cell_log2))) + (partition ? 1 : 0);
    r.blocks = (r.keys + kScanTile - 1) / kScanTile;
    r.bytes = align256(4 * n) /*keys*/ + align256(4 * r.keys) /*histogram*/ + align256(4 * r.blocks) /*block sums*/ +
              align256(16 * n) /*records*/ + align256(4 * n) /*ids*/;
    return r;
}

} // namespace

size_t reorder_scratch_bytes(uint64_t n, uint32_t W, uint32_t H, int cell_log2) {
    const int lx = key_bits(W, cell_log2), ly = key_bits(H, cell_log2);
    if (lx > 16 || ly > 16) return 0;
    return reorder_sizes(n, W, H, cell_log2, false).bytes;
}

cudaError_t launch_reorder(const AgentsSoA& a, const AgentsSoA& to, uint32_t W, uint32_t H, int cell_log2,
                           ReorderScratch& scratch, cudaStream_t s, uint64_t visited) {
    if (a.n == 0) return cudaSuccess;
    if (!to.ids) return cudaErrorInvalidValue;
    if (cell_log2 < 0) cell_log2 = 0;
    if (cell_log2 > 15) cell_log2 = 15;
    const int lx = key_bits(W, cell_log2), ly = key_bits(H, cell_log2);
    if (lx > 16 || ly > 16) return cudaErrorInvalidValue;
    const bool partition = visited < a.n;
    if (partition && (lx > 15 || ly > 15)) return cudaErrorInvalidValue; // no key left past the Morton codes
    const uint32_t frozen_key = (uint32_t)(1ull << (lx + ly));
    const uint64_t n = a.n;
    const ReorderSizes size = reorder_sizes(n, W, H, cell_log2, partition);
    const uint64_t nb = size.keys, nblk = size.blocks;
    const size_t need = size.bytes;
    if (scratch.bytes < need) {
        if (scratch.buf) dev_free(scratch.buf);
        scratch.buf = nullptr;
        scratch.bytes = 0;
        cudaError_t e = dev_alloc((void**)&scratch.buf, need);
        if (e != cudaSuccess) return e;
        scratch.bytes = need;
    }
    char* p = (char*)scratch.buf;
    uint32_t* keys = (uint32_t*)p; p += align256(4 * n);
    uint32_t* hist = (uint32_t*)p; p += align256(4 * nb);
    uint32_t* bsum = (uint32_t*)p; p += align256(4 * nblk);
    float4* rec = (float4*)p; p += align256(16 * n);
    uint32_t* rid = (uint32_t*)p;

    cudaError_t e = cudaMemsetAsync(hist, 0, 4 * nb, s);
    if (e != cudaSuccess) return e;
    unsigned blocks = (unsigned)((n + 255) / 256);
    key_hist_kernel<<<blocks, 256, 0, s>>>(a.x, a.y, a.ids, visited, frozen_key, n, (int)W, (int)H, cell_log2, lx < ly ? lx : ly,
                                          keys, hist);
    scan_reduce_kernel<<<(unsigned)nblk, kScanThreads, 0, s>>>(hist, nb, bsum);
    scan_block_sums_kernel<<<1, kScanThreads, 0, s>>>(bsum, (uint32_t)nblk);
    scan_apply_kernel<<<(unsigned)nblk, kScanThreads, 0, s>>>(hist, nb, bsum);
    scatter_kernel<<<blocks, 256, 0, s>>>(a.x, a.y, a.th, a.v, a.ids, keys, n, hist, rec, rid);
    unpack_kernel<<<blocks, 256, 0, s>>>(rec, rid, n, to.x, to.y, to.th, to.v, to.ids);
    return cudaGetLastError();
}

} // namespace slime
