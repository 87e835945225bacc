// ytgb_schedule.cuh -- the order in which a render's blocks take its tiles.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <string>

#include "ytgb.h"
#include "ytgb_internal.h"

namespace {

// Tiles cost very different times (an AMR volume's refined regions are crossed
// by many small bricks), and blocks are handed out in grid order: where heavy
// tiles came late, some SMs worked on them long after the others had run dry
// (busiest SM / mean of the 1024^2 AMR frame 1.11, interpolated projection
// 1.17, ten samples per cell 1.37, light source 1.54, the 1024^2 octree frame
// 1.17).  So each tile's work is estimated (from the bricks' pixel rectangles;
// from the octree's cells) and the heavy tiles go first.  Any order gives the
// same image.
// Four steps of cost: more of them part neighbours that share bricks in the
// caches (2 to 16 steps lie within 3 %).
constexpr int SORT_BLOCK = 1024, SORT_BUCKETS = 4;
// (tile numbers and their places are held in 16 bits)
constexpr int MAX_SCHEDULED = 65535;
// Forming the order takes some 30 us, so it is left out where that was not won
// back: with no more tiles than two waves of resident blocks (800 tiles: 3 to 20 %
// lost), with fewer cells of an octree (10,000: 0 to 13 % lost, with one scene 8 %
// won) and from a camera inside it (5 to 14 % lost).  Where it is formed, time in
// grid order / in this order over 90 octree and 132 AMR frames from 320^2 to 1600^2:
// 1.05 on average, 0.92 (an almost uniform octree, 0.8 ms) to 1.43 (a camera from
// which most of the image is empty).
constexpr int ORDER_WAVES = 2;
constexpr int ORDER_CELLS = 1 << 16;
__device__ __forceinline__ int cost_bucket(unsigned c, float scale) {
    const int b = (int)((float)c * scale);
    return SORT_BUCKETS - 1 - (b < SORT_BUCKETS - 1 ? b : SORT_BUCKETS - 1);
}

// tiles[place] = tile, by descending cost in SORT_BUCKETS steps of the largest;
// tiles of one step keep their order, and so their neighbours in the caches.
// One block, a stable counting sort: each warp counts, then places, a run of
// tiles 32 at a time, lanes of one bucket together.  (With a run per thread the
// reads did not coalesce: 8 us more for the 8192 tiles of a 1024^2 frame.)
__global__ void __launch_bounds__(SORT_BLOCK) tile_sort_kernel(const unsigned *cost, int n, unsigned short *tiles) {
    constexpr int WARPS = SORT_BLOCK / 32;
    __shared__ unsigned place[SORT_BUCKETS * WARPS];  // [bucket][warp]
    __shared__ unsigned part[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int run = ((n + WARPS - 1) / WARPS + 31) & ~31;
    const int lo = min(warp * run, n), hi = min(lo + run, n);
    unsigned m = 0;
#pragma unroll 8
    for (int i = t; i < n; i += SORT_BLOCK) m = max(m, cost[i]);
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) part[warp] = m;
    if (t < SORT_BUCKETS * WARPS) place[t] = 0;
    __syncthreads();
    m = __reduce_max_sync(0xffffffffu, part[lane]);
    const float scale = m ? (float)SORT_BUCKETS / (float)m : 0.f;
    // (lanes past the run's end: a bucket of their own, not counted)
    for (int base = lo; base < hi; base += 32) {
        const int i = base + lane;
        const int b = i < hi ? cost_bucket(cost[i], scale) : SORT_BUCKETS;
        const unsigned same = __match_any_sync(0xffffffffu, b);
        if (i < hi && lane == __ffs(same) - 1) place[b * WARPS + warp] += __popc(same);
        __syncwarp();
    }
    __syncthreads();
    // exclusive prefix sums over (bucket, warp)
    const unsigned own = t < SORT_BUCKETS * WARPS ? place[t] : 0u;
    unsigned pre = own;
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, pre, d);
        if (lane >= d) pre += u;
    }
    if (lane == 31) part[warp] = pre;
    __syncthreads();
    unsigned before = lane < warp ? part[lane] : 0u;
    before = __reduce_add_sync(0xffffffffu, before);
    if (t < SORT_BUCKETS * WARPS) place[t] = before + pre - own;
    __syncthreads();
    for (int base = lo; base < hi; base += 32) {
        const int i = base + lane;
        const int b = i < hi ? cost_bucket(cost[i], scale) : SORT_BUCKETS;
        const unsigned same = __match_any_sync(0xffffffffu, b);
        unsigned *at = place + b * WARPS + warp;
        if (i < hi) tiles[*at + __popc(same & ((1u << lane) - 1u))] = (unsigned short)i;
        __syncwarp();
        if (i < hi && lane == __ffs(same) - 1) *at += __popc(same);
        __syncwarp();
    }
}

// A render's scratch memory (device): its tiles' costs, then their order.
struct Scratch {
    void *mem;
    size_t bytes;
};

constexpr size_t scratch_bytes(long long n_tiles) { return (size_t)n_tiles * 6; }

int sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// tiles: the order of n tiles whose costs are in scratch memory, behind them.
int sort_tiles(const Scratch &w, int n, cudaStream_t s, const unsigned short **tiles, const char *what) {
    unsigned short *out = (unsigned short *)((unsigned *)w.mem + n);
    tile_sort_kernel<<<1, SORT_BLOCK, 0, s>>>((const unsigned *)w.mem, n, out);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        ytgb_set_error(std::string(what) + ": " + cudaGetErrorString(e));
        return YTGB_ERR_CUDA;
    }
    *tiles = out;
    return YTGB_OK;
}

}  // namespace
