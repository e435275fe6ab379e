// Exclusive scan of a generated sequence in two launches: totals per tile, then each tile
// scans itself and hands every element its prefix. A block of the second launch adds up the
// totals of the tiles before its own, so nothing waits on another block; above SCAN_DIRECT
// tiles the totals are scanned first, by the same two launches.
//   In:  uint32_t operator()(int i) const             the i-th value
//   Out: void operator()(int i, uint32_t v, uint32_t prefix) const
//        void total(uint32_t sum) const               called once
// The build's two scans, with an array for every stage, were 13 launches and 108 us of the
// launch list at N = 4M, 38 us at N = 10000; generated in place they are 4, 56 and 24 us.
#pragma once

#include "pt_prims.cuh"

namespace pt {
namespace scan {

constexpr int THREADS = 256;
constexpr int ITEMS = 16;  // values per thread
constexpr int TILE = THREADS * ITEMS;
constexpr int SCAN_DIRECT = 2048;

__device__ __forceinline__ uint32_t warp_incl(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive scan of one value per thread over the block; *total gets the sum.
__device__ __forceinline__ uint32_t block_excl(uint32_t v, uint32_t *total) {
    __shared__ uint32_t wsum[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t incl = warp_incl(v);
    __syncthreads();  // an earlier call's wsum is read
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t before = 0, sum = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
        const uint32_t s = wsum[w];
        if (w < warp) before += s;
        sum += s;
    }
    *total = sum;
    return before + incl - v;
}

// Warp w of the tile owns its w-th run of 32 x ITEMS values, read 32 at a time.
__device__ __forceinline__ int first_item(int tile) {
    return tile * TILE + (threadIdx.x >> 5) * (32 * ITEMS) + (threadIdx.x & 31);
}

template <class In>
__global__ void __launch_bounds__(THREADS) tile_sums(In in, int n, uint32_t *__restrict__ sums) {
    after_previous();
    const int i0 = first_item(blockIdx.x);
    uint32_t s = 0;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
        if (i0 + 32 * r < n) s += in(i0 + 32 * r);
    uint32_t total;
    block_excl(s, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

template <class In, class Out>
__global__ void __launch_bounds__(THREADS)
    scan_apply(In in, Out out, int n, const uint32_t *__restrict__ sums, int scanned) {
    after_previous();
    uint32_t before = 0;
    if (scanned) {
        before = sums[blockIdx.x];
    } else {
        uint32_t s = 0;
        for (int b = threadIdx.x; b < int(blockIdx.x); b += THREADS) s += sums[b];
        block_excl(s, &before);
    }
    const int i0 = first_item(blockIdx.x);
    uint32_t v[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) v[r] = i0 + 32 * r < n ? in(i0 + 32 * r) : 0u;
    // prefixes within the warp's run: lanes first, then rounds
    uint32_t pre[ITEMS], run = 0;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t incl = warp_incl(v[r]);
        pre[r] = run + incl - v[r];
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    uint32_t total;
    const uint32_t mine = block_excl((threadIdx.x & 31) == 0 ? run : 0u, &total);
    const uint32_t base = before + __shfl_sync(0xffffffffu, mine, 0);
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
        if (i0 + 32 * r < n) out(i0 + 32 * r, v[r], base + pre[r]);
    if (threadIdx.x == 0 && (blockIdx.x + 1) * TILE >= n) out.total(before + total);
}

struct ReadU32 {
    const uint32_t *p;
    __device__ uint32_t operator()(int i) const { return p[i]; }
};
struct WriteU32 {  // out[n] gets the total
    uint32_t *p;
    int n;
    __device__ void operator()(int i, uint32_t, uint32_t prefix) const { p[i] = prefix; }
    __device__ void total(uint32_t sum) const { p[n] = sum; }
};

// Words of scratch for n values: the tiles' totals, and their scan where they are many.
inline size_t scratch_words(int n) {
    size_t words = 0;
    for (long long m = n;;) {
        m = (m + TILE - 1) / TILE;
        words += 2 * size_t(m) + 2;
        if (m <= SCAN_DIRECT) return words;
    }
}

template <class In, class Out>
int run(pt_ctx *ctx, const In &in, const Out &out, int n, uint32_t *tmp) {
    const int tiles = (n + TILE - 1) / TILE;
    uint32_t *sums = tmp;
    launch_next(tile_sums<In>, tiles, THREADS, 0, ctx->stream, in, n, sums);
    PT_TRY(check_launch(ctx, "tile_sums"));
    const uint32_t *pre = sums;
    if (tiles > SCAN_DIRECT) {
        uint32_t *scanned = tmp + tiles;
        PT_TRY(run(ctx, ReadU32{sums}, WriteU32{scanned, tiles}, tiles, tmp + 2 * size_t(tiles) + 2));
        pre = scanned;
    }
    launch_next(scan_apply<In, Out>, tiles, THREADS, 0, ctx->stream, in, out, n, pre, int(tiles > SCAN_DIRECT));
    return check_launch(ctx, "scan_apply");
}

}  // namespace scan

// Scans n > 0 generated values on ctx->stream.
template <class In, class Out>
int scan_generated(pt_ctx *ctx, PrimScratch &s, const In &in, const Out &out, int n) {
    PT_TRY(ensure_buf(ctx, s.scan, scan::scratch_words(n) * sizeof(uint32_t)));
    return scan::run(ctx, in, out, n, static_cast<uint32_t *>(s.scan.ptr));
}

}  // namespace pt
