// Stable radix sort of 63-bit keys and their bodies' indices, written for the Barnes-Hut build.
//
// The upper bits (see head_shift) are sorted by LSD passes of 8-bit digits; bodies that share
// them are few and next to each other then, and rs_finish orders each such run by the whole
// key. The runs that are too long for it (a cluster far smaller than 2^-13 of the box) it puts
// on a list; rs_runs, launched in any case, sorts these by their lower digits, a block or a
// cluster of blocks to a run. Where much of a large input is in such runs (a sample of the keys
// tells) three passes over the lower bits come first instead. Nothing in a sort waits on a
// block that may not be running.
//
// A pass ranks keys stably inside a tile (each warp its own run of keys, with warp
// match/popc), so equal digits keep their input order, stages the tile in shared memory in
// digit order and writes every digit's run contiguously. Up to 262144 keys a pass is
// one launch: every block adds up the tiles' digit counts itself, and counts the digits of
// the next pass as it writes. Above, a histogram pass (per-tile counts) and a row scan (one
// block per digit value over the tiles) come before the scatter.
#include "pt_prims.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace pt {
namespace prims {

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// ---- radix sort ------------------------------------------------------------
constexpr int RS_THREADS = 256;
constexpr int RS_ROUNDS = 8;  // keys per thread of a tile
constexpr int RS_TILE = RS_THREADS * RS_ROUNDS;
constexpr int RS_WARPS = RS_THREADS / 32;

// Keys per thread of a tile of the direct passes, or 0 from where a pass takes three launches.
// Few tiles keep the sum over them short, many keep the chip busy. A whole call at 10000 bodies
// takes 179 us with tiles of 256 keys and 187 with 2048, at 65536 274 with 1024 and 280 with
// 2048 (318 with 256), at 131072 350 with 2048 and 355 with 1024; at 262144 534 against 541
// with three launches a pass.
static int direct_rounds(int n) { return n <= 64 * 256 ? 1 : n <= 64 * 1024 ? 4 : n <= 128 * 2048 ? 8 : 0; }

// Exclusive scan of one value per thread over the 256 threads of a block; wsum holds
// RS_WARPS + 1 words. Every thread of the block must call it.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *wsum, uint32_t *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t incl = warp_incl_scan(v);
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < RS_WARPS ? wsum[lane] : 0u;
        const uint32_t wi = warp_incl_scan(w);
        if (lane < RS_WARPS) wsum[lane] = wi - w;
        if (lane == RS_WARPS - 1) wsum[RS_WARPS] = wi;
    }
    __syncthreads();
    const uint32_t r = wsum[warp] + incl - v;
    if (total) *total = wsum[RS_WARPS];
    __syncthreads();
    return r;
}

__device__ __forceinline__ uint32_t digit_of(uint64_t key, int shift) { return uint32_t(key >> shift) & 255u; }

// hist[d * nblocks + b] = count of digit d in tile b.
__device__ __forceinline__ void hist_tile(const uint64_t *__restrict__ keys, int n, int shift,
                                          uint32_t *__restrict__ hist, int nblocks, int b, uint32_t *cnt) {
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const size_t base = size_t(b) * RS_TILE;
#pragma unroll 4
    for (int r = 0; r < RS_ROUNDS; ++r) {
        const size_t i = base + size_t(r) * RS_THREADS + threadIdx.x;
        if (i < size_t(n)) atomicAdd(&cnt[digit_of(__ldcg(keys + i), shift)], 1u);
    }
    __syncthreads();
    hist[size_t(threadIdx.x) * nblocks + b] = cnt[threadIdx.x];
}

// Where bodies crowd (*deep), LOW_PASSES over the lower bits come before the passes of three
// launches over the upper ones, which then start from the other pair of buffers. (In long runs
// for a few clusters of blocks a large tree's bodies take longer than in the passes that the whole
// chip makes: builds without and with them, us, N = 1M in two knots 1e-5 of the box wide 1018 /
// 499, a Plummer sphere with one body 2e4 away 887 / 444; 4M 3387 / 1268 and 3160 / 1452. The
// launches that find nothing to do cost every other build above 262144 bodies 8 us, of 190 and more.)
constexpr int LOW_PASSES = 3;

// A pass of three launches, from pair `in` of the buffers (the other if *deep) to the other.
// first: unless *deep, a key's value is its index.
struct Pass {
    uint64_t *k0, *k1;
    uint32_t *v0, *v1;
    const int *deep;
    int shift, in;
    bool first;
};

__global__ void __launch_bounds__(RS_THREADS) rs_hist(Pass p, int n, uint32_t *__restrict__ hist, int nblocks) {
    after_previous();
    __shared__ uint32_t cnt[256];
    hist_tile(p.in ^ *p.deep ? p.k1 : p.k0, n, p.shift, hist, nblocks, blockIdx.x, cnt);
}

// Digit d: offs[d * nblocks + b] = count of digit d in tiles before b, rowsum[d] = count of
// digit d.
__device__ __forceinline__ void scan_row(const uint32_t *__restrict__ hist, uint32_t *__restrict__ offs,
                                         uint32_t *__restrict__ rowsum, int nblocks, int d, uint32_t *wsum) {
    const uint32_t *row = hist + size_t(d) * nblocks;
    uint32_t *orow = offs + size_t(d) * nblocks;
    const int q = (nblocks + RS_THREADS - 1) / RS_THREADS;
    const int b0 = min(nblocks, int(threadIdx.x) * q), b1 = min(nblocks, b0 + q);
    uint32_t s = 0;
    for (int b = b0; b < b1; ++b) s += __ldcg(row + b);
    uint32_t total;
    uint32_t acc = block_excl_scan(s, wsum, &total);
    for (int b = b0; b < b1; ++b) {
        const uint32_t h = __ldcg(row + b);
        orow[b] = acc;
        acc += h;
    }
    if (threadIdx.x == 0) rowsum[d] = total;
}

__global__ void __launch_bounds__(RS_THREADS)
    rs_rowscan(const uint32_t *__restrict__ hist, uint32_t *__restrict__ offs, uint32_t *__restrict__ rowsum,
               int nblocks) {
    after_previous();
    __shared__ uint32_t wsum[RS_WARPS + 1];
    scan_row(hist, offs, rowsum, nblocks, blockIdx.x, wsum);
}

template <int ROUNDS>
struct ScatterShared {
    uint64_t skeys[RS_THREADS * ROUNDS];
    uint32_t svals[RS_THREADS * ROUNDS];
    alignas(16) uint32_t wcnt[RS_WARPS][256];
    uint32_t tstart[256], gbase[256];
    uint32_t wsum[RS_WARPS + 1];
};

// Tile b's part of a pass: ranks its keys stably by digit, stages them in shared memory in
// digit order, then writes each digit's run to its global range (consecutive threads write
// consecutive addresses). Warp w owns the tile's w-th run of 32 * RS_ROUNDS keys and ranks
// them round by round with warp match/popc against its own digit counters (no block barrier
// between rounds); one scan over the warps per digit then orders the warps, so equal digits
// keep their input order. gstart(t): where digit t's keys of this tile go. vin null: a key's
// value is its index. next: null, or the digit counts by tile of the pass at next_shift. (All
// reads go to L2: within rs_runs other blocks have written what an earlier pass read.)
template <int ROUNDS, class Start>
__device__ __forceinline__ void scatter_tile(ScatterShared<ROUNDS> &S, const uint64_t *kin, const uint32_t *vin,
                                             uint64_t *kout, uint32_t *vout, int n, int shift, int b,
                                             const Start &gstart, uint32_t *next, int next_shift) {
    constexpr int TILE = RS_THREADS * ROUNDS;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const size_t wbase = size_t(b) * TILE + size_t(warp) * (32 * ROUNDS);
    uint64_t key[ROUNDS];
    uint32_t val[ROUNDS], rank[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const size_t i = wbase + size_t(r) * 32 + lane;
        const bool valid = i < size_t(n);
        key[r] = valid ? __ldcg(kin + i) : 0ull;
        val[r] = valid ? (vin ? __ldcg(vin + i) : uint32_t(i)) : 0u;
    }
    S.gbase[t] = gstart(t);
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) S.wcnt[w][t] = 0;
    __syncthreads();
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const bool valid = wbase + size_t(r) * 32 + lane < size_t(n);
        const uint32_t d = valid ? digit_of(key[r], shift) : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        // keys of digit d in this warp's earlier rounds, then the lanes below
        const uint32_t before = valid ? S.wcnt[warp][d] : 0u;
        __syncwarp();
        if (valid && (peers & lt) == 0u) S.wcnt[warp][d] = before + __popc(peers);
        __syncwarp();
        rank[r] = before + __popc(peers & lt);
    }
    __syncthreads();
    // digit t: the warps' starts within the digit, then the digit's start in the tile
    uint32_t tot = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
        const uint32_t c = S.wcnt[w][t];
        S.wcnt[w][t] = tot;
        tot += c;
    }
    S.tstart[t] = block_excl_scan(tot, S.wsum, nullptr);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        if (wbase + size_t(r) * 32 + lane < size_t(n)) {
            const uint32_t d = digit_of(key[r], shift);
            const uint32_t pos = S.tstart[d] + S.wcnt[warp][d] + rank[r];
            S.skeys[pos] = key[r];
            S.svals[pos] = val[r];
        }
    }
    __syncthreads();
    const int cnt = int(min(size_t(TILE), size_t(n) - size_t(b) * TILE));
    for (int i = t; i < cnt; i += RS_THREADS) {
        const uint64_t k = S.skeys[i];
        const uint32_t d = digit_of(k, shift);
        const uint32_t pos = S.gbase[d] + (uint32_t(i) - S.tstart[d]);
        kout[pos] = k;
        vout[pos] = S.svals[i];
        if (next) atomicAdd(&next[(pos / TILE) * 256 + digit_of(k, next_shift)], 1u);
    }
}

__global__ void __launch_bounds__(RS_THREADS)
    rs_scatter(Pass p, int n, const uint32_t *__restrict__ offs, const uint32_t *__restrict__ rowsum, int nblocks) {
    after_previous();
    __shared__ ScatterShared<RS_ROUNDS> S;
    const int b = blockIdx.x, deep = *p.deep, in = p.in ^ deep;
    const uint32_t *vin = p.first && !deep ? nullptr : in ? p.v1 : p.v0;
    // all smaller digits, then earlier tiles
    scatter_tile(S, in ? p.k1 : p.k0, vin, in ? p.k0 : p.k1, in ? p.v0 : p.v1, n, p.shift, b,
                 [&](int t) { return block_excl_scan(rowsum[t], S.wsum, nullptr) + offs[size_t(t) * nblocks + b]; },
                 nullptr, 0);
}

// The passes over the lower bits take two launches: counts by tile and by span of tiles, then
// every block adds up the spans and the tiles of its own span. Most calls need none of them, so
// they are few, with few blocks, and leave at once.
struct LowPass {
    const uint64_t *kin;
    const uint32_t *vin;
    uint64_t *kout;
    uint32_t *vout;
    const int *deep;
    int n, shift, tiles, span;
    uint32_t *cnt, *sum;  // [tile][256], [span][256] (zero)
};

__global__ void __launch_bounds__(RS_THREADS) rs_low_count(LowPass p) {
    after_previous();
    if (!*p.deep) return;
    __shared__ uint32_t cnt[256];
    const int t = threadIdx.x;
    for (int b = blockIdx.x; b < p.tiles; b += gridDim.x) {
        cnt[t] = 0;
        __syncthreads();
        const size_t end = min(size_t(p.n), size_t(b + 1) * RS_TILE);
#pragma unroll 4
        for (size_t i = size_t(b) * RS_TILE + t; i < end; i += RS_THREADS)
            atomicAdd(&cnt[digit_of(__ldcg(p.kin + i), p.shift)], 1u);
        __syncthreads();
        const uint32_t c = cnt[t];
        p.cnt[size_t(b) * 256 + t] = c;
        if (c) atomicAdd(&p.sum[size_t(b / p.span) * 256 + t], c);
    }
}

__global__ void __launch_bounds__(RS_THREADS) rs_low_scatter(LowPass p) {
    after_previous();
    if (!*p.deep) return;
    __shared__ ScatterShared<RS_ROUNDS> S;
    for (int b = blockIdx.x; b < p.tiles; b += gridDim.x) {
        scatter_tile(S, p.kin, p.vin, p.kout, p.vout, p.n, p.shift, b,
                     [&](int t) {
                         const int mine = b / p.span, spans = (p.tiles + p.span - 1) / p.span;
                         uint32_t before = 0, total = 0;
#pragma unroll 8
                         for (int j = 0; j < spans; ++j) {
                             const uint32_t c = p.sum[size_t(j) * 256 + t];
                             if (j < mine) before += c;
                             total += c;
                         }
#pragma unroll 8
                         for (int j = mine * p.span; j < b; ++j) before += p.cnt[size_t(j) * 256 + t];
                         return block_excl_scan(total, S.wsum, nullptr) + before;
                     },
                     nullptr, 0);
        __syncthreads();
    }
}

// One pass in one launch: hist[b * 256 + d] holds the tiles' digit counts.
template <int ROUNDS>
__global__ void __launch_bounds__(RS_THREADS)
    rs_pass(const uint64_t *__restrict__ kin, const uint32_t *__restrict__ vin, uint64_t *__restrict__ kout,
            uint32_t *__restrict__ vout, int n, int shift, const uint32_t *__restrict__ hist, int nblocks,
            uint32_t *__restrict__ next, int next_shift) {
    after_previous();
    __shared__ ScatterShared<ROUNDS> S;
    const int b = blockIdx.x;
    scatter_tile(S, kin, vin, kout, vout, n, shift, b,
                 [&](int t) {
                     // four digits a load, every fourth tile
                     const int g = t >> 6, q = t & 63;
                     uint4 before = make_uint4(0, 0, 0, 0), total = before;
#pragma unroll 8
                     for (int j = g; j < nblocks; j += 4) {
                         const uint4 h = reinterpret_cast<const uint4 *>(hist)[j * 64 + q];
                         if (j < b) {
                             before.x += h.x;
                             before.y += h.y;
                             before.z += h.z;
                             before.w += h.w;
                         }
                         total.x += h.x;
                         total.y += h.y;
                         total.z += h.z;
                         total.w += h.w;
                     }
                     reinterpret_cast<uint4 *>(S.wcnt[g])[q] = before;
                     reinterpret_cast<uint4 *>(S.wcnt[4 + g])[q] = total;
                     __syncthreads();
                     const uint32_t sum = S.wcnt[4][t] + S.wcnt[5][t] + S.wcnt[6][t] + S.wcnt[7][t];
                     const uint32_t mine = S.wcnt[0][t] + S.wcnt[1][t] + S.wcnt[2][t] + S.wcnt[3][t];
                     return block_excl_scan(sum, S.wsum, nullptr) + mine;
                 },
                 next, next_shift);
}

// Orders every run of keys with the same upper bits (key >> shift) by the whole key, stably:
// each key counts those of its run that come before it. A run of more than RUN_LIMIT + 1 keys is
// left to rs_runs: its first key puts it on the list of those for a block, or of those longer than
// BLOCK_RUN, for a cluster. (Builds at limits of 48 / 128 / 256, us: N = 262144 in knots of
// some 60 bodies 531 / 377 / 378, 100 477 / 397 / 388, 200 451 / 477 / 432, 400 399 / 425 / 462.)
constexpr int RUN_LIMIT = 128;
constexpr int BLOCK_RUN = 2 * RS_TILE;

struct RunLists {  // the first keys of the long runs; count: [0] those for a block, [1] for a cluster
    int *count, *block, *cluster;
};

__global__ void __launch_bounds__(256)
    rs_finish(const uint64_t *__restrict__ kin, const uint32_t *__restrict__ vin, int n, int shift,
              uint64_t *__restrict__ kout, uint32_t *__restrict__ vout, const int *__restrict__ deep, RunLists runs) {
    after_previous();
    if (deep && *deep) return;  // sorted by all bits, and in (kout, vout)
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const uint64_t k = kin[i], h = k >> shift;
    const auto same = [&](int j) { return j >= 0 && j < n && (kin[j] >> shift) == h; };
    int lo = i, before = 0;
    const bool below = same(i - 1), above = same(i + 1);
    if (below || above) {
        if (same(i - RUN_LIMIT)) return;  // in a long run
        if (same(i + RUN_LIMIT)) {
            if (!below) {  // its first key
                const bool big = same(i + BLOCK_RUN);
                (big ? runs.cluster : runs.block)[atomicAdd(runs.count + big, 1)] = i;
            }
            return;
        }
        for (; same(lo - 1); --lo) before += kin[lo - 1] <= k;  // (ends within RUN_LIMIT)
        for (int hi = i; same(hi + 1); ++hi) before += kin[hi + 1] < k;
    }
    const int pos = lo + before;  // in the run
    kout[pos] = k;
    vout[pos] = vin[i];
}

// The long runs of (kb, vb) go sorted to (ka, va): three LSD passes over the bits below those
// that a run's keys share, kb -> ka -> kb -> ka within the run's range. A block, or each
// block of a cluster, takes neighbouring tiles and ranks them one after the other; where a
// digit's keys of a block start it knows from the digit counts of the cluster's blocks
// (distributed shared memory). A cluster's blocks run together by themselves, so its barrier
// needs no room on the chip beyond eight blocks and no limit.
constexpr int RUN_CLUSTER = 8, RUN_PASSES = 3;

struct RunShared {
    ScatterShared<RS_ROUNDS> tile;
    uint32_t cnt[256];
};

// The first key behind the run that starts at `start` (which holds start + RUN_LIMIT); `end`: a
// bound of it. Every thread of the block must call it.
__device__ __forceinline__ int run_end(const uint64_t *keys, int start, int end, int shift) {
    const uint64_t h = __ldcg(keys + start) >> shift;
    int lo = start + RUN_LIMIT, hi = end;  // lo is in the run, hi is not
    while (hi - lo > 1) {
        const int step = (hi - lo + RS_THREADS - 1) / RS_THREADS;
        const long long i = lo + (long long)(threadIdx.x + 1) * step;
        const int in = __syncthreads_count(i < hi && (__ldcg(keys + i) >> shift) == h);
        hi = int(min((long long)hi, lo + (long long)(in + 1) * step));
        lo += in * step;
    }
    return hi;
}

template <class Cluster>
__device__ __forceinline__ void sort_run(RunShared &S, uint64_t *ka, uint32_t *va, uint64_t *kb, uint32_t *vb,
                                         int len, const Cluster &cluster) {
    const int t = threadIdx.x, rank = cluster.rank();
    const int tiles = (len + RS_TILE - 1) / RS_TILE, per = (tiles + cluster.size() - 1) / cluster.size();
    const int t0 = min(tiles, rank * per), t1 = min(tiles, t0 + per);
    for (int p = 0; p < RUN_PASSES; ++p) {
        const uint64_t *kin = p & 1 ? ka : kb;
        const uint32_t *vin = p & 1 ? va : vb;
        S.cnt[t] = 0;
        __syncthreads();
        const int end = min(len, t1 * RS_TILE);
#pragma unroll 8
        for (int i = t0 * RS_TILE + t; i < end; i += RS_THREADS) atomicAdd(&S.cnt[digit_of(__ldcg(kin + i), 8 * p)], 1u);
        cluster.sync();
        uint32_t before = 0, total = 0;
        for (int r = 0; r < cluster.size(); ++r) {
            const uint32_t c = cluster.count(&S.cnt[t], r);
            if (r < rank) before += c;
            total += c;
        }
        uint32_t start = block_excl_scan(total, S.tile.wsum, nullptr) + before;
        for (int b = t0; b < t1; ++b) {
            scatter_tile(S.tile, kin, vin, p & 1 ? kb : ka, p & 1 ? vb : va, len, 8 * p, b, [&](int) { return start; },
                         nullptr, 0);
            const uint32_t next = t < 255 ? S.tile.tstart[t + 1] : uint32_t(min(RS_TILE, len - b * RS_TILE));
            start += next - S.tile.tstart[t];
            __syncthreads();
        }
        cluster.sync();  // the pass is written and the counts are read
    }
}

struct OneBlock {
    __device__ int rank() const { return 0; }
    __device__ int size() const { return 1; }
    __device__ void sync() const { __syncthreads(); }
    __device__ uint32_t count(const uint32_t *c, int) const { return *c; }
};
struct BlockCluster {
    cooperative_groups::cluster_group group = cooperative_groups::this_cluster();
    __device__ int rank() const { return int(group.block_rank()); }
    __device__ int size() const { return RUN_CLUSTER; }
    __device__ void sync() const { group.sync(); }
    __device__ uint32_t count(uint32_t *c, int r) const { return *group.map_shared_rank(c, r); }
};

__global__ void __cluster_dims__(RUN_CLUSTER, 1, 1) __launch_bounds__(RS_THREADS)
    rs_runs(uint64_t *ka, uint32_t *va, uint64_t *kb, uint32_t *vb, int n, int shift, RunLists runs) {
    after_previous();
    __shared__ RunShared S;
    const int few = runs.count[0], many = runs.count[1];
    const BlockCluster cluster;
    for (int r = blockIdx.x / RUN_CLUSTER; r < many; r += gridDim.x / RUN_CLUSTER) {
        const int i = runs.cluster[r], end = run_end(kb, i, n, shift);
        sort_run(S, ka + i, va + i, kb + i, vb + i, end - i, cluster);
    }
    for (int r = blockIdx.x; r < few; r += gridDim.x) {
        const int i = runs.block[r], end = run_end(kb, i, min(n, i + BLOCK_RUN), shift);
        sort_run(S, ka + i, va + i, kb + i, vb + i, end - i, OneBlock{});
    }
}

}  // namespace prims

// The first sorted bit of n keys: five digits from the top (13 octree levels and a bit) leave
// runs of a few bodies at 4M bulge+disk; a sixth from 8M on.
static int head_shift(int n, int bits) { return std::max(0, bits - 8 * (n >= (1 << 23) ? 6 : 5)); }
static_assert(63 - 8 * 5 <= 8 * prims::RUN_PASSES && 63 - 8 * 5 <= 8 * prims::LOW_PASSES, "all lower bits are sorted");
static_assert(prims::LOW_PASSES % 2 == 1, "the upper passes then start from the other pair");

namespace prims {
// How a sort of n keys is laid out: tiles of the direct passes (rounds = 0: three launches a
// pass) and words of histograms.
struct SortPlan {
    int shift, passes, rounds, tile, tiles, blocks;
    int span, spans;  // tiles to a span of the low passes
    size_t nhist, sums, words;  // words: those of the low passes' spans from sums on, then the flags
    SortPlan(int n, int bits)
        : shift(head_shift(n, bits)),
          passes((bits - shift + 7) / 8),
          rounds(direct_rounds(n)),
          tile(RS_THREADS * (rounds ? rounds : RS_ROUNDS)),
          tiles((n + tile - 1) / tile),
          blocks((n + RS_TILE - 1) / RS_TILE),
          span(blocks <= 4096 ? 64 : 512),
          spans((blocks + span - 1) / span),
          nhist(256 * size_t(blocks)) {
        // counts per pass of the direct passes, or counts, offsets and row sums; where these
        // were, the lists of long runs; then the lengths of the lists and the deep flag
        sums = rounds ? size_t(passes) * 256 * tiles : 2 * nhist + 256;
        words = sums + (rounds ? 0 : LOW_PASSES * 256 * size_t(spans)) + 64;
    }
};
}  // namespace prims

int radix_sort_prepare(pt_ctx *ctx, PrimScratch &s, int n, int bits, RadixFirst *first) {
    using namespace prims;
    const SortPlan p(n, bits);
    PT_TRY(ensure_buf(ctx, s.keys2, sizeof(uint64_t) * size_t(n)));
    PT_TRY(ensure_buf(ctx, s.vals2, sizeof(uint32_t) * size_t(n)));
    PT_TRY(ensure_buf(ctx, s.hist, sizeof(uint32_t) * p.words));
    uint32_t *hist = static_cast<uint32_t *>(s.hist.ptr);
    first->zero = p.rounds ? hist : hist + p.sums;
    first->zero_words = int(p.rounds ? p.words : p.words - p.sums);
    // an odd number of passes ends in the pair that the finishing pass reads
    first->keys = (p.passes & 1) ? nullptr : static_cast<uint64_t *>(s.keys2.ptr);
    first->hist = p.rounds ? hist : nullptr;
    first->shift = p.shift;
    first->tile = p.tile;
    first->deep = p.rounds ? nullptr : reinterpret_cast<int *>(hist + (p.words - 64)) + 2;
    return PT_OK;
}

int radix_sort_u64(pt_ctx *ctx, PrimScratch &s, uint64_t *keys, uint32_t *vals, int n, int bits) {
    using namespace prims;
    const SortPlan sp(n, bits);
    const int nblocks = sp.blocks, shift0 = sp.shift, passes = sp.passes;
    uint32_t *hist = static_cast<uint32_t *>(s.hist.ptr);
    uint32_t *offs = hist + sp.nhist, *rowsum = offs + sp.nhist;
    uint64_t *kb = static_cast<uint64_t *>(s.keys2.ptr), *k[2] = {keys, kb};
    uint32_t *vb = static_cast<uint32_t *>(s.vals2.ptr), *v[2] = {vals, vb};
    cudaStream_t st = ctx->stream;
    int *flags = reinterpret_cast<int *>(hist + (sp.words - 64));
    const int in0 = (passes & 1) ? 0 : 1;  // the passes end in (kb, vb)
    if (sp.rounds) {
        for (int p = 0, in = in0; p < passes; ++p, in ^= 1) {
            const int shift = shift0 + 8 * p;
            const size_t direct = 256 * size_t(sp.tiles);
            uint32_t *next = p + 1 < passes ? hist + (p + 1) * direct : nullptr;
            launch_next(sp.rounds == 1   ? rs_pass<1>
                        : sp.rounds == 4 ? rs_pass<4>
                                         : rs_pass<8>,
                        sp.tiles, RS_THREADS, 0, st, k[in], p == 0 ? nullptr : v[in], k[in ^ 1], v[in ^ 1], n, shift,
                        hist + p * direct, sp.tiles, next, shift + 8);
            PT_TRY(check_launch(ctx, "rs_pass"));
        }
    } else {
        const int few = std::min(nblocks, 4 * std::max(1, ctx->sm_count));
        for (int p = 0, in = in0; p < LOW_PASSES; ++p, in ^= 1) {
            // the lowest bits, the middle ones and those up to shift0, overlapping
            const LowPass q{k[in],     p == 0 ? nullptr : v[in],
                            k[in ^ 1], v[in ^ 1],
                            flags + 2, n,
                            p * (shift0 - 8) / (LOW_PASSES - 1), nblocks,
                            sp.span,   hist,
                            hist + sp.sums + p * 256 * size_t(sp.spans)};
            launch_next(rs_low_count, few, RS_THREADS, 0, st, q);
            PT_TRY(check_launch(ctx, "rs_low_count"));
            launch_next(rs_low_scatter, few, RS_THREADS, 0, st, q);
            PT_TRY(check_launch(ctx, "rs_low_scatter"));
        }
        Pass q{k[0], k[1], v[0], v[1], flags + 2};
        for (int p = 0; p < passes; ++p) {
            q.shift = shift0 + 8 * p;
            q.in = in0 ^ (p & 1);
            q.first = p == 0;
            launch_next(rs_hist, nblocks, RS_THREADS, 0, st, q, n, hist, nblocks);
            PT_TRY(check_launch(ctx, "rs_hist"));
            launch_next(rs_rowscan, 256, RS_THREADS, 0, st, hist, offs, rowsum, nblocks);
            PT_TRY(check_launch(ctx, "rs_rowscan"));
            launch_next(rs_scatter, nblocks, RS_THREADS, 0, st, q, n, offs, rowsum, nblocks);
            PT_TRY(check_launch(ctx, "rs_scatter"));
        }
    }
    int *lists = reinterpret_cast<int *>(hist);  // the passes' counts are read
    const RunLists runs{flags, lists, lists + n / (RUN_LIMIT + 1) + 1};
    launch_next(rs_finish, (n + 255) / 256, 256, 0, st, kb, vb, n, shift0, keys, vals,
                sp.rounds ? nullptr : flags + 2, runs);
    PT_TRY(check_launch(ctx, "rs_finish"));
    // runs for a block are shorter than two tiles and longer than half a block's threads: one
    // block to 256 keys, up to four an SM
    const int grid = std::min(n / 256, 4 * std::max(1, ctx->sm_count)) / RUN_CLUSTER * RUN_CLUSTER;
    launch_next(rs_runs, std::max(RUN_CLUSTER, grid), RS_THREADS, 0, st, keys, vals, kb, vb, n, shift0, runs);
    return check_launch(ctx, "rs_runs");
}

void prim_free(pt_ctx *ctx, PrimScratch &s) {
    free_buf(ctx, s.scan);
    free_buf(ctx, s.hist);
    free_buf(ctx, s.keys2);
    free_buf(ctx, s.vals2);
}

}  // namespace pt
