// cuda::BarnesHut { theta }: on-device octree build and a warp-synchronous walk.
//
// The tree is the reference's orthtree (particular/src/tree/mod.rs:91-138) built in
// parallel instead of recursively:
//  1. root_box : the square root box of BoundingBox::square_with
//                (particular/src/tree/partition.rs:274-292), in the same f32 ops.
//  2. make_keys: each body replays the reference's subdivision for 21 levels
//                (centre = (min+max)/2, child bit = pos < centre, tree/mod.rs:116-124,
//                partition.rs:332-359), giving a 63-bit key whose prefixes are exactly
//                the reference's cells. The digit stored is 7 - orthant, so ascending
//                keys follow the reference's LIFO visiting order (children pushed 0..7,
//                popped 7..0, sequential.rs:489-495).
//  3. radix sort of (key, body) pairs; bodies gathered into key order.
//  4. equal keys collapse into one leaf unit (coincident bodies, or bodies closer
//     than 2^-21 of the root box: deeper than the key resolves).
//  5. Karras (2012) binary radix tree over the unique keys; a binary node is an
//     octree cell where its common-prefix level changes. Single-child chains of the
//     reference tree disappear: accepting a chain cell or its only child adds the
//     same (COM, M), so the result is unchanged.
//  6. cells are laid out in depth-first preorder with skip pointers (index after
//     the subtree), leaves interleaved.
//  7. moments (mass, centre of mass, second moment -> traceless quadrupole) bottom-up
//     (parallel-axis theorem), in compensated FP32 for f32 trees and FP64 for DVec3 trees:
//     the cells inside a chunk of 512 units by the block that lays the chunk out, from
//     shared memory, the few larger ones block of chunks by block of chunks.
#include "pt_bh.cuh"
#include "pt_scan.cuh"

#include <type_traits>

namespace pt {
namespace bh {

// ---- 1. root box -----------------------------------------------------------
// Also clears the sort's words and, where err is not null, the error word. The last block to
// end folds the blocks' extents (min/max: exact in any order) and forms the reference's square
// root box in the same launch: box = {min x,y,z, max x,y,z} of BoundingBox::square_with, centre
// = midpoint of the AABB, half = (max extent + 0) / 2 (MidPoint::half), min/max = centre -/+
// half. done: zero before and after. One launch instead of two and a memset: 274 -> 267 us of
// a call with 65536 bodies.
template <class T>
__global__ void __launch_bounds__(256)
    root_box(const typename Prec<T>::V4 *__restrict__ src, int n, T *part, T *__restrict__ box,
             uint32_t *__restrict__ zero, int zero_words, int *__restrict__ err, unsigned *done) {
    using P = Prec<T>;
    after_previous();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (err && tid == 0) *err = 0;
    for (int i = tid; i < zero_words; i += gridDim.x * blockDim.x) zero[i] = 0u;
    T mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = tid; i < n; i += gridDim.x * blockDim.x) {
        const typename P::V4 p = src[i];
        mn[0] = P::min(mn[0], p.x);
        mn[1] = P::min(mn[1], p.y);
        mn[2] = P::min(mn[2], p.z);
        mx[0] = P::max(mx[0], p.x);
        mx[1] = P::max(mx[1], p.y);
        mx[2] = P::max(mx[2], p.z);
    }
    __shared__ T s[6][8];
    __shared__ bool last;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the block's extents, in thread 0
    auto fold = [&]() {
        for (int o = 16; o > 0; o >>= 1)
            for (int a = 0; a < 3; ++a) {
                mn[a] = P::min(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
                mx[a] = P::max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
            }
        if (lane == 0)
            for (int a = 0; a < 3; ++a) {
                s[a][warp] = mn[a];
                s[3 + a][warp] = mx[a];
            }
        __syncthreads();
        if (threadIdx.x != 0) return;
        for (int w = 1; w < 8; ++w)
            for (int a = 0; a < 3; ++a) {
                mn[a] = P::min(mn[a], s[a][w]);
                mx[a] = P::max(mx[a], s[3 + a][w]);
            }
    };
    fold();
    if (threadIdx.x == 0) {
        for (int a = 0; a < 3; ++a) {
            part[blockIdx.x * 6 + a] = mn[a];
            part[blockIdx.x * 6 + 3 + a] = mx[a];
        }
        __threadfence();
        last = atomicInc(done, gridDim.x - 1) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    for (int b = threadIdx.x; b < int(gridDim.x); b += blockDim.x)
        for (int a = 0; a < 3; ++a) {
            mn[a] = P::min(mn[a], __ldcg(part + b * 6 + a));
            mx[a] = P::max(mx[a], __ldcg(part + b * 6 + 3 + a));
        }
    fold();
    if (threadIdx.x != 0) return;
    T half = 0;
    T c[3];
    for (int a = 0; a < 3; ++a) {
        c[a] = P::mul(P::add(mn[a], mx[a]), T(0.5));
        half = P::max(half, P::sub(mx[a], mn[a]));
    }
    half = P::mul(P::add(half, T(0)), T(0.5));
    for (int a = 0; a < 3; ++a) {
        box[a] = P::sub(c[a], half);
        box[3 + a] = P::add(c[a], half);
    }
}

// ---- 2. keys ---------------------------------------------------------------
template <class T>
__device__ __forceinline__ uint64_t key_of(T px, T py, T pz, const T *box) {
    using P = Prec<T>;
    T mn0 = box[0], mn1 = box[1], mn2 = box[2], mx0 = box[3], mx1 = box[4], mx2 = box[5];
    uint64_t key = 0;
#pragma unroll 3
    for (int l = 0; l < LEVELS; ++l) {
        const T c0 = P::mul(P::add(mn0, mx0), T(0.5));
        const T c1 = P::mul(P::add(mn1, mx1), T(0.5));
        const T c2 = P::mul(P::add(mn2, mx2), T(0.5));
        const int b0 = px < c0, b1 = py < c1, b2 = pz < c2;
        if (b0) mx0 = c0; else mn0 = c0;
        if (b1) mx1 = c1; else mn1 = c1;
        if (b2) mx2 = c2; else mn2 = c2;
        const int o = b0 | (b1 << 1) | (b2 << 2);
        key = (key << 3) | uint64_t(7 - o);
    }
    return key;
}

// Sets *deep where the bodies crowd into cells that the sort's upper bits (key >> shift) do not
// tell apart, some CROWD of them or more to a cell. SAMPLES bodies are looked at: of these,
// SAMPLES^2 / 2 x (the mean run) / n share their cell with an earlier one. One block; it costs the
// smallest call that has it 4 us and larger ones, where it ends before the other blocks, nothing.
// CROWD: runs of a thread per key (up to 129) cost less than the three passes of the whole
// chip, longer ones more (N = 1M in knots of some 60 bodies, below the line, 654 us, of some
// 200, above it, 647, which took 962 without the passes).
constexpr int SAMPLES = 1024, CROWD = 100;

template <class T>
__device__ __forceinline__ void sample_keys(const typename Prec<T>::V4 *__restrict__ bodies, int n, const T *box,
                                            int shift, int *deep) {
    constexpr unsigned long long EMPTY = ~0ull;
    __shared__ unsigned long long seen[2 * SAMPLES];
    __shared__ int shared;
    for (int i = threadIdx.x; i < 2 * SAMPLES; i += blockDim.x) seen[i] = EMPTY;
    if (threadIdx.x == 0) shared = 0;
    __syncthreads();
    unsigned long long h[SAMPLES / 256];
#pragma unroll
    for (int s = 0; s < SAMPLES / 256; ++s) {
        const typename Prec<T>::V4 p = bodies[(long long)(256 * s + threadIdx.x) * n / SAMPLES];
        h[s] = key_of<T>(p.x, p.y, p.z, box) >> shift;
    }
#pragma unroll
    for (int s = 0; s < SAMPLES / 256; ++s)
        for (unsigned at = unsigned((h[s] * 0x9e3779b97f4a7c15ull) >> 32);; ++at) {
            const unsigned long long was = atomicCAS(&seen[at % (2 * SAMPLES)], EMPTY, h[s]);
            if (was == h[s]) atomicAdd(&shared, 1);
            if (was == EMPTY || was == h[s]) break;
        }
    __syncthreads();
    if (threadIdx.x == 0 && (long long)shared * n >= (long long)CROWD * SAMPLES * SAMPLES / 2) *deep = 1;
}

// hist (small n): the counts of the sort's first digit by tile of keys. SAMPLE (large n): the
// first block samples instead.
template <class T, bool SAMPLE>
__global__ void __launch_bounds__(256)
    make_keys(const typename Prec<T>::V4 *__restrict__ bodies, int n, const T *__restrict__ box_g,
              uint64_t *__restrict__ keys, uint32_t *__restrict__ hist, int shift, int tile, int *deep) {
    after_previous();
    __shared__ T box[6];
    if (threadIdx.x < 6) box[threadIdx.x] = box_g[threadIdx.x];
    __syncthreads();
    if (SAMPLE && blockIdx.x == 0) return sample_keys<T>(bodies, n, box, shift, deep);
    const int i = (blockIdx.x - SAMPLE) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const typename Prec<T>::V4 p = bodies[i];
    const uint64_t k = key_of<T>(p.x, p.y, p.z, box);
    keys[i] = k;
    if (hist) atomicAdd(&hist[(i / tile) * 256 + (int(k >> shift) & 255)], 1u);
}

template <class T>
static int launch_make_keys(pt_ctx *ctx, const typename Prec<T>::V4 *bodies, int n, const T *box, uint64_t *keys,
                            const RadixFirst &rf) {
    launch_next(rf.deep ? make_keys<T, true> : make_keys<T, false>, blocks(n) + (rf.deep ? 1 : 0), 256, 0, ctx->stream,
                bodies, n, box, rf.keys ? rf.keys : keys, rf.hist, rf.shift, rf.tile, rf.deep);
    return check_launch(ctx, "make_keys");
}

// The walk's counters (counters + 4 ints) start from zero.
__device__ __forceinline__ void clear_stats(int *counters, int i) {
    if (i < WALK_STATS) (reinterpret_cast<unsigned long long *>(counters) + 2)[i] = 0ull;
}

template <class V4>
__global__ void gather_bodies(const V4 *__restrict__ src, const uint32_t *__restrict__ idx, int n,
                              V4 *__restrict__ out, int *__restrict__ counters) {
    after_previous();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    clear_stats(counters, k);
    if (k < n) out[k] = src[idx[k]];
}

// ---- 4. unique keys -> leaf units ------------------------------------------
// A scan over the sorted bodies of "the first body of its key" numbers the units.
struct UnitHead {
    const uint64_t *keys;
    __device__ uint32_t operator()(int k) const { return (k == 0 || keys[k] != keys[k - 1]) ? 1u : 0u; }
};
// counters[0] = M (units)
struct UnitFill {
    const uint64_t *keys;
    int n;
    uint64_t *ukey;
    uint32_t *ufirst;
    int *counters;
    __device__ void operator()(int k, uint32_t head, uint32_t u) const {
        if (!head) return;
        ukey[u] = keys[k];
        ufirst[u] = uint32_t(k);
    }
    __device__ void total(uint32_t M) const {
        ufirst[M] = uint32_t(n);
        counters[0] = int(M);
    }
};

// ---- 5. Karras binary radix tree ---------------------------------------------
__device__ __forceinline__ int kdelta(const uint64_t *__restrict__ k, int M, int i, int j) {
    if (j < 0 || j >= M) return -1;
    return __clzll(k[i] ^ k[j]) - 1;  // bit 63 is always 0: prefix length of the 63-bit keys
}

// The moments are combined block by block of units (section 7): chunks of CHUNK units first,
// then, stage by stage, blocks of SPAN_FAN of the blocks before. A cell's stage is the first
// whose blocks hold its whole range.
constexpr int CHUNK_SHIFT = 9;
constexpr int CHUNK = 1 << CHUNK_SHIFT;
constexpr int FAN_SHIFT = 6;
// A cell of stage s >= 1 holds one of its block's 63 inner boundaries between blocks of the
// stage before, and a boundary has one such cell per level at most.
constexpr int SPAN_CAP = ((1 << FAN_SHIFT) - 1) * LEVELS;

__host__ __device__ constexpr int stage_shift(int stage) { return CHUNK_SHIFT + FAN_SHIFT * stage; }
__host__ __device__ inline int stage_blocks(int n, int stage) { return int(((long long)n + (1ll << stage_shift(stage)) - 1) >> stage_shift(stage)); }
// Blocks of the stages 1 .. stage - 1 come first in the arrays of the blocks' cells.
__host__ __device__ inline int stage_first(int n, int stage) {
    int f = 0;
    for (int s = 1; s < stage; ++s) f += stage_blocks(n, s);
    return f;
}
// Stages after the chunks' until one block holds all n units.
inline int stages(int n) {
    int s = 0;
    while (stage_blocks(n, s) > 1) ++s;
    return s;
}
__device__ __forceinline__ int stage_of(int first, int last) {
    int s = 0;
    while (((long long)first >> stage_shift(s)) != ((long long)last >> stage_shift(s))) ++s;
    return s;
}

// Binary node i: its range, its split's children's parents, and whether it is an octree
// cell: the root, or a node whose common-prefix level (delta / 3) exceeds its parent's. The
// parent's prefix is the longer of those that the range shares with its neighbours, so no
// second pass over the parents is needed. top[i] = 1 + stage for a cell, else 0. Thread i
// also clears what the next pass counts, and moves body i of the key order to its place: a
// random read beside the search's chain of dependent ones.
template <class V4>
__global__ void karras(const V4 *__restrict__ src, const uint32_t *__restrict__ idx, V4 *__restrict__ sbody,
                       const uint64_t *__restrict__ ukey, const int *__restrict__ counters, int n,
                       int *__restrict__ bfirst, int *__restrict__ blast, int *__restrict__ bdelta,
                       int *__restrict__ bparent, int *__restrict__ lparent, uint8_t *__restrict__ top,
                       uint32_t *__restrict__ starts, uint32_t *__restrict__ kmask, int *__restrict__ nspan,
                       int span_blocks) {
    after_previous();
    const int M = counters[0];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) sbody[i] = src[idx[i]];
    if (i <= n) starts[i] = 0u;
    if (i < span_blocks) nspan[i] = 0;
    if (i >= M - 1) return;
    const int dn = kdelta(ukey, M, i, i + 1), dp = kdelta(ukey, M, i, i - 1);
    const int d = dn >= dp ? 1 : -1;
    const int dmin = min(dn, dp);
    int lmax = 2;
    while (kdelta(ukey, M, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (kdelta(ukey, M, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = kdelta(ukey, M, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (kdelta(ukey, M, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int first = min(i, j), last = max(i, j);
    bfirst[i] = first;
    blast[i] = last;
    bdelta[i] = dnode;
    if (first == gamma) lparent[gamma] = i; else bparent[gamma] = i;
    if (last == gamma + 1) lparent[gamma + 1] = i; else bparent[gamma + 1] = i;
    if (i == 0) bparent[0] = -1;
    const int dparent = max(dmin, kdelta(ukey, M, j, j + d));
    uint8_t c = 0;
    if (i == 0 || dparent / 3 < dnode / 3) {
        const int stage = stage_of(first, last);
        if (stage > 0) kmask[i] = 0u;
        c = uint8_t(1 + stage);
    }
    top[i] = c;
}

__device__ __forceinline__ int climb(int p, const uint8_t *__restrict__ top, const int *__restrict__ bparent) {
    while (!top[p]) p = bparent[p];
    return p;
}

// The octant digit of a key at an octree level.
__device__ __forceinline__ int digit_at(uint64_t key, int level) {
    return int((key >> (3 * (LEVELS - 1 - level))) & 7u);
}

// Octree parents and the levels of the cells starting at each unit (a bit each); a cell that
// spans chunks enters its block's list, and its children that come from earlier stages the
// digits of its child list.
__global__ void octree_links(const int *__restrict__ counters, int n, const int *__restrict__ bfirst,
                             const int *__restrict__ bparent, const int *__restrict__ lparent,
                             const uint8_t *__restrict__ top, const int *__restrict__ bdelta,
                             const uint64_t *__restrict__ ukey, int *__restrict__ oparent, int *__restrict__ loparent,
                             uint32_t *__restrict__ starts, uint32_t *__restrict__ kmask, int *__restrict__ nspan,
                             int *__restrict__ spans) {
    after_previous();
    const int M = counters[0];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < M - 1 && top[k]) {
        const int op = (k == 0) ? -1 : climb(bparent[k], top, bparent);
        const int b = bfirst[k];
        oparent[k] = op;
        atomicOr(&starts[b], 1u << (bdelta[k] / 3));
        if (op >= 0 && top[op] > top[k]) atomicOr(&kmask[op], 1u << digit_at(ukey[b], bdelta[op] / 3));
        const int stage = top[k] - 1;
        if (stage > 0) {
            const int blk = stage_first(n, stage) + int((long long)b >> stage_shift(stage));
            spans[size_t(blk) * SPAN_CAP + atomicAdd(&nspan[blk], 1)] = k;
        }
    }
    if (k < M) {
        const int op = (M == 1) ? -1 : climb(lparent[k], top, bparent);
        loparent[k] = op;
        if (op >= 0 && top[op] > 1) atomicOr(&kmask[op], 1u << digit_at(ukey[k], bdelta[op] / 3));
    }
}

// The number of cells that start at each unit.
struct CellStarts {
    const uint32_t *starts;
    __device__ uint32_t operator()(int b) const { return uint32_t(__popc(starts[b])); }
};

// ---- 7. moments ------------------------------------------------------------
// The leaves, then the cells, each after all its children, the children always summed in
// preorder, so the order of every sum is fixed by the tree. A block of threads combines the
// cells of one stage that lie in its block of units, deepest level first, from records in
// shared memory: the chunks' in the layout pass, the few that span chunks stage by stage
// (cells_span). Records that cross between stages are read through L2 (ld.global.cg).
__device__ __forceinline__ float4 ld_cg(const float4 *p) { return __ldcg(p); }
__device__ __forceinline__ double4_32a ld_cg(const double4_32a *p) {
    const double2 a = __ldcg(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
    double4_32a r;
    r.x = a.x, r.y = a.y, r.z = b.x, r.w = b.y;
    return r;
}
__device__ __forceinline__ Moments ld_cg(const Moments *p) {
    const double2 *q = reinterpret_cast<const double2 *>(p);
    double2 v[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) v[i] = __ldcg(q + i);
    Moments r;
    r.m = v[0].x, r.cx = v[0].y, r.cy = v[1].x, r.cz = v[1].y;
    r.sxx = v[2].x, r.sxy = v[2].y, r.sxz = v[3].x, r.syy = v[3].y, r.syz = v[4].x, r.szz = v[4].y;
    r.count = v[5].x, r.pad = v[5].y;
    return r;
}

// Cell record of f32 trees, in FP32. The centre of mass and the mass are unevaluated
// sums hi + lo with hi = nodeA, and a child's offset from its parent's geometric
// centre G is formed as (hi - G) + lo: hi and G lie within a cell width of each
// other, so every sum below is relative to the cell width, not to the position.
struct Rec32 {
    float4 lo;  // centre of mass - nodeA.xyz, mass - nodeA.w
    float4 s0;  // second moment about the centre of mass: xx xy xz yy
    float4 s1;  // yz zz, body count (int bits), 0
};

// Knuth's TwoSum: returns s = fl(a + b) and sets e with s + e == a + b exactly.
__device__ __forceinline__ float two_sum(float a, float b, float &e) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return s;
}

__device__ __forceinline__ void store_quad(float4 *nodeQ, int pk, float sxx, float sxy, float sxz, float syy,
                                           float syz, float szz) {
    const float tr = sxx + syy + szz;
    nodeQ[2 * pk] = make_float4(3.f * sxx - tr, 3.f * sxy, 3.f * sxz, 3.f * syy - tr);
    nodeQ[2 * pk + 1] = make_float4(3.f * syz, 3.f * szz - tr, 0.f, 0.f);
}

__device__ __forceinline__ double4_32a store_cell(const Moments &m, int pk, Moments *mom, double4_32a *nodeA, float4 *) {
    mom[pk] = m;
    return nodeA[pk] = Prec<double>::make(m.cx, m.cy, m.cz, m.m);  // the f64 method is monopole only
}

__device__ __forceinline__ float4 store_cell(const Moments &m, int pk, Rec32 *rec, float4 *nodeA, float4 *nodeQ) {
    const float hx = float(m.cx), hy = float(m.cy), hz = float(m.cz), hm = float(m.m);
    const float4 a = make_float4(hx, hy, hz, hm);
    nodeA[pk] = a;
    rec[pk].lo = make_float4(float(m.cx - hx), float(m.cy - hy), float(m.cz - hz), float(m.m - hm));
    rec[pk].s0 = make_float4(float(m.sxx), float(m.sxy), float(m.sxz), float(m.syy));
    rec[pk].s1 = make_float4(float(m.syz), float(m.szz), __int_as_float(int(m.count)), 0.f);
    store_quad(nodeQ, pk, float(m.sxx), float(m.sxy), float(m.sxz), float(m.syy), float(m.syz), float(m.szz));
    return a;
}

// Leaves: a single body is its own cell data (no record: parents read nodeA; no
// quadrupole: the walks read it for cells only); several (coincident, or closer
// than the key resolution) get FP64 moments.
template <class V4, class R>
__device__ __forceinline__ V4 leaf(int pk, int f, int e, const V4 *__restrict__ sbody, R *rec, V4 *nodeA, float4 *nodeQ) {
    if (e - f == 1) {
        const V4 p = sbody[f];
        nodeA[pk] = p;
        return p;
    }
    Moments m{};
    double sx = 0, sy = 0, sz = 0;
    for (int b = f; b < e; ++b) {
        const V4 p = sbody[b];
        m.m += p.w;
        sx += double(p.w) * p.x;
        sy += double(p.w) * p.y;
        sz += double(p.w) * p.z;
    }
    m.count = e - f;
    if (m.m != 0.0) {
        m.cx = sx / m.m;
        m.cy = sy / m.m;
        m.cz = sz / m.m;
    } else {  // massless: plain mean (gravity/impls/mod.rs:127-129)
        for (int b = f; b < e; ++b) {
            const V4 p = sbody[b];
            m.cx += p.x;
            m.cy += p.y;
            m.cz += p.z;
        }
        m.cx /= m.count;
        m.cy /= m.count;
        m.cz /= m.count;
    }
    for (int b = f; b < e; ++b) {
        const V4 p = sbody[b];
        const double dx = p.x - m.cx, dy = p.y - m.cy, dz = p.z - m.cz;
        m.sxx += p.w * dx * dx;
        m.sxy += p.w * dx * dy;
        m.sxz += p.w * dx * dz;
        m.syy += p.w * dy * dy;
        m.syz += p.w * dy * dz;
        m.szz += p.w * dz * dz;
    }
    return store_cell(m, pk, rec, nodeA, nodeQ);
}

// One child of a cell, for the combination below.
struct Child32 {
    float4 a, lo, s0, s1;  // nodeA and Rec32
};
template <class T>
using ChildOf = typename std::conditional<sizeof(T) == 4, Child32, Moments>::type;

// A single body, and a cell or several-body leaf from its record in global memory.
__device__ __forceinline__ void child_single(float4 b, Child32 &c) {
    c.a = b;
    c.lo = c.s0 = make_float4(0.f, 0.f, 0.f, 0.f);
    c.s1 = make_float4(0.f, 0.f, __int_as_float(1), 0.f);
}
__device__ __forceinline__ void child_single(const double4_32a &b, Moments &c) {
    c = Moments{};
    c.cx = b.x, c.cy = b.y, c.cz = b.z, c.m = b.w, c.count = 1.0;
}
__device__ __forceinline__ void child_record(float4 a, const Rec32 *r, Child32 &c) {
    c.a = a;
    c.lo = ld_cg(&r->lo);
    c.s0 = ld_cg(&r->s0);
    c.s1 = ld_cg(&r->s1);
}
__device__ __forceinline__ void child_record(const double4_32a &, const Moments *r, Moments &c) { c = ld_cg(r); }

// f32 trees: one pass over the children in FP32, sums about the cell's geometric
// centre G, then moved to the centre of mass C by the parallel-axis rule
// S_C = S_G - P P^T / M with P = sum m (c - G) = M (C - G). *a gets nodeA.
template <class Child>
__device__ __forceinline__ Rec32 combine(float4 g, const Child &child, float4 *a) {
    float mh = 0.f, ml = 0.f, px = 0.f, py = 0.f, pz = 0.f;
    float sxx = 0.f, sxy = 0.f, sxz = 0.f, syy = 0.f, syz = 0.f, szz = 0.f;
    int count = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        Child32 c;
        if (!child(i, c)) continue;
        const float dx = __fsub_rn(c.a.x, g.x) + c.lo.x, dy = __fsub_rn(c.a.y, g.y) + c.lo.y,
                    dz = __fsub_rn(c.a.z, g.z) + c.lo.z;
        float e;
        mh = two_sum(mh, c.a.w, e);
        ml += e + c.lo.w;
        const float mx = c.a.w * dx, my = c.a.w * dy, mz = c.a.w * dz;
        px += mx;
        py += my;
        pz += mz;
        sxx += c.s0.x + mx * dx;
        sxy += c.s0.y + mx * dy;
        sxz += c.s0.z + mx * dz;
        syy += c.s0.w + my * dy;
        syz += c.s1.x + my * dz;
        szz += c.s1.y + mz * dz;
        count += __float_as_int(c.s1.z);
    }
    float e;
    const float M = two_sum(mh, ml, e);
    const float Ml = e;
    float ox, oy, oz;
    if (M != 0.f) {
        const float inv = 1.f / M;
        ox = px * inv, oy = py * inv, oz = pz * inv;  // C - G
        sxx -= px * ox;
        sxy -= px * oy;
        sxz -= px * oz;
        syy -= py * oy;
        syz -= py * oz;
        szz -= pz * oz;
    } else {  // massless: plain mean of the bodies (gravity/impls/mod.rs:127-129), a rare second pass
        float ux = 0.f, uy = 0.f, uz = 0.f;
        for (int i = 0; i < 8; ++i) {
            Child32 c;
            if (!child(i, c)) continue;
            const float cn = float(__float_as_int(c.s1.z));
            ux += cn * (__fsub_rn(c.a.x, g.x) + c.lo.x);
            uy += cn * (__fsub_rn(c.a.y, g.y) + c.lo.y);
            uz += cn * (__fsub_rn(c.a.z, g.z) + c.lo.z);
        }
        ox = ux / float(count), oy = uy / float(count), oz = uz / float(count);
    }
    float ex, ey, ez;
    const float hx = two_sum(g.x, ox, ex), hy = two_sum(g.y, oy, ey), hz = two_sum(g.z, oz, ez);
    *a = make_float4(hx, hy, hz, M);
    Rec32 r;
    r.lo = make_float4(ex, ey, ez, Ml);
    r.s0 = make_float4(sxx, sxy, sxz, syy);
    r.s1 = make_float4(syz, szz, __int_as_float(count), 0.f);
    return r;
}

// f64 trees (DVec3 bodies): the same combination in FP64.
template <class Child>
__device__ __forceinline__ Moments combine(double4_32a g, const Child &child, double4_32a *a) {
    const double gx = g.x, gy = g.y, gz = g.z;
    Moments m{};
    double px = 0, py = 0, pz = 0;
    for (int i = 0; i < 8; ++i) {
        Moments c;
        if (!child(i, c)) continue;
        const double dx = c.cx - gx, dy = c.cy - gy, dz = c.cz - gz;
        m.m += c.m;
        m.count += c.count;
        const double mx = c.m * dx, my = c.m * dy, mz = c.m * dz;
        px += mx;
        py += my;
        pz += mz;
        m.sxx += c.sxx + mx * dx;
        m.sxy += c.sxy + mx * dy;
        m.sxz += c.sxz + mx * dz;
        m.syy += c.syy + my * dy;
        m.syz += c.syz + my * dz;
        m.szz += c.szz + mz * dz;
    }
    if (m.m != 0.0) {
        const double inv = 1.0 / m.m;
        const double ox = px * inv, oy = py * inv, oz = pz * inv;  // C - G
        m.cx = gx + ox;
        m.cy = gy + oy;
        m.cz = gz + oz;
        m.sxx -= px * ox;
        m.sxy -= px * oy;
        m.sxz -= px * oz;
        m.syy -= py * oy;
        m.syz -= py * oz;
        m.szz -= pz * oz;
    } else {  // massless: plain mean of the bodies (gravity/impls/mod.rs:127-129), a rare second pass
        double ux = 0, uy = 0, uz = 0;
        for (int i = 0; i < 8; ++i) {
            Moments c;
            if (!child(i, c)) continue;
            ux += c.count * (c.cx - gx);
            uy += c.count * (c.cy - gy);
            uz += c.count * (c.cz - gz);
        }
        m.cx = gx + ux / m.count;
        m.cy = gy + uy / m.count;
        m.cz = gz + uz / m.count;
    }
    *a = Prec<double>::make(m.cx, m.cy, m.cz, m.m);
    return m;
}

// The same combinations by eight neighbouring lanes, one child to a lane (has: this lane has
// one): the children's loads are all in flight and their sums form a tree, the same one
// every time. All 32 lanes of the warp take part, each eight of them with a cell of its own;
// every lane gets the result.
__device__ __forceinline__ float sum8(float v) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double sum8(double v) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ int sum8(int v) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ Rec32 combine8(float4 g, bool has, const Child32 &c, float4 *a) {
    float dx = 0.f, dy = 0.f, dz = 0.f, m = 0.f, ml = 0.f;
    int cn = 0;
    if (has) {
        dx = __fsub_rn(c.a.x, g.x) + c.lo.x;
        dy = __fsub_rn(c.a.y, g.y) + c.lo.y;
        dz = __fsub_rn(c.a.z, g.z) + c.lo.z;
        m = c.a.w;
        ml = c.lo.w;
        cn = __float_as_int(c.s1.z);
    }
    const float mx = m * dx, my = m * dy, mz = m * dz;
    const float px = sum8(mx), py = sum8(my), pz = sum8(mz);
    float sxx = sum8((has ? c.s0.x : 0.f) + mx * dx), sxy = sum8((has ? c.s0.y : 0.f) + mx * dy),
          sxz = sum8((has ? c.s0.z : 0.f) + mx * dz), syy = sum8((has ? c.s0.w : 0.f) + my * dy),
          syz = sum8((has ? c.s1.x : 0.f) + my * dz), szz = sum8((has ? c.s1.y : 0.f) + mz * dz);
    const int count = sum8(cn);
    float mh = m, e;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, mh, o), ol = __shfl_xor_sync(0xffffffffu, ml, o);
        mh = two_sum(mh, oh, e);
        ml = (ml + ol) + e;
    }
    const float M = two_sum(mh, ml, e);
    const float Ml = e;
    float ux = 0.f, uy = 0.f, uz = 0.f;
    if (__any_sync(0xffffffffu, M == 0.f)) {  // massless: plain mean of the bodies (gravity/impls/mod.rs:127-129)
        ux = sum8(float(cn) * dx);
        uy = sum8(float(cn) * dy);
        uz = sum8(float(cn) * dz);
    }
    float ox, oy, oz;
    if (M != 0.f) {
        const float inv = 1.f / M;
        ox = px * inv, oy = py * inv, oz = pz * inv;  // C - G
        sxx -= px * ox;
        sxy -= px * oy;
        sxz -= px * oz;
        syy -= py * oy;
        syz -= py * oz;
        szz -= pz * oz;
    } else {
        const float k = float(max(count, 1));
        ox = ux / k, oy = uy / k, oz = uz / k;
    }
    float ex, ey, ez;
    const float hx = two_sum(g.x, ox, ex), hy = two_sum(g.y, oy, ey), hz = two_sum(g.z, oz, ez);
    *a = make_float4(hx, hy, hz, M);
    Rec32 r;
    r.lo = make_float4(ex, ey, ez, Ml);
    r.s0 = make_float4(sxx, sxy, sxz, syy);
    r.s1 = make_float4(syz, szz, __int_as_float(count), 0.f);
    return r;
}

__device__ __forceinline__ Moments combine8(double4_32a g, bool has, const Moments &c, double4_32a *a) {
    double dx = 0, dy = 0, dz = 0, m = 0, cn = 0;
    if (has) dx = c.cx - g.x, dy = c.cy - g.y, dz = c.cz - g.z, m = c.m, cn = c.count;
    const double mx = m * dx, my = m * dy, mz = m * dz;
    Moments r{};
    r.m = sum8(m);
    r.count = sum8(cn);
    const double px = sum8(mx), py = sum8(my), pz = sum8(mz);
    r.sxx = sum8((has ? c.sxx : 0.0) + mx * dx), r.sxy = sum8((has ? c.sxy : 0.0) + mx * dy);
    r.sxz = sum8((has ? c.sxz : 0.0) + mx * dz), r.syy = sum8((has ? c.syy : 0.0) + my * dy);
    r.syz = sum8((has ? c.syz : 0.0) + my * dz), r.szz = sum8((has ? c.szz : 0.0) + mz * dz);
    double ux = 0, uy = 0, uz = 0;
    if (__any_sync(0xffffffffu, r.m == 0.0)) ux = sum8(cn * dx), uy = sum8(cn * dy), uz = sum8(cn * dz);
    if (r.m != 0.0) {
        const double inv = 1.0 / r.m;
        const double ox = px * inv, oy = py * inv, oz = pz * inv;  // C - G
        r.cx = g.x + ox;
        r.cy = g.y + oy;
        r.cz = g.z + oz;
        r.sxx -= px * ox;
        r.sxy -= px * oy;
        r.sxz -= px * oz;
        r.syy -= py * oy;
        r.syz -= py * oz;
        r.szz -= pz * oz;
    } else {
        const double k = fmax(r.count, 1.0);
        r.cx = g.x + ux / k;
        r.cy = g.y + uy / k;
        r.cz = g.z + uz / k;
    }
    *a = Prec<double>::make(r.cx, r.cy, r.cz, r.m);
    return r;
}

// A combined cell's node data (w its width). A cell's nodeB.w (a leaf's body count) holds
// (M w^3)^(2/5): the error-bound opening radius^2 is this times (alpha |a|)^(-2/5) of the
// walking group.
__device__ __forceinline__ void put_cell(int pk, float w, float4 a, const Rec32 &r, float4 *nodeA, float4 *nodeQ,
                                         int4 *nodeB) {
    nodeA[pk] = a;
    nodeB[pk].w = __float_as_int(a.w > 0.f ? __powf(a.w * w * w * w, 0.4f) : 0.f);
    store_quad(nodeQ, pk, r.s0.x, r.s0.y, r.s0.z, r.s0.w, r.s1.x, r.s1.y);
}
__device__ __forceinline__ void put_cell(int pk, double, double4_32a a, const Moments &, double4_32a *nodeA, float4 *,
                                         int4 *) {
    nodeA[pk] = a;  // the f64 method is monopole only
}

template <class T>
using Record = typename std::conditional<sizeof(T) == 4, Rec32, Moments>::type;

// Records of N cells in shared memory. Until a cell is combined its record holds its box
// (centre, width).
template <class T, int N>
struct Records;
template <int N>
struct Records<float, N> {
    float4 f[4][N];  // nodeA, lo, s0, s1
    __device__ __forceinline__ void set_box(int l, float4 g) { f[0][l] = g; }
    __device__ __forceinline__ float4 box(int l) const { return f[0][l]; }
    __device__ __forceinline__ void set(int l, float4 a, const Rec32 &r) {
        f[0][l] = a, f[1][l] = r.lo, f[2][l] = r.s0, f[3][l] = r.s1;
    }
    __device__ __forceinline__ void get(int l, Child32 &c) const {
        c.a = f[0][l], c.lo = f[1][l], c.s0 = f[2][l], c.s1 = f[3][l];
    }
};
template <int N>
struct Records<double, N> {
    double f[11][N];
    __device__ __forceinline__ void set_box(int l, double4_32a g) {
        f[0][l] = g.x, f[1][l] = g.y, f[2][l] = g.z, f[3][l] = g.w;
    }
    __device__ __forceinline__ double4_32a box(int l) const { return Prec<double>::make(f[0][l], f[1][l], f[2][l], f[3][l]); }
    __device__ __forceinline__ void set(int l, double4_32a, const Moments &r) {
        f[0][l] = r.m, f[1][l] = r.cx, f[2][l] = r.cy, f[3][l] = r.cz, f[4][l] = r.sxx, f[5][l] = r.sxy;
        f[6][l] = r.sxz, f[7][l] = r.syy, f[8][l] = r.syz, f[9][l] = r.szz, f[10][l] = r.count;
    }
    __device__ __forceinline__ void get(int l, Moments &c) const {
        c.m = f[0][l], c.cx = f[1][l], c.cy = f[2][l], c.cz = f[3][l], c.sxx = f[4][l], c.sxy = f[5][l];
        c.sxz = f[6][l], c.syy = f[7][l], c.syz = f[8][l], c.szz = f[9][l], c.count = f[10][l];
    }
};

// Cells bucketed by octree level in shared memory: count with add(), then every thread of the
// block calls offsets(), then place().
template <int N>
struct LevelLists {
    uint16_t list[N];
    int cnt[LEVELS], start[LEVELS + 1];
    __device__ __forceinline__ void clear() {
        if (threadIdx.x < LEVELS) cnt[threadIdx.x] = 0;
    }
    __device__ __forceinline__ int add(int level) { return atomicAdd(&cnt[level], 1); }
    __device__ __forceinline__ void offsets() {
        __syncthreads();
        if (threadIdx.x == 0) {
            int acc = 0;
            for (int L = 0; L < LEVELS; ++L) {
                start[L] = acc;
                acc += cnt[L];
            }
            start[LEVELS] = acc;
        }
        __syncthreads();
    }
    __device__ __forceinline__ void place(int level, int rank, int l) { list[start[level] + rank] = uint16_t(l); }
};

// Child entries by octant digit, which is the children's preorder: a local cell, or a local
// unit, of several bodies or one.
constexpr unsigned KID_NONE = 0xffffu, KID_CELL = 0x8000u, KID_BUCKET = 0x4000u, KID_INDEX = 0x3fffu;
static_assert(CHUNK <= int(KID_INDEX) && SPAN_CAP <= int(KID_INDEX), "local indices fit the child entries");

template <class T>
struct alignas(32) Chunk {
    typename Prec<T>::V4 body[CHUNK];
    Records<T, CHUNK> rec;
    alignas(16) uint16_t kid[CHUNK][8];
    int pre[CHUNK];      // the cells' preorder indices
    LevelLists<CHUNK> lists;
    uint8_t out[CHUNK];  // the cell's parent is of a later stage: its record goes to global memory
};

// A chunk cell's children.
template <class T>
struct ChunkKids {
    const Chunk<T> &C;
    int l;
    const Record<T> *grec;  // several-body leaves have their record in global memory
    const uint32_t *pscan, *starts;
    int c0;
    __device__ __forceinline__ bool operator()(int i, ChildOf<T> &c) const {
        const unsigned e = C.kid[l][i];
        if (e == KID_NONE) return false;
        const int x = int(e & KID_INDEX), u = c0 + x;
        if (e & KID_CELL) C.rec.get(x, c);
        else if (e & KID_BUCKET) child_record(C.body[x], grec + (u + int(pscan[u]) + __popc(starts[u])), c);
        else child_single(C.body[x], c);
        return true;
    }
};

// ---- 6. preorder layout, the leaves' records and the chunks' cells ------------
// nodeB = {width bits, skip, first body (-1: internal cell), body count}.
// counters[1] = T (cells + leaves), counters[2] = internal cells.
// A block lays out the nodes of one chunk of CHUNK units (a binary node's index is one end of
// its range, so a chunk's inner cells are among its own indices) and then combines the
// chunk's inner cells level by level from shared memory. (As two passes over global memory, a
// layout and a launch per level, they took 193 + 478 us of the launch list at N = 4M, 51 + 225
// at N = 1M and 7 + 102 at N = 10000; layout and cells_span take 283 + 86, 84 + 58 and 22 +
// 15.) A block waits on its own chain of loads, four blocks to an SM.
constexpr int CHUNK_THREADS = 256;
constexpr int SPREAD = 8;

template <class T>
__global__ void __launch_bounds__(CHUNK_THREADS)
    layout(int *counters, const int *__restrict__ bfirst, const int *__restrict__ blast,
           const int *__restrict__ bdelta, const uint8_t *__restrict__ top, const int *__restrict__ oparent,
           const uint32_t *__restrict__ starts, const uint32_t *__restrict__ pscan, const uint64_t *__restrict__ ukey,
           const uint32_t *__restrict__ ufirst, const T *__restrict__ box, int *__restrict__ pre, int4 *nodeB,
           typename Prec<T>::V4 *__restrict__ nodeG, int2 *__restrict__ nodeR, const int *__restrict__ loparent,
           int *__restrict__ kid, const typename Prec<T>::V4 *__restrict__ sbody, Record<T> *rec,
           typename Prec<T>::V4 *nodeA, float4 *nodeQ) {
    after_previous();
    using P = Prec<T>;
    constexpr int PER = CHUNK / CHUNK_THREADS;
    extern __shared__ __align__(32) unsigned char block_raw[];
    Chunk<T> &C = *reinterpret_cast<Chunk<T> *>(block_raw);
    const int M = counters[0];
    // Neighbouring chunks go to blocks SPREAD apart: where bodies share keys only the first few
    // chunks hold units, and the first blocks start on the same SMs (1M bodies within 1e-5 of the
    // box: build 2.13 ms in block order, 0.91 so).
    const int c0 = int(blockIdx.x % SPREAD * (gridDim.x / SPREAD) + blockIdx.x / SPREAD) << CHUNK_SHIFT;
    if (c0 >= M) return;
    if (blockIdx.x == 0) clear_stats(counters, threadIdx.x);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        counters[1] = M + int(pscan[M]);
        counters[2] = int(pscan[M]);
    }
    C.lists.clear();
    for (int i = threadIdx.x; i < CHUNK; i += CHUNK_THREADS)
        reinterpret_cast<uint4 *>(C.kid)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    __syncthreads();
    int lvl[PER], rank[PER];  // a chunk cell's octree level and rank among the chunk's of that level
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int lk = q * CHUNK_THREADS + threadIdx.x;
        const int k = c0 + lk;
        lvl[q] = -1;
        const int cls = k < M - 1 ? top[k] : 0;
        if (cls) {
            const int b = bfirst[k], after = blast[k] + 1, op = oparent[k];
            const int L = bdelta[k] / 3;
            // the unit's shallower cells come first
            const int pk = b + int(pscan[b]) + __popc(starts[b] & ((1u << L) - 1u));
            const int skip = after + int(pscan[after]);
            // Cell box at level L along the key's path: BoundingBox::width() of the
            // reference cell (partition.rs:322-327) and its centre, replayed in the same
            // f32 ops.
            const uint64_t key = ukey[b];
            T mn0 = box[0], mn1 = box[1], mn2 = box[2], mx0 = box[3], mx1 = box[4], mx2 = box[5];
            for (int l = 0; l < L; ++l) {
                const int o = 7 - digit_at(key, l);
                const T x = P::mul(P::add(mn0, mx0), T(0.5));
                const T y = P::mul(P::add(mn1, mx1), T(0.5));
                const T z = P::mul(P::add(mn2, mx2), T(0.5));
                if (o & 1) mx0 = x; else mn0 = x;
                if (o & 2) mx1 = y; else mn1 = y;
                if (o & 4) mx2 = z; else mn2 = z;
            }
            const T w = P::sub(mx0, mn0);
            const auto g = P::make(T(0.5) * (mn0 + mx0), T(0.5) * (mn1 + mx1), T(0.5) * (mn2 + mx2), w);
            // the f32 walk reads the width from nodeB.x; the f64 walk from nodeG.w
            nodeB[pk] = make_int4(sizeof(T) == 4 ? __float_as_int(float(w)) : 0, skip, -1, 0);
            nodeG[pk] = g;
            nodeR[pk] = make_int2(int(ufirst[b]), int(ufirst[after]));
            const bool out = op >= 0 && top[op] > cls;
            const int digit = op >= 0 ? digit_at(key, bdelta[op] / 3) : 0;
            if (out) kid[8 * size_t(op) + digit] = 2 * pk;
            if (cls == 1) {
                if (op >= 0 && !out) C.kid[op - c0][digit] = uint16_t(KID_CELL | unsigned(lk));
                C.pre[lk] = pk;
                C.out[lk] = out;
                C.rec.set_box(lk, g);
                lvl[q] = L;
                rank[q] = C.lists.add(L);
            } else {
                pre[k] = pk;
            }
        }
        if (k < M) {
            const int pk = k + int(pscan[k]) + __popc(starts[k]);
            const int f = int(ufirst[k]);
            const int nb = int(ufirst[k + 1]) - f;
            nodeB[pk] = make_int4(0, pk + 1, f, nb);
            // (no nodeG / nodeR for leaves: the cell centre and body range are read for
            // cells only, by the f64 walk's widths and the learned features and samples)
            const int op = loparent[k];
            C.body[lk] = leaf(pk, f, f + nb, sbody, rec, nodeA, nodeQ);  // the leaf's moment record
            if (op >= 0) {
                const int digit = digit_at(ukey[k], bdelta[op] / 3);
                if (top[op] > 1) kid[8 * size_t(op) + digit] = 2 * pk + (nb == 1 ? 1 : 0);
                else C.kid[op - c0][digit] = uint16_t((nb == 1 ? 0u : KID_BUCKET) | unsigned(lk));
            }
        }
    }
    C.lists.offsets();
#pragma unroll
    for (int q = 0; q < PER; ++q)
        if (lvl[q] >= 0) C.lists.place(lvl[q], rank[q], q * CHUNK_THREADS + threadIdx.x);
    for (int L = LEVELS - 1; L >= 0; --L) {
        const int s = C.lists.start[L], e = C.lists.start[L + 1];
        if (s == e) continue;
        __syncthreads();  // the list; the records of the levels below
        for (int i = s + threadIdx.x; i < e; i += CHUNK_THREADS) {
            const int l = C.lists.list[i], pk = C.pre[l];
            const auto g = C.rec.box(l);
            typename P::V4 a;
            const Record<T> r = combine(g, ChunkKids<T>{C, l, rec, pscan, starts, c0}, &a);
            put_cell(pk, g.w, a, r, nodeA, nodeQ, nodeB);
            if (C.out[l]) rec[pk] = r;
            C.rec.set(l, a, r);
        }
    }
}

// The cells that span blocks of the stage before and lie in one of this stage's, a block of
// threads for each such block. Children of the same stage are in shared memory, the others
// have their records in global memory. (Climbing from child to parent through global memory
// took 62 us at N = 10000 and 128 us at N = 4M, a cluster going level by level 177 us there:
// a step up costs some five trips to L2 and two fences, 6 us. From shared memory, eight lanes
// to a cell: 15 us at N = 10000, 29 + 35 + 22 us for the three stages at N = 4M.)
constexpr int SPAN_THREADS = 512;

template <class T>
struct alignas(32) SpanBlock {
    Records<T, SPAN_CAP> rec;
    int kid[SPAN_CAP][8];  // 2 x preorder index + 1 for a single body, -1 none, -2 - x: local cell x
    int pre[SPAN_CAP];     // preorder indices
    LevelLists<SPAN_CAP> lists;
    uint8_t out[SPAN_CAP]; // the cell's parent is of a later stage: its record goes to global memory
};

template <class T>
__global__ void __launch_bounds__(SPAN_THREADS)
    cells_span(int n, int stage, const int *__restrict__ nspan, const int *__restrict__ spans,
               const int *__restrict__ bfirst, const int *__restrict__ bdelta, const uint8_t *__restrict__ top,
               const uint64_t *__restrict__ ukey, const int *__restrict__ oparent, const int *__restrict__ pre,
               const int *__restrict__ kid, const uint32_t *__restrict__ kmask, int *slot,
               const typename Prec<T>::V4 *__restrict__ nodeG, Record<T> *rec, typename Prec<T>::V4 *nodeA,
               float4 *nodeQ, int4 *nodeB) {
    after_previous();
    extern __shared__ __align__(32) unsigned char block_raw[];
    SpanBlock<T> &C = *reinterpret_cast<SpanBlock<T> *>(block_raw);
    const int blk = stage_first(n, stage) + blockIdx.x;
    const int m = min(nspan[blk], SPAN_CAP);
    if (m == 0) return;
    constexpr int PER = (SPAN_CAP + SPAN_THREADS - 1) / SPAN_THREADS;
    const int *cells = spans + size_t(blk) * SPAN_CAP;
    C.lists.clear();
    for (int x = threadIdx.x; x < 8 * m; x += SPAN_THREADS) {
        const int i = x >> 3, d = x & 7, k = cells[i];
        C.kid[i][d] = (kmask[k] >> d) & 1u ? kid[8 * size_t(k) + d] : -1;
        if (d == 0) slot[k] = i;
    }
    __syncthreads();
    int lvl[PER], rank[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int i = q * SPAN_THREADS + threadIdx.x;
        if (i >= m) break;
        const int k = cells[i], op = oparent[k], pk = pre[k];
        const bool same = op >= 0 && top[op] == top[k];
        C.pre[i] = pk;
        C.out[i] = op >= 0 && !same;
        C.rec.set_box(i, nodeG[pk]);
        lvl[q] = bdelta[k] / 3;
        rank[q] = C.lists.add(lvl[q]);
        if (same) C.kid[slot[op]][digit_at(ukey[bfirst[k]], bdelta[op] / 3)] = -2 - i;
    }
    C.lists.offsets();
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int i = q * SPAN_THREADS + threadIdx.x;
        if (i >= m) break;
        C.lists.place(lvl[q], rank[q], i);
    }
    const int lane = threadIdx.x & 31, d = lane & 7;
    for (int L = LEVELS - 1; L >= 0; --L) {
        const int s = C.lists.start[L], e = C.lists.start[L + 1];
        if (s == e) continue;
        __syncthreads();  // the list; the records of the levels below
        for (int i0 = s + (threadIdx.x >> 5) * 4; i0 < e; i0 += SPAN_THREADS / 8) {  // four cells to a warp
            const bool valid = i0 + (lane >> 3) < e;
            const int l = C.lists.list[valid ? i0 + (lane >> 3) : i0], x = C.kid[l][d];
            const auto g = C.rec.box(l);
            ChildOf<T> c;
            if (x >= 0) {
                const auto ca = ld_cg(nodeA + (x >> 1));
                if (x & 1) child_single(ca, c);
                else child_record(ca, rec + (x >> 1), c);
            } else if (x < -1) {
                C.rec.get(-2 - x, c);
            }
            typename Prec<T>::V4 a;
            const Record<T> r = combine8(g, x != -1, c, &a);
            if (valid && d == 0) {
                const int pk = C.pre[l];
                put_cell(pk, g.w, a, r, nodeA, nodeQ, nodeB);
                if (C.out[l]) rec[pk] = r;
                C.rec.set(l, a, r);
            }
        }
    }
}

template <class T>
int build_t(pt_ctx *ctx, State &S, const typename Prec<T>::V4 *d_src, int n) {
    using V4 = typename Prec<T>::V4;
    constexpr bool F64 = sizeof(T) == 8;
    // the f64 method keeps its own body, node and box arrays (the rest is shared)
    DevBuf &sb = F64 ? S.sbody64 : S.sbody;
    DevBuf &nA = F64 ? S.nodeA64 : S.nodeA;
    DevBuf &nG = F64 ? S.nodeG64 : S.nodeG;
    cudaStream_t st = ctx->stream;
    const size_t N = size_t(n);
    const int nb = std::min(1024, blocks(n));  // of root_box
    PT_TRY(ensure_buf(ctx, S.box_part, sizeof(T) * 6 * size_t(nb)));
    PT_TRY(ensure_buf(ctx, S.box, sizeof(T) * 8));
    PT_TRY(ensure_buf(ctx, S.keys, sizeof(uint64_t) * N));
    PT_TRY(ensure_buf(ctx, S.idx, sizeof(uint32_t) * N));
    PT_TRY(ensure_buf(ctx, sb, sizeof(V4) * N));
    PT_TRY(ensure_buf(ctx, S.ukey, sizeof(uint64_t) * N));
    PT_TRY(ensure_buf(ctx, S.ufirst, sizeof(uint32_t) * (N + 1)));
    PT_TRY(ensure_buf(ctx, S.bfirst, sizeof(int) * N));
    PT_TRY(ensure_buf(ctx, S.blast, sizeof(int) * N));
    PT_TRY(ensure_buf(ctx, S.bdelta, sizeof(int) * N));
    PT_TRY(ensure_buf(ctx, S.bparent, sizeof(int) * N));
    PT_TRY(ensure_buf(ctx, S.lparent, sizeof(int) * N));
    PT_TRY(ensure_buf(ctx, S.top, N));
    PT_TRY(ensure_buf(ctx, S.oparent, sizeof(int) * N));
    PT_TRY(ensure_buf(ctx, S.loparent, sizeof(int) * N));
    PT_TRY(ensure_buf(ctx, S.starts, sizeof(uint32_t) * (N + 1)));
    PT_TRY(ensure_buf(ctx, S.pscan, sizeof(uint32_t) * (N + 2)));
    PT_TRY(ensure_buf(ctx, S.pre, sizeof(int) * N));
    PT_TRY(ensure_buf(ctx, S.kmask, sizeof(uint32_t) * N));
    PT_TRY(ensure_buf(ctx, S.slot, sizeof(int) * N));
    PT_TRY(ensure_buf(ctx, S.kid, sizeof(int) * 8 * N));
    PT_TRY(ensure_buf(ctx, nA, sizeof(V4) * 2 * N));
    PT_TRY(ensure_buf(ctx, S.nodeB, sizeof(int4) * 2 * N));
    if (!F64) PT_TRY(ensure_buf(ctx, S.nodeQ, sizeof(float4) * 4 * N));
    PT_TRY(ensure_buf(ctx, nG, sizeof(V4) * 2 * N));
    float4 *nodeQ = F64 ? nullptr : as<float4>(S.nodeQ);
    PT_TRY(ensure_buf(ctx, S.nodeR, sizeof(int2) * 2 * N));
    PT_TRY(ensure_buf(ctx, S.mom, sizeof(Record<T>) * 2 * N));
    PT_TRY(ensure_counters(ctx, S));

    RadixFirst rf{};
    PT_TRY(radix_sort_prepare(ctx, S.prims, n, 3 * LEVELS, &rf));
    int *counters = as<int>(S.counters);
    launch_next(root_box<T>, nb, 256, 0, st, d_src, n, as<T>(S.box_part), as<T>(S.box), rf.zero, rf.zero_words,
                ctx->keep_errors ? nullptr : counters + 3, reinterpret_cast<unsigned *>(counters) + ROOT_BOX_DONE);
    PT_TRY(check_launch(ctx, "root_box"));
    PT_TRY(launch_make_keys<T>(ctx, d_src, n, as<T>(S.box), as<uint64_t>(S.keys), rf));
    PT_TRY(radix_sort_u64(ctx, S.prims, as<uint64_t>(S.keys), as<uint32_t>(S.idx), n, 3 * LEVELS));
    PT_TRY(scan_generated(ctx, S.prims, UnitHead{as<uint64_t>(S.keys)},
                          UnitFill{as<uint64_t>(S.keys), n, as<uint64_t>(S.ukey), as<uint32_t>(S.ufirst), counters}, n));
    const int nstages = stages(n), span_blocks = stage_first(n, nstages + 1);
    PT_TRY(ensure_buf(ctx, S.nspan, sizeof(int) * size_t(std::max(1, span_blocks))));
    PT_TRY(ensure_buf(ctx, S.spans, sizeof(int) * size_t(std::max(1, span_blocks)) * SPAN_CAP));
    launch_next(karras<V4>, blocks(n + 1), 256, 0, st, d_src, as<uint32_t>(S.idx), as<V4>(sb), as<uint64_t>(S.ukey),
                counters, n, as<int>(S.bfirst), as<int>(S.blast), as<int>(S.bdelta), as<int>(S.bparent),
                as<int>(S.lparent), as<uint8_t>(S.top), as<uint32_t>(S.starts), as<uint32_t>(S.kmask),
                as<int>(S.nspan), span_blocks);
    PT_TRY(check_launch(ctx, "karras"));
    launch_next(octree_links, blocks(n), 256, 0, st, counters, n, as<int>(S.bfirst), as<int>(S.bparent), as<int>(S.lparent),
                                           as<uint8_t>(S.top), as<int>(S.bdelta), as<uint64_t>(S.ukey),
                                           as<int>(S.oparent), as<int>(S.loparent), as<uint32_t>(S.starts),
                                           as<uint32_t>(S.kmask), as<int>(S.nspan), as<int>(S.spans));
    PT_TRY(check_launch(ctx, "octree_links"));
    PT_TRY(scan_generated(ctx, S.prims, CellStarts{as<uint32_t>(S.starts)},
                          scan::WriteU32{as<uint32_t>(S.pscan), n + 1}, n + 1));
    const int chunks = ((n + CHUNK - 1) / CHUNK + SPREAD - 1) / SPREAD * SPREAD;
    PT_CUDA(cudaFuncSetAttribute(layout<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(Chunk<T>))));
    launch_next(
        layout<T>, chunks, CHUNK_THREADS, sizeof(Chunk<T>), st, counters, as<int>(S.bfirst), as<int>(S.blast), as<int>(S.bdelta), as<uint8_t>(S.top), as<int>(S.oparent),
        as<uint32_t>(S.starts), as<uint32_t>(S.pscan), as<uint64_t>(S.ukey), as<uint32_t>(S.ufirst), as<T>(S.box),
        as<int>(S.pre), as<int4>(S.nodeB), as<V4>(nG), as<int2>(S.nodeR), as<int>(S.loparent), as<int>(S.kid),
        as<V4>(sb), as<Record<T>>(S.mom), as<V4>(nA), nodeQ);
    PT_TRY(check_launch(ctx, "layout"));
    if (nstages > 0)
        PT_CUDA(cudaFuncSetAttribute(cells_span<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(sizeof(SpanBlock<T>))));
    for (int stage = 1; stage <= nstages; ++stage) {
        launch_next(
            cells_span<T>, stage_blocks(n, stage), SPAN_THREADS, sizeof(SpanBlock<T>), st, n, stage, as<int>(S.nspan), as<int>(S.spans), as<int>(S.bfirst), as<int>(S.bdelta), as<uint8_t>(S.top),
            as<uint64_t>(S.ukey), as<int>(S.oparent), as<int>(S.pre), as<int>(S.kid), as<uint32_t>(S.kmask),
            as<int>(S.slot), as<V4>(nG), as<Record<T>>(S.mom), as<V4>(nA), nodeQ, as<int4>(S.nodeB));
        PT_TRY(check_launch(ctx, "cells_span"));
    }
    S.last_n_src = n;
    S.f64 = F64;
    S.user_tree = false;
    ++S.generation;
    return PT_OK;
}

int build(pt_ctx *ctx, State &S, const float4 *d_src, int n) { return build_t<float>(ctx, S, d_src, n); }

// Sorts separate targets along the same keys (same root box) for coherent warps.
template <class T>
int sort_targets_t(pt_ctx *ctx, State &S, const typename Prec<T>::V4 *d_aff, int n) {
    using V4 = typename Prec<T>::V4;
    DevBuf &tb = sizeof(T) == 8 ? S.tbody64 : S.tbody;
    cudaStream_t st = ctx->stream;
    PT_TRY(ensure_buf(ctx, S.tkeys, sizeof(uint64_t) * size_t(n)));
    PT_TRY(ensure_buf(ctx, S.tidx, sizeof(uint32_t) * size_t(n)));
    PT_TRY(ensure_buf(ctx, tb, sizeof(V4) * size_t(n)));
    RadixFirst rf{};
    PT_TRY(radix_sort_prepare(ctx, S.prims, n, 3 * LEVELS, &rf));
    PT_CUDA(cudaMemsetAsync(rf.zero, 0, sizeof(uint32_t) * size_t(rf.zero_words), st));
    PT_TRY(launch_make_keys<T>(ctx, d_aff, n, as<T>(S.box), as<uint64_t>(S.tkeys), rf));
    PT_TRY(radix_sort_u64(ctx, S.prims, as<uint64_t>(S.tkeys), as<uint32_t>(S.tidx), n, 3 * LEVELS));
    launch_next(gather_bodies<V4>, blocks(n), 256, 0, st, d_aff, as<uint32_t>(S.tidx), n, as<V4>(tb), as<int>(S.counters));
    return check_launch(ctx, "gather_bodies(targets)");
}

int sort_targets(pt_ctx *ctx, State &S, const float4 *d_aff, int n) {
    return sort_targets_t<float>(ctx, S, d_aff, n);
}


template int build_t<double>(pt_ctx *, State &, const Prec<double>::V4 *, int);
template int sort_targets_t<double>(pt_ctx *, State &, const Prec<double>::V4 *, int);

}  // namespace bh
}  // namespace pt
