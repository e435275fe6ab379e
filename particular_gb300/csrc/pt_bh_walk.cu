// cuda::BarnesHut walks over the tree of pt_bh_build.cu (sequential.rs:466-505):
//  * bh_walk_masked: the default method, the reference's per-body rule with one
//    shared traversal per warp (accept/open masks on stack ranges and list entries);
//  * bh_walk_group (PT_BH_GROUP): a cell opened for all 64 bodies of a warp when any
//    of them opens it, lists evaluated densely, optional quadrupoles, local
//    expansions of far nodes (PT_BH_LOCAL), the error-bound opening radius
//    (PT_BH_RELATIVE, with its per-group estimate bh_group_scale) and the learned
//    correction's records;
//  * bh_walk64: the reference rule over DVec3 bodies in double;
//  * lane_walk: the per-body cursor walk the others fall back to when a stack runs out.
#include "pt_bh_group.cuh"

namespace pt {
namespace bh {

// ---- learned correction: evaluation of the group walk's records ----------------
// One warp per chunk (grid-stride): features of the 128 recorded cells at the group
// centre, four 32-row tensor-core batches, the chunk's sum into part[chunk]. (It holds
// 2 CTAs per SM at ~242 registers; capped at 168 for 3 CTAs it spills 128 bytes and
// the learned step at N = 4M went from 9.95 to 10.69 ms.)
// Cells whose size/distance ratio at the group centre lies outside the range the
// model was trained on ([lo, hi]) get no correction.
__global__ void __launch_bounds__(128) bh_learned_eval(LearnedRecords L, const float4 *__restrict__ nodeA,
                                                      const float4 *__restrict__ nodeQ,
                                                      const float4 *__restrict__ nodeG,
                                                      const uint32_t *__restrict__ W, const float *__restrict__ bias,
                                                      float lo, float hi) {
    __shared__ float X[4][32 * mlp::TC_XS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int used = min(*L.used, L.cap);
    const float sc = __ldg(bias + mlp::TC_SCALE);
    float *Xw = X[warp];
    for (int c = blockIdx.x * 4 + warp; c < used; c += gridDim.x * 4) {
        const float4 gc = L.centre[L.chunk_group[c]];
        float rx = 0.f, ry = 0.f, rz = 0.f;
        for (int b = 0; b < LCHUNK / 32; ++b) {
            const int node = L.rec[size_t(c) * LCHUNK + b * 32 + lane];
            if (__ballot_sync(0xffffffffu, node >= 0) == 0u) break;  // padding fills the chunk's tail
            float f[mlp::IN];
            float a = 0.f;  // M / |r|^2 of this row's cell, 0 = no correction
            if (node >= 0) {
                const float4 A = __ldg(nodeA + node);
                const float4 q0 = __ldg(nodeQ + 2 * node), q1 = __ldg(nodeQ + 2 * node + 1);
                const float q[6] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y};
                const float r2 = mlp::features(gc.x, gc.y, gc.z, A, q, __ldg(nodeG + node), f);
                if (f[3] >= lo && f[3] <= hi) a = A.w / r2;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) Xw[lane * mlp::TC_XS + i] = (i < mlp::IN && a != 0.f) ? f[i] : 0.f;
            __syncwarp();
            float y[2][4];
            mlp::tc_batch(Xw, W, bias, y);
            __syncwarp();
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float s = __shfl_sync(0xffffffffu, a, 16 * mt + 8 * h + g);
                    if (t == 0) {
                        rx = fmaf(y[mt][2 * h], s, rx);
                        ry = fmaf(y[mt][2 * h + 1], s, ry);
                    } else if (t == 1) {
                        rz = fmaf(y[mt][2 * h], s, rz);
                    }
                }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            rx += __shfl_xor_sync(0xffffffffu, rx, off);
            ry += __shfl_xor_sync(0xffffffffu, ry, off);
            rz += __shfl_xor_sync(0xffffffffu, rz, off);
        }
        if (lane == 0) L.part[c] = make_float4(rx * sc, ry * sc, rz * sc, 0.f);
    }
}

// out[target] += the sum of its group's chunk corrections, in chain order.
__global__ void bh_learned_apply(LearnedRecords L, const uint32_t *__restrict__ tidx, int n_aff, int group_shift,
                                 float *__restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_aff) return;
    float cx = 0.f, cy = 0.f, cz = 0.f;
    // chunk indices grow along a chain (each is taken after its predecessor)
    for (int c = L.head[t >> group_shift], prev = -1; c > prev && c < L.cap; prev = c, c = L.next[c]) {
        const float4 v = L.part[c];
        cx += v.x;
        cy += v.y;
        cz += v.z;
    }
    const uint32_t o = tidx[t];
    out[3 * size_t(o) + 0] += cx;
    out[3 * size_t(o) + 1] += cy;
    out[3 * size_t(o) + 2] += cz;
}

// ---- estimate of |a| per group ------------------------------------------------
// PT_BH_RELATIVE: |a| estimated at the centre of each group's box by a walk at theta
// = 1.5 with monopoles; gscale[g] = 1 / (alpha |a|), the factor of the group walk's
// error bound. (At N = 4M bulge+disk, estimates from theta 1.0 and 1.5 walks select
// the same cells up to 0.2 %; 1.5 visits about half the nodes.)
// The per-point cursor walk: the node index only grows, so the loop ends.
__device__ __forceinline__ void scale_cursor_walk(float cx, float cy, float cz, const float4 *__restrict__ nodeA,
                                                  const int4 *__restrict__ nodeB, int T, float eps2, float &ax,
                                                  float &ay, float &az) {
    for (int node = 0; node < T;) {
        const float4 A = __ldg(nodeA + node);
        const int4 B = __ldg(nodeB + node);
        const float dx = A.x - cx, dy = A.y - cy, dz = A.z - cz;
        const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        if (B.z < 0) {
            const float w = __int_as_float(B.x);
            if (2.25f * d2 < w * w) {  // theta = 1.5: open
                ++node;
                continue;
            }
        }
        if (d2 > 0.f) {
            const float inv = rsqrt_ftz(d2 + eps2);
            const float s = (A.w * inv) * (inv * inv);
            ax = fmaf(dx, s, ax);
            ay = fmaf(dy, s, ay);
            az = fmaf(dz, s, az);
        }
        node = B.y;
    }
}

// One thread per group: the group's box, then the cursor walk from its centre. (One
// warp per group walking with a range stack, one node per lane and pop, was slower at
// N = 4M: the walk phase, which includes this kernel, went from 5.68 to 5.85 ms. Its
// 65536 warps take several waves, each pop a round trip to L2, while the threads'
// cursor walks mostly hit L1 in the tree's upper levels. Eight threads per group, each
// walking one of the root's children's subtrees, took the same 0.124 ms: the group's
// own octant holds most of the visits. Four lanes per group popping up to four ranges
// of a shared-memory stack per step took 0.18 ms: a walk from one point keeps few
// ranges open, so the steps stayed nearly as many and each cost more.)
__global__ void __launch_bounds__(128)
    bh_group_scale(const float4 *__restrict__ tbody, int n_aff, const float4 *__restrict__ nodeA,
                   const int4 *__restrict__ nodeB, const int *__restrict__ counters, float eps2, float alpha,
                   float *__restrict__ gscale) {
    after_previous();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int g0 = g * GW_GROUP;
    if (g0 >= n_aff) return;
    const int g1 = min(n_aff, g0 + GW_GROUP);
    float4 p = tbody[g0];
    float mn0 = p.x, mn1 = p.y, mn2 = p.z, mx0 = p.x, mx1 = p.y, mx2 = p.z;
    for (int t = g0 + 1; t < g1; ++t) {
        p = tbody[t];
        mn0 = fminf(mn0, p.x), mn1 = fminf(mn1, p.y), mn2 = fminf(mn2, p.z);
        mx0 = fmaxf(mx0, p.x), mx1 = fmaxf(mx1, p.y), mx2 = fmaxf(mx2, p.z);
    }
    float ax = 0.f, ay = 0.f, az = 0.f;
    scale_cursor_walk(0.5f * (mn0 + mx0), 0.5f * (mn1 + mx1), 0.5f * (mn2 + mx2), nodeA, nodeB, counters[1], eps2,
                      ax, ay, az);
    const float a = sqrtf(fmaf(ax, ax, fmaf(ay, ay, az * az)));
    gscale[g] = 1.f / (alpha * fmaxf(a, 1e-30f));
}

// Two octaves of the scale (positive, or infinite) to a bucket, the largest first.
constexpr int ORDER_BUCKETS = 128;  // a float's upper seven exponent bits
__device__ __forceinline__ int order_bucket(float scale) {
    return ORDER_BUCKETS - 1 - ((__float_as_int(scale) & 0x7fffffff) >> 24);
}

// The groups by descending key, for the walk to take them in: one that opens many cells and
// starts last holds up the call. In the error-bound walk the key is the group's scale: one whose
// error bound is small next to its forces opens the most (rank correlation with its walk 0.75).
// Within a bucket they stay in tree order: neighbours still share what they read, and the order
// is the same every time, which the masked walk needs, for it halves the groups that come last
// and that shows in the rounding of their sums. A stable counting sort by one block, a warp to
// each 32nd of the groups: 5.1 us for the 4096 groups of N = 262144, 10.5 for 16384 and 25 for
// 65536. (Many blocks with a counter per bucket, so in no fixed order, took 3.8 to 4.8 us;
// but in tree order the walk at N = 4M takes 5.08 ms, 5.2 in theirs.) Whole error-bound call
// in tree order alone and by key, us: N = 262144 974 / 872, 524288 1513 / 1209, 1048576 1824 /
// 1825, 2097152 3880 / 3290, 4194304 6008 / 5998.
constexpr int ORDER_WARPS = 32, ORDER_BATCH = 8;

__global__ void __launch_bounds__(32 * ORDER_WARPS)
    bh_group_order(const float *__restrict__ key, int groups, int *__restrict__ gorder) {
    after_previous();
    constexpr int PER = ORDER_BUCKETS / ORDER_WARPS;  // buckets a warp scans
    __shared__ unsigned place[ORDER_WARPS][ORDER_BUCKETS + 1], first[ORDER_BUCKETS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per = (groups + 32 * ORDER_WARPS - 1) / (32 * ORDER_WARPS) * 32;
    const int g0 = min(groups, warp * per), g1 = min(groups, g0 + per);
    int bucket[ORDER_BATCH];  // of the groups i0 + 32 r + lane
    auto load = [&](int i0) {
#pragma unroll
        for (int r = 0; r < ORDER_BATCH; ++r) {
            const int i = i0 + 32 * r + lane;
            bucket[r] = i < g1 ? order_bucket(key[i]) : -1;
        }
    };
    for (int b = lane; b < ORDER_BUCKETS; b += 32) place[warp][b] = 0;
    load(g0);
    __syncwarp();
    for (int i0 = g0;;) {
#pragma unroll
        for (int r = 0; r < ORDER_BATCH; ++r)
            if (bucket[r] >= 0) atomicAdd(&place[warp][bucket[r]], 1u);
        if ((i0 += 32 * ORDER_BATCH) >= g1) break;
        load(i0);
    }
    __syncthreads();
    // where each warp's groups of a bucket go: lane w holds warp w's count
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int b = PER * warp + k;
        const unsigned c = place[lane][b];
        unsigned incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        place[lane][b] = incl - c;
        if (lane == 31) first[b] = incl;
    }
    __syncthreads();
    if (warp == 0) {  // the buckets' starts, PER to a lane
        unsigned c[PER], sum = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            c[k] = sum;
            sum += first[PER * lane + k];
        }
        unsigned incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
#pragma unroll
        for (int k = 0; k < PER; ++k) first[PER * lane + k] = incl - sum + c[k];
    }
    __syncthreads();
    if (per > 32 * ORDER_BATCH) load(g0);  // else the buckets are still there
    for (int i0 = g0;;) {
#pragma unroll
        for (int r = 0; r < ORDER_BATCH; ++r) {
            if (i0 + 32 * r >= g1) break;
            const int b = bucket[r];
            const unsigned peers = __match_any_sync(0xffffffffu, b), below = peers & ((1u << lane) - 1u);
            const unsigned at = b >= 0 ? place[warp][b] : 0u;
            __syncwarp();
            if (b >= 0) {
                gorder[first[b] + at + __popc(below)] = i0 + 32 * r + lane;
                if (below == 0u) place[warp][b] = at + __popc(peers);
            }
            __syncwarp();
        }
        if ((i0 += 32 * ORDER_BATCH) >= g1) break;
        load(i0);
    }
}

// The key of the walks by opening angle: a group's squared width over its squared distance from
// the root's centre of mass, the angle under which the mass sees it (rank correlation with the
// walk 0.57 to 0.68; of the longest 5 % of the walks, 74 to 90 % are in the first fifth). Whole
// call in tree order and so ordered, us: masked N = 131072 theta 0.8 347 / 334, N = 262144 theta
// 0.5 1018 / 964, N = 1M 3226 / 3170; group walk N = 262144 theta 0.6 725 / 699, N = 524288 with
// local expansions 1435 / 1319, N = 1M 3000 / 2930. (The error-bound walk by this key: N = 1M
// 1825 -> 1739, 4M 6015 -> 6127.)
__global__ void __launch_bounds__(256)
    bh_group_width(const float4 *__restrict__ tbody, int n_aff, int groups, int size,
                   const float4 *__restrict__ nodeA, float *__restrict__ ratio) {
    after_previous();
    const int lanes = min(32, size);  // a power of two
    const float4 root = nodeA[0];
    const int step = gridDim.x * blockDim.x / lanes;
    const int l = threadIdx.x % lanes;
    const int rounds = (groups + step - 1) / step;
    int g = (blockIdx.x * blockDim.x + threadIdx.x) / lanes;
    for (int r = 0; r < rounds; ++r, g += step) {  // as many for every thread: the shuffles need the warp
        float mn0 = INFINITY, mn1 = INFINITY, mn2 = INFINITY, mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY;
        if (g < groups)
            for (int t = g * size + l; t < min(n_aff, (g + 1) * size); t += lanes) {
                const float4 p = tbody[t];
                mn0 = fminf(mn0, p.x), mn1 = fminf(mn1, p.y), mn2 = fminf(mn2, p.z);
                mx0 = fmaxf(mx0, p.x), mx1 = fmaxf(mx1, p.y), mx2 = fmaxf(mx2, p.z);
            }
        for (int o = lanes / 2; o > 0; o >>= 1) {
            mn0 = fminf(mn0, __shfl_xor_sync(0xffffffffu, mn0, o));
            mn1 = fminf(mn1, __shfl_xor_sync(0xffffffffu, mn1, o));
            mn2 = fminf(mn2, __shfl_xor_sync(0xffffffffu, mn2, o));
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
            mx2 = fmaxf(mx2, __shfl_xor_sync(0xffffffffu, mx2, o));
        }
        if (l == 0 && g < groups) {
            const float w0 = mx0 - mn0, w1 = mx1 - mn1, w2 = mx2 - mn2;
            const float d0 = 0.5f * (mn0 + mx0) - root.x, d1 = 0.5f * (mn1 + mx1) - root.y,
                        d2 = 0.5f * (mn2 + mx2) - root.z;
            const float s = fmaf(w0, w0, fmaf(w1, w1, w2 * w2)) / fmaf(d0, d0, fmaf(d1, d1, d2 * d2));
            // two buckets an octave from 2^-20 to 2^12, as order_bucket takes two octaves
            const float q = fminf(fmaxf(s, 9.5367431640625e-7f), 4096.f);
            ratio[g] = __int_as_float(((__float_as_int(q) - 0x35800000) >> 22) << 24);
        }
    }
}

// ---- masked group walk: the reference's rule, per body, with shared traversal ----
// The default method (no PT_BH_GROUP). One warp walks for 64 key-adjacent
// bodies (two per lane; fewer in small calls) like bh_walk_group, but every stack range carries the
// masks of the bodies that still descend into it, and every list entry the masks of
// the bodies that accept it: each body's accepted set is exactly the reference's
// (sequential.rs:470-505: skip a node at d^2 == 0, open a cell when theta^2 d^2 <
// w^2, else accept). A list entry is evaluated for every body and weighted by the
// body's mask bit. Sums run in list order instead of the reference's visit order
// (rounding-level differences).
// One warp (group) per CTA, so that a finished group's slot is refilled at once (walk at N =
// 4M, 4 / 2 / 1 warps per CTA: theta 0.5 14.57 / 14.46 / 14.26 ms, with quadrupoles 22.79 /
// 22.60 / 22.64, theta 0.3 40.06 / 40.36 / 39.87).
// Stack ranges per warp of the masked walk: 320 fit 20 one-warp CTAs per SM in shared
// memory (384: 18). Walk at N = 4M, 384 -> 320: theta 0.5 13.96 -> 13.81 ms, with
// quadrupoles 22.51 -> 22.38, theta 0.3 39.40 -> 39.03 (12 of 65536 warps then run out
// of stack and take the per-body cursor walk: the same accepted sets).
#ifndef PT_MW_STACK
#define PT_MW_STACK 320
#endif
constexpr int MW_STACK = PT_MW_STACK;
// List capacities of the masked walk (88 cells / 112 bodies, for 21 warps per SM, and
// 17 with quadrupoles, measured 0.3-0.6 % slower).
#ifndef PT_MW_CELLS
#define PT_MW_CELLS 96
#endif
#ifndef PT_MW_BODIES
#define PT_MW_BODIES 128
#endif
// A warp walks for 32 TPL / LPB bodies: TPL bodies to a lane, mask word i covering bodies g0 +
// 32 i + lane, or, in small calls, one body to LPB lanes, which carry the same mask bits,
// vote alike and split the list entries among them.

// Entry pair (packed lo/hi) for one body, weighted by the body's bits of the two
// entries' masks (qm = the pair's mask words for this body's word).
template <int NF>
__device__ __forceinline__ void eval_pair_masked(const f2 *q, f2 qm, f2 px, f2 py, f2 pz, f2 e2, f2 &ax, f2 &ay,
                                                 f2 &az) {
    const unsigned mine = 1u << (threadIdx.x & 31);
    float m0, m1;
    upk2(qm, m0, m1);
    const f2 dx = sub2(q[0], px);
    const f2 dy = sub2(q[1], py);
    const f2 dz = sub2(q[2], pz);
    const f2 r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, e2)));
    float r0, r1;
    upk2(r2, r0, r1);
    float i0 = rsqrt_ftz(r0), i1 = rsqrt_ftz(r1);
    // a body outside the entry's mask adds exactly 0 (a body at r = 0 is never in it); a select
    // on the mask word, where a factor made of the bit took a conversion on the MUFU pipe
    i0 = (__float_as_uint(m0) & mine) ? i0 : 0.0f;
    i1 = (__float_as_uint(m1) & mine) ? i1 : 0.0f;
    const f2 inv = pk2(i0, i1);
    const f2 inv2 = mul2(inv, inv);
    const f2 sc = mul2(mul2(q[3], inv), inv2);
    if constexpr (NF == 10) {
        const f2 ux = fma2(q[4], dx, fma2(q[5], dy, mul2(q[6], dz)));
        const f2 uy = fma2(q[5], dx, fma2(q[7], dy, mul2(q[8], dz)));
        const f2 uz = fma2(q[6], dx, fma2(q[8], dy, mul2(q[9], dz)));
        const f2 c = fma2(dx, ux, fma2(dy, uy, mul2(dz, uz)));
        const f2 inv5 = mul2(mul2(inv2, inv2), inv);
        const f2 k = mul2(c, mul2(inv2, pk2(-2.5f, -2.5f)));
        const f2 s2 = fma2(inv5, k, sc);
        ax = fma2(dx, s2, fma2(inv5, ux, ax));
        ay = fma2(dy, s2, fma2(inv5, uy, ay));
        az = fma2(dz, s2, fma2(inv5, uz, az));
    } else {
        ax = fma2(dx, sc, ax);
        ay = fma2(dy, sc, ay);
        az = fma2(dz, sc, az);
    }
}

// Lists hold NF fields, then TPL mask words per entry.
template <int NF, int TPL, int LPB, int CAP>
__device__ __forceinline__ void eval_list_masked(IList<NF + TPL, CAP> &Lst, int cnt, const f2 (&px)[TPL],
                                                 const f2 (&py)[TPL], const f2 (&pz)[TPL], f2 e2,
                                                 RegSums<TPL> &acc) {
    const int lane = threadIdx.x & 31;
    f2 ax[TPL], ay[TPL], az[TPL];
#pragma unroll
    for (int i = 0; i < TPL; ++i) ax[i] = ay[i] = az[i] = pk2(0.f, 0.f);
    __syncwarp();
    const int end = (cnt + 2 * LPB - 1) / (2 * LPB) * (2 * LPB);
    if (end != cnt) {  // pad: far away, massless, empty masks
        for (int x = lane; x < (NF + TPL) * (end - cnt); x += 32)
            Lst.put(x % (NF + TPL), cnt + x / (NF + TPL), (x % (NF + TPL) < 3) ? 1e30f : 0.0f);
        __syncwarp();
    }
#pragma unroll 2
    for (int e = 2 * (lane % LPB); e < end; e += 2 * LPB) {
        f2 q[NF + TPL];
        Lst.pair(e, q);
#pragma unroll
        for (int i = 0; i < TPL; ++i)
            eval_pair_masked<NF>(q, q[NF + i], px[i], py[i], pz[i], e2, ax[i], ay[i], az[i]);
    }
#pragma unroll
    for (int i = 0; i < TPL; ++i) acc.fold(i, ax[i], ay[i], az[i]);
    __syncwarp();
}

// Shared memory of a warp that walks for `BODIES` bodies (64 to 2).
template <bool QUAD, int BODIES>
struct Masked {
    static constexpr int TPL = BODIES == 64 ? 2 : 1, LPB = BODIES >= 32 ? 1 : 32 / BODIES;
    static_assert(32 * TPL / LPB == BODIES && LPB <= 16, "64 to 2 bodies");
    static constexpr int NFC = QUAD ? 10 : 4;
    // (smaller lists with one body per lane, whose fewer registers leave room for more warps)
    static constexpr int CELLS = TPL == 1 ? 64 : PT_MW_CELLS, LEAVES = TPL == 1 ? 96 : PT_MW_BODIES;
    static constexpr int PAD = LPB > 1 ? 2 * LPB - 2 : 0;
    using CellList = IList<NFC + TPL, CELLS + PAD>;  // + the masks of the accepting bodies
    using BodyList = IList<4 + TPL, LEAVES + PAD>;
    // (first, end, mask word 0, mask word 1); one more: a pop from a full stack votes on two nodes
    int4 stack[MW_STACK + 1];
    alignas(16) CellList cells;
    alignas(16) BodyList leaves;
};

// The walk for the bodies from g0 on.
template <bool QUAD, int NB>
__device__ __forceinline__ void
    walk_masked(Masked<QUAD, NB> &Sh, int g0, const float4 *__restrict__ tbody, const uint32_t *__restrict__ tidx,
                int n_aff, const float4 *__restrict__ nodeA, const int4 *__restrict__ nodeB,
                const float4 *__restrict__ nodeQ, const float4 *__restrict__ sbody,
                const int *__restrict__ counters, float th2, float eps2, float *__restrict__ out,
                unsigned long long *__restrict__ stats) {
    using M = Masked<QUAD, NB>;
    constexpr int NFC = M::NFC, TPL = M::TPL, LPB = M::LPB, CELLS = M::CELLS, BODIES = M::LEAVES;
    int4 *stack = Sh.stack;
    auto &Lc = Sh.cells;
    auto &Lb = Sh.leaves;
    const int lane = threadIdx.x;
    float4 p[TPL];
    bool valid[TPL];
    unsigned vmask[TPL];
#pragma unroll
    for (int i = 0; i < TPL; ++i) {
        const int t = g0 + 32 * i + lane / LPB;
        valid[i] = t < n_aff;
        p[i] = tbody[valid[i] ? t : g0];
        vmask[i] = __ballot_sync(0xffffffffu, valid[i]);
    }
    const unsigned lt = (1u << lane) - 1u;
    const int T = counters[1];
    const float4 pl = p[TPL - 1];
    float mn0 = fminf(p[0].x, pl.x), mn1 = fminf(p[0].y, pl.y), mn2 = fminf(p[0].z, pl.z);
    float mx0 = fmaxf(p[0].x, pl.x), mx1 = fmaxf(p[0].y, pl.y), mx2 = fmaxf(p[0].z, pl.z);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn0 = fminf(mn0, __shfl_xor_sync(0xffffffffu, mn0, o));
        mn1 = fminf(mn1, __shfl_xor_sync(0xffffffffu, mn1, o));
        mn2 = fminf(mn2, __shfl_xor_sync(0xffffffffu, mn2, o));
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
        mx2 = fmaxf(mx2, __shfl_xor_sync(0xffffffffu, mx2, o));
    }
    const f2 e2 = pk2(eps2, eps2);
    f2 px[TPL], py[TPL], pz[TPL];
    RegSums<TPL> bsum;  // the bodies' compensated sums over the evaluated lists
    bsum.zero();
#pragma unroll
    for (int i = 0; i < TPL; ++i) {
        px[i] = pk2(p[i].x, p[i].x);
        py[i] = pk2(p[i].y, p[i].y);
        pz[i] = pk2(p[i].z, p[i].z);
    }
    if (lane == 0) stack[0] = make_int4(0, T, int(vmask[0]), TPL == 2 ? int(vmask[TPL - 1]) : 0);
    __syncwarp();
    int S = 1, Nc = 0, Nb = 0;
    unsigned long long acc_pairs = 0, cell_pairs = 0, visit_pairs = 0;
    bool failed = false;
    while (S > 0) {
        const int k = min(min(32, S), max(1, (MW_STACK - S) / 2));
        const bool first = lane < k;
        int4 r = first ? stack[S - 1 - lane] : make_int4(0, 0, 0, 0);
        __syncwarp();
        S -= k;
        int node = r.x;
        float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
        int4 B = make_int4(0, 0, 0, 0);
        if (first) {
            A = __ldg(nodeA + node);
            B = __ldg(nodeB + node);
        }
        // A pop of fewer than 32 ranges leaves lanes idle: lane k + i then also takes
        // the second node of range i (its first node's skip pointer) with the range's
        // masks, and the rest of the range passes to it. Each range still pushes at
        // most three ranges, within the room k was sized for (2 per popped range).
        bool second = false;
        if (k < 32) {
            const int src = lane >= k ? lane - k : lane;
            const int nxt = __shfl_sync(0xffffffffu, B.y, src);
            const int end = __shfl_sync(0xffffffffu, r.y, src);
            const int m0 = __shfl_sync(0xffffffffu, r.z, src), m1 = __shfl_sync(0xffffffffu, r.w, src);
            if (lane >= k && src < k && nxt < end) {
                second = true;
                node = nxt;
                r = make_int4(nxt, end, m0, m1);
                A = __ldg(nodeA + node);
                B = __ldg(nodeB + node);
            }
        }
        const unsigned msecond = __ballot_sync(0xffffffffu, second);
        // its rest went to lane + k
        const bool handed = first && lane + k < 32 && ((msecond >> (lane + k)) & 1u);
        const bool have = first || second;
        const unsigned mk0 = unsigned(r.z), mk1 = unsigned(r.w);
        visit_pairs += __popc(mk0) + __popc(mk1);
        // Per node: which of its bodies open it and which accept it. The bodies' box
        // settles most nodes; a node whose centre of mass lies inside the box (a body
        // may coincide with it: skipped) or whose rule differs across the box is
        // voted on, each lane testing its own bodies.
        const bool cell = B.z < 0;
        const float w = cell ? __int_as_float(B.x) : 0.f;
        unsigned op0 = 0, op1 = 0, ac0 = 0, ac1 = 0;
        bool need = false;
        if (have && (mk0 | mk1)) {
            const float e0 = fmaxf(fmaxf(mn0 - A.x, A.x - mx0), 0.f);
            const float e1 = fmaxf(fmaxf(mn1 - A.y, A.y - mx1), 0.f);
            const float e2b = fmaxf(fmaxf(mn2 - A.z, A.z - mx2), 0.f);
            const float db2 = fmaf(e0, e0, fmaf(e1, e1, e2b * e2b));
            const bool inside = !(db2 > 0.0f);
            if (inside) {
                need = true;
            } else if (!cell || !(th2 * db2 < w * w)) {  // every body accepts
                ac0 = mk0;
                ac1 = mk1;
            } else {
                const float f0 = fmaxf(A.x - mn0, mx0 - A.x);
                const float f1 = fmaxf(A.y - mn1, mx1 - A.y);
                const float f2b = fmaxf(A.z - mn2, mx2 - A.z);
                if (th2 * fmaf(f0, f0, fmaf(f1, f1, f2b * f2b)) < w * w) {  // every body opens
                    op0 = mk0;
                    op1 = mk1;
                } else {
                    need = true;
                }
            }
        }
        // The voted nodes are read back from the stack's free slots (the popped ranges' and
        // the room k left above them, for 2 k nodes at most). A leaf's width is
        // 0: no body opens it.
        unsigned vm = __ballot_sync(0xffffffffu, need);
        if (need) stack[S + __popc(vm & lt)] = make_int4(__float_as_int(A.x), __float_as_int(A.y), __float_as_int(A.z),
                                                         __float_as_int(w * w));
        __syncwarp();
        for (int v = S; vm; ++v) {
            const int j = __ffs(vm) - 1;
            vm &= vm - 1;
            const int4 c = stack[v];
            const float cx = __int_as_float(c.x), cy = __int_as_float(c.y), cz = __int_as_float(c.z),
                        cw2 = __int_as_float(c.w);
            const unsigned mj0 = __shfl_sync(0xffffffffu, mk0, j);
            const f2 dx = sub2(pk2(cx, cx), pk2(p[0].x, pl.x));
            const f2 dy = sub2(pk2(cy, cy), pk2(p[0].y, pl.y));
            const f2 dz = sub2(pk2(cz, cz), pk2(p[0].z, pl.z));
            float d0, d1;
            upk2(fma2(dx, dx, fma2(dy, dy, mul2(dz, dz))), d0, d1);
            const unsigned om0 = mj0 & __ballot_sync(0xffffffffu, d0 > 0.0f && th2 * d0 < cw2);
            const unsigned am0 = mj0 & ~om0 & __ballot_sync(0xffffffffu, d0 > 0.0f);
            unsigned om1 = 0u, am1 = 0u;
            if (TPL == 2) {
                const unsigned mj1 = __shfl_sync(0xffffffffu, mk1, j);
                om1 = mj1 & __ballot_sync(0xffffffffu, d1 > 0.0f && th2 * d1 < cw2);
                am1 = mj1 & ~om1 & __ballot_sync(0xffffffffu, d1 > 0.0f);
            }
            if (lane == j) {
                op0 = om0;
                op1 = om1;
                ac0 = am0;
                ac1 = am1;
            }
        }
        __syncwarp();
        // push: later siblings share the parent's masks; children get the opening bodies
        const bool rest = have && !handed && (mk0 | mk1) && B.y < r.y;
        const bool opn = (op0 | op1) != 0u;
        const unsigned mrest = __ballot_sync(0xffffffffu, rest), mopen = __ballot_sync(0xffffffffu, opn);
        const int total = __popc(mrest) + __popc(mopen);
        if (S + total > MW_STACK) {
            failed = true;
            break;
        }
        int slot = S + __popc(mrest & lt) + __popc(mopen & lt);
        if (rest) stack[slot++] = make_int4(B.y, r.y, int(mk0), int(mk1));
        if (opn) stack[slot++] = make_int4(node + 1, B.y, int(op0), int(op1));
        S += total;
        const int na = __popc(ac0) + __popc(ac1);
        acc_pairs += na;
        const bool accd = na != 0;
        const bool bucket = accd && !cell && B.w > 1;
        const bool cellacc = accd && cell;
        const bool bodyacc = accd && !cell && B.w == 1;
        if (cellacc) cell_pairs += na;
        const unsigned mc = __ballot_sync(0xffffffffu, cellacc);
        const int nc1 = __popc(mc);
        if (Nc + nc1 > CELLS) {
            eval_list_masked<NFC, TPL, LPB>(Lc, Nc, px, py, pz, e2, bsum);
            Nc = 0;
        }
        if (cellacc) {
            const int e = Nc + __popc(mc & lt);
            Lc.put(0, e, A.x);
            Lc.put(1, e, A.y);
            Lc.put(2, e, A.z);
            Lc.put(3, e, A.w);
            if constexpr (QUAD) {  // negated: the list evaluation's form
                const float4 q0 = __ldg(nodeQ + 2 * node);
                const float4 q1 = __ldg(nodeQ + 2 * node + 1);
                Lc.put(4, e, -q0.x);
                Lc.put(5, e, -q0.y);
                Lc.put(6, e, -q0.z);
                Lc.put(7, e, -q0.w);
                Lc.put(8, e, -q1.x);
                Lc.put(9, e, -q1.y);
            }
            Lc.put(NFC, e, __uint_as_float(ac0));
            if (TPL == 2) Lc.put(NFC + 1, e, __uint_as_float(ac1));
        }
        Nc += nc1;
        const unsigned mb1 = __ballot_sync(0xffffffffu, bodyacc);
        const int nb1 = __popc(mb1);
        if (Nb + nb1 > BODIES) {
            eval_list_masked<4, TPL, LPB>(Lb, Nb, px, py, pz, e2, bsum);
            Nb = 0;
        }
        if (bodyacc) {
            const int e = Nb + __popc(mb1 & lt);
            Lb.put(0, e, A.x);
            Lb.put(1, e, A.y);
            Lb.put(2, e, A.z);
            Lb.put(3, e, A.w);
            Lb.put(4, e, __uint_as_float(ac0));
            if (TPL == 2) Lb.put(5, e, __uint_as_float(ac1));
        }
        Nb += nb1;
        unsigned mbk = __ballot_sync(0xffffffffu, bucket);
        while (mbk) {  // leaves holding several bodies: one entry per body, the leaf's masks
            const int src = __ffs(mbk) - 1;
            mbk &= mbk - 1;
            const int f = __shfl_sync(0xffffffffu, B.z, src);
            const int c = __shfl_sync(0xffffffffu, B.w, src);
            const unsigned b0 = __shfl_sync(0xffffffffu, ac0, src), b1 = __shfl_sync(0xffffffffu, ac1, src);
            for (int base = 0; base < c; base += 32) {
                const int n = min(32, c - base);
                if (Nb + n > BODIES) {
                    eval_list_masked<4, TPL, LPB>(Lb, Nb, px, py, pz, e2, bsum);
                    Nb = 0;
                }
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane < n) q = __ldg(sbody + f + base + lane);
                unsigned q0 = b0, q1 = b1;
                // A body does not meet itself in the leaf: only one in the group's box can be at
                // a body of the group. (Voting on every leaf body: 1M bodies, all but 20 within
                // 1e-5 of the box, 14.5 ms a walk, and 8.9 like this.) With softening it may: it
                // adds 0 times a factor that is finite for eps >= 1e-6 and masses up to 1e20. (With
                // the votes and without, us a walk: 524288 bodies in two knots 1e-5 of the box wide
                // 1014 / 968, 1M 1985 / 1875, 1M in knots of some 200 718 / 644.)
                const float e0 = fmaxf(fmaxf(mn0 - q.x, q.x - mx0), 0.0f);
                const float e1 = fmaxf(fmaxf(mn1 - q.y, q.y - mx1), 0.0f);
                const float e2b = fmaxf(fmaxf(mn2 - q.z, q.z - mx2), 0.0f);
                const bool in_box = lane < n && !(fmaf(e0, e0, fmaf(e1, e1, e2b * e2b)) > 0.0f);
                unsigned vote = eps2 >= 1e-12f ? 0u : __ballot_sync(0xffffffffu, in_box);
                while (vote) {
                    const int j = __ffs(vote) - 1;
                    vote &= vote - 1;
                    const float cx = __shfl_sync(0xffffffffu, q.x, j), cy = __shfl_sync(0xffffffffu, q.y, j),
                                cz = __shfl_sync(0xffffffffu, q.z, j);
                    const float x0 = cx - p[0].x, y0 = cy - p[0].y, z0 = cz - p[0].z;
                    const float x1 = cx - pl.x, y1 = cy - pl.y, z1 = cz - pl.z;
                    const unsigned m0 = __ballot_sync(0xffffffffu, fmaf(x0, x0, fmaf(y0, y0, z0 * z0)) > 0.f);
                    const unsigned m1 = __ballot_sync(0xffffffffu, fmaf(x1, x1, fmaf(y1, y1, z1 * z1)) > 0.f);
                    if (lane == j) q0 = b0 & m0, q1 = b1 & m1;
                }
                if (lane < n) {
                    Lb.put(0, Nb + lane, q.x);
                    Lb.put(1, Nb + lane, q.y);
                    Lb.put(2, Nb + lane, q.z);
                    Lb.put(3, Nb + lane, q.w);
                    Lb.put(4, Nb + lane, __uint_as_float(q0));
                    if (TPL == 2) Lb.put(5, Nb + lane, __uint_as_float(q1));
                }
                Nb += n;
            }
        }
        __syncwarp();
    }
    eval_list_masked<NFC, TPL, LPB>(Lc, Nc, px, py, pz, e2, bsum);
    eval_list_masked<4, TPL, LPB>(Lb, Nb, px, py, pz, e2, bsum);
    float rx[TPL], ry[TPL], rz[TPL];
#pragma unroll
    for (int i = 0; i < TPL; ++i) {
        if (LPB > 1) bsum.template gather<LPB>(i);
        bsum.total(i, rx[i], ry[i], rz[i]);
    }
    if (failed) {  // the stack ran out: the per-body cursor walk instead (warp-uniform)
        unsigned na = 0, nv = 0, nc = 0;
#pragma unroll
        for (int i = 0; i < TPL; ++i) {
            rx[i] = ry[i] = rz[i] = 0.f;
            lane_walk<QUAD>(p[i], valid[i], T, nodeA, nodeB, nodeQ, sbody, th2, eps2, rx[i], ry[i], rz[i], na, nv,
                            nc);
        }
        acc_pairs = na;
        cell_pairs = nc;
        visit_pairs = nv;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {  // per-lane counts -> the warp's
        acc_pairs += __shfl_xor_sync(0xffffffffu, acc_pairs, o);
        cell_pairs += __shfl_xor_sync(0xffffffffu, cell_pairs, o);
        visit_pairs += __shfl_xor_sync(0xffffffffu, visit_pairs, o);
    }
#pragma unroll
    for (int i = 0; i < TPL; ++i)
        if (valid[i]) {
            if (LPB > 1 && lane % LPB != 0) continue;
            const uint32_t o = tidx[g0 + 32 * i + lane / LPB];
            out[3 * size_t(o) + 0] = rx[i];
            out[3 * size_t(o) + 1] = ry[i];
            out[3 * size_t(o) + 2] = rz[i];
        }
    if (stats && lane == 0) {
        atomicAdd(stats + 0, acc_pairs / LPB);
        atomicAdd(stats + 1, visit_pairs / LPB);
        atomicAdd(stats + 2, 1ull);
        atomicAdd(stats + 5, cell_pairs / LPB);
        if (failed) atomicAdd(stats + 6, 1ull);
    }
}

// BIG bodies a warp for the first big_groups blocks, SMALL for the rest: the last warps to
// start are short, so that the chip does not idle for the length of a whole warp's walk at
// the end.
template <bool QUAD, int BIG, int SMALL>
__global__ void __launch_bounds__(32)
    bh_walk_masked(int big_groups, const int *__restrict__ order, const float4 *__restrict__ tbody, const uint32_t *__restrict__ tidx, int n_aff,
                   const float4 *__restrict__ nodeA, const int4 *__restrict__ nodeB,
                   const float4 *__restrict__ nodeQ, const float4 *__restrict__ sbody,
                   const int *__restrict__ counters, float th2, float eps2, float *__restrict__ out,
                   unsigned long long *__restrict__ stats) {
    after_previous();
    __shared__ union {
        __align__(16) unsigned char raw[1];
        Masked<QUAD, BIG> big;
        Masked<QUAD, SMALL> small;
    } Sh;
    const int b = blockIdx.x;
    if (BIG == SMALL || b < big_groups) {
        const int g0 = (order ? order[b] : b) * BIG;
        if (unsigned(g0) < unsigned(n_aff))
            walk_masked<QUAD, BIG>(Sh.big, g0, tbody, tidx, n_aff, nodeA, nodeB, nodeQ, sbody, counters, th2, eps2,
                                   out, stats);
    } else {
        const int half = b - big_groups, whole = big_groups + (half >> 1);
        const int g0 = (order ? order[whole] : whole) * BIG + (half & 1) * SMALL;
        if (unsigned(g0) < unsigned(n_aff))
            walk_masked<QUAD, SMALL>(Sh.small, g0, tbody, tidx, n_aff, nodeA, nodeB, nodeQ, sbody, counters, th2, eps2,
                                     out, stats);
    }
}

// ---- the reference rule over DVec3 bodies (f64 method) -------------------------
// As bh_walk_masked with one body per lane, in double: node data, widths and the
// per-pair kernel (impl_acceleration_cpu_scalar!(DVec3, f64): d * (m / (n_s sqrt n_s)))
// are f64; accepted sets per body are the reference's. Monopole only, as the reference.
constexpr int W64_STACK = 384;

// m / (n_s sqrt(n_s)) without the FP64 square root and divide, which cost more than the rest
// of the pair on a pipe that does two lane-operations a cycle: an FP32 reciprocal root y of
// n_s, then the binomial series of n_s^(-3/2) = y^3 (1 - e)^(-3/2) about e = 1 - n_s y^2,
// y^3 (1 + 3/2 e + 15/8 e^2). y has 24 bits, so y^2 is exact; |e| < 7e-7, so the series'
// remainder is below 2^-60. The rounding errors left are those of the four operations that
// the square root, product, divide form has too: against 80-bit values over 2e6 random pairs
// 0.734 units of 2^-53 rms, where sqrt and divide give 0.735. Conversions and compares run on
// the integer pipe, by the bits: on the FP64 pipe they were 5 of a pair's 22 operations (whole
// host call at N = 50021, theta 0.5, 4.86 -> 3.91 ms, 10000 at 0.6 0.79 -> 0.71).
__device__ __forceinline__ double inv_cube64(double ns, double m) {
    const unsigned hi = __double2hiint(ns), lo = __double2loint(ns);
    // 2^-119 <= ns < 2^119 by its exponent; outside FP32's range:
    if (hi - ((1023u - 119u) << 20) >= (238u << 20)) return __ddiv_rn(m, __dmul_rn(ns, __dsqrt_rn(ns)));
    // ns to FP32 (a half rounded up) and y back by their bits: the exponents differ by 896
    const float nf = __uint_as_float(__funnelshift_l(lo, hi, 3) - (896u << 23) + ((lo >> 28) & 1u));
    const unsigned yb = __float_as_uint(rsqrt_ftz(nf));
    const double y = __hiloint2double((yb >> 3) + (896u << 20), yb << 29);
    const double y2 = y * y;
    const double e = fma(-ns, y2, 1.0);
    const double my3 = m * (y2 * y);
    return fma(my3, e * fma(1.875, e, 1.5), my3);
}

__device__ __forceinline__ void pair64(double px, double py, double pz, double cx, double cy, double cz, double m,
                                       double eps2, double &ax, double &ay, double &az) {
    const double dx = cx - px, dy = cy - py, dz = cz - pz;
    const double n = fma(dx, dx, fma(dy, dy, dz * dz));
    if (__double_as_longlong(n) == 0) return;  // checked: d itself, which is zero (n is not -0)
    const double s = inv_cube64(n + eps2, m);
    ax = fma(dx, s, ax);
    ay = fma(dy, s, ay);
    az = fma(dz, s, az);
}

struct List64 {
    static constexpr int CAP = 128;
    double f[4][CAP];
    unsigned mask[CAP];
};

// Transposes a 32 x 32 bit matrix held as one row per lane: afterwards bit r of lane c is
// what bit c of lane r was.
__device__ __forceinline__ unsigned transpose32(unsigned x) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
        const unsigned m = 0xffffffffu / ((1u << j) + 1u);  // the columns c with (c & j) == 0
        const unsigned y = __shfl_xor_sync(0xffffffffu, x, j);
        x = lane & j ? (x & ~m) | ((y & ~m) >> j) : (x & m) | ((y & m) << j);
    }
    return x;
}

// Each lane evaluates its own body's accepted entries of the list, in list order. The pair
// costs 17 lane-operations of an FP64 pipe that does two a cycle, so a lane whose body
// does not accept an entry goes on to its own next entry instead of waiting for the lanes
// whose bodies do: the list takes as many rounds as the body with the most accepted entries
// has, not as many as it holds. (Entry by entry with the mask's lanes on, N = 50021 at theta
// 0.5 took 11.9 ms through the host API, and 8.3 ms like this.) With LPB lanes to a body,
// lane % LPB takes the entries e with e % LPB equal to it.
template <int LPB>
__device__ __forceinline__ void eval_list64(const List64 &Lst, int cnt, double px, double py, double pz, double eps2,
                                            double &ax, double &ay, double &az) {
    const int lane = threadIdx.x & 31;
    constexpr int WORDS = List64::CAP / 32;
    constexpr unsigned share = 0xffffffffu / ((1u << LPB) - 1u);  // every LPB-th bit
    __syncwarp();
    unsigned w[WORDS];  // bit e of word k: this lane's body accepts entry 32 k + e
#pragma unroll
    for (int k = 0; k < WORDS; ++k)
        w[k] = transpose32(32 * k + lane < cnt ? Lst.mask[32 * k + lane] : 0u) & (share << (lane % LPB));
    for (;;) {
        int e = -1;
#pragma unroll
        for (int k = 0; k < WORDS; ++k)
            if (e < 0 && w[k]) {
                e = 32 * k + __ffs(w[k]) - 1;
                w[k] &= w[k] - 1;
            }
        if (__all_sync(0xffffffffu, e < 0)) break;
        if (e >= 0) pair64(px, py, pz, Lst.f[0][e], Lst.f[1][e], Lst.f[2][e], Lst.f[3][e], eps2, ax, ay, az);
    }
    __syncwarp();
}

// One warp per CTA, so that a finished warp's slot is refilled at once. LPB lanes share a
// body (32 / LPB bodies per warp): they vote alike and split its accepted entries.
template <int LPB>
__global__ void __launch_bounds__(32)
    bh_walk64(const double4_32a *__restrict__ tbody, const uint32_t *__restrict__ tidx, int n_aff,
              const double4_32a *__restrict__ nodeA, const int4 *__restrict__ nodeB,
              const double4_32a *__restrict__ nodeG, const double4_32a *__restrict__ sbody,
              const int *__restrict__ counters, double th2, double eps2, double *__restrict__ out,
              unsigned long long *__restrict__ stats, int *__restrict__ err) {
    after_previous();
    __shared__ int4 stack[W64_STACK];
    __shared__ List64 Lst;
    __shared__ float4 vote[64];
    const int lane = threadIdx.x;
    const int group = blockIdx.x;
    constexpr int BODIES = 32 / LPB;
    if (group * BODIES >= n_aff) return;
    const int t = group * BODIES + lane / LPB;
    const bool valid = t < n_aff;
    const double4_32a p = tbody[valid ? t : group * BODIES];
    const unsigned lt = (1u << lane) - 1u;
    const unsigned valid_mask = __ballot_sync(0xffffffffu, valid);
    const int T = counters[1];
    double mn0 = p.x, mn1 = p.y, mn2 = p.z, mx0 = p.x, mx1 = p.y, mx2 = p.z;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn0 = fmin(mn0, __shfl_xor_sync(0xffffffffu, mn0, o));
        mn1 = fmin(mn1, __shfl_xor_sync(0xffffffffu, mn1, o));
        mn2 = fmin(mn2, __shfl_xor_sync(0xffffffffu, mn2, o));
        mx0 = fmax(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
        mx1 = fmax(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
        mx2 = fmax(mx2, __shfl_xor_sync(0xffffffffu, mx2, o));
    }
    // for the decisions: this lane's body and the box's half widths about its centre, in FP32
    const double g0 = 0.5 * (mn0 + mx0), g1 = 0.5 * (mn1 + mx1), g2 = 0.5 * (mn2 + mx2);
    const float px = float(p.x - g0), py = float(p.y - g1), pz = float(p.z - g2);
    float h0 = fabsf(px), h1 = fabsf(py), h2 = fabsf(pz);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        h0 = fmaxf(h0, __shfl_xor_sync(0xffffffffu, h0, o));
        h1 = fmaxf(h1, __shfl_xor_sync(0xffffffffu, h1, o));
        h2 = fmaxf(h2, __shfl_xor_sync(0xffffffffu, h2, o));
    }
    const float rg2 = fmaf(h0, h0, fmaf(h1, h1, h2 * h2));
    const float th2f = float(th2);
    const bool th2_ok = th2 == 0.0 || th2f > 1e-30f;
    double ax = 0.0, ay = 0.0, az = 0.0;
    if (lane == 0) stack[0] = make_int4(0, T, int(valid_mask), 0);
    __syncwarp();
    int S = 1, Nl = 0;
    unsigned long long acc_pairs = 0, visit_pairs = 0;
    bool failed = false;
    while (S > 0) {
        const int k = min(min(32, S), max(1, (W64_STACK - S) / 2));
        const bool have = lane < k;
        const int4 r = have ? stack[S - 1 - lane] : make_int4(0, 0, 0, 0);
        __syncwarp();
        S -= k;
        const int node = r.x;
        const unsigned mask = unsigned(r.z);
        double4_32a A;
        A.x = A.y = A.z = A.w = 0.0;
        int4 B = make_int4(0, 0, 0, 0);
        double w = 0.0;
        if (have) {
            A = nodeA[node];
            B = __ldg(nodeB + node);
            if (B.z < 0) w = nodeG[node].w;
        }
        visit_pairs += __popc(mask);
        const bool cell = B.z < 0;
        unsigned open_m = 0, acc_m = 0;
        bool need = false;
        // The box, then each node that it leaves open the bodies, decide in FP32. With c and b
        // the node and a body (or a point of the box) about the box's centre, rounded to 24 bits
        // each, |c - b|^2 is off by less than 2^-20 (|c|^2 + |b|^2), its product with theta^2 by
        // 2^-22 of the same more and w^2 by 2^-22 of itself (and by 1e-37 where they are
        // denormal). Within twice that of the decision (or of zero distance, or where a product
        // could overflow) the bodies decide in FP64, so that the accepted sets stay the
        // reference's. A vote in FP64 keeps that pipe, two lane-operations a cycle, for a
        // quarter of what a pair does: whole host call at N = 50021, theta 0.5, 6.15 -> 5.23 ms,
        // 10000 at 0.6 1.20 -> 0.93; the box in FP32 too: 4.86 and 0.79.
        if (have && mask) {
            const float cx = float(A.x - g0), cy = float(A.y - g1), cz = float(A.z - g2), wf = float(w);
            const float c2 = fmaf(cx, cx, fmaf(cy, cy, cz * cz)) + rg2, lim = wf * wf;
            const bool ok = th2_ok && c2 < 1e37f && lim < 1e37f;
            const float zero = ok ? fmaf(c2, 0x1p-19f, 1e-36f) : INFINITY;
            const float line = fmaf(fmaf(th2f, c2, lim), 0x1p-19f, fmaf(th2f, 1e-36f, 1e-36f));
            const float x0 = fabsf(cx), x1 = fabsf(cy), x2 = fabsf(cz);
            const float n0 = fmaxf(x0 - h0, 0.f), n1 = fmaxf(x1 - h1, 0.f), n2 = fmaxf(x2 - h2, 0.f);
            const float near2 = fmaf(n0, n0, fmaf(n1, n1, n2 * n2));
            const float far2 = fmaf(x0 + h0, x0 + h0, fmaf(x1 + h1, x1 + h1, (x2 + h2) * (x2 + h2)));
            need = true;
            if (near2 > zero) {
                if (!cell || fmaf(th2f, near2, -lim) > line) {
                    acc_m = mask;
                    need = false;
                } else if (fmaf(th2f, far2, -lim) < -line) {
                    open_m = mask;
                    need = false;
                }
            }
            if (need) {
                vote[2 * lane] = make_float4(cx, cy, cz, cell ? lim : -1.f);
                vote[2 * lane + 1] = make_float4(zero, line, __uint_as_float(mask), 0.f);
            }
        }
        unsigned vm = __ballot_sync(0xffffffffu, need);
        __syncwarp();
        while (vm) {
            const int j = __ffs(vm) - 1;
            vm &= vm - 1;
            const float4 v0 = vote[2 * j], v1 = vote[2 * j + 1];
            const float fx = v0.x - px, fy = v0.y - py, fz = v0.z - pz;
            const float f2 = fmaf(fx, fx, fmaf(fy, fy, fz * fz)), side = fmaf(th2f, f2, -v0.w);
            const bool in = (__float_as_uint(v1.z) >> lane) & 1u;
            const bool leaf = v0.w < 0.f;
            if (__all_sync(0xffffffffu, !in || (f2 > v1.x && (leaf || fabsf(side) > v1.y)))) {
                const unsigned om = __ballot_sync(0xffffffffu, in && !leaf && side < 0.f);
                if (lane == j) {
                    open_m = om;
                    acc_m = mask & ~om;
                }
                continue;
            }
            const double cx = __shfl_sync(0xffffffffu, A.x, j), cy = __shfl_sync(0xffffffffu, A.y, j);
            const double cz = __shfl_sync(0xffffffffu, A.z, j), cw = __shfl_sync(0xffffffffu, w, j);
            const unsigned mj = __shfl_sync(0xffffffffu, mask, j);
            const bool cj = __shfl_sync(0xffffffffu, cell, j);
            // the reference's d^2: (com - body) squared, x, y, z in order
            const double dx = __dsub_rn(cx, p.x), dy = __dsub_rn(cy, p.y), dz = __dsub_rn(cz, p.z);
            const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
            const bool mine = (mj >> lane) & 1u;
            const bool o = mine && cj && d2 > 0.0 && __dmul_rn(th2, d2) < __dmul_rn(cw, cw);
            const bool a = mine && !o && d2 > 0.0;
            const unsigned om = __ballot_sync(0xffffffffu, o), am = __ballot_sync(0xffffffffu, a);
            if (lane == j) {
                open_m = om;
                acc_m = am;
            }
        }
        const bool rest = have && mask && B.y < r.y;
        const bool opn = open_m != 0u;
        const unsigned mrest = __ballot_sync(0xffffffffu, rest), mopen = __ballot_sync(0xffffffffu, opn);
        const int total = __popc(mrest) + __popc(mopen);
        int slot = S + __popc(mrest & lt) + __popc(mopen & lt);
        if (slot + int(rest) + int(opn) > W64_STACK) {
            failed = true;
        } else {
            if (rest) stack[slot++] = make_int4(B.y, r.y, int(mask), 0);
            if (opn) stack[slot++] = make_int4(node + 1, B.y, int(open_m), 0);
        }
        if (__any_sync(0xffffffffu, failed)) {
            failed = true;
            break;
        }
        S += total;
        acc_pairs += __popc(acc_m);
        // accepted cells and single bodies: one list entry with the accepting mask;
        // several-body leaves: one entry per body
        const bool single = acc_m != 0u && (cell || B.w == 1);
        const unsigned ms = __ballot_sync(0xffffffffu, single);
        const int ns = __popc(ms);
        if (Nl + ns > List64::CAP) {
            eval_list64<LPB>(Lst, Nl, p.x, p.y, p.z, eps2, ax, ay, az);
            Nl = 0;
        }
        if (single) {
            const int e = Nl + __popc(ms & lt);
            Lst.f[0][e] = A.x;
            Lst.f[1][e] = A.y;
            Lst.f[2][e] = A.z;
            Lst.f[3][e] = A.w;
            Lst.mask[e] = acc_m;
        }
        Nl += ns;
        unsigned mbk = __ballot_sync(0xffffffffu, acc_m != 0u && !cell && B.w > 1);
        while (mbk) {
            const int src = __ffs(mbk) - 1;
            mbk &= mbk - 1;
            const int f = __shfl_sync(0xffffffffu, B.z, src), c = __shfl_sync(0xffffffffu, B.w, src);
            const unsigned bm = __shfl_sync(0xffffffffu, acc_m, src);
            for (int base = 0; base < c; base += 32) {
                const int n = min(32, c - base);
                if (Nl + n > List64::CAP) {
                    eval_list64<LPB>(Lst, Nl, p.x, p.y, p.z, eps2, ax, ay, az);
                    Nl = 0;
                }
                if (lane < n) {
                    const double4_32a q = sbody[f + base + lane];
                    Lst.f[0][Nl + lane] = q.x;
                    Lst.f[1][Nl + lane] = q.y;
                    Lst.f[2][Nl + lane] = q.z;
                    Lst.f[3][Nl + lane] = q.w;
                    Lst.mask[Nl + lane] = bm;
                }
                Nl += n;
            }
        }
        __syncwarp();
    }
    eval_list64<LPB>(Lst, Nl, p.x, p.y, p.z, eps2, ax, ay, az);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        acc_pairs += __shfl_xor_sync(0xffffffffu, acc_pairs, o);
        visit_pairs += __shfl_xor_sync(0xffffffffu, visit_pairs, o);
    }
#pragma unroll
    for (int o = 1; o < LPB; o <<= 1) {  // the body's lanes
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
        az += __shfl_xor_sync(0xffffffffu, az, o);
    }
    if (failed) {  // no stackless fallback in f64: the bodies are NaN and the call fails
        ax = ay = az = __longlong_as_double(0x7ff8000000000000ll);
        if (lane == 0) atomicOr(err, 1);
    }
    if (valid && lane % LPB == 0) {
        const uint32_t o = tidx[t];
        out[3 * size_t(o) + 0] = ax;
        out[3 * size_t(o) + 1] = ay;
        out[3 * size_t(o) + 2] = az;
    }
    if (stats && lane == 0) {
        atomicAdd(stats + 0, acc_pairs / LPB);
        atomicAdd(stats + 1, visit_pairs / LPB);
        atomicAdd(stats + 2, 1ull);
    }
}


using WalkKernel = void (*)(int, const int *, const float4 *, const uint32_t *, int, const float4 *, const int4 *, const float4 *,
                            const float4 *, const int *, float, float, float *, unsigned long long *);
template <bool QUAD>
static WalkKernel masked_kernel_q(int big) {
    return big == 64   ? bh_walk_masked<QUAD, 64, 32>
           : big == 32 ? bh_walk_masked<QUAD, 32, 16>
           : big == 16 ? bh_walk_masked<QUAD, 16, 16>
           : big == 8  ? bh_walk_masked<QUAD, 8, 8>
           : big == 4  ? bh_walk_masked<QUAD, 4, 4>
                       : bh_walk_masked<QUAD, 2, 2>;
}

static GroupKernel group_kernel(bool quad, bool guard, bool learned, bool local, bool rel, int team) {
    if (learned) return group_kernel_q<true, false, false, 1>(quad, guard);
    return team > 1 ? group_kernel_team(quad, guard, local, rel, team) : group_kernel_w<1>(quad, guard, local, rel);
}

// Warps per group of the group walk. A group alone waits on its own loads and votes, so while
// there are few groups several warps share each; once every SM has its 20 warps the team's
// barriers only cost. The lines lie where calls of bodies that are their own targets turn (8 / 4
// warps at 300, 340, 360 and 380 groups 218 / 241, 246 / 255, 265 / 260 and 258 / 252; 4 / 1 at 1563,
// 1672 and 1673 546 / 534, 545 / 592 and 561 / 536; theta 0.6, quadrupoles); far-flung probes would
// take the larger team for longer (8 / 4 at 381 groups 463 / 733, 4 / 1 at 1673 797 / 1241).
// Whole call at 1 / 2 / 4 / 8 / 16 warps, us: 79 groups (5003 probes of a
// 1M tree, theta 0.6, quadrupoles) 2141 / 1459 / 880 / 612 / 523; 157 groups (N = 10000) 329
// / 296 / 260 / 244 / 235; 469 groups (N = 30000) 370 / 345 / 309 / 328 / 392; 1563 groups
// (100003 probes) 1113 / 844 / 753 / 1001 / 1446; 2048 groups (N = 131072, theta 0.6) 678 /
// 686 / 732 / 1003 / 1423.
static int team_of(const pt_ctx *ctx, int groups) {
    const int sms = std::max(1, ctx->sm_count);
    return groups <= 5 * sms / 2 ? 8 : groups <= 11 * sms ? 4 : 1;
}

// Bodies per warp of the masked walk. A warp alone waits on its own loads and votes, so small
// calls want many warps with little to evaluate in each: 2 to 16 bodies, 16 to 2 lanes to a
// body, while these warps are (nearly) all resident at once, 20 per SM (host call at 8 / 4 / 2
// bodies, theta 0.7, us: N = 500 104.5 / 100.9 / 100.6; 3000 143 / 139 / 130; 10000 177 / 169 /
// 183; 20000 205 / 220 / 243). 32 bodies, one to a lane,
// meet fewer nodes than 64 (which share a traversal over more bodies) and end sooner; from
// some 110 warps per SM on the traversals saved count for more. Whole call at 64 / 32 / 16 /
// 8 bodies, us: N = 3000 theta 0.7 271 / 232 / 213 / 200; N = 30000 theta 0.5 552 / 436 / 391
// / 392; N = 65536 theta 0.7 422 / 372 / 379 / 424; N = 262144 theta 0.5 1208 / 1163 / 1389 /
// 1829; N = 524288 theta 0.8 1034 / 1027 / 1229 / 1653; N = 1M theta 0.5 3686 / 3759 / 4796 /
// 6834.
// The last five groups per SM are walked in halves, so that the warps that end last are short
// (whole call without, 5 and 10 per SM, us: N = 131072 theta 0.8 339 / 333 / 347; N = 262144
// theta 0.5 970 / 963 / 979; N = 1M theta 0.5 3192 / 3170 / 3182).
struct MaskedPlan {
    int big, big_groups, small_groups;  // bodies per warp of the first groups (then half of it from 32 on)
};

static MaskedPlan masked_plan(const pt_ctx *ctx, int n_aff) {
    const long long sms = std::max(1, ctx->sm_count);
    MaskedPlan p{};
    p.big = n_aff <= 2 * 20 * sms ? 2 : n_aff <= 4 * 20 * sms ? 4 : n_aff <= 8 * 20 * sms ? 8 : n_aff <= 16 * 27 * sms ? 16 : n_aff <= 32 * 110 * sms ? 32 : 64;
    const int all = (n_aff + p.big - 1) / p.big;
    const int halved = p.big >= 32 ? int(5 * sms) : 0;
    p.big_groups = std::max(0, all - halved);
    p.small_groups = halved ? 2 * (all - p.big_groups) : 0;
    return p;
}

int ensure_counters(pt_ctx *ctx, State &S) {
    if (S.counters.ptr) return PT_OK;
    PT_TRY(ensure_buf(ctx, S.counters, COUNTER_BYTES));
    PT_CUDA(cudaMemsetAsync(S.counters.ptr, 0, COUNTER_BYTES, ctx->stream));
    return PT_OK;
}

// Clears the error word (counters[3]) before a walk of separate targets, as a build does by
// itself; within a leapfrog sequence it collects every step's errors.
int clear_errors(pt_ctx *ctx, State &S) {
    PT_TRY(ensure_counters(ctx, S));
    if (!ctx->keep_errors) PT_CUDA(cudaMemsetAsync(as<int>(S.counters) + 3, 0, sizeof(int), ctx->stream));
    return PT_OK;
}

// The order of the groups whose keys are in S.gscale.
static int place_groups(pt_ctx *ctx, State &S, int groups, const int **order) {
    PT_TRY(ensure_buf(ctx, S.gorder, sizeof(int) * size_t(groups)));
    launch_next(bh_group_order, 1, 32 * ORDER_WARPS, 0, ctx->stream, as<float>(S.gscale), groups, as<int>(S.gorder));
    *order = as<int>(S.gorder);
    return check_launch(ctx, "bh_group_order");
}

// The order of groups of `size` bodies by width over distance, or null up to 24 a SM: 20 or 24
// groups of one warp are resident (N = 50000, 3125 groups of 16, took 237 us without and 240 with
// it, N = 65536, 4096 groups, 266 and 265). Groups walked by teams stay below the line and are not
// ordered, although few teams start at once.
static int order_groups(pt_ctx *ctx, State &S, const float4 *tbody, int n_aff, int size, const int **order) {
    const int sms = std::max(1, ctx->sm_count), groups = (n_aff + size - 1) / size;
    *order = nullptr;
    if (groups <= 24 * sms) return PT_OK;
    PT_TRY(ensure_buf(ctx, S.gscale, sizeof(float) * size_t(groups)));
    launch_next(bh_group_width, std::min(2 * sms, blocks(groups * std::min(32, size))), 256, 0, ctx->stream, tbody,
                n_aff, groups, size, as<float4>(S.nodeA), as<float>(S.gscale));
    PT_TRY(check_launch(ctx, "bh_group_width"));
    return place_groups(ctx, S, groups, order);
}

int run(pt_ctx *ctx, const float4 *d_aff, int n_aff, const float4 *d_src, int n_src, float theta,
               float softening, uint32_t flags, float *d_out) {
    cudaStream_t st = ctx->stream;
    if (n_aff == 0) return PT_OK;
    if (n_src == 0) {
        PT_CUDA(cudaMemsetAsync(d_out, 0, sizeof(float) * 3 * size_t(n_aff), st));
        return PT_OK;
    }
    State *Sp = state(ctx);
    if (!Sp) return set_error(PT_ERR_OOM, "Barnes-Hut state allocation failed");
    State &S = *Sp;
    mark(ctx, 0);
    PT_TRY(build(ctx, S, d_src, n_src));
    const bool same = (d_aff == d_src) && (n_aff == n_src);
    const float4 *tbody;
    const uint32_t *tidx;
    if (same) {
        tbody = as<float4>(S.sbody);
        tidx = as<uint32_t>(S.idx);
    } else {
        PT_TRY(sort_targets(ctx, S, d_aff, n_aff));
        tbody = as<float4>(S.tbody);
        tidx = as<uint32_t>(S.tidx);
    }
    return walk(ctx, S, tbody, tidx, n_aff, theta, softening, flags, d_out);
}

// Lanes that share a body in bh_walk64. A warp of a small call is bound by its own FP64 latency,
// so as many lanes, up to 16, as keep every warp resident at once (20 per SM by registers); once
// the chip is full more lanes repeat the traversal but end more evenly: which of the two counts
// for more at a size depends on theta, by 1 to 4 % about the lines. Whole host call, us, at
// 1 / 2 / 4 / 8 / 16 lanes: N = 2000 theta 0.6 - / - / 445 / 373 / 329, 5000 1206 / 787 / 589 /
// 500 / 462, 10000 1462 / 895 / 712 / 651 / 693, 20000 1806 / 1258 / 1101 / 1132 / 1204; N = 50021
// theta 0.5 3918 / 3413 / 3370, theta 0.9 1423 / 1395 / 1416; N = 100000 theta 0.5 7258 / 6923 /
// 6845, theta 0.9 2491 / 2407 / 2490; N = 300000 theta 0.7 10970 / 10961 / 11416; N = 1M theta
// 0.9 22528 / 23063.
static int lanes_per_body64(const pt_ctx *ctx, int n_aff) {
    const long long slots = 20ll * std::max(1, ctx->sm_count) * 32, n = n_aff;
    return 16 * n <= slots ? 16 : 8 * n <= slots ? 8 : 8 * n <= 5 * slots ? 4 : n <= 4 * slots ? 2 : 1;
}

// The f64 method: build over DVec3 bodies, walk with the reference rule in double.
int run64(pt_ctx *ctx, const double4_32a *d_aff, int n_aff, const double4_32a *d_src, int n_src,
                 double theta, double softening, double *d_out) {
    cudaStream_t st = ctx->stream;
    if (n_aff == 0) return PT_OK;
    if (n_src == 0) {
        PT_CUDA(cudaMemsetAsync(d_out, 0, sizeof(double) * 3 * size_t(n_aff), st));
        return PT_OK;
    }
    State *Sp = state(ctx);
    if (!Sp) return set_error(PT_ERR_OOM, "Barnes-Hut state allocation failed");
    State &S = *Sp;
    mark(ctx, 0);
    PT_TRY(build_t<double>(ctx, S, d_src, n_src));
    const bool same = (d_aff == d_src) && (n_aff == n_src);
    if (!same) PT_TRY(sort_targets_t<double>(ctx, S, d_aff, n_aff));
    const double4_32a *tbody = same ? as<double4_32a>(S.sbody64) : as<double4_32a>(S.tbody64);
    const uint32_t *tidx = same ? as<uint32_t>(S.idx) : as<uint32_t>(S.tidx);
    unsigned long long *stats = reinterpret_cast<unsigned long long *>(S.counters.ptr) + 2;
    int *err = as<int>(S.counters) + 3;
    mark(ctx, 1);
    const int lpb = lanes_per_body64(ctx, n_aff);
    auto kern = lpb == 16 ? bh_walk64<16>
                : lpb == 8  ? bh_walk64<8>
                : lpb == 4  ? bh_walk64<4>
                : lpb == 2  ? bh_walk64<2>
                            : bh_walk64<1>;
    launch_next(
        kern, (n_aff + 32 / lpb - 1) / (32 / lpb), 32, 0, st, tbody, tidx, n_aff, as<double4_32a>(S.nodeA64), as<int4>(S.nodeB), as<double4_32a>(S.nodeG64),
        as<double4_32a>(S.sbody64), as<int>(S.counters), theta * theta, softening * softening, d_out, stats, err);
    PT_TRY(check_launch(ctx, "bh_walk64"));
    mark(ctx, 2);
    return PT_OK;
}

// Walks the context's current tree for targets tbody (key-sorted; tidx maps them back
// to the caller's order) and writes accelerations to d_out.
int walk(pt_ctx *ctx, State &S, const float4 *tbody, const uint32_t *tidx, int n_aff, float theta,
                float softening, uint32_t flags, float *d_out) {
    cudaStream_t st = ctx->stream;
    if (S.f64) return set_error(PT_ERR_INVALID, "the context's tree holds DVec3 bodies: walk it with the f64 method");
    // counters: int[4] = {leaves, nodes, cells, error} then u64[8] = {interactions,
    // visits, warps, max group stack, learned records, cell interactions, warps that
    // fell back to the per-body walk, far nodes taken by the local expansion}, cleared by the
    // layout or the targets' gather before
    unsigned long long *stats = reinterpret_cast<unsigned long long *>(S.counters.ptr) + 2;
    int *err = as<int>(S.counters) + 3;
    const float th2 = theta * theta;
    const float eps2 = softening * softening;
    const bool quad = flags & PT_BH_QUADRUPOLE;
    mark(ctx, 1);
    if (flags & PT_BH_GROUP) {
        const int groups = (n_aff + GW_GROUP - 1) / GW_GROUP;
        const bool learned = flags & PT_BH_LEARNED;
        if (learned && !S.mlp_w) return set_error(PT_ERR_INVALID, "PT_BH_LEARNED needs a model (pt_mlp_*)");
        LearnedRecords LR{};
        if (learned) {
            PT_TRY(ensure_buf(ctx, S.lhead, sizeof(int) * size_t(groups)));
            PT_TRY(ensure_buf(ctx, S.lcentre, sizeof(float4) * size_t(groups)));
            PT_TRY(ensure_buf(ctx, S.lused, sizeof(int)));
            if (S.lcap_fixed > 0) S.lcap = S.lcap_fixed;
            else if (S.lcap == 0) S.lcap = std::max(1024, 2 * groups);
        }
        const float *gscale = nullptr;
        const int *gorder = nullptr;
        if (flags & PT_BH_RELATIVE) {
            PT_TRY(ensure_buf(ctx, S.gscale, sizeof(float) * size_t(groups)));
            const bool ordered = groups > 20 * std::max(1, ctx->sm_count);  // more than start at once by single warps
            launch_next(bh_group_scale, blocks(groups, 128), 128, 0, st, tbody, n_aff, as<float4>(S.nodeA),
                        as<int4>(S.nodeB), as<int>(S.counters), eps2, S.rel_alpha, as<float>(S.gscale));
            PT_TRY(check_launch(ctx, "bh_group_scale"));
            gscale = as<float>(S.gscale);
            if (ordered) PT_TRY(place_groups(ctx, S, groups, &gorder));
        } else {
            PT_TRY(order_groups(ctx, S, tbody, n_aff, GW_GROUP, &gorder));
        }
        for (int attempt = 0;; ++attempt) {
            if (learned) {
                PT_TRY(ensure_buf(ctx, S.lrec, sizeof(int) * size_t(S.lcap) * LCHUNK));
                PT_TRY(ensure_buf(ctx, S.lgroup, sizeof(int) * size_t(S.lcap)));
                PT_TRY(ensure_buf(ctx, S.lnext, sizeof(int) * size_t(S.lcap)));
                PT_TRY(ensure_buf(ctx, S.lpart, sizeof(float4) * size_t(S.lcap)));
                LR = LearnedRecords{as<int>(S.lrec),   as<int>(S.lgroup),   as<int>(S.lnext), as<int>(S.lhead),
                                    as<float4>(S.lcentre), as<float4>(S.lpart), as<int>(S.lused), S.lcap};
                PT_CUDA(cudaMemsetAsync(LR.used, 0, sizeof(int), st));
            }
            const int team = learned ? 1 : team_of(ctx, groups);
            launch_next(
                group_kernel(quad, eps2 == 0.0f, learned, flags & PT_BH_LOCAL, gscale != nullptr, team), groups,
                32 * team, 0, st, tbody, tidx, n_aff, as<float4>(S.nodeA), as<int4>(S.nodeB), as<float4>(S.nodeQ), as<float4>(S.nodeG),
                as<float4>(S.sbody), as<int>(S.counters), th2, S.theta_inner * S.theta_inner, LR, eps2, d_out, stats,
                err, S.stack_cap > 0 ? S.stack_cap : INT_MAX, S.local_ratio, gscale, S.rel_mono, gorder);
            PT_TRY(check_launch(ctx, "bh_walk_group"));
            // Outside stream capture (and with the automatic capacity) the record count
            // is checked and the walk rerun with room for all records; otherwise an
            // overflow sets error bit 2, which the callers report as PT_ERR_CAPACITY.
            if (!learned || ctx->capturing || attempt > 0 || S.lcap_fixed > 0) break;
            int used = 0;
            PT_CUDA(cudaMemcpyAsync(&used, LR.used, sizeof(int), cudaMemcpyDeviceToHost, st));
            PT_CUDA(cudaStreamSynchronize(st));
            if (used <= S.lcap) break;
            S.lcap = used + used / 4;
            PT_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
            PT_CUDA(cudaMemsetAsync(stats, 0, WALK_STATS * sizeof(unsigned long long), st));
        }
        if (learned) {
            bh_learned_eval<<<ctx->sm_count * 4, 128, 0, st>>>(LR, as<float4>(S.nodeA), as<float4>(S.nodeQ),
                                                               as<float4>(S.nodeG), S.mlp_w, S.mlp_b,
                                                               S.theta_inner, theta);
            PT_TRY(check_launch(ctx, "bh_learned_eval"));
            bh_learned_apply<<<blocks(n_aff), 256, 0, st>>>(LR, tidx, n_aff, GW_SHIFT, d_out);
            PT_TRY(check_launch(ctx, "bh_learned_apply"));
        }
        PT_TRY(check_launch(ctx, "bh_walk_group"));
        mark(ctx, 2);
        return PT_OK;
    }
    const MaskedPlan p = masked_plan(ctx, n_aff);
    auto kern = quad ? masked_kernel_q<true>(p.big) : masked_kernel_q<false>(p.big);
    const int *order = nullptr;
    PT_TRY(order_groups(ctx, S, tbody, n_aff, p.big, &order));
    launch_next(
        kern, p.big_groups + p.small_groups, 32, 0, st, p.big_groups, order, tbody, tidx, n_aff, as<float4>(S.nodeA), as<int4>(S.nodeB), as<float4>(S.nodeQ), as<float4>(S.sbody),
        as<int>(S.counters), th2, eps2, d_out, stats);
    PT_TRY(check_launch(ctx, "bh_walk_masked"));
    mark(ctx, 2);
    return PT_OK;
}


}  // namespace bh
}  // namespace pt
