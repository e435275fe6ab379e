// The group walk (PT_BH_GROUP) of pt_bh_walk.cu and pt_bh_team.cu, with the interaction
// lists, compensated sums, per-body fallback walk and local expansions it is made of.
#pragma once

#include "pt_bh.cuh"

#include <type_traits>

namespace pt {
namespace bh {

// ---- walk ------------------------------------------------------------------

// PT_BH_RELATIVE: a cell of mass m and width w is also opened within squared distance
// r2, where its truncation bound m w^p / d^(p+2) (p = 3 with quadrupoles, 2 without)
// reaches alpha |a|; ginv = 1 / (alpha |a|) of the target's group, 0 when off.
template <bool QUAD>
__device__ __forceinline__ float rel_r2(float m, float w, float ginv) {
    if (!(ginv > 0.f && m > 0.f)) return 0.f;
    return QUAD ? __powf(m * w * w * w * ginv, 0.4f) : sqrtf(m * w * w * ginv);
}

// The reference's per-body walk (sequential.rs) for this lane's target p, the cursor
// being the warp minimum of the lanes' next nodes: all 32 lanes take part. Adds the
// accepted nodes' accelerations to (ax, ay, az) and counts them.
template <bool QUAD>
__device__ __forceinline__ void lane_walk(float4 p, bool valid, int T, const float4 *__restrict__ nodeA,
                                          const int4 *__restrict__ nodeB, const float4 *__restrict__ nodeQ,
                                          const float4 *__restrict__ sbody, float th2, float eps2, float &ax,
                                          float &ay, float &az, unsigned &nacc, unsigned &nvisit,
                                          unsigned &ncell, float ginv = 0.f) {
    int resume = valid ? 0 : T;
    int node = 0;
    while (node < T) {
        const float4 A = __ldg(nodeA + node);
        const int4 B = __ldg(nodeB + node);
        const bool active = node >= resume;
        float dx = 0.f, dy = 0.f, dz = 0.f, d2 = 0.f;
        bool open = false, zero = false;
        if (active) {
            dx = A.x - p.x;
            dy = A.y - p.y;
            dz = A.z - p.z;
            d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            zero = (d2 == 0.0f);
            const float w = __int_as_float(B.x);
            open = !zero && B.z < 0 && (th2 * d2 < w * w || d2 < rel_r2<QUAD>(A.w, w, ginv));
        }
        int next = resume;
        if (active) {
            ++nvisit;
            if (zero) {
                next = resume = B.y;  // the whole node is skipped (sequential.rs:485-487)
            } else if (open) {
                next = node + 1;
            } else {
                if (B.z >= 0 && B.w > 1) {  // a bucket leaf: its bodies one by one
                    for (int b = B.z; b < B.z + B.w; ++b) {
                        const float4 q = __ldg(sbody + b);
                        const float ex = q.x - p.x, ey = q.y - p.y, ez = q.z - p.z;
                        const float e2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
                        if (e2 == 0.0f) continue;
                        const float inv = rsqrt_ftz(e2 + eps2);
                        const float s = (q.w * inv) * (inv * inv);
                        ax = fmaf(ex, s, ax);
                        ay = fmaf(ey, s, ay);
                        az = fmaf(ez, s, az);
                    }
                } else {
                    const float inv = rsqrt_ftz(d2 + eps2);
                    const float inv2 = inv * inv;
                    const float s = (A.w * inv) * inv2;
                    ax = fmaf(dx, s, ax);
                    ay = fmaf(dy, s, ay);
                    az = fmaf(dz, s, az);
                    if (QUAD && B.z < 0) {  // traceless quadrupole of the cell
                        const float4 q0 = __ldg(nodeQ + 2 * node);
                        const float4 q1 = __ldg(nodeQ + 2 * node + 1);
                        // q0 = (Qxx, Qxy, Qxz, Qyy), q1 = (Qyz, Qzz)
                        const float qx = fmaf(q0.x, dx, fmaf(q0.y, dy, q0.z * dz));
                        const float qy = fmaf(q0.y, dx, fmaf(q0.w, dy, q1.x * dz));
                        const float qz = fmaf(q0.z, dx, fmaf(q1.x, dy, q1.y * dz));
                        const float dqd = fmaf(dx, qx, fmaf(dy, qy, dz * qz));
                        const float inv5 = inv2 * inv2 * inv;
                        const float c7 = 2.5f * dqd * inv5 * inv2;
                        ax += fmaf(c7, dx, -qx * inv5);
                        ay += fmaf(c7, dy, -qy * inv5);
                        az += fmaf(c7, dz, -qz * inv5);
                    }
                }
                ++nacc;
                ncell += B.z < 0;
                next = resume = B.y;
            }
        }
        node = __reduce_min_sync(0xffffffffu, next);
    }
}

// ---- group walk (PT_BH_GROUP) ----------------------------------------------
// One warp walks for 32 x GW_TPL (64) key-adjacent targets. Each step pops up to 32
// nodes from a shared-memory stack of sibling ranges (independent loads, one per
// lane), opens a cell when the reference's per-body rule opens it for at least one of
// the targets (so never less accurate than that rule), and appends accepted nodes to
// shared-memory interaction lists. A full list is evaluated densely: every lane runs
// its targets against all entries, two entries per packed f32x2 instruction.
// Warps (groups) per CTA of the group walk. A CTA's slot is held until its slowest
// warp ends, so with one warp per CTA no warp slot idles behind a neighbouring group's
// longer walk; the local-expansion lists are sized (64 cells, 80 bodies) so that 20
// one-warp CTAs fit an SM's shared memory. Measured at N = 4M (walk ms): headline
// configuration 5.40 with 2 warps per CTA (72 / 96 entries) -> 5.25 with 1 (then 64 / 88);
// quadrupole + group + local at theta 0.52 12.19 -> 11.74; quadrupole + group at theta
// 0.52 16.30 -> 15.19 (4 warps per CTA: 5.47, 12.43, 16.40). Persistent warps taking
// groups from a counter instead spilled (96 -> 116 bytes) and were slower (5.85 ms).

// In small calls W = 4 or 8 warps walk for one group together: they share the stack, each pops,
// votes and evaluates a share of the nodes for all 64 targets, and their sums are added up at
// the end, in warp order. The opened and accepted nodes are the same.
constexpr int GW_TEAM_STACK = 768;

template <int W>
__device__ __forceinline__ void team_sync() {
    if (W > 1) __syncthreads();
    else __syncwarp();
}

// Interaction lists. Cells carry their quadrupole when QUAD; single bodies never need one.
// pair(): two entries' fields, packed.
template <int NF, int CAP_>
struct IList {  // an array per field
    static constexpr int FIELDS = NF, CAP = CAP_;
    float f[NF][CAP + 2];
    __device__ __forceinline__ void put(int k, int e, float x) { f[k][e] = x; }
    __device__ __forceinline__ void pair(int e, f2 (&q)[NF]) const {
#pragma unroll
        for (int k = 0; k < NF; ++k) q[k] = *reinterpret_cast<const f2 *>(&f[k][e]);
    }
};

// The same with a field's two values of a pair of entries side by side, so that one 16-byte
// read gives two fields. In the walks with local expansions this is the faster of the two (N
// = 4M error bound: walk 5205 -> 5000 us), in the others its wider registers spill or it is 1-3 %
// slower.
template <int NF, int CAP_>
struct PList {
    static_assert(NF % 2 == 0, "two fields to a 16-byte read");
    static constexpr int FIELDS = NF, CAP = CAP_;
    float4 v[(CAP + 2) / 2 * (NF / 2)];
    __device__ __forceinline__ void put(int k, int e, float x) {
        reinterpret_cast<float *>(v)[(e >> 1) * (2 * NF) + 2 * k + (e & 1)] = x;
    }
    __device__ __forceinline__ void pair(int e, f2 (&q)[NF]) const {
        const float4 *p = v + (e >> 1) * (NF / 2);
#pragma unroll
        for (int k = 0; k < NF / 2; ++k) {
            const float4 t = p[k];
            q[2 * k] = pk2(t.x, t.y);
            q[2 * k + 1] = pk2(t.z, t.w);
        }
    }
};

// A body's acceleration as a compensated FP32 sum (running sum s, rounding errors c).
// Each evaluated list chunk (up to 128 entries) is summed in plain FP32 in two packed
// partials and enters the running sum through TwoSum, so the rounding error of the
// total does not grow with the number of chunks: it is that of one chunk's sum.
struct CSum {
    float sx, sy, sz, cx, cy, cz;
};

__device__ __forceinline__ void csum_zero(CSum &a) { a.sx = a.sy = a.sz = a.cx = a.cy = a.cz = 0.f; }

__device__ __forceinline__ void csum_fold(CSum &a, f2 tx, f2 ty, f2 tz) {
    float l, h;
    upk2(tx, l, h);
    two_sum_acc(a.sx, a.cx, l + h);
    upk2(ty, l, h);
    two_sum_acc(a.sy, a.cy, l + h);
    upk2(tz, l, h);
    two_sum_acc(a.sz, a.cz, l + h);
}

// Where a warp keeps its bodies' compensated sums: in registers, or, in the kernel
// whose registers the traversal state fills (the quadrupole group walk with local
// expansions, 96 registers for 20 warps per SM: 56 bytes spilled, walk +15 %), in shared
// memory as [value][lane] (conflict-free; touched once per evaluated chunk; walk +2.5 %
// over plain FP32 sums). Measured at N = 4M: the other group walks +1.2 % in registers
// (+2.7 % in shared memory), the masked walk +1.6 %.
template <int TPL>
struct RegSums {
    CSum c[TPL];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < TPL; ++i) csum_zero(c[i]);
    }
    __device__ __forceinline__ void fold(int i, f2 tx, f2 ty, f2 tz) { csum_fold(c[i], tx, ty, tz); }
    __device__ __forceinline__ void parts(int i, float *v) const {
        v[0] = c[i].sx, v[1] = c[i].sy, v[2] = c[i].sz, v[3] = c[i].cx, v[4] = c[i].cy, v[5] = c[i].cz;
    }
    // adds up the sums of the LPB lanes that share body i; each of them gets the result
    template <int LPB>
    __device__ __forceinline__ void gather(int i) {
        float *s[3] = {&c[i].sx, &c[i].sy, &c[i].sz}, *e[3] = {&c[i].cx, &c[i].cy, &c[i].cz};
#pragma unroll
        for (int o = 1; o < LPB; o <<= 1)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float os = __shfl_xor_sync(0xffffffffu, *s[a], o), oe = __shfl_xor_sync(0xffffffffu, *e[a], o);
                float r = *e[a] + oe;
                two_sum_acc(*s[a], r, os);
                *e[a] = r;
            }
    }
    __device__ __forceinline__ void total(int i, float &x, float &y, float &z) const {
        x = c[i].sx + c[i].cx;
        y = c[i].sy + c[i].cy;
        z = c[i].sz + c[i].cz;
    }
};

template <int TPL>
struct SmemSums {
    float (*v)[32];  // [6 * TPL][32]: per body sx, sy, sz, cx, cy, cz
    int lane;
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int k = 0; k < 6 * TPL; ++k) v[k][lane] = 0.f;
    }
    __device__ __forceinline__ void fold(int i, f2 tx, f2 ty, f2 tz) {
        CSum a;
        a.sx = v[6 * i][lane], a.sy = v[6 * i + 1][lane], a.sz = v[6 * i + 2][lane];
        a.cx = v[6 * i + 3][lane], a.cy = v[6 * i + 4][lane], a.cz = v[6 * i + 5][lane];
        csum_fold(a, tx, ty, tz);
        v[6 * i][lane] = a.sx, v[6 * i + 1][lane] = a.sy, v[6 * i + 2][lane] = a.sz;
        v[6 * i + 3][lane] = a.cx, v[6 * i + 4][lane] = a.cy, v[6 * i + 5][lane] = a.cz;
    }
    __device__ __forceinline__ void parts(int i, float *o) const {
#pragma unroll
        for (int k = 0; k < 6; ++k) o[k] = v[6 * i + k][lane];
    }
    __device__ __forceinline__ void total(int i, float &x, float &y, float &z) const {
        x = v[6 * i][lane] + v[6 * i + 3][lane];
        y = v[6 * i + 1][lane] + v[6 * i + 4][lane];
        z = v[6 * i + 2][lane] + v[6 * i + 5][lane];
    }
};

// Two list entries (packed lo/hi: monopole x, y, z, m and, for NF = 10, the negated
// traceless quadrupole N = -Q as Nxx Nxy Nxz Nyy Nyz Nzz) for one target. With
// u = N d and c = d.u:
//   a += d (m / r^3 + 2.5 (d.Q.d) / r^7) - (Q d) / r^5 = d (sc - 2.5 c / r^7) + u / r^5
template <int NF, bool GUARD>
__device__ __forceinline__ void eval_pair(const f2 (&q)[NF], f2 px, f2 py, f2 pz, f2 e2, f2 &ax, f2 &ay, f2 &az) {
    const f2 dx = sub2(q[0], px);
    const f2 dy = sub2(q[1], py);
    const f2 dz = sub2(q[2], pz);
    const f2 r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, e2)));
    float r0, r1;
    upk2(r2, r0, r1);
    float i0 = rsqrt_ftz(r0), i1 = rsqrt_ftz(r1);
    if (GUARD) {
        i0 = (r0 > 0.0f) ? i0 : 0.0f;
        i1 = (r1 > 0.0f) ? i1 : 0.0f;
    }
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

// Evaluates entries [0, cnt) of a list for this lane's TPL targets, two entries per
// packed instruction; each pair of entries is read from shared memory once for all
// of the lane's targets.
template <bool GUARD, int TPL, class List, class Sums>
__device__ __forceinline__ void eval_list(List &Lst, int cnt, const f2 (&px)[TPL], const f2 (&py)[TPL],
                                          const f2 (&pz)[TPL], f2 e2, Sums &acc) {
    constexpr int NF = List::FIELDS;
    const int lane = threadIdx.x & 31;
    f2 ax[TPL], ay[TPL], az[TPL];
#pragma unroll
    for (int i = 0; i < TPL; ++i) ax[i] = ay[i] = az[i] = pk2(0.f, 0.f);
    __syncwarp();
    if (cnt & 1) {  // pad with a massless entry far away: contributes exactly 0
        if (lane < NF) Lst.put(lane, cnt, (lane < 3) ? 1e30f : 0.0f);
        __syncwarp();
        ++cnt;
    }
#pragma unroll 2
    for (int e = 0; e < cnt; e += 2) {
        f2 q[NF];
        Lst.pair(e, q);
#pragma unroll
        for (int i = 0; i < TPL; ++i) eval_pair<NF, GUARD>(q, px[i], py[i], pz[i], e2, ax[i], ay[i], az[i]);
    }
#pragma unroll
    for (int i = 0; i < TPL; ++i) acc.fold(i, ax[i], ay[i], az[i]);
    __syncwarp();
}

// ---- learned correction: records of marginal cells ---------------------------
// The walk (PT_BH_LEARNED) does not evaluate the network itself: it records the
// node index of every marginal cell (accepted at theta, opened at theta_inner) in
// chunks of LCHUNK entries that each belong to one warp (one group of 64 targets),
// chained per group in walk order, and the group's centre. A tensor-core kernel then
// evaluates all records (bh_learned_eval) and bh_learned_apply adds each group's
// sum, chunk by chunk in chain order, so results do not depend on scheduling.
constexpr int LCHUNK = 128;

struct LearnedRecords {
    int *rec;        // [cap][LCHUNK] node indices, -1 = padding
    int *chunk_group;  // [cap]
    int *next;       // [cap] next chunk of the same group, -1 = last
    int *head;       // [groups] first chunk of the group, -1 = none
    float4 *centre;  // [groups] mean position of the group's targets
    float4 *part;    // [cap] the chunk's summed correction
    int *used;       // chunks handed out (may exceed cap: then nothing past cap is written)
    int cap;
};

// ---- local (Taylor) expansion of far nodes about the group centre -------------
// PT_BH_LOCAL: an accepted node far from the group (group radius R < ratio * d, d
// from the group's box centre g to the node's centre of mass) is not added to the
// interaction lists. The lane that popped it adds the node's softened monopole (+
// quadrupole) field to a second-order expansion of the acceleration about g:
// a(g + r) = a0 + T r + 1/2 H : r r, with
//   a0 = m d s^-3/2,  T_ij = 3m d_i d_j s^-5/2 - m delta_ij s^-3/2,
//   H_ijk = 15m d_i d_j d_k s^-7/2 - 3m s^-5/2 (delta_ij d_k + delta_ik d_j + delta_jk d_i)
// (s = |d|^2 + eps^2: the exact derivatives of the softened kernel), plus the
// quadrupole's a0 and T. The expansion costs one lane ~150 flops per far node
// instead of every target's list entry; its truncation error is ~(R/d)^3.
struct LocalExp {
    float ax, ay, az;                                      // a(g)
    float txx, txy, txz, tyy, tyz, tzz;                    // d a_i / d x_j
    float hxxx, hxxy, hxxz, hxyy, hxyz, hxzz, hyyy, hyyz, hyzz, hzzz;  // d2 a_i / dx_j dx_k
};

// Adds the softened monopole (+ traceless quadrupole q, when given) field of a node
// at offset d = com - g, mass m, to the expansion about g.
__device__ __forceinline__ void local_add(LocalExp &L, float dx, float dy, float dz, float m, float eps2,
                                          const float4 *q0p, const float4 *q1p) {
    const float s = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2)));
    const float inv = rsqrt_ftz(s);
    const float inv2 = inv * inv;
    const float i3 = m * inv * inv2;      // m s^-3/2
    const float i5 = 3.0f * i3 * inv2;    // 3 m s^-5/2
    const float i7 = 5.0f * i5 * inv2;    // 15 m s^-7/2
    L.ax = fmaf(i3, dx, L.ax);
    L.ay = fmaf(i3, dy, L.ay);
    L.az = fmaf(i3, dz, L.az);
    const float xx = dx * dx, yy = dy * dy, zz = dz * dz, xy = dx * dy, xz = dx * dz, yz = dy * dz;
    L.txx += fmaf(i5, xx, -i3);
    L.txy = fmaf(i5, xy, L.txy);
    L.txz = fmaf(i5, xz, L.txz);
    L.tyy += fmaf(i5, yy, -i3);
    L.tyz = fmaf(i5, yz, L.tyz);
    L.tzz += fmaf(i5, zz, -i3);
    const float ax7 = i7 * dx, ay7 = i7 * dy, az7 = i7 * dz;
    L.hxxx += fmaf(ax7, xx, -3.0f * i5 * dx);
    L.hxxy += fmaf(ax7, xy, -i5 * dy);
    L.hxxz += fmaf(ax7, xz, -i5 * dz);
    L.hxyy += fmaf(ax7, yy, -i5 * dx);
    L.hxyz = fmaf(ax7, yz, L.hxyz);
    L.hxzz += fmaf(ax7, zz, -i5 * dx);
    L.hyyy += fmaf(ay7, yy, -3.0f * i5 * dy);
    L.hyyz += fmaf(ay7, yz, -i5 * dz);
    L.hyzz += fmaf(ay7, zz, -i5 * dy);
    L.hzzz += fmaf(az7, zz, -3.0f * i5 * dz);
    if (q0p) {
        const float4 q0 = __ldg(q0p), q1 = __ldg(q1p);  // Qxx Qxy Qxz Qyy | Qyz Qzz
        const float ux = fmaf(q0.x, dx, fmaf(q0.y, dy, q0.z * dz));
        const float uy = fmaf(q0.y, dx, fmaf(q0.w, dy, q1.x * dz));
        const float uz = fmaf(q0.z, dx, fmaf(q1.x, dy, q1.y * dz));
        const float c = fmaf(dx, ux, fmaf(dy, uy, dz * uz));
        const float j5 = inv2 * inv2 * inv, j7 = j5 * inv2, j9 = j7 * inv2;
        const float c7 = 2.5f * c * j7;
        L.ax += fmaf(c7, dx, -ux * j5);
        L.ay += fmaf(c7, dy, -uy * j5);
        L.az += fmaf(c7, dz, -uz * j5);
        const float f5 = 5.0f * j7, g9 = 17.5f * c * j9;
        L.txx += fmaf(q0.x, j5, fmaf(g9, xx, -fmaf(2.0f * f5, ux * dx, c7)));
        L.tyy += fmaf(q0.w, j5, fmaf(g9, yy, -fmaf(2.0f * f5, uy * dy, c7)));
        L.tzz += fmaf(q1.y, j5, fmaf(g9, zz, -fmaf(2.0f * f5, uz * dz, c7)));
        L.txy += fmaf(q0.y, j5, fmaf(g9, xy, -f5 * fmaf(ux, dy, uy * dx)));
        L.txz += fmaf(q0.z, j5, fmaf(g9, xz, -f5 * fmaf(ux, dz, uz * dx)));
        L.tyz += fmaf(q1.x, j5, fmaf(g9, yz, -f5 * fmaf(uy, dz, uz * dy)));
    }
}

__device__ __forceinline__ void local_reduce(LocalExp &L) {
    float *f = &L.ax;
#pragma unroll
    for (int k = 0; k < 19; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) f[k] += __shfl_xor_sync(0xffffffffu, f[k], o);
}

// a(g + d) from the expansion
__device__ __forceinline__ void local_eval(const LocalExp &L, float dx, float dy, float dz, float &ax, float &ay,
                                           float &az) {
    const float xx = dx * dx, yy = dy * dy, zz = dz * dz, xy2 = 2.0f * dx * dy, xz2 = 2.0f * dx * dz,
                yz2 = 2.0f * dy * dz;
    ax = L.ax + fmaf(L.txx, dx, fmaf(L.txy, dy, L.txz * dz)) +
         0.5f * fmaf(L.hxxx, xx, fmaf(L.hxyy, yy, fmaf(L.hxzz, zz, fmaf(L.hxxy, xy2, fmaf(L.hxxz, xz2, L.hxyz * yz2)))));
    ay = L.ay + fmaf(L.txy, dx, fmaf(L.tyy, dy, L.tyz * dz)) +
         0.5f * fmaf(L.hxxy, xx, fmaf(L.hyyy, yy, fmaf(L.hyzz, zz, fmaf(L.hxyy, xy2, fmaf(L.hxyz, xz2, L.hyyz * yz2)))));
    az = L.az + fmaf(L.txz, dx, fmaf(L.tyz, dy, L.tzz * dz)) +
         0.5f * fmaf(L.hxxz, xx, fmaf(L.hyyz, yy, fmaf(L.hzzz, zz, fmaf(L.hxyz, xy2, fmaf(L.hxzz, xz2, L.hyzz * yz2)))));
}

// PT_BH_LOCAL: adds queued far node e (2 x node index + 1 for a cell) to this lane's
// expansion coefficients, kept in shared memory as [coefficient][lane].
template <bool QUAD>
__device__ __forceinline__ void local_add_node(float (*lx)[32], int lane, int e, const float4 *__restrict__ nodeA,
                                               const float4 *__restrict__ nodeQ, float gx, float gy, float gz,
                                               float eps2) {
    const int node = e >> 1;
    const bool q = QUAD && (e & 1);
    const float4 A = __ldg(nodeA + node);
    LocalExp t;
    float *tf = &t.ax;
#pragma unroll
    for (int k = 0; k < 19; ++k) tf[k] = lx[k][lane];
    local_add(t, A.x - gx, A.y - gy, A.z - gz, A.w, eps2, q ? nodeQ + 2 * node : nullptr,
              q ? nodeQ + 2 * node + 1 : nullptr);
#pragma unroll
    for (int k = 0; k < 19; ++k) lx[k][lane] = tf[k];
}

// Targets per lane of the group walk: a warp walks for 32 * GW_TPL key-adjacent
// targets, and each list entry read from shared memory serves all of a lane's
// targets. Measured at N = 4M bulge+disk, theta 0.5, quadrupole: 1 -> 18.3 ms
// (p95 8.2e-4), 2 -> 16.6 ms (7.7e-4), 4 -> 17.7 ms (7.5e-4); the larger box opens
// more cells (13.5e9 -> 15.2e9 -> 17.6e9 pairs) but traversal is shared by more
// targets.
#ifndef PT_GW_TPL
#define PT_GW_TPL 2
#endif
constexpr int GW_TPL = PT_GW_TPL;
constexpr int GW_GROUP = 32 * GW_TPL;
constexpr int GW_SHIFT = GW_TPL == 1 ? 5 : GW_TPL == 2 ? 6 : 7;
static_assert(GW_GROUP == (1 << GW_SHIFT), "targets per lane: 1, 2 or 4");
// PT_BH_LOCAL walk: occupancy (counted in CTAs of 4 warps per SM, so 5 = 20 warps)
// and list capacities. Both registers (96) and shared memory (11 KB per warp) hold it
// at 20 warps per SM; 24 warps with lists of 64 cells and 96 bodies (80 registers, 84
// bytes spilled) measured 6.9 ms against 6.1 ms at N = 4M.
#ifndef PT_GW_LMINB
#define PT_GW_LMINB 5
#endif
#ifndef PT_GW_LCELLS
#define PT_GW_LCELLS 64
#endif
#ifndef PT_GW_LBODIES
#define PT_GW_LBODIES 80
#endif
// Stack ranges per warp of the PT_BH_LOCAL walk. (21 warps per SM, with lists of 56
// cells / 80 bodies and 272 ranges, measured the same as 20: 5.21 against 5.20 ms.)
#ifndef PT_GW_LSTACK
#define PT_GW_LSTACK 288
#endif
// Opened cells with at most this many nodes below them are summed body by body at
// once instead of being walked level by level (loaded 32 nodes per round; 0 = off).
// The calibrated headline at N = 4M (fastest configuration within the error margin)
// for limits 7 / 15 / 31 / 47 / 63 / 95 / 127: 5.26 / 5.65 / 6.07 / 6.10 / 6.05 /
// 5.92 / 5.77 e8 bodies/s.
#ifndef PT_GW_FLAT
#define PT_GW_FLAT 31
#endif
constexpr int GW_FLAT = PT_GW_FLAT;
static_assert(GW_FLAT >= 0 && GW_FLAT <= 1023, "flattened subtree size");
#ifndef PT_GW_MINB
#define PT_GW_MINB (GW_TPL == 1 ? 6 : 5)  // 4-warp CTAs per SM the register budget is set for
#endif
// A team's warps read the cells that they vote on from slots of their own; one warp alone from the
// stack's free slots.
template <int W>
struct VoteSlots {
    float4 vote[32];
    __device__ __forceinline__ float4 *slots(int2 *) { return vote; }
};
template <>
struct VoteSlots<1> {
    __device__ __forceinline__ float4 *slots(int2 *free) { return reinterpret_cast<float4 *>(free); }
};

template <bool QUAD, bool GUARD, bool LEARNED, bool LOCAL, bool REL, int W>
__global__ void __launch_bounds__(32 * W, (LOCAL ? PT_GW_LMINB : PT_GW_MINB) * 4 / W)
    bh_walk_group(const float4 *__restrict__ tbody, const uint32_t *__restrict__ tidx, int n_aff,
                  const float4 *__restrict__ nodeA, const int4 *__restrict__ nodeB, const float4 *__restrict__ nodeQ,
                  const float4 *__restrict__ nodeG, const float4 *__restrict__ sbody, const int *__restrict__ counters,
                  float th2, float th_in2, LearnedRecords LR, float eps2, float *__restrict__ out,
                  unsigned long long *__restrict__ stats, int *__restrict__ err, int stack_cap,
                  float local_ratio, const float *__restrict__ gscale, float mono_beta,
                  const int *__restrict__ gorder) {
    after_previous();
    static_assert(!(LEARNED && LOCAL), "PT_BH_LEARNED and PT_BH_LOCAL are exclusive");
    static_assert(!(LEARNED && REL), "PT_BH_LEARNED and PT_BH_RELATIVE are exclusive");
    static_assert(!(LEARNED && W > 1), "one warp chains a group's records");
    constexpr int NFC = QUAD ? 10 : 4;
    constexpr int TPL = GW_TPL;
    using CellList = typename std::conditional<LOCAL, PList<NFC, PT_GW_LCELLS>, IList<NFC, 96>>::type;
    using BodyList = typename std::conditional<LOCAL, PList<4, PT_GW_LBODIES>, IList<4, 128>>::type;
    // PT_BH_LOCAL keeps its 19 expansion coefficients per lane in shared memory
    // ([coefficient][lane]: no bank conflicts) and queues far nodes (up to 63) so that
    // they are expanded 32 at a time, one per lane, instead of by the few lanes that
    // popped them; the stack is trimmed to 288 ranges so that 20 warps stay resident per SM.
    constexpr int STK = W > 1 ? GW_TEAM_STACK : LOCAL ? PT_GW_LSTACK : GW_STACK;
    // A pop of k <= (cap - S) / 2 ranges leaves 3 k slots free below the cap and may vote on
    // min(32, 2 k) cells of two slots, from an even slot on: 17 slots past the cap at most.
    // (W > 1: the warps have vote slots of their own.)
    constexpr int VOTE_SLACK = W > 1 ? 0 : 18;
    stack_cap = min(stack_cap, STK);
    struct Shared : VoteSlots<W> {
        CellList cells;
        BodyList bodies;
        float lx[LOCAL ? 19 : 1][32];
        float sums[QUAD && LOCAL ? 6 * GW_TPL : 1][32];
        int far[LOCAL ? 64 : 1];
    };
    // 20 warps per SM by shared memory too: 228 KB, of which a block takes 1 KB more than it
    // declares, in steps of 128 bytes (16 bytes more, and 19 are resident: a whole call with the
    // error bound at N = 4M takes 6040 us, and 5999 with 20)
    static_assert(!(QUAD && LOCAL && W == 1) ||
                      20 * ((sizeof(Shared) + sizeof(int2) * (STK + VOTE_SLACK) + 1024 + 127) / 128 * 128) <= 228 * 1024,
                  "shared memory for 20 warps per SM");
    __shared__ __align__(16) int2 stack[STK + VOTE_SLACK];
    __shared__ __align__(16) Shared s_warp[W];
    __shared__ int s_push[W];
    const int warp = W > 1 ? threadIdx.x >> 5 : 0, lane = threadIdx.x & 31;
    const int group = gorder ? gorder[blockIdx.x] : blockIdx.x;
    const int g0 = group * GW_GROUP;
    if (unsigned(g0) >= unsigned(n_aff)) return;
    Shared &my = s_warp[warp];
    // this lane's targets: g0 + lane, g0 + 32 + lane, ...
    float4 p[TPL];
    bool valid[TPL];
#pragma unroll
    for (int i = 0; i < TPL; ++i) {
        const int t = g0 + 32 * i + lane;
        valid[i] = t < n_aff;
        p[i] = tbody[valid[i] ? t : g0];
    }
    const int nvalid = min(GW_GROUP, n_aff - g0);
    const unsigned lt = (1u << lane) - 1u;
    // PT_BH_RELATIVE: 1 / (alpha |a|) of this group (warp-uniform), and its 2/5 power,
    // the factor of a cell's (M w^3)^(2/5) kept in its nodeB.w
    const float ginv = (REL && !QUAD) ? gscale[group] : 0.f;
    const float gq = (REL && QUAD) ? __powf(gscale[group], 0.4f) : 0.f;
    // PT_BH_RELATIVE with quadrupoles: an accepted cell whose monopole truncation bound
    // M w^2 / d^4 (the quadrupole term it would drop) stays within mono_beta alpha |a|
    // from every body of the group enters the body list, without its quadrupole.
    const float gmono = (REL && QUAD && mono_beta > 0.f) ? gscale[group] / mono_beta : 0.f;
    const int T = counters[1];
    CellList &Lc = my.cells;
    BodyList &Lb = my.bodies;

    // the bounding box of the group's targets: it settles most opening decisions
    // without the per-target vote
    float mn0 = p[0].x, mn1 = p[0].y, mn2 = p[0].z, mx0 = p[0].x, mx1 = p[0].y, mx2 = p[0].z;
#pragma unroll
    for (int i = 1; i < TPL; ++i) {
        mn0 = fminf(mn0, p[i].x), mn1 = fminf(mn1, p[i].y), mn2 = fminf(mn2, p[i].z);
        mx0 = fmaxf(mx0, p[i].x), mx1 = fmaxf(mx1, p[i].y), mx2 = fmaxf(mx2, p[i].z);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn0 = fminf(mn0, __shfl_xor_sync(0xffffffffu, mn0, o));
        mn1 = fminf(mn1, __shfl_xor_sync(0xffffffffu, mn1, o));
        mn2 = fminf(mn2, __shfl_xor_sync(0xffffffffu, mn2, o));
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
        mx2 = fmaxf(mx2, __shfl_xor_sync(0xffffffffu, mx2, o));
    }
    // the group centre, where learned corrections are evaluated
    float gcx = 0.f, gcy = 0.f, gcz = 0.f;
    if (LEARNED) {
#pragma unroll
        for (int i = 0; i < TPL; ++i)
            if (valid[i]) gcx += p[i].x, gcy += p[i].y, gcz += p[i].z;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            gcx += __shfl_xor_sync(0xffffffffu, gcx, o);
            gcy += __shfl_xor_sync(0xffffffffu, gcy, o);
            gcz += __shfl_xor_sync(0xffffffffu, gcz, o);
        }
        const float nv = float(nvalid);
        gcx /= nv;
        gcy /= nv;
        gcz /= nv;
    }
    // PT_BH_LOCAL: the expansion centre g (box centre) and the far radius^2
    const float lgx = 0.5f * (mn0 + mx0), lgy = 0.5f * (mn1 + mx1), lgz = 0.5f * (mn2 + mx2);
    const float rg2 = 0.25f * fmaf(mx0 - mn0, mx0 - mn0, fmaf(mx1 - mn1, mx1 - mn1, (mx2 - mn2) * (mx2 - mn2)));
    const float far2 = LOCAL ? rg2 / (local_ratio * local_ratio) : 0.f;
    if (LOCAL)
        for (int k = 0; k < 19; ++k) my.lx[k][lane] = 0.f;
    unsigned nlocal = 0, nlocalq = 0;  // warp-uniform: far nodes, those with a quadrupole
    int Nf = 0;                     // queued far nodes
    // learned: the warp's current record chunk and its fill; the previous chunk links to
    // the next one (head of the group's chain first)
    int chunk = -1, fill = LCHUNK;
    unsigned long long learned = 0;

    const f2 e2 = pk2(eps2, eps2);
    // the lane's two targets packed, for the opening vote
    const f2 vx01 = pk2(p[0].x, p[TPL - 1].x), vy01 = pk2(p[0].y, p[TPL - 1].y), vz01 = pk2(p[0].z, p[TPL - 1].z);
    f2 px[TPL], py[TPL], pz[TPL];
    // the bodies' compensated sums over the evaluated lists
    using Sums = typename std::conditional<QUAD && LOCAL, SmemSums<TPL>, RegSums<TPL>>::type;
    Sums bsum;
    if constexpr (QUAD && LOCAL) bsum = Sums{my.sums, lane};
    bsum.zero();
#pragma unroll
    for (int i = 0; i < TPL; ++i) {
        px[i] = pk2(p[i].x, p[i].x);
        py[i] = pk2(p[i].y, p[i].y);
        pz[i] = pk2(p[i].z, p[i].z);
    }
    // Stack entries are sibling ranges (first, end): `first` is the next node to
    // visit, its later siblings follow by skip pointers up to `end`. A pop visits one
    // node of a range (two when lanes are idle) and pushes back its remaining
    // siblings and, for each opened cell, its children (pre+1, skip). The stack
    // therefore stays within about 32 ranges per tree level.
    if (threadIdx.x == 0) stack[0] = make_int2(0, T);
    team_sync<W>();
    int S = 1, Nc = 0, Nb = 0, maxS = 1;
    unsigned entries = 0, visits = 0, centries = 0;
    bool failed = false;
    while (S > 0) {
        // each pop pushes at most two ranges: never more than the room left. W warps share the
        // popped ranges evenly.
        const int kt = min(min(32 * W, S), max(1, (stack_cap - S) / 2));
        const int k = W > 1 ? (kt + W - 1 - warp) / W : kt;
        const int before = W > 1 ? warp * (kt / W) + min(warp, kt % W) : 0;
        const bool first = lane < k;
        int2 range = first ? stack[S - 1 - before - lane] : make_int2(0, 0);
        __syncwarp();
        S -= kt;
        int node = range.x;
        float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
        int4 B = make_int4(0, 0, 0, 0);
        bool open = false;
        if (first) {
            A = __ldg(nodeA + node);
            B = __ldg(nodeB + node);
        }
        // A pop of fewer than 32 ranges leaves lanes idle: lane k + i then also takes
        // the second node of range i (its first node's skip pointer), and the rest of
        // the range passes to it. Each range still pushes at most three ranges, within
        // the room k was sized for (2 per popped range).
        bool second = false;
        if (k < 32) {
            const int src = lane >= k ? lane - k : lane;
            const int nxt = __shfl_sync(0xffffffffu, B.y, src);
            const int end = __shfl_sync(0xffffffffu, range.y, src);
            if (lane >= k && src < k && nxt < end) {
                second = true;
                node = nxt;
                range = make_int2(nxt, end);
                A = __ldg(nodeA + node);
                B = __ldg(nodeB + node);
            }
        }
        const unsigned msecond = __ballot_sync(0xffffffffu, second);
        // its rest went to lane + k
        const bool handed = first && lane + k < 32 && ((msecond >> (lane + k)) & 1u);
        const bool have = first || second;
        visits += k + __popc(msecond);
        // Open iff the per-body rule opens for at least one target: some target with
        // nonzero d^2 (targets with d^2 == 0 skip the cell under that rule and do not
        // vote) and theta^2 d^2 < w^2. Settled without a vote: cells accepted even from
        // the nearest point of the targets' box (maybe false) and cells opened even
        // from its farthest corner (sure). Rounding is monotone, so these box bounds
        // never contradict the per-target values. The remaining cells are voted on one
        // at a time: each lane tests its own target, a ballot collects the votes.
        // PT_BH_RELATIVE adds a second opening radius per cell (rr2), tested the same way.
        bool maybe = false, sure = false, monoq = false;
        float w = 0.f, rr2 = 0.f;
        if (have && B.z < 0) {
            w = __int_as_float(B.x);
            if (REL) rr2 = QUAD ? __int_as_float(B.w) * gq : rel_r2<false>(A.w, w, ginv);
            const float e0 = fmaxf(fmaxf(mn0 - A.x, A.x - mx0), 0.f);
            const float e1 = fmaxf(fmaxf(mn1 - A.y, A.y - mx1), 0.f);
            const float e2b = fmaxf(fmaxf(mn2 - A.z, A.z - mx2), 0.f);
            const float emin2 = fmaf(e0, e0, fmaf(e1, e1, e2b * e2b));
            maybe = (LEARNED ? th_in2 : th2) * emin2 < w * w || (REL && emin2 < rr2);
            if (REL && QUAD) monoq = emin2 * emin2 >= A.w * w * w * gmono && gmono > 0.f;
            const float f0 = fmaxf(A.x - mn0, mx0 - A.x);
            const float f1 = fmaxf(A.y - mn1, mx1 - A.y);
            const float f2b = fmaxf(A.z - mn2, mx2 - A.z);
            const float dmax2 = fmaf(f0, f0, fmaf(f1, f1, f2b * f2b));
            // dmax2 > 0: some target is off the centre of mass
            sure = dmax2 > 0.0f && (th2 * dmax2 < w * w || (REL && dmax2 < rr2));
        }
        open = sure;
        bool marginal = false;
        // the cells to vote on are read back from the stack's free slots, two each
        unsigned amb = __ballot_sync(0xffffffffu, maybe && !sure);
        float4 *voted = my.slots(stack + ((S + 1) & ~1));
        if (maybe && !sure) voted[__popc(amb & lt)] = make_float4(A.x, A.y, A.z, w * w);
        __syncwarp();
        for (int v = 0; amb; ++v) {
            const int j = __ffs(amb) - 1;
            amb &= amb - 1;
            const float4 cell = voted[v];
            const float cx = cell.x, cy = cell.y, cz = cell.z, cw2 = cell.w;
            const float crr = REL ? __shfl_sync(0xffffffffu, rr2, j) : 0.f;
            bool o1 = false, i1 = false;
            if constexpr (TPL == 2) {  // both targets in one packed pass (same IEEE ops)
                const f2 dx = sub2(pk2(cx, cx), vx01), dy = sub2(pk2(cy, cy), vy01), dz = sub2(pk2(cz, cz), vz01);
                float d0, d1;
                upk2(fma2(dx, dx, fma2(dy, dy, mul2(dz, dz))), d0, d1);
                o1 = (d0 > 0.0f && (th2 * d0 < cw2 || (REL && d0 < crr))) ||
                     (d1 > 0.0f && (th2 * d1 < cw2 || (REL && d1 < crr)));
                if (LEARNED) i1 = (d0 > 0.0f && th_in2 * d0 < cw2) || (d1 > 0.0f && th_in2 * d1 < cw2);
            } else {
#pragma unroll
                for (int i = 0; i < TPL; ++i) {
                    const float dx = cx - p[i].x, dy = cy - p[i].y, dz = cz - p[i].z;
                    const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                    o1 |= d2 > 0.0f && (th2 * d2 < cw2 || (REL && d2 < crr));
                    if (LEARNED) i1 |= d2 > 0.0f && th_in2 * d2 < cw2;
                }
            }
            const unsigned vo = __ballot_sync(0xffffffffu, o1);
            if (lane == j) open = vo != 0u;
            if (LEARNED) {
                // accepted by every target, but opened by one at theta_inner
                const unsigned vi = __ballot_sync(0xffffffffu, i1);
                if (lane == j) marginal = vo == 0u && vi != 0u && A.w > 0.0f;
            }
        }
        __syncwarp();
        if (LEARNED) {
            const unsigned mm = __ballot_sync(0xffffffffu, marginal);
            const int nm = __popc(mm);
            if (nm && fill + nm > LCHUNK) {
                // pad the current chunk's tail, take the next chunk and link it
                if (chunk >= 0 && chunk < LR.cap)
                    for (int i = fill + lane; i < LCHUNK; i += 32) LR.rec[size_t(chunk) * LCHUNK + i] = -1;
                int nc = 0;
                if (lane == 0) nc = atomicAdd(LR.used, 1);
                nc = __shfl_sync(0xffffffffu, nc, 0);
                if (lane == 0) {
                    if (nc < LR.cap) {
                        LR.chunk_group[nc] = group;
                        LR.next[nc] = -1;
                    } else {
                        atomicOr(err, 2);
                    }
                    if (chunk < 0) LR.head[group] = nc;
                    else if (chunk < LR.cap) LR.next[chunk] = nc;
                }
                chunk = nc;
                fill = 0;
            }
            if (marginal && chunk < LR.cap) LR.rec[size_t(chunk) * LCHUNK + fill + __popc(mm & lt)] = node;
            fill += nm;
            learned += nm;
        }
        const bool rest = have && !handed && B.y < range.y;  // later siblings remain
        // An opened cell with at most GW_FLAT nodes below it is not pushed: the bodies
        // of its leaves go straight to the body list (below). Exact sums instead of its
        // descendants' multipoles, so never less accurate; it saves the pops and votes
        // of the tree's last levels.
        const bool flat = GW_FLAT > 0 && open && B.y - node - 1 <= GW_FLAT;
        const bool kids = open && !flat;
        // each lane's pushes follow those of the lanes below it
        const unsigned mrest = __ballot_sync(0xffffffffu, rest), mopen = __ballot_sync(0xffffffffu, kids);
        int total = __popc(mrest) + __popc(mopen), slot = S;
        if (W > 1) {  // the warps' pushes follow each other
            if (lane == 0) s_push[warp] = total;
            __syncthreads();  // and every warp has read its ranges
            total = 0;
#pragma unroll
            for (int v = 0; v < W; ++v) {
                if (v == warp) slot += total;
                total += s_push[v];
            }
        }
        if (S + total > stack_cap) {
            failed = true;  // never written out of bounds
            break;
        }
        slot += __popc(mrest & lt) + __popc(mopen & lt);
        if (rest) stack[slot++] = make_int2(B.y, range.y);
        if (kids) stack[slot++] = make_int2(node + 1, B.y);  // children on top: popped first
        S += total;
        maxS = max(maxS, S);
        const bool acc = have && !open;
        bool farc = false;
        if (LOCAL && acc && (B.z < 0 || B.w == 1) && A.w != 0.0f) {  // cells and single bodies
            const float dx = A.x - lgx, dy = A.y - lgy, dz = A.z - lgz;
            farc = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > far2;
        }
        if (LOCAL) {
            const unsigned mf = __ballot_sync(0xffffffffu, farc);
            if (mf) {
                // the low bit asks for the cell's quadrupole (not for monopole-only cells)
                const bool farq = farc && B.z < 0 && !monoq;
                if (farc) my.far[Nf + __popc(mf & lt)] = 2 * node + (farq ? 1 : 0);
                if (QUAD) nlocalq += __popc(__ballot_sync(0xffffffffu, farq));
                Nf += __popc(mf);
                nlocal += __popc(mf);
                __syncwarp();
                if (Nf >= 32) {  // the newest 32: one per lane
                    Nf -= 32;
                    local_add_node<QUAD>(my.lx, lane, my.far[Nf + lane], nodeA, nodeQ, lgx, lgy, lgz,
                                         eps2);
                    __syncwarp();
                }
            }
        }
        const bool bucket = acc && B.z >= 0 && B.w > 1;
        const bool cellacc = acc && B.z < 0 && !farc && !monoq;
        // single bodies, and cells whose quadrupole term is negligible (monoq): monopoles
        const bool bodyacc = acc && (B.z >= 0 ? B.w == 1 : monoq) && !farc;
        // accepted cells -> the cell list (with their quadrupoles)
        const unsigned mc = __ballot_sync(0xffffffffu, cellacc);
        const int nc1 = __popc(mc);
        if (Nc + nc1 > CellList::CAP) {
            eval_list<GUARD, TPL>(Lc, Nc, px, py, pz, e2, bsum);
            entries += Nc;
            centries += Nc;
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
        }
        Nc += nc1;
        // accepted single-body leaves -> the body list (monopole only)
        const unsigned mb1 = __ballot_sync(0xffffffffu, bodyacc);
        const int nb1 = __popc(mb1);
        if (Nb + nb1 > BodyList::CAP) {
            eval_list<GUARD, TPL>(Lb, Nb, px, py, pz, e2, bsum);
            entries += Nb;
            Nb = 0;
        }
        if (bodyacc) {
            const int e = Nb + __popc(mb1 & lt);
            Lb.put(0, e, A.x);
            Lb.put(1, e, A.y);
            Lb.put(2, e, A.z);
            Lb.put(3, e, A.w);
        }
        Nb += nb1;
        // bodies [f, f + c) of the key-ordered array -> the body list (warp-uniform f, c)
        auto append_bodies = [&](int f, int c) {
            for (int base = 0; base < c; base += 32) {
                const int n = min(32, c - base);
                if (Nb + n > BodyList::CAP) {
                    eval_list<GUARD, TPL>(Lb, Nb, px, py, pz, e2, bsum);
                    entries += Nb;
                    Nb = 0;
                }
                if (lane < n) {
                    const float4 q = __ldg(sbody + f + base + lane);
                    Lb.put(0, Nb + lane, q.x);
                    Lb.put(1, Nb + lane, q.y);
                    Lb.put(2, Nb + lane, q.z);
                    Lb.put(3, Nb + lane, q.w);
                }
                Nb += n;
            }
        };
        unsigned mb = __ballot_sync(0xffffffffu, bucket);
        while (mb) {  // leaves holding several bodies: one entry per body
            const int src = __ffs(mb) - 1;
            mb &= mb - 1;
            append_bodies(__shfl_sync(0xffffffffu, B.z, src), __shfl_sync(0xffffffffu, B.w, src));
        }
        // Small opened subtrees, all of this pop's at once: their nodes are numbered
        // across the warp (a prefix sum of the subtrees' sizes) and loaded 32 at a
        // time, one per lane; the leaves' bodies go to the body list.
        if (GW_FLAT > 0 && __any_sync(0xffffffffu, flat)) {
            const int fcnt = flat ? B.y - node - 1 : 0;
            int fincl = fcnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, fincl, o);
                if (lane >= o) fincl += t;
            }
            const int ftot = __shfl_sync(0xffffffffu, fincl, 31);
            visits += ftot;
            for (int fb = 0; fb < ftot; fb += 32) {
                const int j = fb + lane;
                // the subtree holding node j: the number of lanes whose prefix ends at or before j
                int o = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1) {
                    const int v = __shfl_sync(0xffffffffu, fincl, o + step - 1);
                    if (v <= j) o += step;
                }
                o = min(o, 31);
                const int first = __shfl_sync(0xffffffffu, node, o) + 1;
                const int before = __shfl_sync(0xffffffffu, fincl, o) - __shfl_sync(0xffffffffu, fcnt, o);
                const int nd = first + j - before;
                int4 lb = make_int4(0, 0, -1, 0);
                float4 la = make_float4(0.f, 0.f, 0.f, 0.f);
                if (j < ftot) lb = __ldg(nodeB + nd);
                const bool one = lb.z >= 0 && lb.w == 1;  // a single-body leaf: its record is the body
                if (one) la = __ldg(nodeA + nd);
                const unsigned m1 = __ballot_sync(0xffffffffu, one);
                const int n1 = __popc(m1);
                if (Nb + n1 > BodyList::CAP) {
                    eval_list<GUARD, TPL>(Lb, Nb, px, py, pz, e2, bsum);
                    entries += Nb;
                    Nb = 0;
                }
                if (one) {
                    const int e = Nb + __popc(m1 & lt);
                    Lb.put(0, e, la.x);
                    Lb.put(1, e, la.y);
                    Lb.put(2, e, la.z);
                    Lb.put(3, e, la.w);
                }
                Nb += n1;
                unsigned mm = __ballot_sync(0xffffffffu, lb.z >= 0 && lb.w > 1);
                while (mm) {
                    const int s2 = __ffs(mm) - 1;
                    mm &= mm - 1;
                    append_bodies(__shfl_sync(0xffffffffu, lb.z, s2), __shfl_sync(0xffffffffu, lb.w, s2));
                }
            }
        }
        team_sync<W>();  // the pushes
    }
    eval_list<GUARD, TPL>(Lc, Nc, px, py, pz, e2, bsum);
    eval_list<GUARD, TPL>(Lb, Nb, px, py, pz, e2, bsum);
    entries += Nc + Nb;
    centries += Nc;
    float rx[TPL], ry[TPL], rz[TPL];
    float lx[TPL], ly[TPL], lz[TPL];  // the local expansion's share
#pragma unroll
    for (int i = 0; i < TPL; ++i) lx[i] = ly[i] = lz[i] = 0.f;
    if (LOCAL) {
        if (lane < Nf) local_add_node<QUAD>(my.lx, lane, my.far[lane], nodeA, nodeQ, lgx, lgy, lgz, eps2);
        __syncwarp();
        LocalExp LX;
        float *lf = &LX.ax;
#pragma unroll
        for (int k = 0; k < 19; ++k) lf[k] = my.lx[k][lane];
        local_reduce(LX);
#pragma unroll
        for (int i = 0; i < TPL; ++i)
            local_eval(LX, p[i].x - lgx, p[i].y - lgy, p[i].z - lgz, lx[i], ly[i], lz[i]);
    }
    if (W > 1) {  // the warps' compensated sums and expansions, added up in warp order
        float (*x)[9 * TPL][32] = reinterpret_cast<float (*)[9 * TPL][32]>(s_warp);
        static_assert(sizeof(float) * 9 * TPL * 32 <= sizeof(Shared), "the lists' space holds a warp's sums");
        float v[TPL][9];
#pragma unroll
        for (int i = 0; i < TPL; ++i) {
            bsum.parts(i, v[i]);
            v[i][6] = lx[i], v[i][7] = ly[i], v[i][8] = lz[i];
        }
        __syncthreads();  // every warp is done with its lists
#pragma unroll
        for (int i = 0; i < TPL; ++i)
#pragma unroll
            for (int q = 0; q < 9; ++q) x[warp][9 * i + q][lane] = v[i][q];
        __syncthreads();
        if (warp == 0)
#pragma unroll
            for (int i = 0; i < TPL; ++i) {
#pragma unroll
                for (int u = 1; u < W; ++u)
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        two_sum_acc(v[i][a], v[i][3 + a], x[u][9 * i + a][lane]);
                        v[i][3 + a] += x[u][9 * i + 3 + a][lane];
                        v[i][6 + a] += x[u][9 * i + 6 + a][lane];
                    }
                lx[i] = v[i][6], ly[i] = v[i][7], lz[i] = v[i][8];
            }
#pragma unroll
        for (int i = 0; i < TPL; ++i) rx[i] = v[i][0] + v[i][3], ry[i] = v[i][1] + v[i][4], rz[i] = v[i][2] + v[i][5];
    } else {
#pragma unroll
        for (int i = 0; i < TPL; ++i) bsum.total(i, rx[i], ry[i], rz[i]);
    }
    if (LOCAL)
#pragma unroll
        for (int i = 0; i < TPL; ++i) rx[i] += lx[i], ry[i] += ly[i], rz[i] += lz[i];
    const unsigned long long nv = unsigned(nvalid);
    unsigned long long s_acc = entries * nv, s_vis = visits * nv, s_cell = centries * nv;
    if (failed) {
        // The stack ran out (failed is uniform): the targets take the reference's per-body
        // walk instead, which needs no stack.
        if (W > 1 && warp != 0) return;
        unsigned na = 0, nvis = 0, nc = 0;
#pragma unroll
        for (int i = 0; i < TPL; ++i) {
            rx[i] = ry[i] = rz[i] = 0.f;
            lane_walk<QUAD>(p[i], valid[i], T, nodeA, nodeB, nodeQ, sbody, th2, eps2, rx[i], ry[i], rz[i], na, nvis,
                            nc, REL ? gscale[group] : 0.f);
        }
        unsigned long long a = na, v = nvis, c = nc;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            v += __shfl_xor_sync(0xffffffffu, v, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        s_acc = a;
        s_vis = v;
        s_cell = c;
    }
    if (LEARNED) {
        if (chunk >= 0 && chunk < LR.cap)
            for (int i = fill + lane; i < LCHUNK; i += 32) LR.rec[size_t(chunk) * LCHUNK + i] = -1;
        if (lane == 0) {
            if (chunk < 0 || failed) LR.head[group] = -1;  // a fallback warp keeps the plain result
            LR.centre[group] = make_float4(gcx, gcy, gcz, 0.f);
        }
    }
#pragma unroll
    for (int i = 0; i < TPL; ++i)
        if (valid[i] && warp == 0) {
            const uint32_t o = tidx[g0 + 32 * i + lane];
            out[3 * size_t(o) + 0] = rx[i];
            out[3 * size_t(o) + 1] = ry[i];
            out[3 * size_t(o) + 2] = rz[i];
        }
    if (stats && lane == 0) {
        atomicAdd(stats + 0, s_acc);
        atomicAdd(stats + 1, s_vis);
        if (LEARNED) atomicAdd(stats + 4, learned);
        if (LOCAL && !failed) {
            atomicAdd(stats + 7, nlocal);
            if (QUAD) atomicAdd(stats + 8, nlocalq);
        }
        atomicAdd(stats + 5, s_cell);
        if (warp == 0) atomicAdd(stats + 2, 1ull);
        atomicMax(stats + 3, (unsigned long long)maxS);
        if (failed) atomicAdd(stats + 6, 1ull);
    }
}

using GroupKernel = void (*)(const float4 *, const uint32_t *, int, const float4 *, const int4 *, const float4 *,
                             const float4 *, const float4 *, const int *, float, float, LearnedRecords, float,
                             float *, unsigned long long *, int *, int, float, const float *, float, const int *);

template <bool LEARNED, bool LOCAL, bool REL, int W>
inline GroupKernel group_kernel_q(bool quad, bool guard) {
    if (quad)
        return guard ? bh_walk_group<true, true, LEARNED, LOCAL, REL, W> : bh_walk_group<true, false, LEARNED, LOCAL, REL, W>;
    return guard ? bh_walk_group<false, true, LEARNED, LOCAL, REL, W> : bh_walk_group<false, false, LEARNED, LOCAL, REL, W>;
}

template <int W>
inline GroupKernel group_kernel_w(bool quad, bool guard, bool local, bool rel) {
    if (local)
        return rel ? group_kernel_q<false, true, true, W>(quad, guard) : group_kernel_q<false, true, false, W>(quad, guard);
    return rel ? group_kernel_q<false, false, true, W>(quad, guard) : group_kernel_q<false, false, false, W>(quad, guard);
}

// The kernels of 4 and 8 warps per group (pt_bh_team.cu).
GroupKernel group_kernel_team(bool quad, bool guard, bool local, bool rel, int team);

}  // namespace bh
}  // namespace pt
