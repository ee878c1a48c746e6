// ge_gwalk.cu -- the group walk of the mixed-precision mode.
//
// No counterpart in the reference: its walk (physics.cpp:91-205,
// physics3D.cpp:131-253) is one traversal per particle.  Here one warp walks
// the tree once for a group of at most GS = 32 x PPL particles that share a
// small cell of the tree (k_make_groups):
//   * the group's bounding box decides the opening test for all of them: a
//     node is accepted when b^2 < dmin^2 + eps2, dmin the distance from its
//     centre of mass to the box and b the node's opening radius (ge_moments.cu),
//     which is at least as strict as every member's own test;
//   * up to 32 candidate nodes are tested at once, one per lane, taken from a
//     per-warp work stack in shared memory (moved to the warp's stack in
//     global memory when it outgrows it);
//   * accepted nodes (centre of mass, mass, second moments) and the
//     particles of opened leaves are staged in shared memory and, when a list
//     fills up or the walk ends, every lane evaluates them for its own
//     particles (monopole + softened quadrupole for nodes, the softened pair
//     force for particles; the particle itself is skipped);
//   * each lane sums a list pass in FP32 and adds that sum to its running
//     total with Kahan compensation.
// What bounds it: the FP32 pipe.  A node costs 31 packed instructions for two
// particles of a lane in 3D (21 in 2D), a leaf particle 12 (9); an FMA of three
// fresh registers issues every 1.7 cycles, the packed one every 3.0 (1.0 and
// 2.0 with one of them reused), so packing pays by halving the other issue
// slots.  Measured against one scalar particle at a time, 128 particles to a
// warp, single leaves staged one by one (walk stage, 3D theta 0.5 groups of
// 128 and 2D theta 0.7 groups of 64): 1M 3D 7.01 -> 6.24 ms, 262k 4.54 -> 2.48,
// 30k 0.84 -> 0.42; 1M 2D 0.551 -> 0.475 ms, 100k 0.126 -> 0.078.  Rejected:
// all four particles of a 128-group in one warp (1M 3D 6.17 ms, 262k 2.72, 30k
// 0.58: one traversal less, half the warps).
// Which nodes a particle interacts with depends only on its group, not on the
// traversal order, so the interaction set is deterministic; only the FP32
// summation order within a list pass follows the traversal.
#include <cfloat>
#include <type_traits>

#include "ge_bh.h"
#include "ge_device.cuh"
#include "ge_internal.h"

namespace ge {

constexpr int kGWWarps = 4;
constexpr int kGWThreads = kGWWarps * 32;
constexpr int kGWNodes = 64;           // staged accepted nodes per warp
constexpr int kGWParts = 64;           // staged leaf particles per warp
// sources per trip of the packed loops: independent chains (a lone warp at the
// end of a launch waits on its own latency), in the registers of four blocks
constexpr int kUnroll = 4;
constexpr uint32_t kGWStack = 2048;    // work stack entries per warp (global memory)
// the work stack lives in shared memory while it fits (the deepest measured
// stacks: ~170 entries in 2D, ~800 in 3D at theta 0.5, ~1400 at theta 0.3)
// and moves to the warp's global stack when it would not (with 768 entries the
// deepest 3D walks at theta 0.5 do; 1024 take the same time: 4M 22.38 / 22.39 ms)
template <int D> struct GWShared { static constexpr uint32_t value = D == 2 ? 256u : 768u; };
constexpr int kMetaGroupCtr = 10;      // tree meta word: next group to walk
constexpr int kMetaGroupCount = 11;    // tree meta word: groups made
constexpr int kMetaSlotsW = 9;         // tree meta word: node slots of the last build

// A staged accepted node: c = (hi - o) + lo, its centre of mass from the
// group's centre o; J = 7.5 I, its second moments; t = -1.5 tr(I).  With DUP
// (two particles per lane) every value is stored twice, so that one 16-byte
// load brings two operands of the packed arithmetic.
template <int D, bool DUP> struct GWSmem;
template <>
struct GWSmem<2, false> {
    float4 nA[kGWNodes];   // {c.x, c.y, m, Jxx}
    float4 nB[kGWNodes];   // {Jxy, Jyy, t, 0}
    float4 pA[kGWParts];   // {x - o, m}
    uint32_t pI[kGWParts]; // particle slot
};
template <>
struct GWSmem<3, false> {
    float4 nA[kGWNodes];   // {c.x, c.y, c.z, m}
    float4 nB[kGWNodes];   // {Jxx, Jyz, t, 0}
    float4 nC[kGWNodes];   // {Jyy, Jzz, Jxy, Jxz}
    float4 pA[kGWParts];
    uint32_t pI[kGWParts];
};
template <>
struct GWSmem<2, true> {
    float4 n[3][kGWNodes];   // pairs (c.x, c.y), (m, t), (Jxx, Jxy)
    float2 n1[kGWNodes];     // pair Jyy
    float4 p[1][kGWParts];   // pairs (x - o, y - o)
    float2 p1[kGWParts];     // pair m
    uint32_t pI[kGWParts];
};
template <>
struct GWSmem<3, true> {
    float4 n[5][kGWNodes];   // pairs (c.x, c.y), (c.z, m), (Jxx, Jxy), (Jxz, Jyy), (Jyz, Jzz)
    float2 n1[kGWNodes];     // pair t
    float4 p[2][kGWParts];   // pairs (x - o, y - o), (z - o, m)
    uint32_t pI[kGWParts];
};

__device__ __forceinline__ float4 dup2(float a, float b) { return make_float4(a, a, b, b); }

struct GWNode {
    float c[3], m, jxx, jxy, jxz, jyy, jyz, jzz, t;
};

template <int D, bool DUP>
__device__ __forceinline__ void put_node(GWSmem<D, DUP> &sm, int q, const GWNode &v) {
    if constexpr (DUP && D == 2) {
        sm.n[0][q] = dup2(v.c[0], v.c[1]);
        sm.n[1][q] = dup2(v.m, v.t);
        sm.n[2][q] = dup2(v.jxx, v.jxy);
        sm.n1[q] = make_float2(v.jyy, v.jyy);
    } else if constexpr (DUP) {
        sm.n[0][q] = dup2(v.c[0], v.c[1]);
        sm.n[1][q] = dup2(v.c[2], v.m);
        sm.n[2][q] = dup2(v.jxx, v.jxy);
        sm.n[3][q] = dup2(v.jxz, v.jyy);
        sm.n[4][q] = dup2(v.jyz, v.jzz);
        sm.n1[q] = make_float2(v.t, v.t);
    } else if constexpr (D == 2) {
        sm.nA[q] = make_float4(v.c[0], v.c[1], v.m, v.jxx);
        sm.nB[q] = make_float4(v.jxy, v.jyy, v.t, 0.0f);
    } else {
        sm.nA[q] = make_float4(v.c[0], v.c[1], v.c[2], v.m);
        sm.nB[q] = make_float4(v.jxx, v.jyz, v.t, 0.0f);
        sm.nC[q] = make_float4(v.jyy, v.jzz, v.jxy, v.jxz);
    }
}

template <int D, bool DUP>
__device__ __forceinline__ GWNode get_node(const GWSmem<D, DUP> &sm, int j) {
    GWNode v;
    if constexpr (DUP && D == 2) {
        const float4 a = sm.n[0][j], b = sm.n[1][j], c = sm.n[2][j];
        v = GWNode{{a.x, a.z, 0.0f}, b.x, c.x, c.z, 0.0f, sm.n1[j].x, 0.0f, 0.0f, b.z};
    } else if constexpr (DUP) {
        const float4 a = sm.n[0][j], b = sm.n[1][j], c = sm.n[2][j], d = sm.n[3][j],
                     e = sm.n[4][j];
        v = GWNode{{a.x, a.z, b.x}, b.z, c.x, c.z, d.x, d.z, e.x, e.z, sm.n1[j].x};
    } else if constexpr (D == 2) {
        const float4 a = sm.nA[j], b = sm.nB[j];
        v = GWNode{{a.x, a.y, 0.0f}, a.z, a.w, b.x, 0.0f, b.y, 0.0f, 0.0f, b.z};
    } else {
        const float4 a = sm.nA[j], b = sm.nB[j], c = sm.nC[j];
        v = GWNode{{a.x, a.y, a.z}, a.w, b.x, c.z, c.w, c.x, b.y, c.y, b.z};
    }
    return v;
}

template <int D, bool DUP>
__device__ __forceinline__ void put_part(GWSmem<D, DUP> &sm, int q, float x, float y, float z,
                                         float m, uint32_t slot) {
    if constexpr (DUP && D == 2) {
        sm.p[0][q] = dup2(x, y);
        sm.p1[q] = make_float2(m, m);
    } else if constexpr (DUP) {
        sm.p[0][q] = dup2(x, y);
        sm.p[1][q] = dup2(z, m);
    } else {
        sm.pA[q] = make_float4(x, y, z, m);
    }
    sm.pI[q] = slot;
}

template <int D, bool DUP>
__device__ __forceinline__ float4 get_part(const GWSmem<D, DUP> &sm, int j) {
    if constexpr (DUP && D == 2) {
        const float4 a = sm.p[0][j];
        return make_float4(a.x, a.z, 0.0f, sm.p1[j].x);
    } else if constexpr (DUP) {
        const float4 a = sm.p[0][j], b = sm.p[1][j];
        return make_float4(a.x, a.z, b.x, b.z);
    } else {
        return sm.pA[j];
    }
}

__device__ __forceinline__ float rsqrt_fast(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <int PPL>
struct GroupState {
    float x[PPL][3];
    float f[PPL][3], fc[PPL][3];   // running sums and their Kahan compensation
    float u[PPL], uc[PPL];         // potential pass: sum of m / r terms (phi = -G u)
    uint32_t idx[PPL];
    bool act[PPL];
    unsigned long long count;
};

// accepted nodes for the first NK of a lane's particles: monopole +
// quadrupole of the softened kernel (with POT, the potential instead:
// M / r + 1.5 (d.I.d) / r^5 - 0.5 tr(I) / r^3).  The moments are staged as
// J = 7.5 I with t = -1.5 tr(I), so that
//   a = (M / r^3 + (d.J.d / r^2 + t) / r^5) d - 0.4 (J d) / r^5.
template <int D, int NK, int PPL, bool DUP, bool POT>
__device__ __forceinline__ void flush_nodes(const GWSmem<D, DUP> &sm, int nl, GroupState<PPL> &g,
                                            float eps2, bool count) {
    float acc[NK][3], pu[NK];
#pragma unroll
    for (int k = 0; k < NK; k++) {
        pu[k] = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; a++) acc[k][a] = 0.0f;
    }
    for (int j = 0; j < nl; j++) {
        const GWNode v = get_node(sm, j);
#pragma unroll
        for (int k = 0; k < NK; k++) {
            float d[3];
            d[0] = v.c[0] - g.x[k][0];
            d[1] = v.c[1] - g.x[k][1];
            d[2] = D == 3 ? v.c[2] - g.x[k][2] : 0.0f;
            float rr = __fmaf_rn(d[1], d[1], eps2);
            if (D == 3) rr = __fmaf_rn(d[2], d[2], rr);
            rr = __fmaf_rn(d[0], d[0], rr);
            const float inv = rsqrt_fast(rr);
            const float inv2 = inv * inv, inv3 = inv2 * inv, inv5 = inv3 * inv2;
            float Jd[3];
            if (D == 2) {
                Jd[0] = __fmaf_rn(v.jxx, d[0], v.jxy * d[1]);
                Jd[1] = __fmaf_rn(v.jxy, d[0], v.jyy * d[1]);
                Jd[2] = 0.0f;
            } else {
                Jd[0] = __fmaf_rn(v.jxx, d[0], __fmaf_rn(v.jxy, d[1], v.jxz * d[2]));
                Jd[1] = __fmaf_rn(v.jxy, d[0], __fmaf_rn(v.jyy, d[1], v.jyz * d[2]));
                Jd[2] = __fmaf_rn(v.jxz, d[0], __fmaf_rn(v.jyz, d[1], v.jzz * d[2]));
            }
            float dJd = __fmaf_rn(d[1], Jd[1], d[0] * Jd[0]);
            if (D == 3) dJd = __fmaf_rn(d[2], Jd[2], dJd);
            if (POT) {   // 1.5 d.I.d = 0.2 d.J.d, -0.5 tr = t / 3
                pu[k] += v.m * inv + 0.2f * dJd * inv5 + (v.t * (1.0f / 3.0f)) * inv3;
                continue;
            }
            const float q = __fmaf_rn(dJd, inv2, v.t);
            const float cm = __fmaf_rn(q, inv5, v.m * inv3);
            const float ci = -0.4f * inv5;
#pragma unroll
            for (int a = 0; a < D; a++) acc[k][a] = __fmaf_rn(ci, Jd[a], __fmaf_rn(cm, d[a], acc[k][a]));
        }
    }
#pragma unroll
    for (int k = 0; k < NK; k++) {
        if (POT) kahan_add(g.u[k], g.uc[k], pu[k]);
#pragma unroll
        for (int a = 0; a < D; a++)
            if (!POT) kahan_add(g.f[k][a], g.fc[k][a], acc[k][a]);
        if (count && g.act[k]) g.count += (unsigned long long)nl;
    }
}

// particles of opened leaves: the softened pair force (with POT, m / r), the
// particle itself skipped
template <int D, int NK, int PPL, bool DUP, bool POT>
__device__ __forceinline__ void flush_parts(const GWSmem<D, DUP> &sm, int pl, GroupState<PPL> &g,
                                            float eps2, bool count) {
    float acc[NK][3], pu[NK];
    uint32_t self_hits = 0;
#pragma unroll
    for (int k = 0; k < NK; k++) {
        pu[k] = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; a++) acc[k][a] = 0.0f;
    }
    if (!POT && !count && eps2 > 0.0f) {
        // the particle's own term is exactly zero (d = 0: its staged offset
        // is its own offset, bit for bit), so no pair needs the test
        for (int j = 0; j < pl; j++) {
            const float4 P = get_part(sm, j);
#pragma unroll
            for (int k = 0; k < NK; k++) {
                float d[3];
                d[0] = P.x - g.x[k][0];
                d[1] = P.y - g.x[k][1];
                d[2] = D == 3 ? P.z - g.x[k][2] : 0.0f;
                float rr = __fmaf_rn(d[1], d[1], eps2);
                if (D == 3) rr = __fmaf_rn(d[2], d[2], rr);
                rr = __fmaf_rn(d[0], d[0], rr);
                const float inv = rsqrt_fast(rr);
                const float fm = P.w * (inv * inv * inv);
#pragma unroll
                for (int a = 0; a < D; a++) acc[k][a] = __fmaf_rn(d[a], fm, acc[k][a]);
            }
        }
    } else
    for (int j = 0; j < pl; j++) {
        const float4 P = get_part(sm, j);
        const uint32_t pj = sm.pI[j];
#pragma unroll
        for (int k = 0; k < NK; k++) {
            float d[3];
            d[0] = P.x - g.x[k][0];
            d[1] = P.y - g.x[k][1];
            d[2] = D == 3 ? P.z - g.x[k][2] : 0.0f;
            float rr = d[0] * d[0] + d[1] * d[1] + eps2;
            if (D == 3) rr += d[2] * d[2];
            const float inv = rsqrt_fast(rr);
            const bool self = pj == g.idx[k];
            self_hits += (self && g.act[k]) ? 1u : 0u;
            if (POT) {
                pu[k] += self ? 0.0f : P.w * inv;
                continue;
            }
            const float fm = self ? 0.0f : P.w * (inv * inv * inv);
#pragma unroll
            for (int a = 0; a < D; a++) acc[k][a] += d[a] * fm;
        }
    }
#pragma unroll
    for (int k = 0; k < NK; k++) {
        if (POT) kahan_add(g.u[k], g.uc[k], pu[k]);
#pragma unroll
        for (int a = 0; a < D; a++)
            if (!POT) kahan_add(g.f[k][a], g.fc[k][a], acc[k][a]);
        if (count && g.act[k]) g.count += (unsigned long long)pl;
    }
    if (count) g.count -= self_hits;
}

// The same two passes for both particles of a lane in packed arithmetic
// (f32x2: one instruction, two roundings, each as the scalar one's), so every
// result is the scalar passes' bit for bit.
template <int D>
__device__ __forceinline__ void flush_nodes_x2(const GWSmem<D, true> &sm, int nl,
                                               GroupState<2> &g, float eps2) {
    f32x2 nx[D], acc[D];
#pragma unroll
    for (int a = 0; a < D; a++) {
        nx[a] = pack2(-g.x[0][a], -g.x[1][a]);
        acc[a] = pack2(0.0f, 0.0f);
    }
    const f32x2 e2 = pack2(eps2, eps2), m04 = pack2(-0.4f, -0.4f);
#pragma unroll kUnroll
    for (int j = 0; j < nl; j++) {
        f32x2 d[D], Jd[D], m, t;
        const ulonglong2 v0 = *reinterpret_cast<const ulonglong2 *>(&sm.n[0][j]);
        const ulonglong2 v1 = *reinterpret_cast<const ulonglong2 *>(&sm.n[1][j]);
        const ulonglong2 v2 = *reinterpret_cast<const ulonglong2 *>(&sm.n[2][j]);
        const f32x2 w = *reinterpret_cast<const f32x2 *>(&sm.n1[j]);
        d[0] = add2(v0.x, nx[0]);
        d[1] = add2(v0.y, nx[1]);
        f32x2 rr = fma2(d[1], d[1], e2);
        if constexpr (D == 3) {
            d[2] = add2(v1.x, nx[2]);
            rr = fma2(d[2], d[2], rr);
        }
        rr = fma2(d[0], d[0], rr);
        float r0, r1;
        unpack2(rr, r0, r1);
        const f32x2 inv = pack2(rsqrt_fast(r0), rsqrt_fast(r1));
        const f32x2 inv2 = mul2(inv, inv), inv3 = mul2(inv2, inv), inv5 = mul2(inv3, inv2);
        if constexpr (D == 2) {
            m = v1.x; t = v1.y;
            Jd[0] = fma2(v2.x, d[0], mul2(v2.y, d[1]));
            Jd[1] = fma2(v2.y, d[0], mul2(w, d[1]));
        } else {
            const ulonglong2 v3 = *reinterpret_cast<const ulonglong2 *>(&sm.n[3][j]);
            const ulonglong2 v4 = *reinterpret_cast<const ulonglong2 *>(&sm.n[4][j]);
            m = v1.y; t = w;
            Jd[0] = fma2(v2.x, d[0], fma2(v2.y, d[1], mul2(v3.x, d[2])));
            Jd[1] = fma2(v2.y, d[0], fma2(v3.y, d[1], mul2(v4.x, d[2])));
            Jd[2] = fma2(v3.x, d[0], fma2(v4.x, d[1], mul2(v4.y, d[2])));
        }
        f32x2 dJd = fma2(d[1], Jd[1], mul2(d[0], Jd[0]));
        if constexpr (D == 3) dJd = fma2(d[2], Jd[2], dJd);
        const f32x2 q = fma2(dJd, inv2, t);
        const f32x2 cm = fma2(q, inv5, mul2(m, inv3));
        const f32x2 ci = mul2(m04, inv5);
#pragma unroll
        for (int a = 0; a < D; a++) acc[a] = fma2(ci, Jd[a], fma2(cm, d[a], acc[a]));
    }
#pragma unroll
    for (int a = 0; a < D; a++) {
        float s0, s1;
        unpack2(acc[a], s0, s1);
        kahan_add(g.f[0][a], g.fc[0][a], s0);
        kahan_add(g.f[1][a], g.fc[1][a], s1);
    }
}

// eps2 > 0 (no self test, as in flush_parts)
template <int D>
__device__ __forceinline__ void flush_parts_x2(const GWSmem<D, true> &sm, int pl,
                                               GroupState<2> &g, float eps2) {
    f32x2 nx[D], acc[D];
#pragma unroll
    for (int a = 0; a < D; a++) {
        nx[a] = pack2(-g.x[0][a], -g.x[1][a]);
        acc[a] = pack2(0.0f, 0.0f);
    }
    const f32x2 e2 = pack2(eps2, eps2);
#pragma unroll kUnroll
    for (int j = 0; j < pl; j++) {
        f32x2 d[D], m;
        const ulonglong2 v0 = *reinterpret_cast<const ulonglong2 *>(&sm.p[0][j]);
        d[0] = add2(v0.x, nx[0]);
        d[1] = add2(v0.y, nx[1]);
        f32x2 rr = fma2(d[1], d[1], e2);
        if constexpr (D == 3) {
            const ulonglong2 v1 = *reinterpret_cast<const ulonglong2 *>(&sm.p[1][j]);
            d[2] = add2(v1.x, nx[2]);
            rr = fma2(d[2], d[2], rr);
            m = v1.y;
        } else {
            m = *reinterpret_cast<const f32x2 *>(&sm.p1[j]);
        }
        rr = fma2(d[0], d[0], rr);
        float r0, r1;
        unpack2(rr, r0, r1);
        const f32x2 inv = pack2(rsqrt_fast(r0), rsqrt_fast(r1));
        const f32x2 fm = mul2(m, mul2(mul2(inv, inv), inv));
#pragma unroll
        for (int a = 0; a < D; a++) acc[a] = fma2(d[a], fm, acc[a]);
    }
#pragma unroll
    for (int a = 0; a < D; a++) {
        float s0, s1;
        unpack2(acc[a], s0, s1);
        kahan_add(g.f[0][a], g.fc[0][a], s0);
        kahan_add(g.f[1][a], g.fc[1][a], s1);
    }
}

// The staged lists for a lane's particles: nk (warp-uniform) of them are in
// use, one when the item holds at most 32 particles.
template <int D, int PPL, bool DUP, bool COUNT, bool POT>
__device__ __forceinline__ void eval_nodes(const GWSmem<D, DUP> &sm, int nl, GroupState<PPL> &g,
                                           float eps2, int nk) {
    if constexpr (PPL == 2) {
        if (nk == 2) {
            if constexpr (!COUNT && !POT) flush_nodes_x2<D>(sm, nl, g, eps2);
            else flush_nodes<D, 2, 2, DUP, POT>(sm, nl, g, eps2, COUNT);
            return;
        }
    }
    flush_nodes<D, 1, PPL, DUP, POT>(sm, nl, g, eps2, COUNT);
}
template <int D, int PPL, bool DUP, bool COUNT, bool POT>
__device__ __forceinline__ void eval_parts(const GWSmem<D, DUP> &sm, int pl, GroupState<PPL> &g,
                                           float eps2, int nk) {
    if constexpr (PPL == 2) {
        if (nk == 2) {
            if constexpr (!COUNT && !POT) {
                if (eps2 > 0.0f) {
                    flush_parts_x2<D>(sm, pl, g, eps2);
                    return;
                }
            }
            flush_parts<D, 2, 2, DUP, POT>(sm, pl, g, eps2, COUNT);
            return;
        }
    }
    flush_parts<D, 1, PPL, DUP, POT>(sm, pl, g, eps2, COUNT);
}

// Groups: every particle belongs to exactly one node that holds at most GS
// particles while its parent holds more (or that is its simulation's root);
// runs of such nodes that are adjacent children of one parent are packed
// into one group while the run holds at most GS particles.  A group is then
// a contiguous particle range inside one cell (its parent's), so its
// bounding box stays compact.  A leaf of more than GS particles (a cell at
// the minimum size) is cut into GS-particle pieces.  A sparse child (below)
// is split down its subtree instead.  The groups depend only on the tree, so
// a simulation forms the same groups alone and in a batch.
__device__ __forceinline__ void emit_group(const Tree &t, uint32_t a, uint32_t b) {
    const uint32_t k = atomicAdd(&t.meta[kMetaGroupCount], 1u);
    t.grp[k] = make_uint2(a, b);
}

// A node of c particles and cell size s is sparse, relative to a parent of
// C particles and size S, when its particles' mean spacing is more than four
// times the parent's: (s / S)^D C > 4^D c.  A group made of it would have a
// box far larger than the matter around it warrants (halo and tidal-tail
// particles in a cell beside a dense disk: one such group of 57 particles
// spread over 6 x 10 units opened ~11,000 particles for every member and
// held one warp for 3.5 ms), so it is split down its subtree, depth first
// with a stack of 256 entries, into nodes dense enough by the same reference,
// or leaves (the node whole when the stack is full).
template <int D>
__device__ __forceinline__ bool sparse_node(float s, uint32_t c, float S, uint32_t C) {
    const double r = (double)s / (double)S;
    const double rd = D == 2 ? r * r : r * r * r;
    return rd * (double)C > (D == 2 ? 16.0 : 64.0) * (double)c;
}

template <int D>
__device__ void emit_split(const Tree &t, uint32_t node, float S, uint32_t C) {
    constexpr int kStack = 256;
    uint32_t stack[kStack];
    int top = 0;
    stack[top++] = node;
    while (top > 0) {
        const uint32_t k = stack[--top];
        const uint4 inf = __ldcg(&t.info[k]);
        if (inf.w <= inf.z) continue;
        const int nc = __popc(inf.y);
        // a leaf, a node dense enough, or (stack full) the node whole
        if (!inf.y || !sparse_node<D>(__ldcg(&t.cell[k]).w, inf.w - inf.z, S, C) ||
            top + nc > kStack) {
            emit_group(t, inf.z, inf.w);
            continue;
        }
        for (int q = nc - 1; q >= 0; q--) stack[top++] = inf.x + (uint32_t)q;
    }
}

template <int D>
__global__ void k_make_groups(Tree t, uint32_t GS) {
    dep_wait();
    const uint32_t slots = __ldcg(&t.meta[kMetaSlotsW]);
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < slots; k += stride) {
        const uint4 inf = __ldcg(&t.info[k]);
        if (inf.w <= inf.z) continue;   // hole
        const uint32_t cnt = inf.w - inf.z;
        if (cnt <= GS) {
            if (__ldcg(&t.aux[k]).z == kEmpty) emit_group(t, inf.z, inf.w);   // a small root
            continue;
        }
        if (!inf.y) {   // a leaf larger than a group
            for (uint32_t a = inf.z; a < inf.w; a += GS) emit_group(t, a, min(a + GS, inf.w));
            continue;
        }
        const int nc = __popc(inf.y);
        const float S = __ldcg(&t.cell[k]).w;
        uint32_t ra = 0, rb = 0;   // current run of small adjacent children
        for (int c = 0; c < nc; c++) {
            const uint32_t ck = inf.x + (uint32_t)c;
            const uint4 ci = __ldcg(&t.info[ck]);
            const uint32_t cc = ci.w - ci.z;
            if (cc > GS) {
                if (rb > ra) emit_group(t, ra, rb);
                ra = rb = 0;
                continue;
            }
            if (ci.y && sparse_node<D>(__ldcg(&t.cell[ck]).w, cc, S, cnt)) {
                if (rb > ra) emit_group(t, ra, rb);
                ra = rb = 0;
                emit_split<D>(t, ck, S, cnt);
                continue;
            }
            if (rb > ra && rb == ci.z && (ci.w - ra) <= GS) {
                rb = ci.w;
            } else {
                if (rb > ra) emit_group(t, ra, rb);
                ra = ci.z;
                rb = ci.w;
            }
        }
        if (rb > ra) emit_group(t, ra, rb);
    }
}

// One particle per lane: how the walk hides its latency.  Small launches load
// the next candidates ahead, in the registers of four blocks per SM; from some
// 200,000 particles on six blocks per SM hide more, which have no registers for
// that and stage a round's nodes before its children are pushed (BUSY).  Walk of
// groups of 32 (us, ahead / BUSY): 3D theta 0.7 10k 172 / 199, 100k 500 / 524, 200k
// 868 / 829, 500k 1966 / 1772, 1M 3855 / 3446, 2D 60k 61 / 69, 200k 139 / 137, 1M 574 /
// 549.
constexpr int kBusyGroups = 200000;
static bool gw_busy(int n) { return n >= kBusyGroups; }

// GSC: the group size in 32-particle chunks.  A work item is PPL = min(GSC, 2)
// of a group's chunks: every item of a group takes the whole group's box, so
// it meets the same sources in the same order as one warp that walked for all
// of them would, and an item without particles is passed over.
template <int D, int GSC, bool COUNT, bool POT = false, bool BUSY = false>
__global__ void __launch_bounds__(kGWThreads, BUSY ? 6 : 4)
k_group_walk(State s, StepParams p, Segs sg_tab, Tree t, int integrate_end,
             unsigned long long *inter, uint32_t *err, double *epot = nullptr) {
    dep_wait();
    constexpr int PPL = GSC > 1 ? 2 : 1, kItems = GSC / PPL;
    constexpr bool DUP = PPL == 2;
    __shared__ GWSmem<D, DUP> smem[kGWWarps];
    __shared__ uint32_t s_stack[kGWWarps][GWShared<D>::value];
    GWSmem<D, DUP> &sm = smem[threadIdx.x >> 5];
    uint32_t *stk = s_stack[threadIdx.x >> 5];
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t *wl = t.wl + (size_t)gwarp * kGWStack;
    const uint32_t nitems = __ldcg(&t.meta[kMetaGroupCount]) * kItems;
    const float eps2 = p.eps2;
    const float *pos[3] = {s.x, s.y, s.z};
    GroupState<PPL> g;
    g.count = 0;
    while (true) {
        uint32_t item = 0;
        if (lane == 0) item = atomicAdd(&t.meta[kMetaGroupCtr], 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= nitems) break;
        // last group first: a thread that splits a sparse child emits its groups
        // late, and they meet the most sources
        item = nitems - 1u - item;
        const uint2 range = __ldcg(&t.grp[item / kItems]);
        const uint32_t base = range.x + (item % kItems) * (PPL * 32u), seg_end = range.y;
        if (base >= seg_end) continue;
        const int nk = PPL == 2 && seg_end - base > 32u ? 2 : 1;
        const uint32_t sg = sg_tab.seg_of ? sg_tab.seg_of[base] : 0u;
        float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
#pragma unroll
        for (int c = 0; c < GSC; c++) {   // the group's box
            const uint32_t i = range.x + (uint32_t)c * 32u + lane;
            if (i < seg_end)
#pragma unroll
                for (int a = 0; a < D; a++) {
                    const float v = pos[a][i];
                    lo[a] = fminf(lo[a], v);
                    hi[a] = fmaxf(hi[a], v);
                }
        }
#pragma unroll
        for (int k = 0; k < PPL; k++) {
            const uint32_t i = base + (uint32_t)k * 32u + lane;
            g.idx[k] = i;
            g.act[k] = i < seg_end;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                g.x[k][a] = (g.act[k] && a < D) ? pos[a][i] : 0.0f;
                g.f[k][a] = 0.0f;
                g.fc[k][a] = 0.0f;
            }
            g.u[k] = 0.0f;
            g.uc[k] = 0.0f;
        }
#pragma unroll
        for (int a = 0; a < D; a++)
            for (int o = 16; o > 0; o >>= 1) {
                lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
                hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
            }
        // the list terms are evaluated from the group's centre o: members
        // and staged sources are stored as offsets from it (the opening test
        // keeps the absolute box)
        float oc[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int a = 0; a < D; a++) oc[a] = 0.5f * (lo[a] + hi[a]);
#pragma unroll
        for (int k = 0; k < PPL; k++)
#pragma unroll
            for (int a = 0; a < D; a++) g.x[k][a] -= oc[a];
        int nl = 0, pl = 0;
        // a round's candidates, one per lane, and what their test needs; unless
        // BUSY the next round's are loaded before this round's lists are filled and
        // evaluated, so their latency passes meanwhile
        uint32_t top = 0, c = lane == 0 ? sg : kEmpty;   // the simulation's root node slot
        bool spilled = false;   // warp-uniform: the stack is in wl (global)
        bool overflow = false;
        float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 E2 = make_float2(0.f, 0.f);
        uint4 inf = make_uint4(0u, 0u, 0u, 0u);
        auto load = [&]() {
            if (c == kEmpty) return;
            A = __ldg(&t.gw[c]);
            inf = __ldg(&t.info[c]);
            if (D == 3) E2 = __ldg(&t.gq2[c]);
        };
        load();
        while (__any_sync(0xffffffffu, c != kEmpty)) {
            int kind = 0;   // 1 accepted node, 2 opened leaf, 3 opened internal node
            if (c != kEmpty) {
                const float m = D == 2 ? A.z : A.w;
                const float b2 = D == 2 ? A.w : E2.y;
                if (m > 0.0f) {
                    const float com[3] = {A.x, A.y, A.z};
                    float dm = eps2;
#pragma unroll
                    for (int a = 0; a < D; a++) {
                        const float e = fmaxf(fmaxf(lo[a] - com[a], com[a] - hi[a]), 0.0f);
                        dm = __fmaf_rn(e, e, dm);
                    }
                    kind = b2 < dm ? 1 : (inf.y ? 3 : 2);
                }
            }
            // children of opened internal nodes onto the work stack (false: it is
            // full), from whose top the next round's candidates come
            auto push = [&]() {
                const uint32_t nch = kind == 3 ? (uint32_t)__popc(inf.y) : 0u;
                uint32_t incl = nch;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= (unsigned)o) incl += v;
                }
                const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
                if (!spilled && top + tot > GWShared<D>::value) {   // warp-uniform: move to wl
                    for (uint32_t q = lane; q < top; q += 32) wl[q] = stk[q];
                    spilled = true;
                    __syncwarp();
                }
                if (top + tot > kGWStack) return false;   // warp-uniform
                if (spilled)
                    for (uint32_t q = 0; q < nch; q++) wl[top + incl - nch + q] = inf.x + q;
                else
                    for (uint32_t q = 0; q < nch; q++) stk[top + incl - nch + q] = inf.x + q;
                top += tot;
                __syncwarp();
                return true;
            };
            auto take = [&]() {
                const uint32_t some = min(top, 32u);
                top -= some;
                c = lane < some ? (spilled ? __ldcg(&wl[top + lane]) : stk[top + lane]) : kEmpty;
            };
            // an accepted node's entry and moments
            const uint32_t ce = c;
            const float4 Ae = A;
            float4 Bq = make_float4(0.f, 0.f, 0.f, 0.f), Cq = Bq;
            float Eq = 0.0f;
            auto moments = [&]() {
                if (kind != 1) return;
                Bq = __ldg(&t.gq0[ce]);
                if (D == 3) Cq = __ldg(&t.gq1[ce]);
                Eq = D == 3 ? E2.x : __ldg(&t.gq2[ce]).x;
            };
            uint32_t pc = 0, pbeg = 0;   // the particles of an opened leaf
            auto leaf = [&]() {
                pc = kind == 2 ? inf.w - inf.z : 0u;
                pbeg = inf.z;
            };
            if (!BUSY) {
                if (!push()) {
                    overflow = true;
                    break;
                }
                moments();
                leaf();
                take();
                load();
            } else {
                moments();
            }
            // accepted nodes into the node list
            const unsigned accb = __ballot_sync(0xffffffffu, kind == 1);
            if (nl + __popc(accb) > kGWNodes) {
                eval_nodes<D, PPL, DUP, COUNT, POT>(sm, nl, g, eps2, nk);
                nl = 0;
                __syncwarp();
            }
            if (kind == 1) {
                const int q = nl + __popc(accb & lt);
                // staged for flush_nodes: J = 7.5 I and t = -1.5 tr(I)
                float tr;
                if (D == 2) {   // {lo.x, lo.y, Ixx, Ixy}, Iyy
                    tr = Bq.z + Eq;
                    Bq.z *= 7.5f; Bq.w *= 7.5f; Eq *= 7.5f;
                } else {        // {lo.xyz, Ixx}, {Iyy, Izz, Ixy, Ixz}, Iyz
                    tr = Bq.w + Cq.x + Cq.y;
                    Bq.w *= 7.5f; Cq.x *= 7.5f; Cq.y *= 7.5f; Cq.z *= 7.5f; Cq.w *= 7.5f; Eq *= 7.5f;
                }
                const float cx = (Ae.x - oc[0]) + Bq.x, cy = (Ae.y - oc[1]) + Bq.y;
                GWNode v;
                if (D == 2)
                    v = GWNode{{cx, cy, 0.0f}, Ae.z, Bq.z, Bq.w, 0.0f, Eq, 0.0f, 0.0f, -1.5f * tr};
                else
                    v = GWNode{{cx, cy, (Ae.z - oc[2]) + Bq.z}, Ae.w, Bq.w, Cq.z, Cq.w, Cq.x, Eq,
                               Cq.y, -1.5f * tr};
                put_node<D, DUP>(sm, q, v);
            }
            nl += __popc(accb);
            if (BUSY) {
                if (!push()) {
                    overflow = true;
                    break;
                }
                take();
                leaf();
            }
            // particles of opened leaves into the particle list, which is
            // evaluated whenever it is full: the leaves' particles are numbered
            // through (in lane order) and each lane takes every 32nd of them
            if (__any_sync(0xffffffffu, pc > 0u)) {
                uint32_t pin = pc;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, pin, o);
                    if (lane >= (unsigned)o) pin += v;
                }
                const uint32_t ptot = __shfl_sync(0xffffffffu, pin, 31);
                const uint32_t first = pbeg - (pin - pc);   // particle r of this lane's: first + r
                uint32_t r0 = 0;
                while (r0 < ptot) {
                    const uint32_t now = min(ptot - r0, (uint32_t)(kGWParts - pl));
                    for (uint32_t b = 0; b < now; b += 32u) {
                        const uint32_t r = r0 + b + lane;
                        uint32_t L = 0;   // the first lane whose inclusive count passes r
#pragma unroll
                        for (uint32_t st = 16; st > 0; st >>= 1)
                            if (__shfl_sync(0xffffffffu, pin, L + st - 1u) <= r) L += st;
                        const uint32_t src = __shfl_sync(0xffffffffu, first, L & 31u) + r;
                        if (b + lane < now)
                            put_part<D, DUP>(sm, pl + (int)(b + lane), s.x[src] - oc[0],
                                             s.y[src] - oc[1], D == 3 ? s.z[src] - oc[2] : 0.0f,
                                             s.m[src], src);
                    }
                    r0 += now;
                    pl += (int)now;
                    if (pl == kGWParts) {
                        __syncwarp();
                        eval_parts<D, PPL, DUP, COUNT, POT>(sm, pl, g, eps2, nk);
                        __syncwarp();
                        pl = 0;
                    }
                }
            }
            __syncwarp();
            if (BUSY) load();
        }
        if (overflow) {
            if (lane == 0) set_err(err, kErrStack);
            nl = 0;
            pl = 0;
        }
        __syncwarp();
        if (nl) eval_nodes<D, PPL, DUP, COUNT, POT>(sm, nl, g, eps2, nk);
        if (pl) eval_parts<D, PPL, DUP, COUNT, POT>(sm, pl, g, eps2, nk);
        __syncwarp();
        if (POT) {   // potential pass: sum_i m_i u_i in FP64, nothing written to the state
            double v = 0.0;
#pragma unroll
            for (int k = 0; k < PPL; k++)
                if (g.act[k]) v += (double)s.m[g.idx[k]] * ((double)g.u[k] - (double)g.uc[k]);
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) atomicAdd(epot, v);
            continue;
        }
        // results and the fused second half kick
#pragma unroll
        for (int k = 0; k < PPL; k++) {
            if (!g.act[k]) continue;
            const uint32_t i = g.idx[k];
            float a3[3];
#pragma unroll
            for (int a = 0; a < D; a++) a3[a] = p.G * (g.f[k][a] - g.fc[k][a]);
            s.ax[i] = a3[0];
            s.ay[i] = a3[1];
            if (D == 3) s.az[i] = a3[2];
            if (integrate_end && !(s.pinned && s.pinned[i])) {
                float *vel[3] = {s.vx, s.vy, s.vz};
                if (s.kvx) {
                    float *kv[3] = {s.kvx, s.kvy, s.kvz};
#pragma unroll
                    for (int a = 0; a < D; a++) kahan_add(vel[a][i], kv[a][i], fmul(a3[a], p.half_dt));
                } else {
#pragma unroll
                    for (int a = 0; a < D; a++) vel[a][i] = fadd(vel[a][i], fmul(a3[a], p.half_dt));
                }
            }
        }
    }
    if (COUNT) {
        unsigned long long v = g.count;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0 && v) atomicAdd(inter, v);
    }
}

static int grid_blocks(int n) {
    int b = (n + 255) / 256;
    if (b > 148 * 8) b = 148 * 8;
    return b < 1 ? 1 : b;
}

template <int D, int GSC, bool COUNT, bool POT = false, bool BUSY = false>
static int resident_blocks() {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &per_sm, k_group_walk<D, GSC, COUNT, POT, BUSY>, kGWThreads, 0) != cudaSuccess)
        return 0;
    return per_sm;
}

template <int D>
static int most_resident() {
    int m = resident_blocks<D, 1, false>();
    m = max(m, resident_blocks<D, 2, false>());
    m = max(m, resident_blocks<D, 4, false>());
    m = max(m, resident_blocks<D, 1, true>());
    m = max(m, resident_blocks<D, 2, true>());
    m = max(m, resident_blocks<D, 4, true>());
    m = max(m, resident_blocks<D, 1, false, false, true>());
    m = max(m, resident_blocks<D, 1, true, false, true>());
    return m;
}

// Warps the group walk keeps resident (its work stacks are sized for them).
int group_walk_warps(int dims, int num_sms) {
    const int per_sm = dims == 2 ? most_resident<2>() : most_resident<3>();
    return per_sm * num_sms * kGWWarps;
}

uint32_t group_walk_stack_entries() { return kGWStack; }

// Blocks of a walk: those it keeps resident, at most one per four groups, which
// number at most n; the work stacks, one per warp, bound them too.
template <int D, int GSC, bool COUNT, bool POT, bool BUSY>
static int gw_blocks(const Tree &t, int n, int num_sms) {
    static const int per_sm = resident_blocks<D, GSC, COUNT, POT, BUSY>();
    const int64_t stacks = t.wl_warps / kGWWarps, groups = ((int64_t)n + kGWWarps - 1) / kGWWarps;
    const int64_t resident = per_sm > 0 ? (int64_t)per_sm * num_sms : stacks;
    return (int)max((int64_t)1, min(min(stacks, resident), groups));
}

template <int D, int GSC, bool COUNT, bool BUSY>
static cudaError_t gw_walk(const State &s, const StepParams &p, const Segs &g, const Tree &t, int ie,
                           unsigned long long *inter, uint32_t *err, int num_sms, cudaStream_t st) {
    double *no_pot = nullptr;
    return launch_dep(k_group_walk<D, GSC, COUNT, false, BUSY>,
                      gw_blocks<D, GSC, COUNT, false, BUSY>(t, p.n, num_sms), kGWThreads, st, s, p,
                      g, t, ie, inter, err, no_pot);
}

template <int D, int GSC, bool COUNT>
static cudaError_t gw_launch(const State &s, const StepParams &p, const Segs &g, const Tree &t,
                             int ie, unsigned long long *inter, uint32_t *err, int num_sms,
                             cudaStream_t st) {
    cudaError_t e = launch_dep(k_make_groups<D>, grid_blocks(p.n), 256, st, t, 32u * GSC);
    if (e != cudaSuccess) return e;
    if constexpr (GSC == 1)
        if (gw_busy(p.n)) return gw_walk<D, GSC, COUNT, true>(s, p, g, t, ie, inter, err, num_sms, st);
    return gw_walk<D, GSC, COUNT, false>(s, p, g, t, ie, inter, err, num_sms, st);
}

template <int D>
static cudaError_t gw_dims(const State &s, const StepParams &p, const Segs &g, const Tree &t,
                           int ie, unsigned long long *inter, uint32_t *err, int num_sms,
                           cudaStream_t st) {
    if (inter) {
        if (p.group_size >= 128) return gw_launch<D, 4, true>(s, p, g, t, ie, inter, err, num_sms, st);
        if (p.group_size >= 64) return gw_launch<D, 2, true>(s, p, g, t, ie, inter, err, num_sms, st);
        return gw_launch<D, 1, true>(s, p, g, t, ie, inter, err, num_sms, st);
    }
    if (p.group_size >= 128) return gw_launch<D, 4, false>(s, p, g, t, ie, inter, err, num_sms, st);
    if (p.group_size >= 64) return gw_launch<D, 2, false>(s, p, g, t, ie, inter, err, num_sms, st);
    return gw_launch<D, 1, false>(s, p, g, t, ie, inter, err, num_sms, st);
}

template <int D, int PPL>
static cudaError_t gw_pot(const State &s, const StepParams &p, const Segs &g, const Tree &t,
                          uint32_t *err, double *epot, int num_sms, cudaStream_t st) {
    k_make_groups<D><<<grid_blocks(p.n), 256, 0, st>>>(t, 32u * PPL);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    auto go = [&](auto busy) {
        constexpr bool BUSY = decltype(busy)::value;
        k_group_walk<D, PPL, false, true, BUSY>
            <<<gw_blocks<D, PPL, false, true, BUSY>(t, p.n, num_sms), kGWThreads, 0, st>>>(
                s, p, g, t, 0, nullptr, err, epot);
    };
    if (gw_busy(p.n)) go(std::true_type{});
    else go(std::false_type{});
    return cudaGetLastError();
}

cudaError_t launch_group_potential(int dims, const State &s, const StepParams &p, const Segs &g,
                                   const Tree &t, uint32_t *counter, uint32_t *err, double *epot,
                                   int num_sms, cudaStream_t st) {
    if (!t.wl || !t.grp || t.wl_warps < (uint32_t)kGWWarps) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(counter, 0, 2 * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(epot, 0, sizeof(double), st)) != cudaSuccess) return e;
    return dims == 2 ? gw_pot<2, 1>(s, p, g, t, err, epot, num_sms, st)
                     : gw_pot<3, 1>(s, p, g, t, err, epot, num_sms, st);
}

cudaError_t launch_group_walk(int dims, const State &s, const StepParams &p, const Segs &g,
                              const Tree &t, bool integrate_end, unsigned long long *inter_count,
                              uint32_t *counter, uint32_t *err, int num_sms, cudaStream_t st) {
    if (!t.wl || !t.grp || t.wl_warps < (uint32_t)kGWWarps) return cudaErrorInvalidValue;
    // counter[0]: next group to walk, counter[1]: groups made
    cudaError_t e = cudaMemsetAsync(counter, 0, 2 * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    const int ie = integrate_end ? 1 : 0;
    return dims == 2 ? gw_dims<2>(s, p, g, t, ie, inter_count, err, num_sms, st)
                     : gw_dims<3>(s, p, g, t, ie, inter_count, err, num_sms, st);
}

}  // namespace ge
