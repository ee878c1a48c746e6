// ge_walk.cu -- the theta-criterion tree walk with softened force.
//
// Reference: Physics::calculateForceFromGrid (GalaxyEngine/src/Physics/physics.cpp:91-205)
// and Physics3D::calculateForceFromGrid3D (physics3D.cpp:131-253).  Per
// particle i the reference scans the pre-order node array: a node of zero mass
// is skipped; with d = com - x_i and r2 = |d|^2 + eps2 the node is accepted as
// a monopole when size^2 < theta^2 * r2; otherwise a leaf is summed directly
// over its particles j != i; otherwise the walk descends.  acc_i = F_i / m_i.
//
// Here every particle walks the depth-first layout built with the tree
// (ge_internal.h) with no stack: each step loads one entry and its skip
// target, evaluates the reference's opening test with the reference's
// rounding (so the interaction set is exactly the reference's), interacts if
// accepted and goes to the skip target, else to the next entry (the first
// child, or a leaf's first particle).  A leaf's particles follow the leaf as
// entries of their own with size^2 = -1, which every test accepts, so the
// direct sum over a leaf is the same loop body (the self term j == i is
// skipped as in the reference); a node of zero mass is laid out as an accepted
// entry without mass, so its subtree is skipped as in the reference.
// Sources are met in the reference's pre-order, so each particle accumulates
// in the reference's order.
//   GE_PREC_EXACT : every interaction with the reference's rounding
//                   (1/sqrtf, products in the reference's order, no FMA):
//                   bit-identical accelerations.
//   GE_PREC_FAST  : approximate reciprocal square root (MUFU, flush-to-zero)
//                   and FMA for the force terms, G applied once.
//   GE_PREC_MIXED : the node entries written by the moment pass
//                   (ge_moments.cu): opening radius instead of size, the
//                   double-float centre of mass, a quadrupole term, and
//                   Kahan-compensated sums of the acceleration terms.
// integrateEnd (physics.cpp:1114-1125) is fused into the epilogue.  A
// simulation below params.direct_below is skipped here (ge_direct.cu).
#include <type_traits>

#include "ge_bh.h"
#include "ge_device.cuh"
#include "ge_internal.h"

namespace ge {

// Threads per block: a block's particles, consecutive in Morton order on one
// SM, share most of their walks through L1.  (1024 in 3D shared more while a
// link had 8 bytes, 1M 1.65 ms against 1.78; with packed links 256 takes 1.56,
// 250k 483 us against 537, 60k 188 against 275, 16k 142 against 227.)
constexpr int kWalkThreads = 256, kWalkThreads2D = 512, kWalkThreadsRows = 1024;
// Whether a build packs its 3D entries (k_build decides): a tree of this many
// particles, with some 0.7 nodes for each, within the words' successors.
// Where the guess is wrong the walk is a slower one with the same bits.
static bool walk_packs(const StepParams &p) {
    return p.min_size >= 1e-18f && p.n < (int)((1u << kPackSkipBits) / 17 * 10);
}
// 3D EXACT, MIXED and heat exchange: blocks of 1024 share more still, and take
// less time where their last row (one block on every SM) is at least nine tenths
// full; with a row that is not, the SMs with one block more than others cost more
// than the sharing gains.  Walk, 256 / 1024 threads (us): EXACT 150k 394 / 390, 160k
// 464 / 607, 300k 773 / 710, 350k 955 / 1007, 450k 1127 / 1078, 605k 1451 / 1402, 1M
// 2355 / 2352; with heat exchange 300k 1489 / 1362; FAST with heat exchange 300k 1008
// / 942, 450k 1530 / 1538, 605k 1914 / 1817.  MIXED takes 38 registers with 256
// threads (faster below its six blocks per SM: 50k 672 / 1057) and 32 with 1024,
// where a row alone on the SMs is slow, so two rows have to be full: 285k 3205 /
// 2365, 300k 3141 / 2483, 450k 3707 / 4164, 605k 5161 / 4670, 900k 7356 / 6928.
// FAST in the plain layout, whose links have 8 bytes, from two rows on whether
// full or not: theta 0.5 450k 3282 / 2708, 1M 6208 / 4860, 0.7 1M 1763 / 1645, 1.0
// 1M 565 / 590 (by pairs 3156, 5242, 1823, 700).
static bool walk_rows(const StepParams &p, int mode, bool temp, int num_sms) {
    const int blocks = (p.n - p.i0 + kWalkThreadsRows - 1) / kWalkThreadsRows;
    if (blocks < 1) return false;
    if (mode == GE_PREC_FAST && !temp) {
        if (walk_packs(p)) return false;
        if (blocks > 2 * num_sms) return true;
    }
    const int row = mode == GE_PREC_MIXED ? 2 * num_sms : num_sms;
    return 10 * ((blocks - 1) % row + 1) >= 9 * row;
}
// 2D, by the launch's particles.  While SMs are left over, larger blocks share
// more (256 -> 512 threads, us: 2k 38.9 -> 36.8, 6k 49.2 -> 45.1, 12k 53.3 ->
// 49.2, 20k 55.3 -> 53.8, 28k 55.8 -> 54.3, 36k the same; with heat exchange 12k
// 133 -> 126; 10 disks of up to 4k 43.1 -> 41.0).  Between one and four blocks of
// 256 per SM some SMs have one more than others, which smaller blocks even out for
// one simulation (256 -> 128: 45k 57.3 -> 55.3, 65k 57.3 -> 53.2, 90k 57.5 -> 55.3,
// 130k 56.7 -> 55.3; theta 0.5 65k 91.0 -> 85.5, 1.0 100k 36.4 -> 37.4; with heat
// exchange 65k 139 -> 131; 36k the same, 190k 65.5 -> 66.6).  In a batch their
// walks share more than that (128 -> 256: 64 disks of up to 1.5k 44.0 -> 41.6, 18 of
// up to 16k 52.1 -> 48.1, 14 of up to 32k 54.8 -> 51.7).  3D gains on neither side
// (20k 157.7, 159.7 with 512; 65k 178.2, 181.7 with 128).
static int walk_threads_2d(int n, bool alone, int num_sms) {
    if (n <= 64 * 512) return 512;
    return alone && n > num_sms * 256 && n <= 4 * num_sms * 256 ? 128 : 256;
}

__device__ __forceinline__ float wrap_d(float d, float dom, float hd) {
    // d -= domain * ((d > half) - (d < -half))   (physics.cpp:118-121), the
    // factor -1, 0 or 1 by selection: its conversion to float would go through
    // the unit that the reciprocal square root needs
    return fsub(d, d > hd ? dom : (d < -hd ? -dom : 0.0f));
}

// Whether no offset from a particle to anything inside its simulation's root
// box can pass half the domain, so that the wrap leaves every offset as it is:
// the particle has 0.95 of half the domain to the box's sides, and the build
// has seen nothing farther outside the box than kBoxSlack (0.049) of it; the
// thousandth between them is for the roundings (coordinates up to twice the
// domain).  In a 3D sphere of 250k reaching 77 % of the domain this holds for
// most particles: walk 566 -> 477 us; a 2D disk of 1M well inside it 421 -> 271
// (no wrap at all: 271).
template <int D>
__device__ __forceinline__ bool never_wraps(const Tree &t, const float4 &box, const StepParams &p,
                                            const float *x) {
    const float lo[3] = {box.x, box.y, box.z};
    bool in = __ldg(&t.meta[kMetaMayWrap]) == 0u;
#pragma unroll
    for (int a = 0; a < D; a++) {
        const float most = 0.95f * p.half_domain[a];
        in = in && x[a] - lo[a] < most && lo[a] + box.w - x[a] < most &&
             fabsf(lo[a]) + box.w < 4.0f * p.half_domain[a];
    }
    return in;
}

__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// skip target and size^2 of an entry: 2D link = skip (size^2 in the source),
// 3D link = {skip, size^2 bits}
__device__ __forceinline__ uint32_t link_skip(uint32_t l) { return l; }
__device__ __forceinline__ uint32_t link_skip(const uint2 &l) { return l.x; }
__device__ __forceinline__ float link_s2(uint32_t, float in_src) { return in_src; }
__device__ __forceinline__ float link_s2(const uint2 &l, float) { return __uint_as_float(l.y); }

template <int D> struct LinkOf;
template <> struct LinkOf<2> { using T = uint32_t; };
template <> struct LinkOf<3> { using T = uint2; };

// The 2D packed walk of entries [k, end) in FAST arithmetic, not periodic,
// eps2 > 0: the terms of massless sources and of the particle itself add
// exactly zero.  x and y go through packed operations (f32x2), each rounded as
// the scalar one.  The loads' L1 wavefronts bound it (79 % of peak; 6.7 per
// load, the lanes of a warp at some five entries), so a quarter fewer
// instructions give little, and nothing below 100k particles: against the
// general loop 1M at theta 0.5 507 -> 503 us, 0.7 290 -> 282, 1.0 165 -> 159, 2M at
// 0.7 546 -> 527.
__device__ __forceinline__ void walk_packed2(const float4 *__restrict__ src, uint32_t k,
                                             uint32_t end, uint32_t rs2_bits, const float *pi,
                                             float eps2, float th2, float *f) {
    const f32x2 np = pack2(-pi[0], -pi[1]);
    f32x2 fxy = pack2(0.0f, 0.0f);
    while (k < end) {
        const ulonglong2 A = __ldg(reinterpret_cast<const ulonglong2 *>(src + k));
        float m, w;
        unpack2(A.y, m, w);
        const uint32_t wb = __float_as_uint(w);
        const f32x2 d = add2(A.x, np);
        float xx, yy;
        unpack2(mul2(d, d), xx, yy);
        const float r2 = fadd(fadd(xx, yy), eps2);
        const bool acc = (int)(rs2_bits - ((wb >> 2) & 0x3F000000u)) < __float_as_int(fmul(th2, r2));
        const float inv = rsqrt_approx(r2);
        const float fm = acc ? m * (inv * inv * inv) : 0.0f;
        fxy = fma2(d, pack2(fm, fm), fxy);
        k += 1u + (acc ? packed_ahead(wb) : 0u);
    }
    unpack2(fxy, f[0], f[1]);
}

// 0: the compiler's choice
constexpr int walk_min_blocks(int dims, int mode, int threads) {
    return dims == 2 || (mode == GE_PREC_MIXED && threads == kWalkThreads) ? 0 : 2048 / threads;
}

template <int D, int MODE, bool COUNT, bool PER, bool POS_EPS, bool TEMP, int THREADS>
__global__ void __launch_bounds__(THREADS, walk_min_blocks(D, MODE, THREADS))
k_walk(State s, StepParams p, Segs g, Tree t, int integrate_end, unsigned long long *inter,
       uint32_t *err) {
    dep_wait();
    using LT = typename LinkOf<D>::T;
    constexpr bool kSelfTest = MODE != GE_PREC_FAST || COUNT || !POS_EPS || TEMP;
    const LT *__restrict__ link = (const LT *)t.link;
    const float4 *__restrict__ src = t.src;
    const int n = p.n;
    const float eps2 = p.eps2, th2 = p.theta2, G = p.G;
    const int i = p.i0 + blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long my_count = 0;
    // particles of simulations that take the direct sum are left to it
    const bool walks = i < n && !(g.direct && __ldg(&g.direct[g.seg_of ? __ldg(&g.seg_of[i]) : 0u]));
    if (walks) {
        float pi[3];
        pi[0] = s.x[i]; pi[1] = s.y[i];
        pi[2] = D == 3 ? s.z[i] : 0.0f;
        const float mi = s.m[i];
        const float gm_i = fmul(G, mi);   // Gf * pmass (exact mode)
        const uint32_t self = kSelfTest ? __ldg(&t.slot_of[i]) : kEmpty;
        float f[3] = {0.f, 0.f, 0.f};
        float fc[3] = {0.f, 0.f, 0.f};   // Kahan compensation (MIXED)
        float ti = TEMP ? __ldg(&t.tv[self]) : 0.0f;   // own temperature, accumulated in walk order
        // the walk of the particle's own segment: its root to the root's successor
        const uint32_t sg = g.seg_of ? __ldg(&g.seg_of[i]) : 0u;
        uint32_t k = __ldg(&g.root_begin[sg]);
        const uint32_t end = __ldg(&g.root_end[sg]);
        uint32_t cnt = 0;
        // packed entries: the successor and the level in one word; the root
        // size of the particle's simulation
        const bool packed = MODE != GE_PREC_MIXED && __ldg(&t.meta[kMetaWalkPacked]) != 0u;
        const float rs = packed ? __ldg(&g.box[sg]).w : 0.0f;
        const uint32_t rs2_bits = __float_as_uint(fmul(rs, rs));   // the root's size^2
        // the loop once per layout, chosen here rather than at every step
        auto walk_range = [&](auto pk, auto wrap) {
            constexpr bool WRAP = decltype(wrap)::value;
            constexpr bool PK = decltype(pk)::value && MODE != GE_PREC_MIXED;
            while (k < end) {
                const float4 A = __ldg(&src[k]);
                const float m = D == 2 ? A.z : A.w;
                float s2;          // a node's size^2 (plain layout: -1 particle, -2 massless)
                uint32_t nxt_skip = 0u;
                uint32_t ahead = 0u;   // packed: entries past the next one to the successor
                bool part;         // a particle's entry
                bool always = false;   // packed: a particle or a massless node
                if constexpr (PK) {
                    const uint32_t wb = D == 2 ? __float_as_uint(A.w)
                                               : __ldg(&((const uint32_t *)t.link)[k]);
                    always = packed_accepts(wb);
                    part = packed_particle(wb);
                    s2 = packed_size2(wb, rs2_bits);   // not used for marked entries
                    ahead = packed_ahead(wb);          // a particle's: none
                } else {
                    const LT L = __ldg(&link[k]);
                    s2 = link_s2(L, A.w);
                    nxt_skip = link_skip(L);
                    part = s2 == -1.0f;
                }
                float d[3];
                d[0] = fsub(A.x, pi[0]);
                d[1] = fsub(A.y, pi[1]);
                d[2] = D == 3 ? fsub(A.z, pi[2]) : 0.0f;
                if (WRAP) {
    #pragma unroll
                    for (int a = 0; a < D; a++) d[a] = wrap_d(d[a], p.domain[a], p.half_domain[a]);
                }
                float r2 = fadd(fmul(d[0], d[0]), fmul(d[1], d[1]));
                if (D == 3) r2 = fadd(r2, fmul(d[2], d[2]));
                r2 = fadd(r2, eps2);
                // MIXED entries hold the squared opening radius, which already
                // includes 1 / theta
                bool acc;
                if constexpr (PK) acc = always || s2 < fmul(th2, r2);   // as -1 / -2 would
                else if constexpr (MODE == GE_PREC_MIXED) acc = s2 < r2;
                else acc = s2 < 0.0f || s2 < fmul(th2, r2);   // (a particle whose r2 is no number, too)
                if (kSelfTest) {
                    // heat exchange (physics.cpp:145-158, 183-191): an accepted node
                    // with mass, or any other particle of an opened leaf (massless
                    // ones included); the others' temperatures as before the walk
                    if (TEMP && acc && k != self && (m != 0.0f || part)) {
                        float inv;
                        if (MODE == GE_PREC_EXACT) inv = fdiv(1.0f, __fsqrt_rn(r2));
                        else inv = rsqrt_approx(r2);
                        const float dist = r2 > 1e-16f ? fdiv(1.0f, inv) : 0.0f;
                        if (dist > 1e-8f) {
                            const float diff = fsub(__ldg(&t.tv[k]), ti);
                            ti = fadd(ti, fmul(fdiv(fmul(p.heat_cond, diff), dist), p.dt));
                        }
                    }
                    if (acc && m != 0.0f && k != self) {
                        if (MODE == GE_PREC_MIXED) {
                            float term[3];
                            if (s2 >= 0.0f) {
                                // node: centre of mass = hi + lo, then monopole +
                                // quadrupole of the softened kernel:
                                //   m d / r^3 - 3 I d / r^5 - 1.5 tr(I) d / r^5
                                //   + 7.5 (d.I.d) d / r^7,   r^2 = |d|^2 + eps2
                                const float4 B = __ldg(&t.mq0[k]);
                                d[0] += B.x; d[1] += B.y;
                                if (D == 3) d[2] += B.z;
                                float rr = d[0] * d[0] + d[1] * d[1] + eps2;
                                if (D == 3) rr += d[2] * d[2];
                                const float inv = rsqrt_approx(rr);
                                const float inv2 = inv * inv, inv3 = inv2 * inv, inv5 = inv3 * inv2;
                                const float inv7 = inv5 * inv2;
                                float Id[3], tr;
                                if (D == 2) {
                                    const float ixx = B.z, ixy = B.w, iyy = __ldg(&t.mq2[k]);
                                    Id[0] = ixx * d[0] + ixy * d[1];
                                    Id[1] = ixy * d[0] + iyy * d[1];
                                    Id[2] = 0.0f;
                                    tr = ixx + iyy;
                                } else {
                                    const float4 C = __ldg(&t.mq1[k]);   // {Iyy, Izz, Ixy, Ixz}
                                    const float ixx = B.w, iyz = __ldg(&t.mq2[k]);
                                    Id[0] = ixx * d[0] + C.z * d[1] + C.w * d[2];
                                    Id[1] = C.z * d[0] + C.x * d[1] + iyz * d[2];
                                    Id[2] = C.w * d[0] + iyz * d[1] + C.y * d[2];
                                    tr = ixx + C.x + C.y;
                                }
                                float dId = d[0] * Id[0] + d[1] * Id[1];
                                if (D == 3) dId += d[2] * Id[2];
                                const float cm = m * inv3 - 1.5f * tr * inv5 + 7.5f * dId * inv7;
                                const float ci = -3.0f * inv5;
    #pragma unroll
                                for (int a = 0; a < D; a++) term[a] = cm * d[a] + ci * Id[a];
                            } else {
                                const float inv = rsqrt_approx(r2);
                                const float fm = m * (inv * inv * inv);
    #pragma unroll
                                for (int a = 0; a < D; a++) term[a] = d[a] * fm;
                            }
    #pragma unroll
                            for (int a = 0; a < D; a++) {   // Kahan summation
                                const float y = fsub(term[a], fc[a]);
                                const float tt = fadd(f[a], y);
                                fc[a] = fsub(fsub(tt, f[a]), y);
                                f[a] = tt;
                            }
                        } else if (MODE == GE_PREC_EXACT) {
                            const float inv = fdiv(1.0f, __fsqrt_rn(r2));
                            const float inv3 = fmul(fmul(inv, inv), inv);
                            const float fm = fmul(fmul(gm_i, m), inv3);
    #pragma unroll
                            for (int a = 0; a < D; a++) f[a] = fadd(f[a], fmul(d[a], fm));
                        } else {
                            const float inv = rsqrt_approx(r2);
                            const float fm = m * (inv * inv * inv);
    #pragma unroll
                            for (int a = 0; a < D; a++) f[a] = fmaf(d[a], fm, f[a]);
                        }
                        if (COUNT) cnt++;
                    }
                } else {
                    // eps2 > 0: the self term (d = 0) and massless sources add exactly
                    // zero, so no test is needed for them
                    const float inv = rsqrt_approx(r2);
                    const float fm = acc ? m * (inv * inv * inv) : 0.0f;
    #pragma unroll
                    for (int a = 0; a < D; a++) f[a] = fmaf(d[a], fm, f[a]);
                }
                // a valid skip lies past k; max() keeps k increasing whatever the
                // layout holds, so the walk ends within end - begin entries (a
                // packed word cannot point back)
                if constexpr (PK) k = k + 1u + (acc ? ahead : 0u);
                else k = max(k + 1, acc && !part ? nxt_skip : k + 1);
            }
        };
        // a periodic walk whose offsets cannot wrap is the plain one; a warp that
        // holds both kinds of particles wraps for all (the same bits) instead of
        // running both loops one after the other
        const bool wraps =
            PER && __any_sync(__activemask(), !never_wraps<D>(t, g.box[sg], p, pi));
        if constexpr (!kSelfTest && D == 2) {
            // As signed words the size^2 of a node and theta^2 r2 compare as
            // the floats do, and a marker level (62 or 63 off the root's
            // exponent) lies below theta^2 r2 whenever it lies below theta^2
            // eps2: one subtraction and one compare decide every entry.
            if (!wraps && packed &&
                (int)(rs2_bits - (kPackMassless << 24)) < __float_as_int(fmul(th2, eps2))) {
                walk_packed2(src, k, end, rs2_bits, pi, eps2, th2, f);
                k = end;
            }
        }
        auto by_layout = [&](auto wrap) {
            if (packed) walk_range(std::true_type{}, wrap);
            else walk_range(std::false_type{}, wrap);
        };
        if constexpr (PER) {
            if (wraps) by_layout(std::true_type{});
            else by_layout(std::false_type{});
        } else {
            by_layout(std::false_type{});
        }
        float a3[3];
#pragma unroll
        for (int a = 0; a < D; a++)
            a3[a] = MODE == GE_PREC_EXACT ? fdiv(f[a], mi)
                  : MODE == GE_PREC_MIXED ? G * fsub(f[a], fc[a]) : G * f[a];
        s.ax[i] = a3[0]; s.ay[i] = a3[1];
        if (D == 3) s.az[i] = a3[2];
        if (TEMP) s.temp[i] = ti;
        if (integrate_end && !(s.pinned && s.pinned[i])) {
            if (MODE == GE_PREC_MIXED && s.kvx) {
                float *vel[3] = {s.vx, s.vy, s.vz}, *kv[3] = {s.kvx, s.kvy, s.kvz};
#pragma unroll
                for (int a = 0; a < D; a++) kahan_add(vel[a][i], kv[a][i], fmul(a3[a], p.half_dt));
            } else {
                s.vx[i] = fadd(s.vx[i], fmul(a3[0], p.half_dt));
                s.vy[i] = fadd(s.vy[i], fmul(a3[1], p.half_dt));
                if (D == 3) s.vz[i] = fadd(s.vz[i], fmul(a3[2], p.half_dt));
            }
        }
        my_count = cnt;
    }
    if (COUNT) {
        for (int o = 16; o > 0; o >>= 1) my_count += __shfl_xor_sync(0xffffffffu, my_count, o);
        if ((threadIdx.x & 31) == 0 && my_count) atomicAdd(inter, my_count);
    }
}

// ---- 3D FAST: two particles per thread --------------------------------------
// Two Morton neighbours visit nearly the same entries (4 % more together than
// either alone), so a thread that walks for both loads each entry once: the
// loads' L1 wavefronts are what bounds the 3D walk.  The thread stands at entry
// k for both; a particle that accepts an entry which the other opens takes the
// monopole and sits out the subtree (until entry ra / rb).  Each particle meets
// exactly its own entries, in its own order, with the single walk's arithmetic:
// the same bits.  Half the threads and a longer step, so it pays where the walks
// are long and many: walk (us), single / pairs, theta 0.7: 60k 190 / 227, 150k
// 268 / 283, 200k 383 / 332, 250k 479 / 397, 1M 1558 / 1334; theta 0.5 1M 5172 /
// 3588; theta 1.0 150k 119 / 150, 400k 283 / 275.  Many small systems in one
// launch gain as one large one does (theta 0.8, 400 of up to 2k 335 / 314, 100 of
// up to 15k 516 / 469).  Periodic systems gain where few of their offsets wrap
// (domain twice the system 250k 495 / 407, 1M 1572 / 1381) and lose where most do
// (a full domain 250k 342 / 372, 1M 1158 / 1228).  Plain entries gain at no size
// worth it (walk_rows), nor does 2D, bound by instructions as much as by L1 (1M
// 277 / 285).
constexpr int kPairThreads = 128;
static bool walk_pairs(const StepParams &p) {
    const int n = p.n - p.i0;
    return walk_packs(p) && (n >= 400000 || (n >= 200000 && p.theta <= 0.8f && !p.periodic));
}

// entry k in either layout: whether a particle at squared distance r2
// (softened) accepts it, and its successor
__device__ __forceinline__ bool entry_accepts3(const Tree &t, uint32_t k, bool packed,
                                               uint32_t rs2_bits, float th2r2, uint32_t &nxt) {
    if (packed) {
        const uint32_t wb = __ldg(&((const uint32_t *)t.link)[k]);
        nxt = k + 1u + packed_ahead(wb);
        return packed_accepts(wb) || packed_size2(wb, rs2_bits) < th2r2;
    }
    const uint2 l = __ldg(&((const uint2 *)t.link)[k]);
    nxt = max(k + 1u, l.x);   // a particle's successor is k + 1
    const float s2 = __uint_as_float(l.y);
    return s2 < 0.0f || s2 < th2r2;
}

template <bool PER>
__global__ void __launch_bounds__(kPairThreads)
k_walk_pair(State s, StepParams p, Segs g, Tree t, int integrate_end) {
    dep_wait();
    const float eps2 = p.eps2, th2 = p.theta2, G = p.G;
    const uint32_t n = (uint32_t)p.n;
    const uint32_t i0 = (uint32_t)p.i0 + 2u * (blockIdx.x * blockDim.x + threadIdx.x);
    if (i0 >= n) return;
    const bool packed = __ldg(&t.meta[kMetaWalkPacked]) != 0u;
    const float4 *__restrict__ src = t.src;
    const uint32_t *__restrict__ link = (const uint32_t *)t.link;
    const uint32_t i[2] = {i0, min(i0 + 1u, n - 1u)};
    uint32_t sg[2];
    bool on[2];   // a particle of the launch that takes the walk
    f32x2 np[2], f[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
    float pz[2], fz[2] = {0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 2; q++) {
        sg[q] = g.seg_of ? __ldg(&g.seg_of[i[q]]) : 0u;
        on[q] = i0 + q < n && !(g.direct && __ldg(&g.direct[sg[q]]));
        np[q] = pack2(-s.x[i[q]], -s.y[i[q]]);
        pz[q] = s.z[i[q]];
    }
    // both together inside one simulation, else one after the other
    const bool one = sg[0] == sg[1];
#pragma unroll 1
    for (int pass = one ? 2 : 0; pass < (one ? 3 : 2); pass++) {
        // the entry each particle is waiting for (kEmpty: not walking now)
        uint32_t r[2] = {on[0] && pass != 1 ? 0u : kEmpty, on[1] && pass != 0 ? 0u : kEmpty};
        if (r[0] & r[1]) continue;   // neither
        const uint32_t sgp = pass == 1 ? sg[1] : sg[0];
        uint32_t k = __ldg(&g.root_begin[sgp]);
        const uint32_t end = __ldg(&g.root_end[sgp]);
        const float rs = __ldg(&g.box[sgp]).w;
        const uint32_t rs2_bits = __float_as_uint(fmul(rs, rs));
        // (the signed compare that decides packed entries, marker levels too, as
        // in the 2D packed walk; otherwise the entry's own test)
        const bool by_word =
            packed && (int)(rs2_bits - (kPackMassless << 24)) < __float_as_int(fmul(th2, eps2));
        auto walk = [&](auto words, auto wrap) {
          constexpr bool WORDS = decltype(words)::value, WRAP = decltype(wrap)::value;
          while (k < end) {
            const ulonglong2 A = __ldg(reinterpret_cast<const ulonglong2 *>(src + k));
            float z, m;
            unpack2(A.y, z, m);
            f32x2 d[2];
            float dz[2], r2[2];
            bool acc[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                d[q] = add2(A.x, np[q]);
                dz[q] = fsub(z, pz[q]);
                if (WRAP) {
                    float dx, dy;
                    unpack2(d[q], dx, dy);
                    d[q] = pack2(wrap_d(dx, p.domain[0], p.half_domain[0]),
                                 wrap_d(dy, p.domain[1], p.half_domain[1]));
                    dz[q] = wrap_d(dz[q], p.domain[2], p.half_domain[2]);
                }
                float xx, yy;
                unpack2(mul2(d[q], d[q]), xx, yy);
                r2[q] = fadd(fadd(fadd(xx, yy), fmul(dz[q], dz[q])), eps2);
            }
            uint32_t nxt;
            if constexpr (WORDS) {
                const uint32_t wb = __ldg(link + k);
                const int s2 = (int)(rs2_bits - ((wb >> 2) & 0x3F000000u));
                nxt = k + 1u + packed_ahead(wb);
#pragma unroll
                for (int q = 0; q < 2; q++) acc[q] = s2 < __float_as_int(fmul(th2, r2[q]));
            } else {
#pragma unroll
                for (int q = 0; q < 2; q++)
                    acc[q] = entry_accepts3(t, k, packed, rs2_bits, fmul(th2, r2[q]), nxt);
            }
            bool open = false;
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const bool here = k >= r[q], take = acc[q] && here;
                const float inv = rsqrt_approx(r2[q]);
                const float fm = take ? m * (inv * inv * inv) : 0.0f;
                f[q] = fma2(d[q], pack2(fm, fm), f[q]);
                fz[q] = fmaf(dz[q], fm, fz[q]);
                r[q] = take ? nxt : r[q];
                open |= here && !acc[q];
            }
            k = open ? k + 1u : nxt;
          }
        };
        auto by_layout = [&](auto wrap) {
            if (by_word) walk(std::true_type{}, wrap);
            else walk(std::false_type{}, wrap);
        };
        bool wraps = false;
        if (PER)
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const float x[3] = {s.x[i[q]], s.y[i[q]], pz[q]};
                wraps = wraps || !never_wraps<3>(t, g.box[sgp], p, x);
            }
        if (PER) wraps = __any_sync(__activemask(), wraps);   // as in the single walk
        if constexpr (PER) {
            if (wraps) by_layout(std::true_type{});
            else by_layout(std::false_type{});
        } else {
            by_layout(std::false_type{});
        }
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
        if (!on[q]) continue;
        float a3[3];
        unpack2(f[q], a3[0], a3[1]);
        a3[0] = G * a3[0];
        a3[1] = G * a3[1];
        a3[2] = G * fz[q];
        s.ax[i[q]] = a3[0]; s.ay[i[q]] = a3[1]; s.az[i[q]] = a3[2];
        if (integrate_end && !(s.pinned && s.pinned[i[q]])) {
            s.vx[i[q]] = fadd(s.vx[i[q]], fmul(a3[0], p.half_dt));
            s.vy[i[q]] = fadd(s.vy[i[q]], fmul(a3[1], p.half_dt));
            s.vz[i[q]] = fadd(s.vz[i[q]], fmul(a3[2], p.half_dt));
        }
    }
}

template <int D, int MODE, bool COUNT, bool PER, bool POS_EPS, bool TEMP = false>
static cudaError_t walk_one(const State &s, const StepParams &p, const Segs &g, const Tree &t,
                            int ie, unsigned long long *inter, uint32_t *err, int num_sms,
                            cudaStream_t st) {
    if constexpr (D == 3 && MODE == GE_PREC_FAST && !COUNT && POS_EPS && !TEMP)
        if (walk_pairs(p))
            return launch_dep(k_walk_pair<PER>, (p.n - p.i0 + 2 * kPairThreads - 1) / (2 * kPairThreads),
                              kPairThreads, st, s, p, g, t, ie);
    const int n = p.n - p.i0;
    auto go = [&](auto bound, int threads) {
        const int blocks = (n + threads - 1) / threads;
        return launch_dep(k_walk<D, MODE, COUNT, PER, POS_EPS, TEMP, decltype(bound)::value>,
                          blocks < 1 ? 1 : blocks, threads, st, s, p, g, t, ie, inter, err);
    };
    if constexpr (D == 2) {
        return go(std::integral_constant<int, kWalkThreads2D>{},
                  MODE != GE_PREC_MIXED ? walk_threads_2d(n, g.S == 1, num_sms) : kWalkThreads);
    } else {
        if (walk_rows(p, MODE, TEMP, num_sms))
            return go(std::integral_constant<int, kWalkThreadsRows>{}, kWalkThreadsRows);
        return go(std::integral_constant<int, kWalkThreads>{}, kWalkThreads);
    }
}

template <int D, int MODE, bool PER>
static cudaError_t walk_eps(const State &s, const StepParams &p, const Segs &g, const Tree &t,
                            int ie, unsigned long long *inter, uint32_t *err, int num_sms,
                            cudaStream_t st) {
    if constexpr (MODE != GE_PREC_MIXED)
        if (s.temp && t.tv) {   // heat exchange (counting included)
            if (inter)
                return walk_one<D, MODE, true, PER, false, true>(s, p, g, t, ie, inter, err, num_sms, st);
            return walk_one<D, MODE, false, PER, false, true>(s, p, g, t, ie, nullptr, err, num_sms, st);
        }
    if (inter) return walk_one<D, MODE, true, PER, false>(s, p, g, t, ie, inter, err, num_sms, st);
    if constexpr (MODE != GE_PREC_MIXED)   // MIXED always tests for the particle itself
        if (p.eps2 > 0.0f)
            return walk_one<D, MODE, false, PER, true>(s, p, g, t, ie, nullptr, err, num_sms, st);
    return walk_one<D, MODE, false, PER, false>(s, p, g, t, ie, nullptr, err, num_sms, st);
}

template <int D, int MODE>
static cudaError_t walk_mode(const State &s, const StepParams &p, const Segs &g, const Tree &t,
                             int ie, unsigned long long *inter, uint32_t *err, int num_sms,
                            cudaStream_t st) {
    if (p.periodic) return walk_eps<D, MODE, true>(s, p, g, t, ie, inter, err, num_sms, st);
    return walk_eps<D, MODE, false>(s, p, g, t, ie, inter, err, num_sms, st);
}

cudaError_t launch_walk(int dims, int precision, const State &s, const StepParams &p,
                        const Segs &g, const Tree &t, bool integrate_end,
                        unsigned long long *inter_count, uint32_t *err, int num_sms,
                        cudaStream_t st) {
    const int ie = integrate_end ? 1 : 0;
    const bool exact = precision == GE_PREC_EXACT;
    if (warp_walk_on(p, precision, s.temp && t.tv))
        return launch_warp_walk(dims, s, p, g, t, integrate_end, inter_count, err, num_sms, st);
    if (precision == GE_PREC_MIXED)
        return dims == 2 ? walk_mode<2, GE_PREC_MIXED>(s, p, g, t, ie, inter_count, err, num_sms, st)
                         : walk_mode<3, GE_PREC_MIXED>(s, p, g, t, ie, inter_count, err, num_sms, st);
    if (dims == 2)
        return exact ? walk_mode<2, GE_PREC_EXACT>(s, p, g, t, ie, inter_count, err, num_sms, st)
                     : walk_mode<2, GE_PREC_FAST>(s, p, g, t, ie, inter_count, err, num_sms, st);
    return exact ? walk_mode<3, GE_PREC_EXACT>(s, p, g, t, ie, inter_count, err, num_sms, st)
                 : walk_mode<3, GE_PREC_FAST>(s, p, g, t, ie, inter_count, err, num_sms, st);
}

}  // namespace ge
