// ge_front_dev.cuh -- device code shared by the passes before the tree build:
// one kernel per pass over all particles (ge_integrate.cu, ge_sort.cu), or one
// thread-block cluster per small simulation (ge_front.cu).
#pragma once
#include "ge_device.cuh"
#include "ge_internal.h"

namespace ge {

// float <-> unsigned with the same order (negative floats reversed)
__device__ __forceinline__ uint32_t f2o(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// pos, vel, acc: particle i's, already loaded
template <int D>
__device__ __forceinline__ void kick_drift(const State &s, const StepParams &p, int i,
                                           float *pos, float *vel, const float *acc) {
    if (s.pvx) {
        s.pvx[i] = vel[0]; s.pvy[i] = vel[1];
        if (D == 3) s.pvz[i] = vel[2];
    }
    if (s.kx) {
        // GE_PREC_MIXED: both updates Kahan-compensated
        float *kp[3] = {s.kx, s.ky, s.kz}, *kv[3] = {s.kvx, s.kvy, s.kvz};
#pragma unroll
        for (int a = 0; a < D; a++) {
            float cv = kv[a][i], cp = kp[a][i];
            kahan_add(vel[a], cv, fmul(acc[a], p.half_dt));
            kahan_add(pos[a], cp, fmul(vel[a], p.dt));
            kv[a][i] = cv;
            kp[a][i] = cp;
        }
    } else {
#pragma unroll
        for (int a = 0; a < D; a++) {
            vel[a] = fadd(vel[a], fmul(acc[a], p.half_dt));   // vel += acc * halfDt
            pos[a] = fadd(pos[a], fmul(vel[a], p.dt));         // pos += vel * dt
        }
    }
    if (p.periodic) {
        if (D == 2) {
            // physics.cpp:1104-1110: domain [0, size)
#pragma unroll
            for (int a = 0; a < 2; a++) {
                if (pos[a] < 0.0f) pos[a] = fadd(pos[a], p.domain[a]);
                else if (pos[a] >= p.domain[a]) pos[a] = fsub(pos[a], p.domain[a]);
            }
        } else {
            // physics3D.cpp:785-802: domain [-size/2, size/2)
#pragma unroll
            for (int a = 0; a < 3; a++) {
                if (pos[a] < -p.half_domain[a]) pos[a] = fadd(pos[a], p.domain[a]);
                else if (pos[a] >= p.half_domain[a]) pos[a] = fsub(pos[a], p.domain[a]);
            }
        }
    }
    s.x[i] = pos[0]; s.y[i] = pos[1];
    s.vx[i] = vel[0]; s.vy[i] = vel[1];
    if (D == 3) { s.z[i] = pos[2]; s.vz[i] = vel[2]; }
}

// boundingBox() / boundingBox3D(): the square (cubic) root box of a min / max
template <int D>
__device__ __forceinline__ float4 root_box(const float *l, const float *h) {
    float size = ref_max(fsub(h[0], l[0]), fsub(h[1], l[1]));
    if (D == 3) size = ref_max(size, fsub(h[2], l[2]));
    const float half = fmul(size, 0.5f);
    float4 bb;
    bb.x = fsub(fmul(fadd(l[0], h[0]), 0.5f), half);
    bb.y = fsub(fmul(fadd(l[1], h[1]), 0.5f), half);
    bb.z = D == 3 ? fsub(fmul(fadd(l[2], h[2]), 0.5f), half) : 0.0f;
    bb.w = size;
    return bb;
}

// Morton key of a position in its simulation's root box
template <int D>
__device__ __forceinline__ uint64_t morton_key(float4 bb, float x, float y, float z) {
    if (D == 2) {
        const float ext = bb.w > 1e-6f ? bb.w : 1e-6f;   // std::max(posSize.z, 1e-6f)
        const uint64_t ix = scale_to_grid(x, bb.x, fadd(bb.x, ext), 262144.0f, 262143ull);
        const uint64_t iy = scale_to_grid(y, bb.y, fadd(bb.y, ext), 262144.0f, 262143ull);
        return spread2(ix) | (spread2(iy) << 1);
    }
    const uint64_t ix = scale_to_grid(x, bb.x, fadd(bb.x, bb.w), 2097151.0f, 2097151ull);
    const uint64_t iy = scale_to_grid(y, bb.y, fadd(bb.y, bb.w), 2097151.0f, 2097151ull);
    const uint64_t iz = scale_to_grid(z, bb.z, fadd(bb.z, bb.w), 2097151.0f, 2097151ull);
    return spread3(ix) | (spread3(iy) << 1) | (spread3(iz) << 2);
}

// The lanes whose BITS-bit digit equals this lane's, among the lanes with
// `valid` set: one ballot per digit bit (the same mask as __match_any_sync
// over the digits, for valid lanes; an invalid lane's mask is not used).
template <int BITS>
__device__ __forceinline__ unsigned digit_peers(uint32_t d, bool valid) {
    unsigned m = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < BITS; b++) {
        const bool bit = (d >> b) & 1u;
        const unsigned bb = __ballot_sync(0xffffffffu, bit);
        m &= bit ? bb : ~bb;
    }
    return m;
}

// State of slot j[u] into slot kk[u] (< n) of `out`, U at a time: all loads
// before any store (the stores could alias the next loads, which would keep
// them apart).  L2: the drift wrote its arrays in this same kernel, from other
// SMs, so they are read past L1.
template <bool L2>
__device__ __forceinline__ float ld_l2(const float *p) {
    return L2 ? __ldcg(p) : *p;
}
template <int D, int U, bool L2>
__device__ __forceinline__ void gather_state(const State &in, const State &out, int with_acc,
                                             const uint32_t *kk, const uint32_t *j, uint32_t n) {
    float x[U], y[U], z[U], vx[U], vy[U], vz[U], m[U], ax[U], ay[U], az[U];
    uint32_t id[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        if (kk[u] >= n) continue;
        const uint32_t q = j[u];
        x[u] = ld_l2<L2>(&in.x[q]); y[u] = ld_l2<L2>(&in.y[q]);
        vx[u] = ld_l2<L2>(&in.vx[q]); vy[u] = ld_l2<L2>(&in.vy[q]);
        m[u] = in.m[q];
        id[u] = in.id[q];
        if (D == 3) { z[u] = ld_l2<L2>(&in.z[q]); vz[u] = ld_l2<L2>(&in.vz[q]); }
        if (with_acc) {
            ax[u] = in.ax[q]; ay[u] = in.ay[q];
            if (D == 3) az[u] = in.az[q];
        }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const uint32_t k = kk[u];
        if (k >= n) continue;
        const uint32_t q = j[u];
        out.x[k] = x[u]; out.y[k] = y[u];
        out.vx[k] = vx[u]; out.vy[k] = vy[u];
        out.m[k] = m[u];
        out.id[k] = id[u];
        if (D == 3) { out.z[k] = z[u]; out.vz[k] = vz[u]; }
        if (with_acc) {
            out.ax[k] = ax[u]; out.ay[k] = ay[u];
            if (D == 3) out.az[k] = az[u];
        }
        if (in.pvx) {
            out.pvx[k] = ld_l2<L2>(&in.pvx[q]); out.pvy[k] = ld_l2<L2>(&in.pvy[q]);
            if (D == 3) out.pvz[k] = ld_l2<L2>(&in.pvz[q]);
        }
        if (in.pinned) out.pinned[k] = in.pinned[q];
        if (in.temp) out.temp[k] = in.temp[q];
        if (in.kx) {
            out.kx[k] = ld_l2<L2>(&in.kx[q]); out.ky[k] = ld_l2<L2>(&in.ky[q]);
            out.kvx[k] = ld_l2<L2>(&in.kvx[q]); out.kvy[k] = ld_l2<L2>(&in.kvy[q]);
            if (D == 3) { out.kz[k] = ld_l2<L2>(&in.kz[q]); out.kvz[k] = ld_l2<L2>(&in.kvz[q]); }
        }
    }
}

}  // namespace ge
