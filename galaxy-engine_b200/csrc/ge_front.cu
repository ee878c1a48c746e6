// ge_front.cu -- everything before the tree build for small simulations, one
// thread-block cluster per simulation: kick + drift, root box, Morton keys,
// the stable radix sort and the gather of the state.
//
// The same steps as the per-pass kernels (ge_integrate.cu, ge_sort.cu), with
// the same operations on every particle, so keys, order and state are equal
// bit for bit.  A simulation of a few thousand particles leaves the per-pass
// kernels nothing to do but wait for one another: nine launches of 5 .. 10 us
// (kick, box, zeroing, keys, four or seven radix passes, gather).  Here its
// particles stay in the registers and shared memory of up to 16 blocks, which
// exchange box corners, digit counts and keys through distributed shared
// memory between cluster barriers; a radix pass is then two barriers.
//
// Block r of the cluster holds the simulation's slots [r T, r T + T), T =
// items * 512, and warp w of the block the 32 * items consecutive slots from
// 32 * items * w, in increasing order of (item, lane): counts taken in that
// order keep the sort stable.
#include <cfloat>
#include <cooperative_groups.h>

#include "ge_device.cuh"
#include "ge_front_dev.cuh"
#include "ge_internal.h"

namespace cg = cooperative_groups;

namespace ge {

constexpr int kFrontThreads = 512;
constexpr int kFrontWarps = kFrontThreads / 32;
constexpr uint32_t kFrontCluster = 1u << (kFrontSizes - 1);   // most blocks per simulation: 16
constexpr int kFrontItems = 4;           // most particles per thread
constexpr int kFrontBits = 9, kFrontRadix = 1 << kFrontBits;   // as the per-pass sort
static_assert(kFrontRadix == kFrontThreads, "one thread per digit");

template <int D, int ITEMS>
struct FrontSmem {
    uint64_t word[kFrontThreads * ITEMS];   // 2D key << 28 | index; 3D key
    uint32_t val[D == 3 ? kFrontThreads * ITEMS : 1];   // 3D index
    uint32_t whist[kFrontWarps][kFrontRadix];
    uint32_t cnt[kFrontRadix], off[kFrontRadix];
    uint32_t scan[kFrontWarps];
    uint32_t lo[3], hi[3];                  // the block's corners (ordered words)
    float4 box;
};

template <int D, int ITEMS>
__global__ void __launch_bounds__(kFrontThreads, 2)
k_front(State in, State out, StepParams p, Segs g, Tree t, uint64_t *keys, uint32_t *vals) {
    dep_wait();
    extern __shared__ __align__(16) unsigned char front_smem[];
    FrontSmem<D, ITEMS> &sm = *reinterpret_cast<FrontSmem<D, ITEMS> *>(front_smem);
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t C = cl.num_blocks(), rank = cl.block_rank();
    const uint32_t sg = blockIdx.x / C;
    const uint32_t lo = seg_lo(g, sg), hi = seg_hi(g, sg, (uint32_t)p.n), ns = hi - lo;
    // this simulation's items per thread: a power of two of at most ITEMS
    uint32_t items = 1, shift = 9;   // T = items * 512 = 1 << shift
    while (items < (uint32_t)ITEMS && items * kFrontThreads * C < ns) { items *= 2; shift++; }
    const uint32_t tid = threadIdx.x, w = tid >> 5, lane = tid & 31u;
    const uint32_t first = (rank << shift) + w * 32u * items + lane;   // item it: first + 32 it

    // kick + drift, and the corners
    float pos[ITEMS][3];
    {
        float cl_[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, ch[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        float vel[ITEMS][3], acc[ITEMS][3];
#pragma unroll
        for (int it = 0; it < ITEMS; it++) {
            const uint32_t r = first + 32u * it, i = lo + r;
            if ((uint32_t)it >= items || r >= ns) continue;
            pos[it][0] = in.x[i]; pos[it][1] = in.y[i];
            vel[it][0] = in.vx[i]; vel[it][1] = in.vy[i];
            acc[it][0] = in.ax[i]; acc[it][1] = in.ay[i];
            pos[it][2] = vel[it][2] = acc[it][2] = 0.0f;
            if (D == 3) { pos[it][2] = in.z[i]; vel[it][2] = in.vz[i]; acc[it][2] = in.az[i]; }
        }
#pragma unroll
        for (int it = 0; it < ITEMS; it++) {
            const uint32_t r = first + 32u * it, i = lo + r;
            if ((uint32_t)it >= items || r >= ns) continue;
            if (!(in.pinned && in.pinned[i])) kick_drift<D>(in, p, (int)i, pos[it], vel[it], acc[it]);
#pragma unroll
            for (int a = 0; a < D; a++) {
                cl_[a] = ref_min(cl_[a], pos[it][a]);
                ch[a] = ref_max(ch[a], pos[it][a]);
            }
        }
        if (tid < 3) { sm.lo[tid] = 0xFFFFFFFFu; sm.hi[tid] = 0u; }
        __syncthreads();
#pragma unroll
        for (int a = 0; a < D; a++) {
            const uint32_t l = __reduce_min_sync(0xffffffffu, f2o(cl_[a]));
            const uint32_t h = __reduce_max_sync(0xffffffffu, f2o(ch[a]));
            if (lane == 0) {
                atomicMin(&sm.lo[a], l);
                atomicMax(&sm.hi[a], h);
            }
        }
    }
    cl.sync();   // every block's corners
    if (w == 0) {
        float l[3] = {0.f, 0.f, 0.f}, h[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int a = 0; a < D; a++) {   // C <= 16 blocks, one per lane
            const uint32_t ul = lane < C ? *cl.map_shared_rank(&sm.lo[a], lane) : 0xFFFFFFFFu;
            const uint32_t uh = lane < C ? *cl.map_shared_rank(&sm.hi[a], lane) : 0u;
            l[a] = o2f(__reduce_min_sync(0xffffffffu, ul));
            h[a] = o2f(__reduce_max_sync(0xffffffffu, uh));
        }
        if (lane == 0) {
            const float4 bb = root_box<D>(l, h);
            sm.box = bb;
            if (rank == 0) {   // the root node: cell = box, range = the simulation
                g.box[sg] = bb;
                t.cell[sg] = bb;
                t.info[sg] = make_uint4(0u, 0u, lo, hi);
            }
        }
    }
    __syncthreads();
    const float4 bb = sm.box;
    uint64_t k[ITEMS];
    uint32_t v[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; it++) {
        const uint32_t r = first + 32u * it, i = lo + r;
        k[it] = 0ull;
        v[it] = i;
        if ((uint32_t)it >= items || r >= ns) continue;
        k[it] = morton_key<D>(bb, pos[it][0], pos[it][1], pos[it][2]);
        if (D == 2) k[it] = (k[it] << 28) | (uint64_t)i;
    }

    constexpr int P = D == 2 ? 4 : 7, S0 = D == 2 ? 28 : 0;
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll 1
    for (int ps = 0; ps < P; ps++) {
        const int sh = S0 + kFrontBits * ps;
        for (int q = lane; q < kFrontRadix; q += 32) sm.whist[w][q] = 0u;
        __syncwarp();
        uint32_t rk[ITEMS];   // rank among the warp's earlier keys of its digit
#pragma unroll
        for (int it = 0; it < ITEMS; it++) {
            rk[it] = 0u;
            if ((uint32_t)it >= items) continue;   // uniform
            const bool ok = first + 32u * it < ns;
            const uint32_t d = (uint32_t)(k[it] >> sh) & (kFrontRadix - 1u);
            const unsigned peers = digit_peers<kFrontBits>(d, ok);
            const int leader = __ffs(peers) - 1;
            uint32_t prev = 0;
            if (ok && (int)lane == leader) {
                prev = sm.whist[w][d];
                sm.whist[w][d] = prev + (uint32_t)__popc(peers);
            }
            prev = __shfl_sync(0xffffffffu, prev, leader & 31);
            rk[it] = prev + (uint32_t)__popc(peers & lt);
            __syncwarp();
        }
        __syncthreads();
        uint32_t sum = 0;   // thread = digit: exclusive over the block's warps
#pragma unroll
        for (int q = 0; q < kFrontWarps; q++) {
            const uint32_t c = sm.whist[q][tid];
            sm.whist[q][tid] = sum;
            sum += c;
        }
        sm.cnt[tid] = sum;
        cl.sync();   // every block's counts are out, and its keys in registers
        uint32_t total = 0, before = 0;
        uint32_t c[kFrontCluster];   // all of them on their way at once
#pragma unroll
        for (uint32_t q = 0; q < kFrontCluster; q++)
            c[q] = q < C ? *cl.map_shared_rank(&sm.cnt[tid], q) : 0u;
#pragma unroll
        for (uint32_t q = 0; q < kFrontCluster; q++) {
            before += q < rank ? c[q] : 0u;
            total += c[q];
        }
        uint32_t incl = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += u;
        }
        if (lane == 31) sm.scan[w] = incl;
        __syncthreads();
        uint32_t base = 0;
#pragma unroll
        for (uint32_t q = 0; q < kFrontWarps; q++) base += q < w ? sm.scan[q] : 0u;
        sm.off[tid] = base + incl - total + before;
        __syncthreads();
#pragma unroll
        for (int it = 0; it < ITEMS; it++) {
            if ((uint32_t)it >= items || first + 32u * it >= ns) continue;
            const uint32_t d = (uint32_t)(k[it] >> sh) & (kFrontRadix - 1u);
            const uint32_t to = sm.off[d] + sm.whist[w][d] + rk[it];   // < ns
            const uint32_t at = to & ((1u << shift) - 1u);
            *cl.map_shared_rank(&sm.word[at], to >> shift) = k[it];
            if (D == 3) *cl.map_shared_rank(&sm.val[at], to >> shift) = v[it];
        }
        cl.sync();   // every key in its place
        if (ps + 1 < P) {
#pragma unroll
            for (int it = 0; it < ITEMS; it++) {
                const uint32_t at = w * 32u * items + lane + 32u * it;
                if ((uint32_t)it >= items || first + 32u * it >= ns) continue;
                k[it] = sm.word[at];
                if (D == 3) v[it] = sm.val[at];
            }
        }
    }

    // the sorted keys for the build, and the state in their order
    constexpr int U = 2;
    for (uint32_t at0 = tid; at0 < (1u << shift); at0 += kFrontThreads * U) {
        uint32_t kk[U], j[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t at = at0 + u * kFrontThreads, r = (rank << shift) + at;
            const bool ok = at < (1u << shift) && r < ns;
            kk[u] = ok ? lo + r : hi;
            j[u] = lo;
            if (!ok) continue;
            const uint64_t word = sm.word[at];
            j[u] = D == 2 ? (uint32_t)(word & 0x0FFFFFFFull) : sm.val[at];
            keys[kk[u]] = word;
            if (D == 3) vals[kk[u]] = j[u];
        }
        gather_state<D, U, true>(in, out, 0, kk, j, hi);
    }
}

template <int D, int ITEMS>
static cudaError_t front_launch(int blocks, int cluster, cudaStream_t st, const State &in,
                                const State &out, const StepParams &p, const Segs &g, const Tree &t,
                                SortScratch &ss) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kFrontThreads);
    cfg.dynamicSmemBytes = sizeof(FrontSmem<D, ITEMS>);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, k_front<D, ITEMS>, in, out, p, g, t, ss.keys[0], ss.vals[0]);
}

// More than 48 KB of shared memory and clusters of 16 blocks (a device that
// refuses those keeps the 8 that every device has).  Both are attributes of the
// kernel on the current device.
template <int D, int ITEMS>
static bool front_attributes() {
    const void *k = (const void *)k_front<D, ITEMS>;
    const bool ok = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(FrontSmem<D, ITEMS>)) == cudaSuccess;
    if (!ok || cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        (void)cudaGetLastError();
    return ok;
}

template <int D>
static void front_limits(FrontLimits &lim) {
    lim.known = true;
    if (!front_attributes<D, 1>() || !front_attributes<D, 2>() || !front_attributes<D, 4>()) return;
    for (int q = 0; q < kFrontSizes; q++) {   // the variant with the most shared memory
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1u << q);
        cfg.blockDim = dim3(kFrontThreads);
        cfg.dynamicSmemBytes = sizeof(FrontSmem<D, kFrontItems>);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1u << q;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, (const void *)k_front<D, kFrontItems>, &cfg) !=
            cudaSuccess) {
            (void)cudaGetLastError();
            fit = 0;
        }
        lim.fit[q] = fit;
    }
}

// Few keys per block keep a pass short, many blocks make its barriers and
// remote stores long (a pass at 16 blocks: 0.7 us of ranking, 2 us for the
// counts, 1.8 us for the keys), and a second block on an SM costs as much as
// the shorter passes gain (10 simulations of 16k in clusters of 16 blocks: kick
// to gather 55 us, of 8 blocks 43).  So: the largest cluster that holds every
// simulation with one block per SM (half of those that fit, which are fewer
// than the SMs allow: a cluster lies inside one GPC, 14 of 16 blocks, 33 of 8,
// 71 of 4).  Where none does, the smallest that holds the largest simulation,
// while at most an eighth more of them than fit wait for the first to end and
// there are no more blocks than fit one by one; else the per-pass kernels.
// Step against those (us):
//   2D 2k 174 -> 154, 16k 179 -> 162, 32k 186 -> 177, 45k 189 -> 193 (8 items)
//   3D 16k 391 -> 356, 60k 465 -> 473
//   2D, 10 of 16k in clusters of 16 / 8 blocks 172 / 159 (per pass 179), 18
//   220 / 203 (218); 72 of 4k in clusters of 4 / 2 190 / 175 (210); 73 of up to
//   8k in clusters of 4 224 (231), 35 of up to 16k of 8 215 (220); 16 of up to
//   32k in clusters of 16 194 (192), 18 217 (205)
int front_plan(int dims, int64_t largest, int64_t sims, FrontLimits &lim) {
    if (sims < 1 || largest > (int64_t)kFrontCluster * kFrontThreads * kFrontItems) return 0;
    if (!lim.known) {
        if (dims == 2) front_limits<2>(lim);
        else front_limits<3>(lim);
    }
    int best = -1;   // log2 of the blocks
    for (int q = kFrontSizes - 1; q >= 0; q--) {
        const int64_t threads = (int64_t)kFrontThreads << q;
        if (threads * kFrontItems < largest) break;
        if (q > 0 && threads / 2 >= largest) continue;   // half of it would do
        if (sims <= lim.fit[q] + lim.fit[q] / 8 && sims << q <= lim.fit[0]) best = q;
        if (2 * sims <= lim.fit[q]) break;
    }
    if (best < 0) return 0;
    int items = 1;
    while (((int64_t)items * kFrontThreads << best) < largest) items *= 2;
    return 256 << best | items;
}

template <int D>
static cudaError_t front_dims(int plan, cudaStream_t st, const State &in, const State &out,
                              const StepParams &p, const Segs &g, const Tree &t, SortScratch &ss) {
    const int c = plan >> 8, blocks = g.S * c;
    switch (plan & 255) {
    case 1: return front_launch<D, 1>(blocks, c, st, in, out, p, g, t, ss);
    case 2: return front_launch<D, 2>(blocks, c, st, in, out, p, g, t, ss);
    case 4: return front_launch<D, 4>(blocks, c, st, in, out, p, g, t, ss);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_front(int dims, int plan, const State &in, const State &out,
                         const StepParams &p, const Segs &g, const Tree &t, SortScratch &ss,
                         cudaStream_t st) {
    return dims == 2 ? front_dims<2>(plan, st, in, out, p, g, t, ss)
                     : front_dims<3>(plan, st, in, out, p, g, t, ss);
}

}  // namespace ge
