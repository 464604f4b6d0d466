// Device helpers and the launch of the on-chip batched kernels (cg_onchip.cu,
// cg_onchip_mixed.cu).
#pragma once

#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "cg_dev.cuh"
#include "cg_onchip.cuh"

namespace cmcg {
namespace {

namespace cgrp = cooperative_groups;

// f(q) for the slots q < nk (nk even, at most NS), four at a time (the last two
// may stand alone) so that a step's loads are in flight together; the branches
// are uniform.
template <int NS, typename F>
__device__ __forceinline__ void oc_slots(int nk, F&& f) {
#pragma unroll
    for (int q0 = 0; q0 < NS; q0 += 4) {
        if (q0 + 2 < nk) {
            f(q0);
            f(q0 + 1);
            f(q0 + 2);
            f(q0 + 3);
        } else if (q0 < nk) {
            f(q0);
            f(q0 + 1);
        }
    }
}

// How the threads that solve one system synchronise: as a CTA, as a cluster of
// CTAs, or as a group of T threads of a 512-thread CTA (a named barrier of its
// own: groups of 256 take barriers 1 and 2, groups of 128 take 3 .. 6, since one
// group may already be split while another still works whole, and a barrier
// must not be used with two thread counts at once).
enum OcScope { OC_CTA, OC_CLUSTER, OC_GROUP };
template <OcScope SC, int T>
__device__ __forceinline__ void oc_sync() {
    if constexpr (SC == OC_CLUSTER) cgrp::this_cluster().sync();
    else if constexpr (SC == OC_CTA) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(512 / T - 1 + static_cast<int>(threadIdx.x) / T), "n"(T) : "memory");
}


// v[j][h] (accumulator h of the thread) summed over all virtual warps, into
// v[j][0] of every thread; red: [NV][kOcWarps] of this CTA or group (kOcWarps: the
// virtual warps at most), written by
// every CTA of the cluster; one barrier. Reused only after another barrier.
template <typename VT, int NV, int T, int H, OcScope SC, int kOcWarps>
__device__ __forceinline__ void oc_sum(VT (&v)[NV][H], VT (&red)[2 * kOcWarps], int rank, int ctas) {
    constexpr int W = T / 32;
    const int lane = threadIdx.x & 31, warp = static_cast<int>(threadIdx.x % T) >> 5;
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
        for (int h = 0; h < H; ++h) v[j][h] = warp_sum(v[j][h]);
    if constexpr (SC == OC_CLUSTER) {
        // lane c stores into CTA c
        if (lane < ctas) {
            VT* dst = cgrp::this_cluster().map_shared_rank(&red[0], lane);
#pragma unroll
            for (int j = 0; j < NV; ++j)
#pragma unroll
                for (int h = 0; h < H; ++h) dst[j * kOcWarps + (h * ctas + rank) * W + warp] = v[j][h];
        }
    } else if (lane == 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j)
#pragma unroll
            for (int h = 0; h < H; ++h) red[j * kOcWarps + h * W + warp] = v[j][h];
    }
    oc_sync<SC, T>();
    const int nw = H * W * (SC == OC_CLUSTER ? ctas : 1);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        VT s = lane < nw ? red[j * kOcWarps + lane] : VT(0);
        if constexpr (SC == OC_CLUSTER && kOcWarps > 32)   // (three or four CTAs)
            if (lane + 32 < nw) s += red[j * kOcWarps + lane + 32];
        v[j][0] = warp_sum(s);
    }
}

// Next work item of the group, CTA or cluster.
template <OcScope SC, int T>
__device__ __forceinline__ int oc_fetch(int32_t* next, int* slot, int rank, int ctas) {
    if (rank == 0 && threadIdx.x % T == 0) {
        const int item = atomicAdd(next, 1);
        if constexpr (SC == OC_CLUSTER)
            for (int c = 0; c < ctas; ++c) *cgrp::this_cluster().map_shared_rank(slot, c) = item;
        else *slot = item;
    }
    oc_sync<SC, T>();
    const int item = *slot;
    oc_sync<SC, T>();
    return item;
}

// The thread's p entries that the ranks below and above (contiguous rows, `own`
// per CTA) gather are stored into their halos too: the store of entry i of P.
template <typename VT>
struct OcHalo {
    VT* below = nullptr;
    VT* above = nullptr;
    int own, reach;
    __device__ __forceinline__ OcHalo(VT* P, int rank, int ctas, int own_, int reach_) : own(own_), reach(reach_) {
        cgrp::cluster_group cl = cgrp::this_cluster();
        if (rank > 0) below = cl.map_shared_rank(P, rank - 1) + own;
        if (rank + 1 < ctas) above = cl.map_shared_rank(P, rank + 1) - own;
    }
    __device__ __forceinline__ void store(int i, VT v) const {
        if (below && i < reach) below[i] = v;
        if (above && i >= own - reach) above[i] = v;
    }
};

// Clusters of the form that can be resident at once (looked up once per device,
// kernel and shape).
cmcg_status onchip_resident(const void* kern, const cudaLaunchConfig_t& cfg, int ctas, int* out) {
    static std::mutex mu;
    static std::map<std::tuple<int, const void*, int, size_t>, int> known;
    int device = 0;
    CMCG_CUDA(cudaGetDevice(&device));
    const auto key = std::make_tuple(device, kern, ctas, cfg.dynamicSmemBytes);
    {
        std::lock_guard<std::mutex> lock(mu);
        const auto it = known.find(key);
        if (it != known.end()) { *out = it->second; return CMCG_OK; }
    }
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        n = 0;
    }
    std::lock_guard<std::mutex> lock(mu);
    known[key] = n;
    *out = n;
    return CMCG_OK;
}

// Starts a persistent kernel of one launch form on `items` work items: as many
// CTAs or clusters as are resident at once. *launched = false where the device
// cannot place a cluster of the form.
cmcg_status onchip_start(const void* kern, void** params, int items, const OnchipForm& f, size_t smem, int sms,
                         cudaStream_t stream, bool* launched) {
    *launched = false;
    if (!kern) return CMCG_OK;
    CMCG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    CMCG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(f.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(f.ctas);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    int groups = sms * f.per_sm;   // CTAs or clusters at once
    if (f.ctas > 1) {
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cfg.gridDim = dim3(static_cast<unsigned>(f.ctas));
        CMCG_TRY(onchip_resident(kern, cfg, f.ctas, &groups));
        if (groups < 1) return CMCG_OK;
    }
    groups = std::max(1, std::min(groups, items));
    cfg.gridDim = dim3(static_cast<unsigned>(groups * f.ctas));
    CMCG_CUDA(cudaLaunchKernelExC(&cfg, kern, params));
    *launched = true;
    return CMCG_OK;
}

}  // namespace
}  // namespace cmcg
