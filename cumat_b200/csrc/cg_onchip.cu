// Batched PCG on the diagonal layout with a system's whole state on the chip.
//
// One CTA, or for large systems a cluster of two (FP32) or two to four (FP64), solves
// one system instance at a time from an atomic work counter. The values are
// staged into shared memory once per system, p lives there with a zero halo for
// the gathers, and r, x, p, the inverse diagonal and q of a thread's rows (up
// to 16 FP32, 8 FP64) in registers: an iteration moves, per row, one p store,
// the gathers and the values through shared memory, and nothing through L2. CTAs
// have 512 threads per SM in every form (128 registers a thread); the latency is
// hidden by the rows of a thread, not by occupancy.
//
// What bounds it: the shared-memory pipe is the busiest unit (5 diagonals FP32: 10 words
// per row and iteration), for 58 .. 65 % of the cycles where a system has one CTA or a
// part of it, 42 .. 46 % in clusters (148 systems of 16,384 rows FP32, of 10,000 FP64).
// The rest is latency: of a step's loads, with 16 warps on an SM, and of three barriers
// an iteration, which in a cluster are cluster barriers with a fence. The kernels it replaces read the values, column indices
// and inverse diagonal from L2 in every iteration (FP32), and r, x and q too
// (FP64, where 148 large systems exceed the L2). Measured, there against here, ms:
// FP32 to 1e-6, 296 systems of 16,384 rows 11.5 / 6.3, 592 of 8100 7.8 / 3.2,
// 1184 of 1024 1.87 / 0.61, 20 of 1600 0.33 / 0.22; FP64 to 1e-10, 296 of 10,000
// 12.9 / 10.9, 592 of 4096 11.1 / 2.7, 20 of 16,384 11.3 / 2.1.
//
// FP32 keeps the sums of the 1024-thread kernel for every form: virtual thread
// v < 1024 owns the rows v + 1024 k and adds them in order; a thread of a
// smaller CTA plays H = 1024 / threads of them with separate accumulators, and
// a pair of CTAs splits the virtual threads, 512 each, so its rows interleave in
// runs of 512 and each CTA holds p of both (the half its neighbour gathers is
// stored into both through distributed shared memory). 32 virtual warps are
// combined by the same shuffle tree in every form, so results do not depend on
// the form. FP64 clusters own contiguous rows and exchange a halo.
#include <algorithm>

#include "cg_dev.cuh"
#include "cg_onchip.cuh"
#include "cg_onchip_dev.cuh"

namespace cmcg {
namespace {

// Scratch of one group of threads (shared memory); FP32 has 32 virtual warps in
// every form, FP64 up to four CTAs of 16.
template <typename VT>
struct alignas(16) OcScratch {
    static constexpr int kOcWarps = sizeof(VT) == 4 ? 32 : 64;
    VT redA[2 * kOcWarps];
    VT redB[2 * kOcWarps];
    int slot;
};
static_assert(sizeof(OcScratch<double>) <= kOnchipStatic64, "");

// Solves the work items [t.lo, t.hi) until none is left. T threads (and, OC_CLUSTER,
// the cluster's CTAs) per system; H: virtual threads a thread plays (FP32; 1
// where the form's own order is used). FP32 clusters interleave (see the file
// comment). sm: the group's dynamic shared memory.
template <typename VT, typename MT, int ND, int T, int H, OcScope SC>
__device__ __forceinline__ void onchip_items(const OnchipArgs<VT, MT>& a, const OnchipItems& t, unsigned char* sm,
                                             OcScratch<VT>& sc) {
    constexpr bool CL = SC == OC_CLUSTER;
    constexpr int NS = kOnchipSlots<VT>;
    constexpr bool IL = CL && sizeof(VT) == 4;   // interleaved pair
    constexpr int ST = IL ? 2 * T : T;           // rows from slot to slot
    constexpr int kOcWarps = OcScratch<VT>::kOcWarps;
    VT(&redA)[2 * kOcWarps] = sc.redA;
    VT(&redB)[2 * kOcWarps] = sc.redB;
    const int tid = threadIdx.x % T;
    int rank = 0, ctas = 1;
    if constexpr (CL) {
        rank = static_cast<int>(cgrp::this_cluster().block_rank());
        ctas = static_cast<int>(cgrp::this_cluster().num_blocks());
    }
    const int M = (a.margin + 3) & ~3;
    VT* const P = reinterpret_cast<VT*>(sm) + M;
    const VT tol = static_cast<VT>(a.tol);
    for (;;) {
        const int item = t.lo + oc_fetch<SC, T>(t.next, &sc.slot, rank, ctas);
        if (item >= t.hi) break;
        const int s = a.order[item / a.ob], bi = item % a.ob, inst = bi * a.n_sys + s;
        const int r0 = a.row_off[s], n = a.row_off[s + 1] - r0;
        const int nk = onchip_slots(n, T, ctas);
        const int own = nk * T;
        // local row of slot q: row0 + ST q; its p entry P[p0 + ST q]
        const int row0 = IL ? rank * T + tid : rank * own + tid;
        const int p0 = IL ? row0 : tid;
        const int pend = IL ? 2 * own : own;
        MT* const vs = reinterpret_cast<MT*>(P + pend + M) + tid;
        const int64_t vo = static_cast<int64_t>(bi) * a.rows;
        const VT* bv = a.b + (a.b_b == 1 ? 0 : vo) + r0;
        const VT* gv = a.guess ? a.guess + (a.g_b == 1 ? 0 : vo) + r0 : nullptr;
        const VT* dg = a.dinv ? a.dinv + (a.dinv_b == 1 ? 0 : vo) + r0 : nullptr;
        VT* xg = a.x + vo + r0;
        const MT* dv = a.vals + (a.mb == 1 ? 0 : static_cast<int64_t>(bi) * a.vstride) + __ldg(a.base + s);
        int po[ND], reach = 0;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const int o = __ldg(a.off + s * kDiaMax + d);
            po[d] = p0 + o;
            reach = max(reach, abs(o));
        }
        const bool mid0 = po[ND / 2] == p0;   // the middle diagonal is the main one
        for (int i = tid; i < M; i += T) P[-1 - i] = P[pend + i] = VT(0);
        VT R[NS], X[NS], Pn[NS], D[NS], Q[NS];
        VT acc[2][H];
#pragma unroll
        for (int h = 0; h < H; ++h) acc[0][h] = acc[1][h] = VT(0);
        // values (0 past the system's end), b, inverse diagonal, r = b - A x0
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            R[q] = X[q] = Pn[q] = VT(0);
            D[q] = VT(1);
            if (q >= nk) continue;
            const int row = row0 + ST * q;
            const bool ok = row < n;
            const MT* vr = dv + static_cast<int64_t>(row / kDiaBlockRows) * ND * kDiaBlockRows + row % kDiaBlockRows;
            MT w[ND];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                w[d] = ok ? __ldg(vr + d * kDiaBlockRows) : MT{};
                vs[(d * nk + q) * T] = w[d];
            }
            if (ok) {
                const VT b_i = bv[row];
                if (dg) D[q] = dg[row];
                if (gv) {
                    VT v = VT(0);
#pragma unroll
                    for (int d = 0; d < ND; ++d) {
                        const int c = row + po[d] - p0;
                        v = fma(mval<VT>(w[d]), c >= 0 && c < n ? gv[c] : VT(0), v);
                    }
                    R[q] = b_i - v;
                    X[q] = gv[row];
                    acc[1][q % H] += R[q] * R[q];
                } else {
                    R[q] = b_i;
                }
                acc[0][q % H] += b_i * b_i;
            }
        }
        // p entries other CTAs of the cluster gather: stored there too
        const OcHalo<VT> halo(P, CL && !IL ? rank : 0, CL && !IL ? ctas : 1, own, reach);
        VT* pair = nullptr;   // IL: p of the pair's other CTA
        bool push = false;
        if constexpr (IL) {
            pair = cgrp::this_cluster().map_shared_rank(P, rank ^ 1);
            push = tid < reach || tid >= T - reach;
        }
        const auto store_p = [&](int q, VT v) {
            const int i = p0 + ST * q;
            P[i] = v;
            if constexpr (IL) {
                if (push) pair[i] = v;
            } else if constexpr (CL) {
                halo.store(i, v);
            }
        };
        oc_sum<VT, 2, T, H, SC, kOcWarps>(acc, redA, rank, ctas);   // (also: the halos are zero in every CTA)
        const VT bb = acc[0][0];
        VT rr = gv ? acc[1][0] : bb;
        const VT thr = tol * tol * bb;
        int32_t status = ST_RUNNING, it = 0;
        if ((a.abs_zero_test && bb < tol * tol) || bb == VT(0)) {
#pragma unroll
            for (int q = 0; q < NS; ++q) X[q] = VT(0);
            status = CMCG_SOLVE_ZERO_RHS;
        } else if (!finite_(rr) || !finite_(bb)) {
            status = CMCG_SOLVE_NON_FINITE;
        } else if (rr < thr) {
            status = CMCG_SOLVE_CONVERGED;
        } else {
            VT rz1[1][H];
#pragma unroll
            for (int h = 0; h < H; ++h) rz1[0][h] = VT(0);
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                if (q >= nk) continue;
                const VT zi = D[q] * R[q];
                Pn[q] = zi;
                store_p(q, zi);
                rz1[0][q % H] += R[q] * zi;
            }
            oc_sum<VT, 1, T, H, SC, kOcWarps>(rz1, redB, rank, ctas);   // (and: p is in place)
            VT rz = rz1[0][0];
            if (!finite_(rz)) status = CMCG_SOLVE_NON_FINITE;
            else if (!(rz > VT(0))) status = CMCG_SOLVE_BREAKDOWN;
            const int64_t maxit = sys_max_iter(a.max_iter, n);
            while (status == ST_RUNNING) {
                if (it >= maxit) { status = CMCG_SOLVE_MAX_ITER; break; }
                VT pq[1][H];
#pragma unroll
                for (int h = 0; h < H; ++h) pq[0][h] = VT(0);
                oc_slots<NS>(nk, [&](int q) {
                    VT v = VT(0);
#pragma unroll
                    for (int d = 0; d < ND; ++d) {
                        const VT pv = d == ND / 2 && mid0 ? Pn[q] : P[po[d] + ST * q];
                        v = fma(mval<VT>(vs[(d * nk + q) * T]), pv, v);
                    }
                    Q[q] = v;
                    pq[0][q % H] += Pn[q] * v;
                });
                oc_sum<VT, 1, T, H, SC, kOcWarps>(pq, redA, rank, ctas);
                const VT alpha = rz / pq[0][0];
                if (!finite_(pq[0][0]) || !finite_(alpha)) { status = CMCG_SOLVE_NON_FINITE; break; }
                if (!(pq[0][0] > VT(0))) { status = CMCG_SOLVE_BREAKDOWN; break; }
                VT s2[2][H];
#pragma unroll
                for (int h = 0; h < H; ++h) s2[0][h] = s2[1][h] = VT(0);
                oc_slots<NS>(nk, [&](int q) {
                    X[q] += alpha * Pn[q];
                    const VT ri = R[q] - alpha * Q[q];
                    R[q] = ri;
                    s2[0][q % H] += ri * ri;
                    s2[1][q % H] += ri * (D[q] * ri);
                });
                oc_sum<VT, 2, T, H, SC, kOcWarps>(s2, redB, rank, ctas);
                rr = s2[0][0];
                const VT rzn = s2[1][0];
                if (!finite_(rr) || !finite_(rzn)) { status = CMCG_SOLVE_NON_FINITE; break; }
                if (rr < thr) { status = CMCG_SOLVE_CONVERGED; break; }
                if (!(rzn > VT(0))) { status = CMCG_SOLVE_BREAKDOWN; break; }
                const VT beta = rzn / rz;
                rz = rzn;
                oc_slots<NS>(nk, [&](int q) {
                    Pn[q] = D[q] * R[q] + beta * Pn[q];
                    store_p(q, Pn[q]);
                });
                oc_sync<SC, T>();
                ++it;
            }
        }
#pragma unroll
        for (int q = 0; q < NS; ++q)
            if (row0 + ST * q < n && q < nk) xg[row0 + ST * q] = X[q];
        if (rank == 0 && tid == 0) {
            a.st.it[inst] = it;
            a.st.status[inst] = status;
            a.st.rr[inst] = static_cast<double>(rr);
            a.st.bb[inst] = static_cast<double>(bb);
            a.st.outer[inst] = 0;
            a.st.err[inst] = (status == CMCG_SOLVE_ZERO_RHS) ? 0.0 : sqrt(static_cast<double>(rr) / static_cast<double>(bb));
        }
        // (the next fetch's barriers separate this system's reads from the next one's stores)
    }
    oc_sync<SC, T>();   // (no CTA goes on while another may still address its shared memory)
}

// One form per launch (FP64).
template <typename VT, typename MT, int ND, int T, bool CL>
__global__ void __launch_bounds__(T, 512 / T) k_onchip(const __grid_constant__ OnchipArgs<VT, MT> a,
                                                       const __grid_constant__ OnchipItems t) {
    extern __shared__ __align__(16) unsigned char oc_smem[];
    __shared__ OcScratch<VT> sc;
    onchip_items<VT, MT, ND, T, 1, CL ? OC_CLUSTER : OC_CTA>(a, t, oc_smem, sc);
}

// All forms in one launch (FP32): every 512-thread CTA first works on the largest
// systems with its pair (CL), then on its own, then as two groups of 256 and at
// last four of 128 threads, each with its part of the shared memory.
template <typename MT, int ND, bool CL>
__global__ void __launch_bounds__(512, 1) k_onchip_all(const __grid_constant__ OnchipArgs<float, MT> a,
                                                       const __grid_constant__ OnchipWork w) {
    extern __shared__ __align__(16) unsigned char oc_smem[];
    __shared__ OcScratch<float> sc;
    if constexpr (CL) onchip_items<float, MT, ND, 512, 1, OC_CLUSTER>(a, w.t[0], oc_smem, sc);
    onchip_items<float, MT, ND, 512, 2, OC_CTA>(a, w.t[1], oc_smem, sc);
    // (a group's scratch is at the start of its part)
    static_assert(sizeof(OcScratch<float>) <= kOnchipGroupScratch, "");
    unsigned char* half = oc_smem + threadIdx.x / 256 * (w.smem / 2);
    onchip_items<float, MT, ND, 256, 4, OC_GROUP>(a, w.t[2], half + kOnchipGroupScratch,
                                                  *reinterpret_cast<OcScratch<float>*>(half));
    unsigned char* quarter = oc_smem + threadIdx.x / 128 * (w.smem / 4);
    onchip_items<float, MT, ND, 128, 8, OC_GROUP>(a, w.t[3], quarter + kOnchipGroupScratch,
                                                  *reinterpret_cast<OcScratch<float>*>(quarter));
}

template <typename VT, typename MT, int ND>
const void* onchip_kernel(const OnchipForm& f) {
    if (f.threads == 512 && f.ctas > 1) return reinterpret_cast<const void*>(k_onchip<VT, MT, ND, 512, true>);
    if (f.threads == 512) return reinterpret_cast<const void*>(k_onchip<VT, MT, ND, 512, false>);
    if (f.threads == 256) return reinterpret_cast<const void*>(k_onchip<VT, MT, ND, 256, false>);
    if (f.threads == 128) return reinterpret_cast<const void*>(k_onchip<VT, MT, ND, 128, false>);
    return nullptr;
}

}  // namespace

#ifdef CMCG_ONCHIP_FP64
template <typename VT, typename MT>
cmcg_status onchip_launch(const OnchipArgs<VT, MT>& a, const OnchipItems& t, const OnchipForm& f, size_t smem, int nd,
                          int sms, cudaStream_t stream, bool* launched) {
    const void* kern = nd == 5 ? onchip_kernel<VT, MT, 5>(f) : nd == 7 ? onchip_kernel<VT, MT, 7>(f) : nullptr;
    OnchipArgs<VT, MT> args = a;
    OnchipItems items = t;
    void* params[] = {&args, &items};
    return onchip_start(kern, params, t.hi - t.lo, f, smem, sms, stream, launched);
}
#define CMCG_ONCHIP_INSTANTIATE(MT)                                                                               \
    template cmcg_status onchip_launch<double, MT>(const OnchipArgs<double, MT>&, const OnchipItems&,             \
                                                   const OnchipForm&, size_t, int, int, cudaStream_t, bool*);
#else
template <typename MT>
cmcg_status onchip_launch_all(const OnchipArgs<float, MT>& a, const OnchipWork& w, int nd, int sms, cudaStream_t stream,
                              bool* launched) {
    const bool pairs = w.t[0].hi > w.t[0].lo;
    const void* kern = nd == 5 ? (pairs ? reinterpret_cast<const void*>(k_onchip_all<MT, 5, true>)
                                        : reinterpret_cast<const void*>(k_onchip_all<MT, 5, false>))
                     : nd == 7 ? (pairs ? reinterpret_cast<const void*>(k_onchip_all<MT, 7, true>)
                                        : reinterpret_cast<const void*>(k_onchip_all<MT, 7, false>))
                               : nullptr;
    OnchipArgs<float, MT> args = a;
    OnchipWork work = w;
    void* params[] = {&args, &work};
    // (a cluster or CTA per item of its first tier, or per group of items of the later ones)
    const int items = pairs ? std::max(w.t[0].hi - w.t[0].lo, (w.t[3].hi - w.t[1].lo + 1) / 2) : w.t[3].hi - w.t[1].lo;
    return onchip_start(kern, params, items, OnchipForm{512, pairs ? 2 : 1, 1}, w.smem, sms, stream, launched);
}
#define CMCG_ONCHIP_INSTANTIATE(MT)                                                                                     \
    template cmcg_status onchip_launch_all<MT>(const OnchipArgs<float, MT>&, const OnchipWork&, int, int, cudaStream_t, \
                                               bool*);
#endif
CMCG_ONCHIP_INSTANTIATE(float)
CMCG_ONCHIP_INSTANTIATE(double)
CMCG_ONCHIP_INSTANTIATE(__nv_bfloat16)

}  // namespace cmcg
