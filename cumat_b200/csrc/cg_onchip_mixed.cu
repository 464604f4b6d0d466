// Mixed-precision batched CG with a system's whole FP32 state on the chip.
//
// The method of k_mixed_fast (cg_mixed.cu): FP32 CG on the Jacobi-scaled system
// S A S, increments xh folded into the FP64 solution with x += S xh, the
// residual replaced by S (b - A x) computed in FP64 whenever it fell by delta.
// The form is that of the plain on-chip kernel (cg_onchip.cu): scaled values and
// p in shared memory, r, xh and q of a thread's rows in registers. An iteration
// moves 9 words per row through the shared-memory pipe (four values, four
// gathers, one p store; 15 in k_mixed_fast) and nothing through L2. That pipe is
// busy for 53 % of the cycles (296 systems of 8100 rows and 592 of 4096, with the
// staging and a replacement in 40 iterations); the rest is latency, as there.
//
// The sums are those of k_mixed_fast's tiers, so results are the same bit for
// bit: one CTA of 512 threads for 4097 .. 8192 rows, else 256 virtual threads
// (CTAs of 256, or groups of 128 that play two each). Larger systems stay on
// k_mixed_fast: what does not fit one CTA's shared memory was slower here, as a
// cluster of two CTAs (its three cluster barriers an iteration took 5,000 of
// 11,000 cycles) and with 32 rows per thread and values from L2 (spills): 296
// systems of 16,384 rows to 1e-10 8.7 ms there, 12.4 ms in the second form. Below:
// 592 systems of 8100 rows 6.2 ms there, 3.9 here.
#include <type_traits>

#include "cg_dev.cuh"
#include "cg_onchip.cuh"
#include "cg_onchip_dev.cuh"

namespace cmcg {
namespace {

// Scratch of one group of threads (shared memory).
struct alignas(16) MixScratch {
    double redD[2 * 32];
    float redA[2 * 32];
    float redB[2 * 32];
    int slot;
    int guard[3];   // progress guard of BF16 inner values (k_mixed_fast)
};
constexpr int kMixGroupScratch = (static_cast<int>(sizeof(MixScratch)) + 15) / 16 * 16;
static_assert(kMixGroupScratch <= kOnchipMixScratch && sizeof(MixScratch) <= kOnchipStaticMix256, "");

// Solves the work items [t.lo, t.hi) until none is left, T threads per system,
// H virtual threads per thread. sm: the group's dynamic shared memory.
template <typename MI, typename MO, int ND, int T, int H, OcScope SC>
__device__ __forceinline__ void onchip_mixed_items(const OnchipMixArgs<MI, MO>& a, const OnchipItems& t,
                                                   unsigned char* sm, MixScratch& sc) {
    constexpr int NS = kOnchipSlots<float>;
    constexpr int kOcWarps = 32, rank = 0, ctas = 1;
    float(&redA)[2 * kOcWarps] = sc.redA;
    float(&redB)[2 * kOcWarps] = sc.redB;
    double(&redD)[2 * kOcWarps] = sc.redD;
    int(&guard)[3] = sc.guard;
    const int tid = threadIdx.x % T;
    const int M = (a.margin + 3) & ~3;
    float* const P = reinterpret_cast<float*>(sm) + M;
    const float d2 = a.delta * a.delta;
    constexpr bool kGuard = std::is_same<MI, __nv_bfloat16>::value;
    for (;;) {
        const int item = t.lo + oc_fetch<SC, T>(t.next, &sc.slot, rank, ctas);
        if (item >= t.hi) break;
        const int s = a.order[item / a.ob], bi = item % a.ob, inst = bi * a.n_sys + s;
        const int r0 = a.row_off[s], n = a.row_off[s + 1] - r0;
        const int nk = onchip_slots(n, T, ctas);
        const int own = nk * T;
        MI* const vs = reinterpret_cast<MI*>(P + own + M) + tid;   // slot q of stored diagonal e: vs[(e nk + q) T]
        const int64_t vo = static_cast<int64_t>(bi) * a.rows;
        const double* sv = a.s + (a.mb == 1 ? 0 : vo) + r0;
        const double* bv = a.b + (a.b_b == 1 ? 0 : vo) + r0;
        double* x = a.x + vo + r0;
        const int64_t base = __ldg(a.base + s);
        const MI* vi = a.vin + (a.mb == 1 ? 0 : static_cast<int64_t>(bi) * a.vin_stride) + base;
        const MO* vO = a.vout + (a.mb == 1 ? 0 : static_cast<int64_t>(bi) * a.vout_stride) + base;
        const bool unit = __ldg(a.unit + (a.mb == 1 ? 0 : bi) * a.n_sys + s) != 0;
        int off[ND];
#pragma unroll
        for (int d = 0; d < ND; ++d) off[d] = __ldg(a.off + s * kDiaMax + d);
        // index of a local row's value of diagonal 0
        const auto vidx = [](int row) {
            return static_cast<int64_t>(row / kDiaBlockRows) * ND * kDiaBlockRows + row % kDiaBlockRows;
        };
        for (int i = tid; i < M; i += T) P[-1 - i] = P[own + i] = 0.0f;
        const MI* const vt = vi + tid;   // slot q of diagonal d: vt[value_at(q, d)]
        const auto value_at = [](int q, int d) {
            return ((q * T) / kDiaBlockRows * ND + d) * kDiaBlockRows + (q * T) % kDiaBlockRows;
        };
        float* const Pt = P + tid;
        float R[NS], X[NS], Q[NS], Pn[NS];
        const auto set_p = [&](int q, float v) {
            Pt[T * q] = v;
            Pn[q] = v;
        };
        double acc[1][H] = {};
        float rz1[1][H] = {};
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            R[q] = X[q] = Pn[q] = 0.0f;
            if (q >= nk) continue;
            const int row = tid + T * q;
            const bool ok = row < n;
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                const int e = d > ND / 2 && unit ? d - 1 : d;   // stored diagonal
                if (!(unit && d == ND / 2)) vs[(e * nk + q) * T] = ok ? __ldg(vt + value_at(q, d)) : MI{};
            }
            float rh = 0.0f;
            if (ok) {
                const double b_i = bv[row];
                x[row] = 0.0;
                rh = static_cast<float>(__ldg(sv + row) * b_i);
                R[q] = rh;
                acc[0][q % H] += b_i * b_i;
                rz1[0][q % H] += rh * rh;
            }
            set_p(q, rh);
        }
        oc_sum<double, 1, T, H, SC, kOcWarps>(acc, redD, rank, ctas);
        oc_sum<float, 1, T, H, SC, kOcWarps>(rz1, redA, rank, ctas);    // (also: p and its halos are in place)
        const double bb = acc[0][0];
        const double thr = a.outer_tol * a.outer_tol * bb;
        double rr64 = bb;
        float rz = rz1[0][0];
        float rmax = rz;            // scaled |r|^2 at the last replacement
        float goal = static_cast<float>(thr / rr64) * rmax;   // scaled |r|^2 that would meet the target
        int32_t status = ST_RUNNING, it = 0, updates = 0;
        if (bb == 0.0) status = CMCG_SOLVE_ZERO_RHS;
        else if (!finite_(bb)) status = CMCG_SOLVE_NON_FINITE;
        else if (rr64 < thr) status = CMCG_SOLVE_CONVERGED;
        else if (!(rz > 0.0f)) status = CMCG_SOLVE_BREAKDOWN;
        const int64_t maxit = sys_max_iter(a.max_inner, n);
        if (kGuard && tid == 0) {
            guard[0] = stall_len(0, 0, a.delta);
            guard[1] = 0;
            guard[2] = 0;
        }
        oc_sync<SC, T>();   // (guard; and redA is read before the first iteration writes it)
        // x += S xh over the thread's rows
        const auto fold = [&] {
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                const int row = tid + T * q;
                if (q < nk && row < n) x[row] += __ldg(sv + row) * static_cast<double>(X[q]);
                X[q] = 0.0f;
            }
            oc_sync<SC, T>();
        };
        // (b - A x)[row] of local row `row` in FP64, entries in ascending offset order
        const auto residual = [&](int row) {
            double v = 0.0;
            const MO* vr = vO + vidx(row);
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                const int c = row + off[d];
                const double xc = c >= 0 && c < n ? x[c] : 0.0;
                v = fma(mval<double>(__ldg(vr + d * kDiaBlockRows)), xc, v);
            }
            return bv[row] - v;
        };
        bool folded = true;
        while (status == ST_RUNNING) {
            if (it >= maxit || updates >= a.max_updates) { status = CMCG_SOLVE_MAX_ITER; break; }
            float pq[1][H] = {};
            const auto product = [&](auto u) {
                constexpr bool U = decltype(u)::value;
                oc_slots<NS>(nk, [&](int q) {
                    float v = 0.0f;
#pragma unroll
                    for (int d = 0; d < ND; ++d) {
                        if (U && d == ND / 2) {
                            v = fmaf(1.0f, Pn[q], v);
                            continue;
                        }
                        const int e = U && d > ND / 2 ? d - 1 : d;
                        v = fmaf(mval<float>(vs[(e * nk + q) * T]), Pt[off[d] + T * q], v);
                    }
                    Q[q] = v;
                    pq[0][q % H] += Pn[q] * v;
                });
            };
            if (unit) product(std::true_type{});
            else product(std::false_type{});
            oc_sum<float, 1, T, H, SC, kOcWarps>(pq, redA, rank, ctas);
            const float alpha = rz / pq[0][0];
            if (!finite_(pq[0][0]) || !finite_(alpha)) { status = CMCG_SOLVE_NON_FINITE; break; }
            if (!(pq[0][0] > 0.0f)) { status = CMCG_SOLVE_BREAKDOWN; break; }
            float s1[1][H] = {};
            oc_slots<NS>(nk, [&](int q) {
                X[q] += alpha * Pn[q];
                const float ri = R[q] - alpha * Q[q];
                R[q] = ri;
                s1[0][q % H] += ri * ri;
            });
            oc_sum<float, 1, T, H, SC, kOcWarps>(s1, redB, rank, ctas);
            ++it;
            folded = false;
            float rzn = s1[0][0];
            if (!finite_(rzn)) { status = CMCG_SOLVE_NON_FINITE; break; }
            // replace the residual when it dropped by delta, or when it suggests
            // that the FP64 residual may have reached the target, or when the
            // cycle has run too long (progress guard)
            if (rzn < d2 * rmax || rzn < goal || (kGuard && it >= guard[0])) {
                fold();
                double t2[2][H] = {};
#pragma unroll
                for (int q = 0; q < NS; ++q) {
                    const int row = tid + T * q;
                    if (q < nk && row < n) {
                        const double r64 = residual(row);
                        const float rh = static_cast<float>(__ldg(sv + row) * r64);
                        R[q] = rh;
                        t2[0][q % H] += r64 * r64;
                        t2[1][q % H] += static_cast<double>(rh) * static_cast<double>(rh);
                    }
                }
                oc_sum<double, 2, T, H, SC, kOcWarps>(t2, redD, rank, ctas);
                ++updates;
                folded = true;
                int stalls = 0;
                if constexpr (kGuard) {
                    stalls = t2[0][0] > kStallRatio * rr64 ? guard[2] + 1 : 0;
                    const int cyc0 = updates == 1 ? it : guard[1];
                    oc_sync<SC, T>();
                    if (tid == 0) {
                        guard[0] = it + stall_len(updates, cyc0, a.delta);
                        guard[1] = cyc0;
                        guard[2] = stalls;
                    }
                }
                rr64 = t2[0][0];
                rzn = static_cast<float>(t2[1][0]);
                rmax = rzn;
                goal = static_cast<float>(thr / rr64) * rmax;
                if (!finite_(rr64)) { status = CMCG_SOLVE_NON_FINITE; break; }
                if (rr64 < thr) { status = CMCG_SOLVE_CONVERGED; break; }
                if (kGuard && stalls >= kStallMax) { status = CMCG_SOLVE_BREAKDOWN; break; }
            }
            if (!(rzn > 0.0f)) { status = CMCG_SOLVE_BREAKDOWN; break; }
            const float beta = rzn / rz;
            rz = rzn;
            oc_slots<NS>(nk, [&](int q) {
                set_p(q, R[q] + beta * Pn[q]);
            });
            oc_sync<SC, T>();
        }
        if (!folded) {
            // fold the pending increments and report the true residual
            fold();
            double t1[1][H] = {};
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                const int row = tid + T * q;
                if (q < nk && row < n) {
                    const double r64 = residual(row);
                    t1[0][q % H] += r64 * r64;
                }
            }
            oc_sum<double, 1, T, H, SC, kOcWarps>(t1, redD, rank, ctas);
            rr64 = t1[0][0];
        }
        if (tid == 0) {
            a.st.it[inst] = it;
            a.st.status[inst] = status;
            a.st.rr[inst] = rr64;
            a.st.bb[inst] = bb;
            a.st.outer[inst] = updates;
            a.st.err[inst] = (status == CMCG_SOLVE_ZERO_RHS) ? 0.0 : sqrt(rr64 / bb);
        }
    }
}

// Systems of 4097 .. 8192 rows, a CTA each, then (large batches) those of at most
// 2048 rows, a group of 128 threads each with a quarter of the shared memory (its
// scratch first).
template <typename MI, typename MO, int ND>
__global__ void __launch_bounds__(512, 1) k_onchip_mixed(const __grid_constant__ OnchipMixArgs<MI, MO> a,
                                                         const __grid_constant__ OnchipItems t512,
                                                         const __grid_constant__ OnchipItems t128, int smem) {
    extern __shared__ __align__(16) unsigned char oc_smem[];
    __shared__ MixScratch sc;
    onchip_mixed_items<MI, MO, ND, 512, 1, OC_CTA>(a, t512, oc_smem, sc);
    unsigned char* quarter = oc_smem + threadIdx.x / 128 * (smem / 4);
    onchip_mixed_items<MI, MO, ND, 128, 2, OC_GROUP>(a, t128, quarter + kOnchipMixScratch,
                                                     *reinterpret_cast<MixScratch*>(quarter));
}

// The others: a CTA of 256 threads each, two per SM.
template <typename MI, typename MO, int ND>
__global__ void __launch_bounds__(256, 2) k_onchip_mixed256(const __grid_constant__ OnchipMixArgs<MI, MO> a,
                                                            const __grid_constant__ OnchipItems t) {
    extern __shared__ __align__(16) unsigned char oc_smem[];
    __shared__ MixScratch sc;
    onchip_mixed_items<MI, MO, ND, 256, 1, OC_CTA>(a, t, oc_smem, sc);
}

}  // namespace

template <typename MI, typename MO>
cmcg_status onchip_mixed_launch(const OnchipMixArgs<MI, MO>& a, const OnchipItems& t512, const OnchipItems& t128, int smem,
                                int nd, int sms, cudaStream_t stream, bool* launched) {
    const void* kern = nd == 5 ? reinterpret_cast<const void*>(k_onchip_mixed<MI, MO, 5>)
                     : nd == 7 ? reinterpret_cast<const void*>(k_onchip_mixed<MI, MO, 7>) : nullptr;
    OnchipMixArgs<MI, MO> args = a;
    OnchipItems i512 = t512, i128 = t128;
    void* params[] = {&args, &i512, &i128, &smem};
    const int items = (t512.hi - t512.lo) + (t128.hi - t128.lo);
    return onchip_start(kern, params, items, OnchipForm{512, 1, 1}, smem, sms, stream, launched);
}

template <typename MI, typename MO>
cmcg_status onchip_mixed_launch256(const OnchipMixArgs<MI, MO>& a, const OnchipItems& t, size_t smem, int nd, int sms,
                                   cudaStream_t stream, bool* launched) {
    const void* kern = nd == 5 ? reinterpret_cast<const void*>(k_onchip_mixed256<MI, MO, 5>)
                     : nd == 7 ? reinterpret_cast<const void*>(k_onchip_mixed256<MI, MO, 7>) : nullptr;
    OnchipMixArgs<MI, MO> args = a;
    OnchipItems items = t;
    void* params[] = {&args, &items};
    return onchip_start(kern, params, t.hi - t.lo, OnchipForm{256, 1, 2}, smem, sms, stream, launched);
}

#define CMCG_ONCHIP_MIXED(MI, MO)                                                                                   \
    template cmcg_status onchip_mixed_launch<MI, MO>(const OnchipMixArgs<MI, MO>&, const OnchipItems&,              \
                                                     const OnchipItems&, int, int, int, cudaStream_t, bool*);       \
    template cmcg_status onchip_mixed_launch256<MI, MO>(const OnchipMixArgs<MI, MO>&, const OnchipItems&, size_t,   \
                                                        int, int, cudaStream_t, bool*);
CMCG_ONCHIP_MIXED(float, float)
CMCG_ONCHIP_MIXED(float, double)
CMCG_ONCHIP_MIXED(__nv_bfloat16, float)
CMCG_ONCHIP_MIXED(__nv_bfloat16, double)

}  // namespace cmcg
