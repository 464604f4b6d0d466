// PCG of one mid-size stencil system spread over many SMs with all its state in
// registers: one cooperative launch for the whole solve.
//
// The cluster solve (cg_cluster.cu) holds such a system in the shared memory of
// at most 16 CTAs and is issue-bound on those SMs (300^2 Poisson FP32: 9.4 us per
// iteration on 11 SMs, 4.7 here). Here every warp of that solve becomes a unit that may
// run anywhere: unit (k, w) is warp w of cluster CTA k, its lane l owns the rows
// k 2^lg + 1024 j + 32 w + l of the system, j < J = 2^lg / 1024, and keeps their
// p, r, x, inverse diagonal and matrix values, and the p entries its products
// gather, in registers. A CTA holds eight units and an SM one CTA: 40 SMs at 100^2, 44
// at 300^2, 64 at most. An iteration is bound by latency (300^2: 21 % of the issue slots
// of its SMs used): two rounds through L2, one per reduction (published and polled as tagged
// words, tagged.cuh). The z entries a neighbour gathers are
// published before the second reduction; every reader forms p = z + beta p for
// itself.
//
// A thread adds exactly the rows the cluster solve's thread adds, in its order;
// a unit's 32 lanes are summed by the same shuffles, the 32 units of a cluster
// CTA by the same tree, and the cluster CTAs in rank order: the results are
// those of the cluster solve bit for bit.
//
// Single buffers are enough: a word is written again only after a reduction that
// every reader joined after reading it. Every poll is bounded; one that runs
// out sets the device error bit of the grid barrier, and the CTA leaves.
#include <algorithm>
#include <cstdlib>

#include "cg_cluster.cuh"
#include "cg_dev.cuh"
#include "cg_wide.cuh"
#include "grid_sync.cuh"
#include "objects.h"
#include "tagged.cuh"

namespace cmcg {
namespace {

// Units (warps) per CTA. Fewer and larger CTAs have fewer pollers per sum; 8 is
// what the registers of the widest form allow. 300^2 Poisson, us per iteration
// with 2 / 4 / 8 units a CTA: 7.1 / 5.5 / 4.8 (two hops over combining warps,
// as in the resident solve: 6.3 / 6.0 / 5.4).
constexpr int kWideMaxWarps = 8;

struct WideArgs {
    int32_t n, lg, clusters, units;
    uint64_t* z;        // [n] tagged z
    uint64_t* words;    // two sets of kWideWords
    int32_t* err;
    BarrierLimits lim;
};

constexpr int kWideWords = kClusterMaxCtas * 32 * 4;   // device words of one sum: two values per unit

struct WideScratch {
    // (two sets, used in turn: a set is rewritten a barrier after its last read)
    double tot[2][2 * kClusterMaxCtas];
    int fail[2];
};

// NV per-thread sums added as cluster_sum adds them, in two steps: every unit
// publishes its 32 lanes' sums, then (between the two a thread may do work that
// does not need the result) every CTA collects. set: 0, 1, 0, 1, ... over the
// calls of a solve.
template <typename VT, int NV>
__device__ __forceinline__ void wide_publish(VT (&v)[NV], const WideArgs& a, int unit, int set, uint32_t tag) {
    uint64_t* const words = a.words + set * kWideWords;
    constexpr int S = NV * kWords<VT>;   // words per unit
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = warp_sum(v[j]);
    if ((threadIdx.x & 31) == 0 && unit >= 0) {
        if constexpr (NV == 2) put_pair(words + static_cast<int64_t>(unit) * S, v[0], v[1], tag);
        else put_value(words + static_cast<int64_t>(unit) * S, v[0], tag);
    }
}

// False when a poll ran out.
template <typename VT, int NV>
__device__ __forceinline__ bool wide_collect(VT (&v)[NV], const WideArgs& a, WideScratch& sc, int set, uint32_t want) {
    constexpr int S = NV * kWords<VT>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint64_t* const words = a.words + set * kWideWords;
    VT* const tot = reinterpret_cast<VT*>(sc.tot[set]);
    TaggedSum<VT, NV> part;
    for (int k = warp; k < a.clusters; k += nw) {
        for (long long spins = 0;; ++spins) {
            const int id = k * 32 + lane;
            part.load(id < a.units, words + static_cast<int64_t>(id) * S, want);   // (no such unit: adds 0)
            if (part.arrived(want)) break;
            if (spins > a.lim.spins) {
                sc.fail[set] = 1;
                if (a.err) atomicOr(a.err, DEVERR_GRID_BARRIER);
                break;
            }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const VT s = warp_sum(part.value(j));
            if (lane == 0) tot[j * kClusterMaxCtas + k] = s;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        VT t = VT(0);
        for (int k = 0; k < a.clusters; ++k) t += tot[j * kClusterMaxCtas + k];
        v[j] = t;
    }
    return sc.fail[set] == 0;
}

template <typename VT, int NV>
__device__ __forceinline__ bool wide_sum(VT (&v)[NV], const WideArgs& a, WideScratch& sc, int unit, int set,
                                         uint32_t tag, uint32_t want) {
    wide_publish<VT, NV>(v, a, unit, set, tag);
    return wide_collect<VT, NV>(v, a, sc, set, want);
}

// The z words of the rows other threads own, read into zn (bit j ND + d of
// `need`: entry (j, d) is gathered), all again until all carry the tag. set:
// the next sum's set, which reports a poll that ran out.
template <typename VT, int ND, int J>
__device__ __forceinline__ void wide_gather(VT (&zn)[J][ND], uint64_t need, const WideArgs& a, WideScratch& sc,
                                            const int (&off)[ND], int row0, int set, uint32_t want) {
    // (at most 28 words in flight: a 256-thread CTA has 255 registers a thread. The widest
    // forms with seven diagonals spill, FP32 J = 8 504 bytes and FP64 J = 4 580; no other does)
    constexpr int JG = J * ND * kWords<VT> <= 28 ? J : J * ND * kWords<VT> <= 56 ? J / 2 : J / 4;
#pragma unroll
    for (int j0 = 0; j0 < J; j0 += JG) {
        TaggedValue<VT> w[JG][ND];
        for (long long spins = 0;; ++spins) {
#pragma unroll
            for (int j = 0; j < JG; ++j)
#pragma unroll
                for (int d = 0; d < ND; ++d)
                    w[j][d].load(need >> ((j0 + j) * ND + d) & 1,
                                 a.z + static_cast<int64_t>(row0 + 1024 * (j0 + j) + off[d]) * kWords<VT>, want);
            bool ok = true;
#pragma unroll
            for (int j = 0; j < JG; ++j)
#pragma unroll
                for (int d = 0; d < ND; ++d) ok &= w[j][d].arrived(want);
            if (ok) break;
            if (spins > a.lim.spins) {
                sc.fail[set] = 1;
                if (a.err) atomicOr(a.err, DEVERR_GRID_BARRIER);
                break;
            }
        }
#pragma unroll
        for (int j = 0; j < JG; ++j)
#pragma unroll
            for (int d = 0; d < ND; ++d) zn[j0 + j][d] = w[j][d].value();
    }
}

template <typename VT, typename MT, int ND, int J>
__global__ void __launch_bounds__(32 * kWideMaxWarps, 1) k_wide_cg(const __grid_constant__ SolveArgs<VT, MT> a,
                                                                   const __grid_constant__ WideArgs w) {
    __shared__ WideScratch sc;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = w.n;
    const int u0 = static_cast<int>(static_cast<int64_t>(blockIdx.x) * w.units / gridDim.x);
    const int u1 = static_cast<int>(static_cast<int64_t>(blockIdx.x + 1) * w.units / gridDim.x);
    const int unit = u0 + warp < u1 ? u0 + warp : -1;
    // the lane's first row; rows of the unit past the cluster CTA's range or
    // the system's end do not exist
    const int row0 = unit >= 0 ? ((unit >> 5) << w.lg) + ((unit & 31) << 5) + lane : n;
    if (threadIdx.x == 0) sc.fail[0] = sc.fail[1] = 0;
    int off[ND];
    // entries this lane gathers itself: of other rows than its own that exist,
    // +-1 only where the neighbouring lane is another warp's
    uint64_t need = 0;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        off[d] = __ldg(a.dia.off + d);
        if (off[d] != 0 && (off[d] != -1 || lane == 0) && (off[d] != 1 || lane == 31)) {
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const int row = row0 + 1024 * j, c = row + off[d];
                if (row < n && c >= 0 && c < n) need |= uint64_t(1) << (j * ND + d);
            }
        }
    }
    const MT* const dv = a.dia.vals + __ldg(a.dia.base);
    const bool jacobi = a.dinv != nullptr;
    MT V[J][ND];
    VT R[J], X[J], D[J], Pn[J], N[J][ND];
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const int row = row0 + 1024 * j;
        const bool ok = row < n;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            V[j][d] = ok ? dv[(static_cast<int64_t>(row / kDiaBlockRows) * ND + d) * kDiaBlockRows + row % kDiaBlockRows]
                         : MT{};
            N[j][d] = VT(0);
        }
        D[j] = ok && jacobi ? a.dinv[row] : VT(1);
        R[j] = X[j] = Pn[j] = VT(0);
    }
    const VT tol = static_cast<VT>(a.tol);
    const int64_t maxit = sys_max_iter(a.max_iter, n);
    // r = b - A x0; |b|^2, |r|^2
    VT acc[2] = {VT(0), VT(0)};
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const int row = row0 + 1024 * j;
        if (row >= n) continue;
        const VT bi = a.b[row];
        if (a.guess) {
            VT v = VT(0);
#pragma unroll
            for (int d = 0; d < ND; ++d) v = fma(mval<VT>(V[j][d]), __ldg(a.guess + min(max(row + off[d], 0), n - 1)), v);
            const VT ri = bi - v;
            R[j] = ri;
            X[j] = a.guess[row];
            acc[0] += bi * bi;
            acc[1] += ri * ri;
        } else {
            R[j] = bi;
            acc[0] += bi * bi;
        }
    }
    __syncthreads();
    uint32_t tag = 1;
    uint32_t want = tag + w.lim.extra;
    int32_t it = 0, status = ST_RUNNING;
    bool live = wide_sum<VT, 2>(acc, w, sc, unit, 0, tag, want);
    const VT bb = acc[0];
    VT rr = a.guess ? acc[1] : bb;
    const VT thr = tol * tol * bb;
    VT rz = VT(0);
    if (!live) {
        // (status stays running: finalised as not converged)
    } else if ((a.abs_zero_test && bb < tol * tol) || bb == VT(0)) {
#pragma unroll
        for (int j = 0; j < J; ++j) X[j] = VT(0);
        status = CMCG_SOLVE_ZERO_RHS;
    } else if (!finite_(rr) || !finite_(bb)) {
        status = CMCG_SOLVE_NON_FINITE;
    } else if (rr < thr) {
        status = CMCG_SOLVE_CONVERGED;
    } else {
        VT rzv[1] = {VT(0)};
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int row = row0 + 1024 * j;
            if (row >= n) continue;
            const VT zi = jacobi ? D[j] * R[j] : R[j];
            Pn[j] = zi;
            put_value(w.z + static_cast<int64_t>(row) * kWords<VT>, zi, tag);
            rzv[0] += R[j] * zi;
        }
        live = wide_sum<VT, 1>(rzv, w, sc, unit, 1, tag, want);
        rz = rzv[0];
        if (!live) {
        } else if (!finite_(rz)) status = CMCG_SOLVE_NON_FINITE;
        else if (!(rz > VT(0))) status = CMCG_SOLVE_BREAKDOWN;
        else wide_gather<VT, ND, J>(N, need, w, sc, off, row0, 0, want);
    }
    while (live && status == ST_RUNNING) {
        if (it >= maxit) { status = CMCG_SOLVE_MAX_ITER; break; }
        ++tag;
        want = tag + w.lim.extra;
        VT Q[J];
        VT pq[1] = {VT(0)};
#pragma unroll
        for (int j = 0; j < J; ++j) Q[j] = VT(0);
        // diagonals in ascending order, all rows of a thread per diagonal
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            if (off[d] == 0) {
#pragma unroll
                for (int j = 0; j < J; ++j) Q[j] = fma(mval<VT>(V[j][d]), Pn[j], Q[j]);
            } else if (off[d] == -1) {
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const VT up = __shfl_up_sync(FULL, Pn[j], 1);
                    Q[j] = fma(mval<VT>(V[j][d]), lane == 0 ? N[j][d] : up, Q[j]);
                }
            } else if (off[d] == 1) {
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const VT dn = __shfl_down_sync(FULL, Pn[j], 1);
                    Q[j] = fma(mval<VT>(V[j][d]), lane == 31 ? N[j][d] : dn, Q[j]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < J; ++j) Q[j] = fma(mval<VT>(V[j][d]), N[j][d], Q[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < J; ++j)
            if (row0 + 1024 * j < n) pq[0] += Pn[j] * Q[j];
        if (!wide_sum<VT, 1>(pq, w, sc, unit, 0, tag, want)) break;
        const VT alpha = rz / pq[0];
        if (!finite_(pq[0]) || !finite_(alpha)) { status = CMCG_SOLVE_NON_FINITE; break; }
        if (!(pq[0] > VT(0))) { status = CMCG_SOLVE_BREAKDOWN; break; }
        VT s2[2] = {VT(0), VT(0)};
        VT Z[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int row = row0 + 1024 * j;
            X[j] += alpha * Pn[j];
            const VT ri = R[j] - alpha * Q[j];
            R[j] = ri;
            Z[j] = jacobi ? D[j] * ri : ri;
            if (row < n) {
                put_value(w.z + static_cast<int64_t>(row) * kWords<VT>, Z[j], tag);
                s2[0] += ri * ri;
                s2[1] += ri * Z[j];
            }
        }
        wide_publish<VT, 2>(s2, w, unit, 1, tag);
        // (the neighbours' z arrives while the sum is under way)
        VT zn[J][ND];
        wide_gather<VT, ND, J>(zn, need, w, sc, off, row0, 1, want);
        if (!wide_collect<VT, 2>(s2, w, sc, 1, want)) break;
        rr = s2[0];
        if (!finite_(rr) || !finite_(s2[1])) { status = CMCG_SOLVE_NON_FINITE; break; }
        if (rr < thr) { status = CMCG_SOLVE_CONVERGED; break; }
        const VT rzn = s2[1];
        if (!(rzn > VT(0))) { status = CMCG_SOLVE_BREAKDOWN; break; }
        const VT beta = rzn / rz;
        rz = rzn;
#pragma unroll
        for (int j = 0; j < J; ++j) {
            Pn[j] = fma(beta, Pn[j], Z[j]);
#pragma unroll
            for (int d = 0; d < ND; ++d) N[j][d] = fma(beta, N[j][d], zn[j][d]);
        }
        ++it;
    }
#pragma unroll
    for (int j = 0; j < J; ++j)
        if (row0 + 1024 * j < n) a.x[row0 + 1024 * j] = X[j];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.st.it[0] = it;
        a.st.status[0] = status;
        a.st.rr[0] = static_cast<double>(rr);
        a.st.bb[0] = static_cast<double>(bb);
        a.st.outer[0] = 0;
    }
}

}  // namespace

size_t wide_ws_bytes(int32_t n, size_t vec_bytes) {
    return sizeof(uint64_t) * (2 * kWideWords + vec_bytes / 4 * static_cast<size_t>(n));
}

template <typename VT, typename MT>
cmcg_status wide_cg_launch(const SolveArgs<VT, MT>& a, int rows_log2, int clusters, int nd, int sms, void* ws,
                           int32_t* err, cudaStream_t st, bool* launched) {
    *launched = false;
    const void* kern = nullptr;
    const int J = 1 << (rows_log2 - 10);
#define CMCG_WIDE_PICK(JJ)                                                          \
    if (J == JJ) kern = nd == 5 ? reinterpret_cast<const void*>(k_wide_cg<VT, MT, 5, JJ>) \
                                : reinterpret_cast<const void*>(k_wide_cg<VT, MT, 7, JJ>)
    CMCG_WIDE_PICK(1);
    CMCG_WIDE_PICK(2);
    CMCG_WIDE_PICK(4);
    if constexpr (sizeof(VT) == 4) CMCG_WIDE_PICK(8);
#undef CMCG_WIDE_PICK
    if (!kern || (nd != 5 && nd != 7)) return CMCG_OK;
    // units with rows: all of the full cluster CTAs, those of the last one
    const int64_t last = a.rows - (static_cast<int64_t>(clusters - 1) << rows_log2);
    const int units = (clusters - 1) * 32 + static_cast<int>(std::min<int64_t>(32, (last + 31) / 32));
    const int grid = std::min((units + kWideMaxWarps - 1) / kWideMaxWarps, sms);
    const int warps = (units + grid - 1) / grid;
    if (warps > kWideMaxWarps) return CMCG_OK;
    int occ = 0;
    CMCG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 32 * warps, 0));
    if (occ * sms < grid) return CMCG_OK;
    CMCG_CUDA(cudaMemsetAsync(ws, 0, wide_ws_bytes(a.rows, sizeof(VT)), st));
    BarrierLimits lim{kGridBarrierSpins, 0u};
    if (const char* e = std::getenv("CUMAT_TEST_GRID_SPINS")) lim.spins = std::max(1LL, std::atoll(e));
    if (const char* e = std::getenv("CUMAT_TEST_GRID_EXTRA")) lim.extra = static_cast<unsigned>(std::max(0, std::atoi(e)));
    uint64_t* const p = static_cast<uint64_t*>(ws);
    WideArgs w{a.rows, rows_log2, clusters, units, p + 2 * kWideWords, p, err, lim};
    SolveArgs<VT, MT> args = a;
    void* params[] = {&args, &w};
    CMCG_CUDA(cudaLaunchCooperativeKernel(kern, grid, 32 * warps, params, 0, st));
    *launched = true;
    return CMCG_OK;
}

#define CMCG_WIDE_INSTANTIATE(VT, MT)                                                                              \
    template cmcg_status wide_cg_launch<VT, MT>(const SolveArgs<VT, MT>&, int, int, int, int, void*, int32_t*, \
                                                cudaStream_t, bool*);
CMCG_WIDE_INSTANTIATE(float, float)
CMCG_WIDE_INSTANTIATE(float, double)
CMCG_WIDE_INSTANTIATE(float, __nv_bfloat16)
CMCG_WIDE_INSTANTIATE(double, float)
CMCG_WIDE_INSTANTIATE(double, double)
CMCG_WIDE_INSTANTIATE(double, __nv_bfloat16)

}  // namespace cmcg
