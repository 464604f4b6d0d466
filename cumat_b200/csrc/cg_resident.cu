// Grid-path PCG of one system kept on the chip: the whole loop is one
// cooperative launch whose CTAs hold their rows' values, p, r and x in shared
// memory and registers, and exchange only boundary entries and partial sums.
//
// What bounds it: nothing is streamed, so an iteration costs its shared-memory
// passes (the product: about 1.2 us for 3500 rows and 5 diagonals a CTA) and
// four hops through L2, two per reduction. At 1024^2 the shared-memory pipe is busy
// for 32 % of the cycles and most of the stalls are at barriers, that is, on the sums.
// The graph loop it replaces launches two kernels an iteration, each a pass over
// L2 with its own ramp and closing sum: 1024^2 Poisson FP32 25 us per iteration,
// 9.8 here; 400^2 21.2 and 7.2.
//
// Work split: CTA c is the grid plan's CTAs 4c .. 4c + 3 (256 threads each), so
// every thread adds exactly the rows it adds there, in the same order, and the
// partial sums are combined by the same tree: results are those of the graph
// loop bit for bit. Row quads of a thread: 4 t + 1024 k, t < 256, as in
// dia_rows_seg and seg_rows_vec.
//
// Exchange through tagged words (tagged.cuh), without fences: in a reduction every
// virtual CTA stores its partial, eight combining warps poll a share each and
// store the totals, and one warp of every CTA polls those eight words: 2 .. 3 us.
// With all CTAs polling all partials (592 words, 148 readers) a sum took 6 us.
// The z = M^-1 r entries another CTA gathers are published before the second
// reduction and read after it.
// A word is written again only after every CTA has passed a reduction that
// follows its last read of it, so single buffers are enough.
//
// Every wait is bounded: a poll that runs out sets the device error bit of the
// grid barrier and the CTA leaves; the others run out the same way, since what a
// poll that ran out was to add is never published.
#include <algorithm>
#include <cstdlib>

#include "cg_dev.cuh"
#include "cg_resident.cuh"
#include "grid_sync.cuh"
#include "tagged.cuh"

namespace cmcg {
namespace {

// ---- shared-memory quads ----------------------------------------------------------

// P[e .. e + 3], e any element (two aligned quads where e is not a multiple of 4)
template <typename VT>
__device__ __forceinline__ void sm_quad(const VT* P, int e, VT (&o)[4]) {
    const int a = e & ~3, m = e & 3;
    V4<VT> u;
    u.load(P + a);
    if (m == 0) {   // uniform: e differs between threads by multiples of 4
#pragma unroll
        for (int q = 0; q < 4; ++q) o[q] = u.v[q];
        return;
    }
    V4<VT> w;
    w.load(P + a + 4);
    if (m == 1) { o[0] = u.v[1]; o[1] = u.v[2]; o[2] = u.v[3]; o[3] = w.v[0]; }
    else if (m == 2) { o[0] = u.v[2]; o[1] = u.v[3]; o[2] = w.v[0]; o[3] = w.v[1]; }
    else { o[0] = u.v[3]; o[1] = w.v[0]; o[2] = w.v[1]; o[3] = w.v[2]; }
}

__device__ __forceinline__ void ld_vals4(Vals4<float>& w, const float* p) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    w.v[0] = t.x; w.v[1] = t.y; w.v[2] = t.z; w.v[3] = t.w;
}
__device__ __forceinline__ void ld_vals4(Vals4<double>& w, const double* p) {
    const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
    w.v[0] = a.x; w.v[1] = a.y; w.v[2] = b.x; w.v[3] = b.y;
}
__device__ __forceinline__ void ld_vals4(Vals4<__nv_bfloat16>& w, const __nv_bfloat16* p) {
    const uint2 t = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&t.x);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&t.y);
    w.v[0] = a.x; w.v[1] = a.y; w.v[2] = b.x; w.v[3] = b.y;
}

// ---- reductions -------------------------------------------------------------------

constexpr int kResWarps = kResThreads / 32;
constexpr int kResPlay = kResVirtual * kTile / kResThreads;   // virtual threads a thread plays (2)

// Scratch of the grid sums (shared memory).
template <typename VT>
struct SumScratch {
    VT warp[2][kResVirtual * (kTile / 32)];   // [value][virtual warp]
    VT fin[2][kTile / 32];                    // [value][combining warp]
    int fail;    // a poll of a sum ran out
    int hfail;   // a poll of a p entry ran out (taken over by the next sum)
};

// Device words of one grid sum: a partial per virtual CTA (up to two FP64
// values), then one per combining warp, each in a 32-byte sector of its own.
constexpr int kSumPartials = kResMaxVirtual * 4;
constexpr int kSumWords = kSumPartials + (kTile / 32) * 4;

// x lives in shared memory where the registers would not hold it: two quads per
// virtual thread, or FP64.
template <typename VT, int K> constexpr bool kXShared = K == 2 || sizeof(VT) == 8;

struct ResidentArgs {
    ResidentGeom g;
    uint64_t* halo;    // [rows] tagged z
    uint64_t* words;   // kSumWords per sum
    int32_t* err;
    BarrierLimits lim;
    int32_t partials[2];   // of a sum of one and of two values (n_virtual; a test waits for one more)
};

// Where this CTA and thread stand in the grid plan.
struct ResidentPos {
    int lo, cnt;                        // the CTA's rows [lo, lo + cnt)
    int a0[kResPlay], a1[kResPlay];     // relative rows of the thread's virtual CTAs
    __device__ __forceinline__ ResidentPos(const ResidentGeom& g) {
        const auto row0 = [&](int v) {
            return min(static_cast<int>(static_cast<int64_t>(min(v, g.n_virtual)) * g.n_tiles / g.n_virtual) * kTile, g.n);
        };
        const int v0 = blockIdx.x * kResVirtual;
        lo = row0(v0);
        cnt = row0(v0 + kResVirtual) - lo;
#pragma unroll
        for (int h = 0; h < kResPlay; ++h) {
            const int v = v0 + (threadIdx.x / kTile) + h * (kResThreads / kTile);
            a0[h] = row0(v) - lo;
            a1[h] = row0(v + 1) - lo;
        }
    }
};

// Polls `load` until the words carry the tag; false (and the error bit) when
// the limit ran out.
template <typename F>
__device__ __forceinline__ bool resident_poll(const ResidentArgs& m, F&& arrived) {
    for (long long spins = 0; !arrived(); ++spins) {
        if (spins > m.lim.spins) {
            if (m.err) atomicOr(m.err, DEVERR_GRID_BARRIER);
            return false;
        }
    }
    return true;
}

// v[j][h] (the thread's h-th virtual thread) summed over the virtual CTAs as the
// grid path sums them: the warps of a virtual CTA by shuffles, its 8 warps by one
// more shuffle tree, then the partials: thread i of 256 adds partials i, i + 256,
// i + 512 in order, and one more block tree. That closing sum's 8 warps are
// spread over 8 CTAs, so each polled word has one reader; their results are
// polled by one warp of every CTA. (With every CTA polling all partials the
// waiting CTAs' polls delay the late ones' stores: 6 us a sum on 148 CTAs, against
// 2 to 3 us for the two hops.) meanwhile() runs between the CTA's own
// publication and the result. False when a poll ran out. ORDER: what any thread
// wrote to global memory before the sum, every thread reads after it (at L2): each
// hop fences between the barrier or poll it follows and its own publication.
template <typename VT, int NV, bool ORDER = false, typename F>
__device__ __forceinline__ bool resident_sum(VT (&v)[NV][kResPlay], SumScratch<VT>& sc, const ResidentArgs& m,
                                             uint64_t* words, uint32_t tag, F&& meanwhile) {
    constexpr int W = kWords<VT> * NV, C = kTile / 32;
    const uint32_t want = tag + m.lim.extra;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nv = m.g.n_virtual;
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
        for (int h = 0; h < kResPlay; ++h) {
            const VT s = warp_sum(v[j][h]);
            if (lane == 0) sc.warp[j][h * kResWarps + warp] = s;
        }
    __syncthreads();
    if (threadIdx.x == 0 && sc.hfail) sc.fail = 1;
    VT r[NV];
    if (warp < kResVirtual) {
        const int vc = blockIdx.x * kResVirtual + warp;
#pragma unroll
        for (int j = 0; j < NV; ++j) r[j] = warp_sum(lane < C ? sc.warp[j][warp * C + lane] : VT(0));
        if (lane == 0 && vc < nv) {
            uint64_t* w = words + static_cast<int64_t>(vc) * W;
            if constexpr (ORDER) __threadfence();
            if constexpr (NV == 2) put_pair(w, r[0], r[1], tag);
            else put_value(w, r[0], tag);
        }
    }
    uint64_t* const fin = words + kSumPartials;
    // combining warp c runs in CTA c G / 8 (G CTAs), as its warp 4 + c
    const int c = warp - kResVirtual;
    if (c >= 0 && c < C && c * static_cast<int>(gridDim.x) / C == static_cast<int>(blockIdx.x)) {
        const int t = c * 32 + lane;
        TaggedSum<VT, NV> part[3];
        const bool got = resident_poll(m, [&] {
#pragma unroll
            for (int k = 0; k < 3; ++k)
                part[k].load(t + k * kTile < m.partials[NV - 1], words + static_cast<int64_t>(t + k * kTile) * W, want);
            return part[0].arrived(want) && part[1].arrived(want) && part[2].arrived(want);
        });
        if (!got) sc.fail = 1;
        if constexpr (ORDER) {
            __threadfence();
            __syncwarp();
        }
        // a total that lacks a partial is not published: the other CTAs run out too
        const bool all = __all_sync(FULL, got);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            VT s = VT(0);
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (t + k * kTile < m.partials[NV - 1]) s += part[k].value(j);
            r[j] = warp_sum(s);
        }
        if (lane == 0 && all) {
            if constexpr (ORDER) __threadfence();
            if constexpr (NV == 2) put_pair(fin + c * 4, r[0], r[1], tag);
            else put_value(fin + c * 4, r[0], tag);
        }
    }
    meanwhile();
    if (warp == kResWarps - 1) {
        TaggedSum<VT, NV> part;
        if (!resident_poll(m, [&] {
                part.load(lane < C, fin + lane * 4, want);
                return part.arrived(want);
            }))
            sc.fail = 1;
        if constexpr (ORDER) __threadfence();
        if (lane < C) {
#pragma unroll
            for (int j = 0; j < NV; ++j) sc.fin[j][lane] = part.value(j);
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j][0] = warp_sum(lane < C ? sc.fin[j][lane] : VT(0));
    return sc.fail == 0;
}

// ---- p entries of other CTAs --------------------------------------------------------

template <typename VT>
__device__ __forceinline__ VT p_next(VT beta, VT pold, VT z) { return fma(beta, pold, z); }

// Pair e (two neighbouring rows, the first even) of the entries this CTA
// gathers from others: relative row j and element of p; false past the last.
struct HaloPair {
    int j, elem;
};
__device__ __forceinline__ bool halo_pair(const ResidentGeom& g, int cnt, int e, HaloPair& h) {
    for (int w = 0; w < g.n_win; ++w) {
        // (a CTA with fewer rows than rpad gathers that many fewer)
        const int w0 = g.win_lo[w], w1 = w0 + g.win_len[w] - (g.rpad - cnt);
        // the parts of the window before and after the own rows
        const int l1 = min(w1, 0), r0 = w0 < cnt ? max(w0, (cnt + 1) & ~1) : w0;
        const int nl = max(0, l1 - w0) >> 1, nr = max(0, w1 - r0) >> 1;
        if (e < nl + nr) {
            h.j = e < nl ? w0 + 2 * e : r0 + 2 * (e - nl);
            h.elem = g.win_base[w] + h.j - w0;
            return true;
        }
        e -= nl + nr;
    }
    return false;
}

constexpr int kHaloHeld = 4;   // pairs of z a thread holds while a sum is under way

// The thread's first kHaloHeld pairs: their places (found once), and z of an
// iteration.
template <typename VT>
struct HaloHeld {
    int row[kHaloHeld], elem[kHaloHeld];   // row < 0: none
    VT a[kHaloHeld], b[kHaloHeld];
    __device__ __forceinline__ void init(const ResidentGeom& g, const ResidentPos& at) {
#pragma unroll
        for (int u = 0; u < kHaloHeld; ++u) {
            HaloPair h;
            row[u] = -1;
            elem[u] = 0;
            if (halo_pair(g, at.cnt, threadIdx.x + u * kResThreads, h)) {
                const int r = at.lo + h.j;
                if (r >= 0 && r < g.n) {
                    row[u] = r;
                    elem[u] = h.elem;
                }
            }
        }
    }
    __device__ __forceinline__ void gather(const ResidentArgs& m, uint32_t want, int* fail) {
        TaggedPair<VT> pr[kHaloHeld];
        if (!resident_poll(m, [&] {
                bool ok = true;
#pragma unroll
                for (int u = 0; u < kHaloHeld; ++u)
                    pr[u].load(row[u] >= 0, row[u] + 1 < m.g.n, m.halo + static_cast<int64_t>(row[u]) * kWords<VT>, want);
#pragma unroll
                for (int u = 0; u < kHaloHeld; ++u) ok &= pr[u].arrived(want);
                return ok;
            }))
            *fail = 1;
#pragma unroll
        for (int u = 0; u < kHaloHeld; ++u) {
            a[u] = pr[u].first();
            b[u] = pr[u].second();
        }
    }
};

// p = z + beta p for the gathered entries: the held pairs, then the others with
// z read now. FIRST: z = M^-1 r from memory (before the first publication).
template <typename VT, bool FIRST>
__device__ __forceinline__ void halo_update(VT* P, const ResidentArgs& m, const ResidentPos& at, HaloHeld<VT>& held,
                                            uint32_t want, VT beta, const VT* r, const VT* dinv, int* fail) {
    const ResidentGeom& g = m.g;
    const auto z0 = [&](int row) { return row < g.n ? (dinv ? dinv[row] * r[row] : r[row]) : VT(0); };
#pragma unroll
    for (int u = 0; u < kHaloHeld; ++u) {
        if (held.row[u] < 0) continue;
        const VT a = FIRST ? z0(held.row[u]) : held.a[u], b = FIRST ? z0(held.row[u] + 1) : held.b[u];
        VT* p = P + held.elem[u];
        p[0] = p_next(beta, p[0], a);
        p[1] = p_next(beta, p[1], b);   // (a row past the system's end stays 0)
    }
    constexpr int U = 4;
    for (int e0 = threadIdx.x + kHaloHeld * kResThreads;; e0 += U * kResThreads) {
        HaloPair h[U];
        bool on[U], any = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            h[u] = HaloPair{0, 0};
            const bool in = halo_pair(g, at.cnt, e0 + u * kResThreads, h[u]);
            any = any || in;
            on[u] = in && at.lo + h[u].j >= 0 && at.lo + h[u].j < g.n;
        }
        if (!any) break;
        VT a[U], b[U];
        if constexpr (FIRST) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                a[u] = on[u] ? z0(at.lo + h[u].j) : VT(0);
                b[u] = on[u] ? z0(at.lo + h[u].j + 1) : VT(0);
            }
        } else {
            TaggedPair<VT> pr[U];
            if (!resident_poll(m, [&] {
                    bool ok = true;
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        pr[u].load(on[u], at.lo + h[u].j + 1 < g.n, m.halo + static_cast<int64_t>(at.lo + h[u].j) * kWords<VT>,
                                   want);
#pragma unroll
                    for (int u = 0; u < U; ++u) ok &= pr[u].arrived(want);
                    return ok;
                }))
                *fail = 1;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                a[u] = pr[u].first();
                b[u] = pr[u].second();
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!on[u]) continue;
            VT* p = P + h[u].elem;
            p[0] = p_next(beta, p[0], a[u]);
            p[1] = p_next(beta, p[1], b[u]);
        }
    }
}

// Publishes z of a row quad where other CTAs may gather it.
template <typename VT>
__device__ __forceinline__ void halo_publish(const ResidentArgs& m, const ResidentPos& at, int li, int end,
                                             const VT (&z)[4], uint32_t tag) {
    if (li < m.g.reach || li + 4 > at.cnt - m.g.reach) {
        uint64_t* w = m.halo + static_cast<int64_t>(at.lo + li) * kWords<VT>;
        if (li + 1 < end) put_pair(w, z[0], z[1], tag);
        else put_value(w, z[0], tag);
        if (li + 3 < end) put_pair(w + 2 * kWords<VT>, z[2], z[3], tag);
        else if (li + 2 < end) put_value(w + 2 * kWords<VT>, z[2], tag);
    }
}

// ---- the product ----------------------------------------------------------------------

// q of the thread's NQ row quads (relative rows li[s], multiples of 4; quads
// past the end give values that are not used), diagonals in ascending order,
// the sums of dia_rows_seg; own receives p of the quads. The quads go through
// one diagonal together, so their loads are in flight at once.
// unit: the middle diagonal is offset 0 with every value 1 and is neither
// stored in shared memory nor loaded.
template <typename VT, typename MT, int ND, int NQ>
__device__ __forceinline__ void quads_product(const VT* P, const MT* vs, const MT* __restrict__ dv,
                                              const ResidentGeom& g, int lo, bool unit, const int (&li)[NQ],
                                              VT (&acc)[NQ][4], VT (&own)[NQ][4]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int s = 0; s < NQ; ++s) {
        V4<VT> t;
        t.load(P + g.own + li[s]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            own[s][q] = t.v[q];
            acc[s][q] = VT(0);
        }
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const int o = g.off[d];
        if (d == ND / 2 && unit) {
#pragma unroll
            for (int s = 0; s < NQ; ++s)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[s][q] = fma(VT(1), own[s][q], acc[s][q]);
            continue;
        }
        const int slot = d > ND / 2 && unit ? d - 1 : d;
        Vals4<MT> w[NQ];
        if (slot < g.smem_diags) {
#pragma unroll
            for (int s = 0; s < NQ; ++s) ld_vals4(w[s], vs + slot * g.rpad + li[s]);
        } else {
#pragma unroll
            for (int s = 0; s < NQ; ++s) {
                const int row = lo + li[s];
                w[s].load(dv + static_cast<int64_t>(row / kDiaBlockRows) * ND * kDiaBlockRows + d * kDiaBlockRows +
                          row % kDiaBlockRows);
            }
        }
        if (o == 0) {
#pragma unroll
            for (int s = 0; s < NQ; ++s)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[s][q] = fma(mval<VT>(w[s].v[q]), own[s][q], acc[s][q]);
        } else if (o == -1) {
#pragma unroll
            for (int s = 0; s < NQ; ++s) {
                VT prev = __shfl_up_sync(FULL, own[s][3], 1);
                if (lane == 0) prev = P[g.own + li[s] - 1];
                acc[s][0] = fma(mval<VT>(w[s].v[0]), prev, acc[s][0]);
#pragma unroll
                for (int q = 1; q < 4; ++q) acc[s][q] = fma(mval<VT>(w[s].v[q]), own[s][q - 1], acc[s][q]);
            }
        } else if (o == 1) {
#pragma unroll
            for (int s = 0; s < NQ; ++s) {
                VT next = __shfl_down_sync(FULL, own[s][0], 1);
                if (lane == 31) next = P[g.own + li[s] + 4];
#pragma unroll
                for (int q = 0; q < 3; ++q) acc[s][q] = fma(mval<VT>(w[s].v[q]), own[s][q + 1], acc[s][q]);
                acc[s][3] = fma(mval<VT>(w[s].v[3]), next, acc[s][3]);
            }
        } else {
#pragma unroll
            for (int s = 0; s < NQ; ++s) {
                VT pv[4];
                sm_quad(P, g.pd[d] + li[s], pv);
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[s][q] = fma(mval<VT>(w[s].v[q]), pv[q], acc[s][q]);
            }
        }
    }
}

// The CTA's rows of the diagonals kept in shared memory.
template <typename MT, int ND>
__device__ __forceinline__ void stage_values(MT* vs, const MT* __restrict__ dv, const ResidentGeom& g, int lo, int cnt,
                                             bool unit) {
    const int nd = unit ? ND - 1 : ND;
    for (int slot = 0; slot < min(g.smem_diags, nd); ++slot) {
        const int d = unit && slot >= ND / 2 ? slot + 1 : slot;
        for (int i = 4 * threadIdx.x; i < cnt; i += 4 * kResThreads) {
            const int row = lo + i;
            Vals4<MT> w;
            w.load(dv + static_cast<int64_t>(row / kDiaBlockRows) * ND * kDiaBlockRows + d * kDiaBlockRows +
                   row % kDiaBlockRows);
#pragma unroll
            for (int q = 0; q < 4; ++q) vs[slot * g.rpad + i + q] = w.v[q];
        }
    }
}

// ---- the solve --------------------------------------------------------------------

// Plain PCG of instance 0, initialised by the grid path's init kernels (x, r,
// |b|^2, |r|^2, r.z and the status are in global memory). K: row quads of a
// virtual thread. STRIDED: the update's sums run over rows t, t + 256, ... of a
// virtual CTA, as the grid path's do where its vectors are not 16-byte aligned
// (r passes through shared memory); otherwise over the quads.
template <typename VT, typename MT, int ND, int K, bool STRIDED>
__global__ void __launch_bounds__(kResThreads, 1) k_resident_cg(const __grid_constant__ SolveArgs<VT, MT> a,
                                                                const __grid_constant__ ResidentArgs m) {
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ SumScratch<VT> sc;
    constexpr int NQ = kResPlay * K;   // quads of a thread: K of each virtual thread
    const ResidentGeom& g = m.g;
    if (ld_status(a.st.status) != ST_RUNNING) return;
    VT* const P = reinterpret_cast<VT*>(res_smem);
    constexpr bool XS = kXShared<VT, K>;
    VT* const RB = P + g.p_elems;                       // STRIDED: rpad entries
    VT* const XB = RB + (STRIDED ? g.rpad : 0);         // XS: rpad entries
    MT* const vs = reinterpret_cast<MT*>(XB + (XS ? g.rpad : 0));
    const int tid = threadIdx.x;
    const int t = tid & (kTile - 1);
    const ResidentPos at(g);
    const int lo = at.lo, cnt = at.cnt;
    const MT* const dv = a.dia.vals + __ldg(a.dia.base);
    const bool jacobi = a.dinv != nullptr;
    if (tid == 0) sc.fail = sc.hfail = 0;
    stage_values<MT, ND>(vs, dv, g, lo, cnt, false);
    for (int i = tid; i < g.p_elems; i += kResThreads) P[i] = VT(0);
    // quad s = h K + k: relative rows li[s] .. li[s] + 3, those below end[s] exist
    int li[NQ], end[NQ];
    VT R[NQ][4], X[XS ? 1 : NQ][4], D[NQ][4], DS[STRIDED ? kResPlay : 1][STRIDED ? 4 * K : 1];
#pragma unroll
    for (int s = 0; s < NQ; ++s) {
        end[s] = at.a1[s / K];
        li[s] = at.a0[s / K] + 4 * t + 4 * kTile * (s % K);
        if (li[s] >= end[s]) { li[s] = 0; end[s] = 0; }   // (no rows: reads in range, nothing written)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool ok = li[s] + q < end[s];
            R[s][q] = ok ? a.r[lo + li[s] + q] : VT(0);
            const VT xi = ok ? a.x[lo + li[s] + q] : VT(0);
            if constexpr (!XS) X[s][q] = xi;
            else if (ok) XB[li[s] + q] = xi;
            D[s][q] = ok && jacobi ? a.dinv[lo + li[s] + q] : VT(1);
        }
    }
    // STRIDED: the inverse diagonal of rows a0 + t + 256 k
    if constexpr (STRIDED) {
#pragma unroll
        for (int h = 0; h < kResPlay; ++h)
#pragma unroll
            for (int k = 0; k < 4 * K; ++k) {
                const int i = at.a0[h] + t + kTile * k;
                DS[h][k] = i < at.a1[h] && jacobi ? a.dinv[lo + i] : VT(1);
            }
    }
    HaloHeld<VT> held;
    held.init(g, at);
    VT rz = static_cast<VT>(a.st.rz[0]), rr = static_cast<VT>(a.st.rr[0]);
    const VT tol = static_cast<VT>(a.tol), bb = static_cast<VT>(a.st.bb[0]);
    const int64_t maxit = sys_max_iter(a.max_iter, g.n);
    int32_t it = 0, status = ST_RUNNING;
    uint32_t tag = 0;
    uint64_t* const words2 = m.words + kSumWords;
    __syncthreads();
    // p_0 = z (beta = 0, p_{-1} = 0)
    halo_update<VT, true>(P, m, at, held, 0u, VT(0), a.r, a.dinv, &sc.hfail);
    VT beta = VT(0);
    while (status == ST_RUNNING) {
        ++tag;
        const uint32_t want = tag + m.lim.extra;
        // own p
#pragma unroll
        for (int s = 0; s < NQ; ++s) {
            if (li[s] < end[s]) {
                V4<VT> p;
                p.load(P + g.own + li[s]);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const VT z = jacobi ? D[s][q] * R[s][q] : R[s][q];
                    p.v[q] = li[s] + q < end[s] ? p_next(beta, p.v[q], z) : VT(0);
                }
                p.store(P + g.own + li[s]);
            }
        }
        __syncthreads();
        // q = A p, p.q
        VT Q[NQ][4];
        VT pq[1][kResPlay];
#pragma unroll
        for (int h = 0; h < kResPlay; ++h) {   // (a virtual thread's quads at a time: registers)
            int lh[K];
            VT qh[K][4], own[K][4];
#pragma unroll
            for (int k = 0; k < K; ++k) lh[k] = li[h * K + k];
            quads_product<VT, MT, ND, K>(P, vs, dv, g, lo, false, lh, qh, own);
            pq[0][h] = VT(0);
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    Q[h * K + k][q] = qh[k][q];
                    if (lh[k] + q < end[h * K + k]) pq[0][h] += own[k][q] * qh[k][q];
                }
        }
        if (!resident_sum<VT, 1>(pq, sc, m, m.words, tag, [] {})) break;
        const VT alpha = rz / pq[0][0];
        if (!finite_(pq[0][0]) || !finite_(alpha)) { status = CMCG_SOLVE_NON_FINITE; break; }
        if (!(pq[0][0] > VT(0))) { status = CMCG_SOLVE_BREAKDOWN; break; }
        // x += alpha p, r -= alpha q, z published where other CTAs gather it
        VT s2[2][kResPlay];
#pragma unroll
        for (int h = 0; h < kResPlay; ++h) s2[0][h] = s2[1][h] = VT(0);
#pragma unroll
        for (int s = 0; s < NQ; ++s) {
            if (li[s] >= end[s]) continue;
            V4<VT> p;
            p.load(P + g.own + li[s]);
            VT z[4];
            if constexpr (XS) {
                V4<VT> x;
                x.load(XB + li[s]);
#pragma unroll
                for (int q = 0; q < 4; ++q) x.v[q] += alpha * p.v[q];
                x.store(XB + li[s]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if constexpr (!XS) X[s][q] += alpha * p.v[q];
                const VT ri = R[s][q] - alpha * Q[s][q];
                R[s][q] = ri;
                z[q] = jacobi ? D[s][q] * ri : ri;
                if (!STRIDED && li[s] + q < end[s]) {
                    s2[0][s / K] += ri * ri;
                    s2[1][s / K] += ri * z[q];
                }
            }
            if constexpr (STRIDED) {
                V4<VT> w;
#pragma unroll
                for (int q = 0; q < 4; ++q) w.v[q] = R[s][q];
                w.store(RB + li[s]);
            }
            halo_publish(m, at, li[s], end[s], z, tag);
        }
        if constexpr (STRIDED) {
            __syncthreads();
#pragma unroll
            for (int h = 0; h < kResPlay; ++h)
#pragma unroll
                for (int k = 0; k < 4 * K; ++k) {
                    const int i = at.a0[h] + t + kTile * k;
                    if (i < at.a1[h]) {
                        const VT ri = RB[i];
                        const VT zi = jacobi ? DS[h][k] * ri : ri;
                        s2[0][h] += ri * ri;
                        s2[1][h] += ri * zi;
                    }
                }
        }
        if (!resident_sum<VT, 2>(s2, sc, m, words2, tag, [&] { held.gather(m, want, &sc.hfail); })) break;
        rr = s2[0][0];
        const VT rzn = s2[1][0];
        if (!finite_(rr) || !finite_(rzn)) { status = CMCG_SOLVE_NON_FINITE; break; }
        if (rr < tol * tol * bb) { status = CMCG_SOLVE_CONVERGED; break; }
        if (!(rzn > VT(0))) { status = CMCG_SOLVE_BREAKDOWN; break; }
        beta = rzn / rz;
        rz = rzn;
        ++it;
        if (it >= maxit) { status = CMCG_SOLVE_MAX_ITER; break; }
        halo_update<VT, false>(P, m, at, held, want, beta, nullptr, nullptr, &sc.hfail);
        // (a poll that ran out is seen by all at the next sum)
    }
#pragma unroll
    for (int s = 0; s < NQ; ++s)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (li[s] + q < end[s]) a.x[lo + li[s] + q] = XS ? XB[li[s] + q] : X[XS ? 0 : s][q];
    if (blockIdx.x == 0 && tid == 0) {
        a.st.it[0] = it;
        a.st.status[0] = status;
        a.st.rr[0] = static_cast<double>(rr);
    }
}

// ---- mixed precision with reliable updates --------------------------------------

// x read by other CTAs after a fold: through L2
struct CgX {
    const double* x;
    __device__ __forceinline__ double operator()(int c) const { return __ldcg(x + c); }
};

// x += S xh over the rows [r0, r1) of a virtual CTA, the virtual thread's own quads
__device__ __noinline__ void resident_fold(double* __restrict__ x64, const double* __restrict__ s,
                                           const float* xh, int r0, int r1) {
    for (int ib = r0 + 4 * (threadIdx.x & (kTile - 1)); ib < r1; ib += 4 * kTile)
        for (int i = ib; i < min(ib + 4, r1); ++i) x64[i] += s[i] * static_cast<double>(xh[i]);
}

// r = S (b - A x) of the same rows, in FP64; acc = |b - A x|^2 and |r|^2
template <typename MI, typename MO>
__device__ __noinline__ double2 resident_residual(const GMixArgs<MI, MO>& m, int r0, int r1) {
    const auto Ao = inst_matrix<MO, CMCG_CSR>(m.mo, 0);
    double s0 = 0.0, s1 = 0.0;
    for (int ib = r0 + 4 * (threadIdx.x & (kTile - 1)); ib < r1; ib += 4 * kTile) {
        double ax[4];
        sell_rows4<double>(Ao.rm, 0, ib, CgX{m.x64}, ax);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (ib + q >= r1) break;
            const double r64 = m.b64[ib + q] - ax[q];
            const float rh = static_cast<float>(m.s[ib + q] * r64);
            m.g.r[ib + q] = rh;
            s0 += r64 * r64;
            s1 += static_cast<double>(rh) * static_cast<double>(rh);
        }
    }
    return make_double2(s0, s1);
}

// Replacement state of the mixed solve (shared memory: the loop keeps its
// registers; written by thread 0 at a replacement).
struct MixState {
    double rr;         // |b - A x|^2 at the last replacement
    float rmax, goal;  // scaled |r|^2 there, and the one that would meet the target
    int32_t force_it;  // iteration that forces a replacement (progress guard, iteration limit)
    int32_t outer, cyc0, stall;
};
__device__ __forceinline__ int32_t next_forced(int32_t it, int32_t outer, int32_t cyc0, float delta, int64_t maxit) {
    const int64_t f = static_cast<int64_t>(it) + stall_len(outer, cyc0, delta);
    return static_cast<int32_t>(f < maxit ? f : maxit);
}

// The grid path's mixed solve (k_gmix_*) of instance 0 in the same form: FP32
// CG on the scaled system with r and the increments xh in registers; at a
// replacement every CTA folds its increments into the FP64 solution in global
// memory, passes one grid sum (which orders the folds before the reads), and
// forms its rows of S (b - A x) in FP64. STRIDED as in k_resident_cg.
template <typename MI, typename MO, int ND, int K, bool STRIDED>
__global__ void __launch_bounds__(kResThreads, 1) k_resident_mixed(const __grid_constant__ GMixArgs<MI, MO> m,
                                                                   const __grid_constant__ ResidentArgs ra) {
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ SumScratch<float> sc;
    __shared__ SumScratch<double> sd;
    __shared__ MixState ms;
    constexpr int NQ = kResPlay * K;
    const SolveArgs<float, MI>& a = m.g;
    const ResidentGeom& g = ra.g;
    if (ld_status(a.st.status) != ST_RUNNING) return;
    float* const P = reinterpret_cast<float*>(res_smem);
    constexpr bool XS = kXShared<float, K>;
    float* const RB = P + g.p_elems;
    float* const XB = RB + (STRIDED ? g.rpad : 0);
    MI* const vs = reinterpret_cast<MI*>(XB + (XS ? g.rpad : 0));
    const int tid = threadIdx.x;
    const int t = tid & (kTile - 1);
    const ResidentPos at(g);
    const int lo = at.lo, cnt = at.cnt;
    const MI* const dv = a.dia.vals + __ldg(a.dia.base);
    const bool unit = a.dia.unit && __ldg(a.dia.unit) != 0;
    if (tid == 0) sc.fail = sc.hfail = sd.fail = sd.hfail = 0;
    stage_values<MI, ND>(vs, dv, g, lo, cnt, unit);
    for (int i = tid; i < g.p_elems; i += kResThreads) P[i] = 0.0f;
    int li[NQ], end[NQ];
    float R[NQ][4], X[XS ? 1 : NQ][4];
#pragma unroll
    for (int s = 0; s < NQ; ++s) {
        end[s] = at.a1[s / K];
        li[s] = at.a0[s / K] + 4 * t + 4 * kTile * (s % K);
        if (li[s] >= end[s]) { li[s] = 0; end[s] = 0; }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            R[s][q] = li[s] + q < end[s] ? a.r[lo + li[s] + q] : 0.0f;
            if constexpr (!XS) X[s][q] = 0.0f;
            else if (li[s] + q < end[s]) XB[li[s] + q] = 0.0f;
        }
    }
    HaloHeld<float> held;
    held.init(g, at);
    float rz = static_cast<float>(a.st.rz[0]);
    if (tid == 0) {
        ms.rmax = static_cast<float>(a.st.rmax[0]);
        ms.goal = static_cast<float>(a.st.goal[0]);
        ms.rr = a.st.rr[0];
        ms.outer = ms.cyc0 = ms.stall = 0;
        ms.force_it = next_forced(0, 0, 0, m.delta, sys_max_iter(a.max_iter, g.n));
    }
    int32_t it = 0, status = ST_RUNNING;
    uint32_t tag = 0, htag = 0;
    uint64_t* const words2 = ra.words + kSumWords;
    uint64_t* const words3 = words2 + kSumWords;
    uint64_t* const words4 = words3 + kSumWords;
    __syncthreads();
    halo_update<float, true>(P, ra, at, held, 0u, 0.0f, a.r, static_cast<const float*>(nullptr), &sc.hfail);
    float beta = 0.0f;
    while (status == ST_RUNNING) {
        ++tag;
#pragma unroll
        for (int s = 0; s < NQ; ++s) {
            if (li[s] < end[s]) {
                V4<float> p;
                p.load(P + g.own + li[s]);
#pragma unroll
                for (int q = 0; q < 4; ++q) p.v[q] = li[s] + q < end[s] ? p_next(beta, p.v[q], R[s][q]) : 0.0f;
                p.store(P + g.own + li[s]);
            }
        }
        __syncthreads();
        float Q[NQ][4];
        float pq[1][kResPlay];
#pragma unroll
        for (int h = 0; h < kResPlay; ++h) {   // (a virtual thread's quads at a time: registers)
            int lh[K];
            float qh[K][4], own[K][4];
#pragma unroll
            for (int k = 0; k < K; ++k) lh[k] = li[h * K + k];
            quads_product<float, MI, ND, K>(P, vs, dv, g, lo, unit, lh, qh, own);
            pq[0][h] = 0.0f;
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    Q[h * K + k][q] = qh[k][q];
                    if (lh[k] + q < end[h * K + k]) pq[0][h] += own[k][q] * qh[k][q];
                }
        }
        if (!resident_sum<float, 1>(pq, sc, ra, ra.words, tag, [] {})) break;
        const float alpha = rz / pq[0][0];
        if (!finite_(pq[0][0]) || !finite_(alpha)) { status = CMCG_SOLVE_NON_FINITE; break; }
        if (!(pq[0][0] > 0.0f)) { status = CMCG_SOLVE_BREAKDOWN; break; }
        ++htag;
        float s1[1][kResPlay];
#pragma unroll
        for (int h = 0; h < kResPlay; ++h) s1[0][h] = 0.0f;
#pragma unroll
        for (int s = 0; s < NQ; ++s) {
            if (li[s] >= end[s]) continue;
            V4<float> p;
            p.load(P + g.own + li[s]);
            if constexpr (XS) {
                V4<float> x;
                x.load(XB + li[s]);
#pragma unroll
                for (int q = 0; q < 4; ++q) x.v[q] += alpha * p.v[q];
                x.store(XB + li[s]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if constexpr (!XS) X[s][q] += alpha * p.v[q];
                R[s][q] -= alpha * Q[s][q];
                if (!STRIDED && li[s] + q < end[s]) s1[0][s / K] += R[s][q] * R[s][q];
            }
            if constexpr (STRIDED) {
                V4<float> w;
#pragma unroll
                for (int q = 0; q < 4; ++q) w.v[q] = R[s][q];
                w.store(RB + li[s]);
            }
            halo_publish(ra, at, li[s], end[s], R[s], htag);
        }
        if constexpr (STRIDED) {
            __syncthreads();
#pragma unroll
            for (int h = 0; h < kResPlay; ++h)
#pragma unroll
                for (int k = 0; k < 4 * K; ++k) {
                    const int i = at.a0[h] + t + kTile * k;
                    if (i < at.a1[h]) s1[0][h] += RB[i] * RB[i];
                }
        }
        const uint32_t hwant = htag + ra.lim.extra;
        if (!resident_sum<float, 1>(s1, sc, ra, words2, tag, [&] { held.gather(ra, hwant, &sc.hfail); })) break;
        const float rzn = s1[0][0];
        ++it;
        if (!finite_(rzn)) { status = CMCG_SOLVE_NON_FINITE; break; }
        if (std::is_same<MI, __nv_bfloat16>::value && it == kCondProbe && ms.outer == 0 &&
            !bf16_condition_ok(rzn / ms.rmax, it)) {
            status = CMCG_SOLVE_BREAKDOWN;
            break;
        }
        float rnew = rzn;
        if (rzn < (m.delta * m.delta) * ms.rmax || rzn < ms.goal || it >= ms.force_it) {
            // x += S xh, then r = S (b - A x) in FP64 (through global memory and
            // calls, so that the FP64 code takes no registers from the loop)
#pragma unroll
            for (int s = 0; s < NQ; ++s)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (li[s] + q < end[s]) {
                        m.xh[lo + li[s] + q] = XS ? XB[li[s] + q] : X[XS ? 0 : s][q];
                        if constexpr (XS) XB[li[s] + q] = 0.0f;
                    }
                    if constexpr (!XS) X[s][q] = 0.0f;
                }
#pragma unroll
            for (int h = 0; h < kResPlay; ++h) resident_fold(m.x64, m.s, m.xh, lo + at.a0[h], lo + at.a1[h]);
            float none[1][kResPlay] = {};
            if (!resident_sum<float, 1, /*ORDER=*/true>(none, sc, ra, words3, tag, [] {})) break;
            ++htag;
            double acc[2][kResPlay];
#pragma unroll
            for (int h = 0; h < kResPlay; ++h) {
                const double2 s = resident_residual<MI, MO>(m, lo + at.a0[h], lo + at.a1[h]);
                acc[0][h] = s.x;
                acc[1][h] = s.y;
            }
#pragma unroll
            for (int s = 0; s < NQ; ++s) {
                if (li[s] >= end[s]) continue;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (li[s] + q < end[s]) R[s][q] = __ldcg(a.r + lo + li[s] + q);
                halo_publish(ra, at, li[s], end[s], R[s], htag);
            }
            if (!resident_sum<double, 2>(acc, sd, ra, words4, tag,
                                         [&] { held.gather(ra, htag + ra.lim.extra, &sc.hfail); }))
                break;
            const double rr64 = acc[0][0], rr_prev = ms.rr;
            rnew = static_cast<float>(acc[1][0]);
            const double thr = m.outer_tol * m.outer_tol * a.st.bb[0];
            const int32_t outer = ms.outer + 1;
            const int32_t stall = rr64 > kStallRatio * rr_prev ? ms.stall + 1 : 0;
            const int32_t cyc0 = outer == 1 ? it : ms.cyc0;
            const int64_t maxit = sys_max_iter(a.max_iter, g.n);
            const double dd = static_cast<double>(m.delta) * m.delta;
            __syncthreads();   // (every thread has read the state)
            if (tid == 0) {
                ms.rr = rr64;
                ms.rmax = rnew;
                ms.goal = static_cast<float>(thr / rr64) * rnew;
                ms.outer = outer;
                ms.stall = stall;
                ms.cyc0 = cyc0;
                ms.force_it = next_forced(it, outer, cyc0, m.delta, maxit);
            }
            if (!finite_(rr64)) status = CMCG_SOLVE_NON_FINITE;
            else if (rr64 < thr) status = CMCG_SOLVE_CONVERGED;
            else if (std::is_same<MI, __nv_bfloat16>::value && rr64 > kBf16Lag * dd * rr_prev)
                status = CMCG_SOLVE_BREAKDOWN;   // BF16 values too coarse for this system
            else if (it >= maxit || outer >= m.max_updates) status = CMCG_SOLVE_MAX_ITER;
            else if (!(rnew > 0.0f) || stall >= kStallMax) status = CMCG_SOLVE_BREAKDOWN;
            if (status != ST_RUNNING) break;
        } else if (!(rzn > 0.0f)) {
            status = CMCG_SOLVE_BREAKDOWN;
            break;
        }
        beta = rnew / rz;
        rz = rnew;
        halo_update<float, false>(P, ra, at, held, htag + ra.lim.extra, beta, nullptr, nullptr, &sc.hfail);
    }
    // increments a breakdown left unfolded: the closing fold takes them
#pragma unroll
    for (int s = 0; s < NQ; ++s)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (li[s] + q < end[s]) m.xh[lo + li[s] + q] = XS ? XB[li[s] + q] : X[XS ? 0 : s][q];
    if (blockIdx.x == 0 && tid == 0) {
        a.st.it[0] = it;
        a.st.status[0] = status;
        a.st.rr[0] = ms.rr;
        a.st.outer[0] = ms.outer;
    }
}

inline int32_t floor4(int32_t v) { return v >= 0 ? v & ~3 : -((-v + 3) & ~3); }

}  // namespace

bool resident_plan(ResidentGeom& g, int32_t n, int32_t n_virtual, int32_t nd, const int32_t* off, int32_t sms,
                   size_t val_bytes, size_t vec_bytes, size_t smem_limit) {
    g = ResidentGeom();
    g.n = n;
    g.n_virtual = n_virtual;
    g.n_tiles = static_cast<int32_t>((static_cast<int64_t>(n) + kTile - 1) / kTile);
    g.ctas = (n_virtual + kResVirtual - 1) / kResVirtual;
    if (n_virtual < 1 || n_virtual > kResMaxVirtual || g.ctas > sms) return false;
    // rows of a virtual CTA and of a CTA at most
    int32_t vt = 0, ct = 0;
    const auto tile0 = [&](int32_t v) {
        return static_cast<int32_t>(static_cast<int64_t>(std::min(v, n_virtual)) * g.n_tiles / n_virtual);
    };
    for (int32_t v = 0; v < n_virtual; ++v) vt = std::max(vt, tile0(v + 1) - tile0(v));
    for (int32_t c = 0; c < g.ctas; ++c) ct = std::max(ct, tile0((c + 1) * kResVirtual) - tile0(c * kResVirtual));
    g.quads = (vt + 3) / 4;
    // registers: two quads per thread of FP32 state, one of FP64
    if (g.quads > (vec_bytes == 4 ? 2 : 1)) return false;
    g.rpad = ct * kTile;
    // windows of p: relative rows [off, off + rpad + 4) of every diagonal and
    // the own rows, merged where they overlap; one extra quad each side for
    // unaligned quads and the +-1 neighbours
    struct Iv { int32_t lo, hi; };
    Iv iv[kDiaMax + 1];
    int32_t m = 0;
    iv[m++] = Iv{-4, g.rpad + 4};
    for (int32_t d = 0; d < nd; ++d) iv[m++] = Iv{floor4(off[d]), floor4(off[d]) + g.rpad + 8};
    std::sort(iv, iv + m, [](const Iv& x, const Iv& y) { return x.lo < y.lo; });
    for (int32_t i = 0; i < m; ++i) {
        if (g.n_win > 0 && iv[i].lo <= g.win_lo[g.n_win - 1] + g.win_len[g.n_win - 1]) {
            const int32_t hi = std::max(g.win_lo[g.n_win - 1] + g.win_len[g.n_win - 1], iv[i].hi);
            g.win_len[g.n_win - 1] = hi - g.win_lo[g.n_win - 1];
        } else {
            if (g.n_win == kResMaxWindows) return false;
            g.win_lo[g.n_win] = iv[i].lo;
            g.win_len[g.n_win++] = iv[i].hi - iv[i].lo;
        }
    }
    int32_t margin = 0;
    for (int32_t w = 0; w < g.n_win; ++w) {
        g.win_base[w] = g.p_elems;
        g.p_elems += g.win_len[w];
    }
    const auto elem = [&](int32_t rel) {
        for (int32_t w = 0; w < g.n_win; ++w)
            if (rel >= g.win_lo[w] && rel < g.win_lo[w] + g.win_len[w]) return g.win_base[w] + rel - g.win_lo[w];
        return -1;
    };
    g.own = elem(0);
    for (int32_t d = 0; d < nd; ++d) {
        g.off[d] = off[d];
        g.pd[d] = elem(off[d]);
        margin = std::max(margin, std::abs(off[d]));
    }
    g.reach = static_cast<int32_t>(std::min<int64_t>(static_cast<int64_t>(margin) + 16, n));
    // 16-byte aligned vectors exist where the rows are a multiple of 16 bytes
    g.strided = (static_cast<size_t>(n) * vec_bytes) % 16 != 0;
    const bool xs = g.quads == 2 || vec_bytes == 8;   // (kXShared)
    const size_t fixed = vec_bytes * (static_cast<size_t>(g.p_elems) + static_cast<size_t>(g.rpad) * (g.strided + xs));
    if (fixed > smem_limit) return false;
    g.smem_diags = static_cast<int32_t>(
        std::min<size_t>(static_cast<size_t>(nd), (smem_limit - fixed) / (val_bytes * static_cast<size_t>(g.rpad))));
    g.smem = fixed + val_bytes * static_cast<size_t>(g.rpad) * g.smem_diags;
    return true;
}

// (16-byte aligned sections)
static size_t even(int32_t v) { return (static_cast<size_t>(v) + 1) & ~size_t(1); }

size_t resident_ws_bytes(const ResidentGeom& g, size_t vec_bytes) {
    const size_t w = vec_bytes / 4;
    return sizeof(uint64_t) * (w * even(g.n) + 4 * kSumWords);   // (the mixed solve has four sums)
}

// Launches `kern` (its arguments: args and the ResidentArgs) cooperatively when
// its CTAs can all be resident.
template <typename A>
static cmcg_status resident_launch(const void* kern, A args, const ResidentGeom& g, size_t vec_bytes, void* ws,
                                   int32_t* err, cudaStream_t st, bool* launched) {
    *launched = false;
    if (!kern) return CMCG_OK;
    CMCG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(g.smem)));
    int occ = 0, dev = 0, sms = 0;
    CMCG_CUDA(cudaGetDevice(&dev));
    CMCG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CMCG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kResThreads, g.smem));
    if (occ * sms < g.ctas) return CMCG_OK;
    CMCG_CUDA(cudaMemsetAsync(ws, 0, resident_ws_bytes(g, vec_bytes), st));
    BarrierLimits lim{kGridBarrierSpins, 0u};
    if (const char* e = std::getenv("CUMAT_TEST_GRID_SPINS")) lim.spins = std::max(1LL, std::atoll(e));
    if (const char* e = std::getenv("CUMAT_TEST_GRID_EXTRA")) lim.extra = static_cast<unsigned>(std::max(0, std::atoi(e)));
    uint64_t* w = static_cast<uint64_t*>(ws);
    ResidentArgs m{g, w, w + vec_bytes / 4 * even(g.n), err, lim, {g.n_virtual, g.n_virtual}};
    if (std::getenv("CUMAT_TEST_GRID_PARTIAL")) m.partials[1] = std::min(g.n_virtual + 1, kResMaxVirtual);
    void* params[] = {&args, &m};
    CMCG_CUDA(cudaLaunchCooperativeKernel(kern, g.ctas, kResThreads, params, g.smem, st));
    *launched = true;
    return CMCG_OK;
}

template <typename VT, typename MT>
cmcg_status resident_cg_launch(const SolveArgs<VT, MT>& a, const ResidentGeom& g, int nd, void* ws, int32_t* err,
                               cudaStream_t st, bool* launched) {
    const void* kern = nullptr;
#define CMCG_RES_PICK(ND, K)                                                                            \
    if (nd == ND && g.quads == K)                                                                       \
    kern = g.strided ? reinterpret_cast<const void*>(k_resident_cg<VT, MT, ND, K, true>)                \
                     : reinterpret_cast<const void*>(k_resident_cg<VT, MT, ND, K, false>)
    CMCG_RES_PICK(5, 1);
    CMCG_RES_PICK(7, 1);
    if constexpr (sizeof(VT) == 4) {
        CMCG_RES_PICK(5, 2);
        CMCG_RES_PICK(7, 2);
    }
#undef CMCG_RES_PICK
    return resident_launch(kern, a, g, sizeof(VT), ws, err, st, launched);
}

template <typename MI, typename MO>
cmcg_status resident_mixed_launch(const GMixArgs<MI, MO>& a, const ResidentGeom& g, int nd, void* ws, int32_t* err,
                                  cudaStream_t st, bool* launched) {
    const void* kern = nullptr;
#define CMCG_RES_PICK(ND, K)                                                                            \
    if (nd == ND && g.quads == K)                                                                       \
    kern = g.strided ? reinterpret_cast<const void*>(k_resident_mixed<MI, MO, ND, K, true>)             \
                     : reinterpret_cast<const void*>(k_resident_mixed<MI, MO, ND, K, false>)
    CMCG_RES_PICK(5, 1);
    CMCG_RES_PICK(7, 1);
    CMCG_RES_PICK(5, 2);
    CMCG_RES_PICK(7, 2);
#undef CMCG_RES_PICK
    return resident_launch(kern, a, g, sizeof(float), ws, err, st, launched);
}

#define CMCG_RES_INSTANTIATE(VT, MT) \
    template cmcg_status resident_cg_launch<VT, MT>(const SolveArgs<VT, MT>&, const ResidentGeom&, int, void*, int32_t*, \
                                                    cudaStream_t, bool*);
CMCG_RES_INSTANTIATE(float, float)
CMCG_RES_INSTANTIATE(float, double)
CMCG_RES_INSTANTIATE(float, __nv_bfloat16)
CMCG_RES_INSTANTIATE(double, float)
CMCG_RES_INSTANTIATE(double, double)
CMCG_RES_INSTANTIATE(double, __nv_bfloat16)
#define CMCG_RES_MIXED(MI, MO) \
    template cmcg_status resident_mixed_launch<MI, MO>(const GMixArgs<MI, MO>&, const ResidentGeom&, int, void*, \
                                                       int32_t*, cudaStream_t, bool*);
CMCG_RES_MIXED(float, float)
CMCG_RES_MIXED(float, double)
CMCG_RES_MIXED(__nv_bfloat16, float)
CMCG_RES_MIXED(__nv_bfloat16, double)

}  // namespace cmcg
