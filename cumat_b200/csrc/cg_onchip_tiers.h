// Launch forms of the on-chip batched kernels (cg_onchip.cu, cg_onchip_mixed.cu)
// and the rule that splits a batch's systems over them. Host code without CUDA, so
// that the rule can be checked by itself.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define CMCG_HD __host__ __device__
#else
#define CMCG_HD
#endif

namespace cmcg {

// Launch forms, largest systems first. A CTA (or a cluster of CTAs) owns up to
// slots * threads * ctas rows.
struct OnchipForm {
    int threads;   // per CTA
    int ctas;      // cluster size
    int per_sm;    // CTAs (or groups of a 512-thread CTA) that share an SM
};
constexpr int kOnchipForms32 = 4;   // FP32 vectors: 16 row slots per thread
constexpr OnchipForm kOnchip32[kOnchipForms32] = {{512, 2, 1}, {512, 1, 1}, {256, 1, 2}, {128, 1, 4}};
constexpr int kOnchipForms64 = 6;   // FP64 vectors: 8 row slots per thread
constexpr OnchipForm kOnchip64[kOnchipForms64] = {{512, 4, 1}, {512, 3, 1}, {512, 2, 1}, {512, 1, 1}, {256, 1, 2},
                                                  {128, 1, 4}};
constexpr int kOnchipFormsMix = 3;  // mixed solve, systems of at most 8192 rows
constexpr OnchipForm kOnchipMix[kOnchipFormsMix] = {{512, 1, 1}, {256, 1, 2}, {128, 1, 4}};
template <typename VT> constexpr int kOnchipSlots = sizeof(VT) == 4 ? 16 : 8;

// The mixed solve's tiers by rows (those of k_mixed_fast, whose order of sums it keeps)
constexpr int kOnchipMixRows = 8192;       // at most: larger systems stay on k_mixed_fast
constexpr int kOnchipMixTinyRows = 4096;   // above: 512 threads

constexpr int kOnchipGroupScratch = 544;   // shared memory of a group's sums (FP32 launch)
constexpr int kOnchipMixScratch = 1056;    // the same, mixed solve
// Static shared memory of a CTA (the kernels' files assert it)
constexpr int kOnchipStatic64 = 2064;      // k_onchip with FP64 vectors
constexpr int kOnchipStaticMix256 = 2048;  // k_onchip_mixed256 (at most)

// Row slots per thread of a system of n rows (a multiple of two, see the kernel).
CMCG_HD inline int onchip_slots(int n, int threads, int ctas) {
    const int per = threads * ctas;
    return ((n + per - 1) / per + 1) & ~1;
}

// Dynamic shared memory of a form for systems of up to max_rows rows with nd
// stored diagonals and offsets of up to margin in the batch; 0 where they are too many rows.
template <typename VT>
inline size_t onchip_smem(const OnchipForm& f, int max_rows, int nd, int margin, size_t val_bytes) {
    const int nk = onchip_slots(max_rows, f.threads, f.ctas);
    if (nk > kOnchipSlots<VT>) return 0;
    const size_t own = static_cast<size_t>(nk) * f.threads;
    // FP32 pairs of CTAs interleave their rows and hold p of both
    const bool interleaved = sizeof(VT) == 4 && f.ctas == 2;
    const size_t p = (interleaved ? 2 * own : own) + 2 * static_cast<size_t>((margin + 3) & ~3);
    return p * sizeof(VT) + own * nd * val_bytes;
}

// Whether a form solves a system of n rows whose largest offset is reach: where a
// cluster's CTAs own contiguous rows (FP64), each exchanges entries with its two
// neighbours only, so the reach ends in the neighbour: within this system's own
// rows per CTA, which may be fewer than the tier's largest system has.
template <typename VT>
inline bool onchip_halo_ok(const OnchipForm& f, int n, int reach) {
    if (sizeof(VT) == 4 || f.ctas == 1) return true;
    return reach <= onchip_slots(n, f.threads, f.ctas) * f.threads;
}

// Dynamic shared memory of a CTA when per_sm of them share an SM: 228 KB, of
// which every CTA takes 1 KB for the system and its static arrays.
inline size_t onchip_smem_limit(int per_sm, int static_bytes) {
    return static_cast<size_t>(228 * 1024 / per_sm - 1024 - static_bytes);
}
// In the launches with FP32 vectors the systems share one CTA's memory, whose
// static arrays are below 1 KB (plain) and 1.1 KB (mixed); a group of its threads
// keeps its scratch in its part.
inline size_t onchip_smem_limit32(int per_sm, bool mixed) {
    const size_t scratch = mixed ? kOnchipMixScratch : kOnchipGroupScratch;
    return static_cast<size_t>((227 * 1024 - (mixed ? 1280 : 1024)) / per_sm) - (per_sm > 1 ? scratch + 16 : 0);
}

// The systems of a batch in size order, from the solver and the pattern's diagonal
// plan.
struct OnchipBatch {
    const int32_t* rows;    // of a system, by position in the size order
    const int32_t* reach;   // its largest |offset|
    int32_t n_sys, first;   // positions [first, n_sys)
    int32_t ob;             // instances per system
    int32_t sms;
    int nd, margin;         // stored diagonals, largest |offset| of all systems
    size_t val_bytes;
    bool mixed;
};

// Tiers of an on-chip batched solve: which systems (positions in the size
// order) run on which launch form, and the form's dynamic shared memory.
struct OnchipTier {
    OnchipForm form;
    int32_t lo, hi;   // work items: position * ob + instance
    size_t smem;
};

// Splits the systems over the forms: each system takes the smallest form that
// holds it (its shared memory, its rows and its halo), since more CTAs of fewer threads
// share an SM there (592 systems of 4096 rows, FP64: 2.7 ms two to an SM, 7.5 ms
// for the next size, 4225 rows, one to an SM); with at most one instance per SM
// the forms that share an SM are left out, which spreads the rows over more
// threads. The fallback for systems no form holds is the kernel each form is
// measured against: FP32 20 .. 128 rows square 1.4 .. 3.6x slower, FP64 1.1 ..
// 6.4x, mixed up to 8192 rows 1.1 .. 1.9x. Empty when a system fits no form, or
// not the one its place in the size order gives it.
template <typename VT, int NF>
std::vector<OnchipTier> onchip_tiers(const OnchipBatch& b, const OnchipForm (&forms)[NF]) {
    std::vector<OnchipTier> tiers;
    const bool few = static_cast<int64_t>(b.n_sys) * b.ob <= b.sms;
    const auto fits = [&](const OnchipForm& f, int rows, int reach) {
        // (the mixed solve's order of sums, k_mixed_fast's, goes by size alone)
        if (b.mixed) {
            if (rows > kOnchipMixRows || (f.threads == 512 ? rows <= kOnchipMixTinyRows : rows > kOnchipMixTinyRows))
                return false;
            if (few && f.threads == 128) return false;
        } else if (few && f.per_sm > 1) {
            return false;
        }
        const size_t s = onchip_smem<VT>(f, rows, b.nd, b.margin, b.val_bytes);
        const bool whole = sizeof(VT) == 8 || (b.mixed && f.threads == 256);   // CTAs of this form share the SM, not a CTA's part
        const size_t limit = whole ? onchip_smem_limit(f.per_sm, sizeof(VT) == 8 ? kOnchipStatic64 : kOnchipStaticMix256)
                                   : onchip_smem_limit32(f.per_sm, b.mixed);
        return s > 0 && s <= limit && onchip_halo_ok<VT>(f, rows, reach);
    };
    int32_t lo = b.first;
    for (int f = 0; f < NF; ++f) {
        // systems up to the last one that the next smaller forms do not hold
        int32_t hi = b.n_sys;
        if (f + 1 < NF) {
            hi = lo;
            for (int32_t i = b.n_sys; i > lo; --i) {
                bool smaller = false;
                for (int g = f + 1; g < NF && !smaller; ++g) smaller = fits(forms[g], b.rows[i - 1], b.reach[i - 1]);
                if (!smaller) { hi = i; break; }
            }
        }
        if (hi <= lo) continue;
        const int rows = *std::max_element(b.rows + lo, b.rows + hi);
        if (!fits(forms[f], rows, 0)) return {};
        for (int32_t i = lo; i < hi; ++i)
            if (!onchip_halo_ok<VT>(forms[f], b.rows[i], b.reach[i])) return {};
        tiers.push_back({forms[f], lo * b.ob, hi * b.ob, onchip_smem<VT>(forms[f], rows, b.nd, b.margin, b.val_bytes)});
        lo = hi;
    }
    return tiers;
}

}  // namespace cmcg
