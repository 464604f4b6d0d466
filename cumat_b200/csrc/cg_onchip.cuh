// Batched PCG with a system's whole state on the chip (cg_onchip.cu).
#pragma once

#include "cg_grid.cuh"
#include "objects.h"

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

// Work items [lo, hi) of a form: (position in the size order) * batches + batch,
// taken from a counter.
struct OnchipItems {
    int32_t* next;
    int32_t lo, hi;
};
constexpr int kOnchipGroupScratch = 544;   // shared memory of a group's sums (FP32 launch)
// All forms of an FP32 launch: a pair of CTAs, a CTA, half and a quarter of one.
struct OnchipWork {
    OnchipItems t[kOnchipForms32];
    int32_t smem;   // dynamic shared memory of a CTA (a multiple of 64)
};

template <typename VT, typename MT>
struct OnchipArgs {
    int32_t rows, n_sys, ob, mb;
    const int32_t* row_off;
    const int32_t* order;          // systems, largest first
    const MT* vals;                // values in the diagonal layout, [mb][vstride]
    int64_t vstride;
    const int64_t* base;           // n_sys
    const int32_t* off;            // n_sys * kDiaMax
    int32_t margin;                // largest |offset|
    const VT* dinv;                // Jacobi inverse diagonal (null: identity)
    int32_t dinv_b;
    const VT* b;
    int32_t b_b;
    const VT* guess;
    int32_t g_b;
    VT* x;                         // [batch][rows]
    double tol;
    int64_t max_iter;
    int32_t abs_zero_test;
    InstState st;
};

// Row slots per thread of a system of n rows (a multiple of two, see the kernel).
__host__ __device__ inline int onchip_slots(int n, int threads, int ctas) {
    const int per = threads * ctas;
    return ((n + per - 1) / per + 1) & ~1;
}

// Dynamic shared memory of a form for systems of up to max_rows rows with nd
// stored diagonals; 0 where the form does not take them (too many rows, or a
// halo wider than a CTA's rows).
template <typename VT>
inline size_t onchip_smem(const OnchipForm& f, int max_rows, int nd, int margin, size_t val_bytes) {
    const int nk = onchip_slots(max_rows, f.threads, f.ctas);
    if (nk > kOnchipSlots<VT>) return 0;
    const size_t own = static_cast<size_t>(nk) * f.threads;
    // FP32 pairs of CTAs interleave their rows and hold p of both
    const bool interleaved = sizeof(VT) == 4 && f.ctas == 2;
    if (!interleaved && f.ctas > 1 && static_cast<size_t>(margin) > own) return 0;
    const size_t p = (interleaved ? 2 * own : own) + 2 * static_cast<size_t>((margin + 3) & ~3);
    return p * sizeof(VT) + own * nd * val_bytes;
}

template <typename VT, typename MT>
cmcg_status onchip_launch(const OnchipArgs<VT, MT>& a, const OnchipItems& t, const OnchipForm& f, size_t smem, int nd,
                          int sms, cudaStream_t stream, bool* launched);
template <typename MT>
cmcg_status onchip_launch_all(const OnchipArgs<float, MT>& a, const OnchipWork& w, int nd, int sms, cudaStream_t stream,
                              bool* launched);

// Mixed precision (FP32 CG on the Jacobi-scaled system, FP64 residual
// replacement).
template <typename MI, typename MO>
struct OnchipMixArgs {
    int32_t rows, n_sys, ob, mb;
    const int32_t* row_off;
    const int32_t* order;
    const MI* vin;                 // scaled inner values, diagonal layout
    int64_t vin_stride;
    const MO* vout;                // unscaled outer values, diagonal layout
    int64_t vout_stride;
    const int32_t* unit;           // [mb][n_sys]: 1 = middle diagonal is offset 0 with all values 1
    const int64_t* base;
    const int32_t* off;
    int32_t margin;
    const double* s;               // scale 1 / sqrt(a_ii) (or 1), [mb][rows]
    const double* b;
    int32_t b_b;
    double* x;
    double outer_tol;
    int64_t max_inner;
    int32_t max_updates;
    float delta;
    InstState st;
};

constexpr int kOnchipMixScratch = 1056;   // shared memory of a group's sums

// Systems of the 512-thread and the 128-thread form (smem: shared memory of a CTA,
// a multiple of 64); systems of the 256-thread form.
template <typename MI, typename MO>
cmcg_status onchip_mixed_launch(const OnchipMixArgs<MI, MO>& a, const OnchipItems& t512, const OnchipItems& t128, int smem,
                                int nd, int sms, cudaStream_t stream, bool* launched);
template <typename MI, typename MO>
cmcg_status onchip_mixed_launch256(const OnchipMixArgs<MI, MO>& a, const OnchipItems& t, size_t smem, int nd, int sms,
                                   cudaStream_t stream, bool* launched);

}  // namespace cmcg
