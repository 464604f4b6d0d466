// Batched PCG with a system's whole state on the chip (cg_onchip.cu).
#pragma once

#include "cg_grid.cuh"
#include "cg_onchip_tiers.h"
#include "objects.h"

namespace cmcg {

// Work items [lo, hi) of a form: (position in the size order) * batches + batch,
// taken from a counter.
struct OnchipItems {
    int32_t* next;
    int32_t lo, hi;
};
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

// Systems of the 512-thread and the 128-thread form (smem: shared memory of a CTA,
// a multiple of 64); systems of the 256-thread form.
template <typename MI, typename MO>
cmcg_status onchip_mixed_launch(const OnchipMixArgs<MI, MO>& a, const OnchipItems& t512, const OnchipItems& t128, int smem,
                                int nd, int sms, cudaStream_t stream, bool* launched);
template <typename MI, typename MO>
cmcg_status onchip_mixed_launch256(const OnchipMixArgs<MI, MO>& a, const OnchipItems& t, size_t smem, int nd, int sms,
                                   cudaStream_t stream, bool* launched);

}  // namespace cmcg
