// One mid-size stencil system spread over up to 64 SMs (cg_wide.cu).
#pragma once

#include "cg_grid.cuh"

namespace cmcg {

// Device memory of a launch: the tagged words of z and of the partial sums.
size_t wide_ws_bytes(int32_t n, size_t vec_bytes);

// Solves instance 0 of `a` (diagonal layout, nd = 5 or 7) with the sums of the
// cluster solve of `clusters` CTAs of 2^rows_log2 rows; *launched = false
// leaves the solve to the cluster.
template <typename VT, typename MT>
cmcg_status wide_cg_launch(const SolveArgs<VT, MT>& a, int rows_log2, int clusters, int nd, int sms, void* ws,
                           int32_t* err, cudaStream_t st, bool* launched);

}  // namespace cmcg
