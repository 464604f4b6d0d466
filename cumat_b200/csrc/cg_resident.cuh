// Chip-resident solve of one large system (cg_resident.cu).
#pragma once

#include "cg_grid.cuh"
#include "objects.h"

namespace cmcg {

constexpr int kResThreads = 512;       // 128 registers a thread (plain FP32, two quads: 128 .. 336 bytes of spills)
constexpr int kResVirtual = 4;         // virtual 256-thread CTAs (of the grid plan) per CTA
constexpr int kResMaxWindows = 8;
constexpr int kResMaxVirtual = 3 * kTile;   // partial sums one combining thread may add: 3

// Geometry of a resident launch (host-built, see resident_plan).
struct ResidentGeom {
    int32_t n = 0;           // rows of the system
    int32_t n_virtual = 0;   // CTAs of the grid plan
    int32_t n_tiles = 0;
    int32_t ctas = 0;        // CTAs of the launch
    int32_t quads = 0;       // row quads per thread (1 or 2)
    int32_t rpad = 0;        // rows a CTA stores per diagonal
    int32_t n_win = 0;       // p windows (rows relative to the CTA's first row)
    int32_t win_lo[kResMaxWindows] = {};    // first relative row (multiple of 4)
    int32_t win_len[kResMaxWindows] = {};   // rows (multiple of 4)
    int32_t win_base[kResMaxWindows] = {};  // first element in shared memory (multiple of 4)
    int32_t p_elems = 0;     // elements of all windows
    int32_t own = 0;         // element of relative row 0
    int32_t pd[kDiaMax] = {};    // element of relative row off[d]
    int32_t off[kDiaMax] = {};
    int32_t reach = 0;       // rows at either end of a CTA that other CTAs may read
    int32_t smem_diags = 0;  // diagonals kept in shared memory, the rest read from L2
    int32_t strided = 0;     // the update's sums run over rows t, t + 256, ... (see the kernel)
    size_t smem = 0;
};

// Fills g for a system of n rows with the given diagonal offsets on a grid
// plan of n_virtual CTAs; false when the system does not fit the chip.
bool resident_plan(ResidentGeom& g, int32_t n, int32_t n_virtual, int32_t nd, const int32_t* off, int32_t sms,
                   size_t val_bytes, size_t vec_bytes, size_t smem_limit);

// Workspace of a launch: p exchange words and partial-sum words.
size_t resident_ws_bytes(const ResidentGeom& g, size_t vec_bytes);

// Runs the PCG loop of the (initialised) instance 0 of `a` in one cooperative
// launch; *launched = false where the CTAs cannot all be resident.
template <typename VT, typename MT>
cmcg_status resident_cg_launch(const SolveArgs<VT, MT>& a, const ResidentGeom& g, int nd, void* ws, int32_t* err,
                               cudaStream_t st, bool* launched);

// The grid path's mixed solve of instance 0 (after k_gmix_init), likewise.
template <typename MI, typename MO>
cmcg_status resident_mixed_launch(const GMixArgs<MI, MO>& a, const ResidentGeom& g, int nd, void* ws, int32_t* err,
                                  cudaStream_t st, bool* launched);

}  // namespace cmcg
