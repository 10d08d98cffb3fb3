// Interval classification and pruning of one level of cells over
// level-ordered clause lists (k_interval_block and k_interval_wide in
// dc_kernels.cu), shared by the octree mesher and the quadtree contourer.
#pragma once
#include "dc_device.cuh"

namespace lfb {

constexpr uint32_t kMaxTapeRegs = 400;   // registers a tape may use in these kernels

struct WideArgs {
    Octree o;
    DevTape bt;
    uint32_t n;                    // clauses of the unpruned tape
    const WideEntry* in_lists;     // lists of this depth's groups
    ListRef root_list;             // the unpruned list (depth 0)
    WideEntry* out_lists;          // lists handed to the next depth
    unsigned long long* out_top;
    uint64_t out_cap;
    int write_lists;
    RegClause* arena;              // register tapes
    unsigned long long* arena_top;
    uint64_t arena_cap;
    // Per-warp global scratch: slot state of long lists, and the two-level
    // bitmap of clause states that orders the register tape (zero between
    // cells).
    float2* S;                     // [warps][n + 3]
    uint8_t* SN;                   // [warps][n + 3]
    uint8_t* pst;                  // [warps][n]
    uint8_t* live;                 // [warps][n]
    uint32_t* newpos;              // [warps][n]
    uint32_t* st2;                 // [warps][nw]   2-bit state per clause
    uint32_t* l1;                  // [warps][nw1]  non-zero words of st2
    uint32_t* wl;                  // [warps][nw]   word list
    uint32_t* status;
    uint32_t* next_cell;           // work counter (zero at launch)
    uint32_t group_shift;          // cells per group: 8 (3) in an octree, 4 (2) in a quadtree
    // Box form (launch_interval_boxes): the unpruned tape pruned for each of
    // n_boxes boxes (lower and upper bound per axis), whatever the sign of its
    // interval, min / max clauses decided only between operands that cannot
    // be NaN.  The arena's tapes start after arena_base clauses.
    const float* boxes;
    uint32_t n_boxes;
    uint32_t arena_base;
    TapeRef* box_tape;
};

/// Bytes of WideArgs' per-warp scratch for `warps` warps over a tape of n
/// clauses, and its pointers into such a block (st2 and l1 must then be
/// zeroed: the last st2_l1_bytes of it).
inline size_t wide_scratch_bytes(uint64_t n, uint64_t warps, size_t* st2_l1_bytes = nullptr)
{
    const uint64_t nw = (n + 15) / 16, nw1 = (nw + 31) / 32;
    const size_t zeroed = (4 * nw + 4 * nw1) * warps;
    if (st2_l1_bytes) *st2_l1_bytes = zeroed;
    return (8 * (n + 3) + 4 * n + 4 * nw) * warps + ((n + 3) + 2 * n) * warps + 16 + zeroed;
}
inline void wide_scratch_carve(WideArgs& W, unsigned char* p, uint64_t n, uint64_t warps)
{
    const uint64_t nw = (n + 15) / 16;
    W.S = reinterpret_cast<float2*>(p);
    W.newpos = reinterpret_cast<uint32_t*>(W.S + (n + 3) * warps);
    W.wl = W.newpos + n * warps;
    W.SN = reinterpret_cast<uint8_t*>(W.wl + nw * warps);
    W.pst = W.SN + (n + 3) * warps;
    W.live = W.pst + n * warps;
    const uintptr_t q = (reinterpret_cast<uintptr_t>(W.live + n * warps) + 15) / 16 * 16;
    W.st2 = reinterpret_cast<uint32_t*>(q);
    W.l1 = W.st2 + nw * warps;
}

/// Runs the level of n_cells cells that W describes (W.o.lv[d]): a block a
/// cell for few cells, a warp a cell otherwise.
cudaError_t launch_interval_lists(const WideArgs& W, int d, uint32_t n_cells, uint32_t scratch_warps,
                                  cudaStream_t s);

/// The box form: scratch slots (blocks) that it wants for a tape of n
/// clauses, and its launch.
uint32_t interval_box_slots(uint32_t n, uint32_t n_boxes);
cudaError_t launch_interval_boxes(const WideArgs& W, uint32_t slots, cudaStream_t s);

}  // namespace lfb
