// The solve plan: supernodes chained into fronts, and the sweeps' task lists (fronts.cpp).
#pragma once

#include <stdint.h>

#include <string>
#include <vector>

#include "fcw_internal.h"

namespace fcw {

// Rows per task (M of the sweep kernels) and the layout of a task's panel: k-major, a depth row
// of panel_ld entries (FP64 rows are padded so that tensor-core fragment reads hit distinct banks).
constexpr int kWidestFront = 3072;  // columns fronts.cu's row merge holds in shared memory
constexpr int kDepthPad = 4;  // a panel's depth is padded with zero rows to a multiple of this
inline int64_t panel_ld(int rows, bool fp64) { return (rows + 7) / 8 * 8 + (fp64 ? 4 : 0); }
inline int64_t padded_depth(int64_t d) { return (d + kDepthPad - 1) / kDepthPad * kDepthPad; }

// Forward: stacked rows [r0, r0 + h) of [inv(L_ss); Q_s] times W. Backward: columns
// [r0, r0 + h) of X_s, depth = the front's rows from r0 down.
struct SweepTask {
    int32_t front, r0, h, depth;   // depth: columns (forward) or front rows (backward) it multiplies
    int32_t c0, ns;                // the front's first column and width
    int32_t wrow;                  // forward: the front's first row of the assembled right-hand sides
    int32_t pad;
    int64_t off64, off32;          // its panel in the FP64 / FP32 arrays
    int64_t row0;                  // front-row index of the front's first row
    int64_t urow;                  // forward: update row of the front's first structure row
};

// Children's update rows that land on a front row: up to three inline, more in `more`.
struct GatherRec {
    int32_t src[3];  // update rows, -1: none
    int32_t more;    // index into Fronts::more (count, then (update row, front) pairs), -1: none
};

struct Fronts {
    int32_t nf = 0, nlevels = 0;
    std::vector<int32_t> c0;        // nf + 1
    std::vector<int32_t> m;         // rows: own columns, then structure
    std::vector<int32_t> parent;
    std::vector<int32_t> sn0;       // nf + 1: first supernode of each front
    std::vector<int32_t> col_front; // n
    std::vector<int64_t> row0;      // nf + 1: offsets into rows
    std::vector<int32_t> rows;      // elimination-order row of each front row
    std::vector<int64_t> uoff;      // nf + 1: first update row
    std::vector<int32_t> level_ptr, level_nodes;
    std::vector<int32_t> pos;       // aligned with Symbolic::rows: each panel row's row in its front
    std::vector<GatherRec> rec;     // per front row
    std::vector<int32_t> rec_child; // 3 per front row: the children's fronts
    std::vector<int32_t> more;
    // task lists: per level, tasks [ptr[l], ptr[l + 1]) of rows[l]-row tasks
    std::vector<SweepTask> fwd, bwd;
    std::vector<int32_t> fwd_ptr, bwd_ptr, fwd_rows, bwd_rows;
    // levels from first_wide on assemble their fronts' right-hand sides into rows of their own
    // (asm_rows, per level [asm_ptr[l], asm_ptr[l + 1])) before the products
    int32_t first_wide = 0;
    std::vector<int32_t> asm_ptr;
    std::vector<int32_t> asm_rows;  // 4 per row: front row index, elimination row, front, -
    int64_t n_urows = 0, n_wrows = 0;
    int64_t fwd64 = 0, bwd64 = 0, fwd32 = 0, bwd32 = 0;  // entries of the panel arrays
    int64_t leaf_fwd64 = 0, leaf_bwd64 = 0, leaf_fwd32 = 0, leaf_bwd32 = 0;  // most of one task of level 0
};

int build_fronts(const Symbolic& S, Fronts& f, std::string& err);

// The leaf level with resident panels (k_leaf, solve.cu): a CTA's warps, a warp's ring of right-hand
// sides (chunks, depth rows per chunk), the columns of a warp's groups, and the shared memory of a CTA,
// of which two fit an SM.
constexpr int kLeafWarps = 8, kLeafStages = 3, kLeafChunk = 16;
constexpr size_t kLeafSmem = 113 * 1024 - 1024;
constexpr int leaf_columns(bool fp64, bool back) { return !fp64 ? 32 : (back ? 16 : 8); }
// panel: entries of the largest task's panel; index_rows: rows whose indices a backward CTA holds
inline size_t leaf_smem(int64_t panel, int columns, size_t entry, int32_t index_rows) {
    return ((size_t)panel + (size_t)kLeafWarps * kLeafStages * kLeafChunk * columns) * entry +
           (size_t)index_rows * sizeof(int32_t);
}
// Least tasks times column rounds (a warp's groups) for which k_leaf is the faster: with fewer, its
// CTAs, each with all of a panel to fetch first, do not fill the chip. 147k vertices FP64, backward:
// 2066 rounds (128 columns) 0.324 against 0.334 ms, 16528 (1024) 1.36 against 1.48; 37k vertices: 1038
// rounds equal, 2076 0.241 against 0.245; 9k vertices, forward: 2096 0.160 against 0.163, 131 0.069
// against 0.064. With reach flags rounds differ in length, so more are needed: 147k vertices 16528
// 1.04 against 1.11 ms, 8264 0.612 against 0.633, 4132 0.403 against 0.400; 37k vertices 4152 0.306
// against 0.297.
constexpr int64_t kLeafRounds = 1184, kLeafRoundsReach = 5920;
inline bool leaves_resident(int64_t tasks, int rounds, size_t smem, bool reach) {
    return smem <= kLeafSmem && tasks * rounds >= (reach ? kLeafRoundsReach : kLeafRounds);
}

}  // namespace fcw
