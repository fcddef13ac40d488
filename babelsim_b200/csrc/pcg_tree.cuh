// Persistent PCG with the aggregation-AMG V-cycle (one damped-Jacobi sweep down and up) whose
// coarse levels stay on chip.
//
// A solve of a small or middling system is bound by latency: a V-cycle is a chain of short
// phases, and each used to cost the barrier plus one L2 round trip (about 0.35 us) for every
// dependent load, slice offset -> column -> value, aggregate list -> member -> residual.
// Here each CTA copies the matrix rows it owns into shared memory once per solve, so a phase is
// a barrier and one round of gathers.
//
// Tree numbering.  From level `top` down to the coarsest, a level's rows stand in the order of
// their aggregates: the members of the next level's row of rank c take positions 4c..4c+3
// (aggregates have at most four members; missing ones leave holes, which hold zeros).  A warp
// then owns whole aggregates: the residual of a level and its restriction are one phase (the
// four members are added by shuffles), and the prolongation is a read of the coarse value of
// rank position/4, with no push and no list.  Levels finer than `top`, whose matrices do not
// fit, keep their own numbering and stream SELL-32 slices from memory (pcg_sell.cuh).
//
// Phases per CG iteration with L levels and top = 0: 2 L; with top > 0 one or two more per
// streamed level.
//
// FP64 only.  An FP32 V-cycle (precision 1 and 2) stays on the streaming kernel: there rounding decides after
// which iteration a solve is accepted, and rows split over lanes, other sums and folded levels round otherwise
// (CG counts of mixed 110k-cell outer iterations moved by one or two in 7 of 16, p by up to 1.5e-9 relative; in FP64,
// 7e-13).  Mixed outer iterations, on chip / streamed: 8k cells 2.8 / 4.6 ms, 33k 4.0 / 6.3, 110k 6.9 / 9.5, 373k
// 17.8 / 21.4.
#pragma once

#include "group.cuh"
#include "pcg_persistent.cuh"
#include "pcg_sell.cuh"
#include "sell.cuh"

#include <vector>

namespace bsg {

constexpr int kMaxTreeLevels = 16;

// One level in tree numbering.  `row`..`memb` are by position, b and w too; e, the level's
// result, is by rank (the positions in order, holes left out).
struct TreeLevel {
    int n = 0;                    // rows
    int npos = 0;                 // positions: 4 x the next level's rows (n on the coarsest level)
    const int* row = nullptr;     // position -> row, -1 in a hole
    const int* rank = nullptr;    // position -> rank, -1 in a hole
    const int* pos = nullptr;     // rank -> position
    const int4* memb = nullptr;   // position -> rows of the finer level it is made of, -1 past the last
    const int* ptr = nullptr;     // CSR of the level, by row
    const int* pcol = nullptr;    // position of each entry's column
    const double* val = nullptr;
    const double* diag = nullptr;
};

struct TreeView {
    int levels = 0;                    // L
    int first = 0;                     // the finest level that has a tree numbering
    double gamma = 1.0;
    double omega = 1.0;
    const TreeLevel* lv = nullptr;     // device array of L (entries below `first` unused)
    const VLevel<double>* nat = nullptr;   // device array of L: the levels in their own numbering
    double* const* vec = nullptr;          // device array of 3 L: b, w, e of every tree level
    const double* dense_inv = nullptr;     // coarsest inverse, n x n row-major (by row)
    const double* folded = nullptr;        // level L - 2: its whole V-cycle as a matrix, rank x position
};

struct TreePcgArgs {
    SellMat<double> A;    // level 0 in its own numbering (top > 0)
    TreeView T;
    int top = 0;      // finest level in tree numbering in this launch
    int n = 0;        // rows of level 0
    const double* b;
    double* x;
    // At least max(n, positions of level 0) entries each.  With level 0 in tree numbering what
    // neighbours gather together lies together: {z, p} of an iteration, and {w, omega / diagonal
    // * q}, each in two buffers that alternate, so a sweep gathers one 16-byte pair per entry
    // instead of two or three values, which counts where every gather goes to L2.  A streamed
    // level 0 keeps its vectors apart (in the same memory): there the pairs' half-written sectors
    // cost more (1M cells: 70 against 58 us per product).
    double *r, *q, *xt;
    double2 *zp0, *zp1, *wq0, *wq1;
    double* partial;
    PcgState* st;
    PhaseLog log;
    int smem = 0;      // bytes of dynamic shared memory for matrix rows
};

// What a launch needs to know of a hierarchy to place it on `ctas` CTAs.
struct TreePlan {
    std::vector<long long> slices;   // per level: slices of 32 positions
    std::vector<double> entries;     // per level: off-diagonal entries, padded to each slice's widest row
    std::vector<int> rows, positions;
    int first = 0;                   // finest level with a tree numbering
    long long nnz = 0;               // off-diagonal entries of level 0
    bool folded = false;             // the V-cycle from level L - 2 down exists as one dense matrix
    // Bytes of shared memory per CTA for the rows of levels [from, levels - 1).
    double bytes(int from, int levels, int ctas) const;
    bool fits(int from, int ctas) const;
    struct Place {
        int top, levels, smem;
    };
    Place place(int ctas) const;
};

// One system: on one thread-block cluster when it is small, else on the whole grid.  Returns its placement.
TreePlan::Place launchTreePcg(Context& ctx, const TreePlan& plan, TreePcgArgs args);

// Systems of a batch, side by side on CTA ranges of one cooperative launch (several launches when
// they outnumber its argument block), each with barriers of its own.
struct TreeBatch {
    std::vector<TreePcgArgs> args;
    std::vector<const TreePlan*> plans;
    std::vector<int> slices;         // level-0 slices, for the CTA shares
    DeviceArray<SegmentBarrier> d_bars;
    int bars_used = 0;               // barriers of the last launch, for its error report
};
void launchTreePcgBatch(Context& ctx, TreeBatch& batch);

}  // namespace bsg
