// Host side of the aggregation-AMG structure: aggregates, coarse patterns, the maps of the numeric
// Galerkin product, and the tree numbering (pcg_tree.cuh).  No device code.
#pragma once

#include <array>
#include <functional>
#include <vector>

namespace bsg {

struct HostCsr {
    int n = 0;
    std::vector<int> ptr, col;
    std::vector<double> diag, val;
};

// Runs f(begin, end, thread) over [0, n) on up to eight host threads, each a contiguous range;
// on the caller alone below `grain` items.
void parallelRanges(int n, int grain, const std::function<void(int, int, int)>& f);
int hostThreads();

// Greedy pairwise matching on strongest negative couplings.
std::vector<int> pairwise(const HostCsr& a, int& n_coarse);

// Coarse row -> its rows, in increasing order.
void aggregateLists(const std::vector<int>& agg, int nc, std::vector<int>& ptr, std::vector<int>& rows);

// Galerkin coarse matrix of piecewise-constant aggregation; slot_target (optional): coarse entry of
// every fine entry, -1 inside an aggregate.
HostCsr coarsen(const HostCsr& a, const std::vector<int>& agg, int nc, std::vector<int>* slot_target);

// Fine entries that make up each coarse entry and each coarse diagonal, in fine-row order.
struct GalerkinMaps {
    std::vector<int> cslot_ptr, cslot_src, cintra_ptr, cintra_src;
};
GalerkinMaps galerkinMaps(const HostCsr& a, const std::vector<int>& target, const std::vector<int>& agg_ptr,
                          const std::vector<int>& agg_rows, int cnnz);

// Tree numbering of one level (see pcg_tree.cuh): `order` is the row of every rank of the next coarser
// level on entry and this level's on return.
struct TreeMaps {
    std::vector<int> row, rank, pos, at;  // position -> row, -> rank; rank -> position; row -> position
};
using Members = std::vector<std::array<int, 4>>;  // a coarse row's fine rows, -1 past the last
Members membersOf(const std::vector<int>& agg, int nc);
TreeMaps treeMaps(int n, const Members& members, std::vector<int>& order);
// Entries of the level's rows by position, padded to the widest row of every 32 positions.
double paddedEntries(const TreeMaps& t, const std::vector<int>& ptr);
// out[4 p ..]: the members of the row at position p; holes are left as they are.
void membersByPosition(const TreeMaps& t, const Members& members, int* out);

}  // namespace bsg
