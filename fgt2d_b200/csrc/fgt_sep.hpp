// Transforms between the leaves' Hermite / Taylor blocks and the cut level's
// plane-wave expansions, one dimension at a time over the subtree of each
// cut-level box (fgt_sep.cu; the 3D kernels: fgt_sep3d.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "fgt_device.hpp"
#include "fgt_plan.hpp"

namespace fgtb {

struct KP;

// Phase rows: a row for every place that a box can have in its root along one
// dimension (SepItem::x), by depth.  Up to depth SEP_DENSE every place of the
// grid has one (row 2^d - 1 + i); in deeper trees, which only callers with a
// tree of their own have, those that occur.
constexpr int SEP_DENSE = 8;
struct SepRows {
  std::vector<int> base;   // first row of every depth
  std::vector<double> at;  // offset of every row from the root's centre over the root's size
};

// The boxes as items, sorted by (rank[depth], root, x, y, z),
// in 2D (rank[depth], root, y, x); roots are the
// boxes of level lroot, numbered from its first.  rank: by depth, equal orders
// next to one another.
void sep_order(const Tree& t, int lroot, const std::vector<int>& boxes, const std::vector<int>& rank,
               uvector<SepItem>& items, SepRows& rows);
// rank of sep_order from the orders by depth (increasing order, then depth)
std::vector<int> sep_rank(const std::vector<int>& order_of_depth);

// Columns (equal root, depth, x, y; 2D: y), slabs (3D: equal root, depth, x)
// and boxes of sorted items with their blocks (leaf.off, leaf.n, taken over;
// the rows are filled here); offsets and sizes per density.  slot: the
// expansion slots by root; without any item root `also` (-1: none) gets an
// empty box.
void sep_lists(int dim, const uvector<SepItem>& items, const SepRows& rows, std::vector<SepLeaf>& leaf,
               const std::vector<int>& order_of_depth, const int* slot, int also, int npw, SepLists& S);

// The phase rows: exp(i t_m sh) of the npw nodes, sh the row's offset over
// sqrt(delta) (bs0: the root's size).
void sep_phases(const HostPlan& H, const SepRows& rows, double bs0, std::vector<double>& ph);

// Flops per density of the way up or down through the lists (a multiply-add:
// 2): products with the node tables and turns to the nodes' phases.
double sep_flops(int dim, bool up, const SepLists& S, int npw);

// 3D (fgt_sep3d.cu)
cudaError_t sep_up_3d(const KP& k, const SepDev& S, const double* hbuf, cudaStream_t st, long long& launches);
cudaError_t sep_down_3d(const KP& k, const SepDev& S, double* lo, cudaStream_t st, long long& launches);

// Upward: Hermite blocks in hbuf -> the expansions k.mp of the boxes' slots.
cudaError_t sep_up(const KP& k, const SepDev& S, const double* hbuf, cudaStream_t st, long long& launches);

// Downward: the expansions k.loc of the boxes' slots -> the columns (t1) of
// every order and the Taylor blocks (lo) of the groups with blocks; 2D blocks
// of at most f32 rows as FP32 pairs.
cudaError_t sep_down(const KP& k, const SepDev& S, double* lo, int f32, cudaStream_t st, long long& launches);

// Evaluation from the columns: the most points of a task, and the tasks of
// one order (Pn: order + 1).
int sep_col_points(int pgh);
cudaError_t sep_eval_cols(const KP& k, const SepDev& S, const ColTask* tasks, int ntask, int Pn, int pgh,
                          cudaStream_t st);

}  // namespace fgtb
