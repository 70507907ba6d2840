// 3D transforms between the leaves' Hermite / Taylor blocks and the cut
// level's plane-wave expansions, one dimension at a time over the subtree of
// each cut-level box (fgt_sep3d.cu).
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "fgt_device.hpp"
#include "fgt_plan.hpp"

namespace fgtb {

struct KP;

// Fills d and x of every item from the tree (root_box[item.root]) and sorts
// the items by (p, d, root, x, y, z).
void sep_sort(const Tree& t, const std::vector<int>& root_box, std::vector<SepItem>& items);

// Columns (equal root, depth, x, y), slabs (equal root, depth, x) and boxes
// of sorted items; offsets and sizes per density.  Every root gets a box,
// with no slabs where it has no leaf; slot: the root's expansion slot.
void sep_lists(const std::vector<SepItem>& items, const std::vector<int>& slot, int npw, SepLists& S);

// Phase rows of depths 0..dmax: row 2^d - 1 + i holds exp(i t_m sh) of the
// npw nodes, sh the offset of box i of 2^d from its root's centre over
// sqrt(delta) (bs0: the root's size).
void sep_phases(const HostPlan& H, int dmax, double bs0, std::vector<double>& ph);

// The leaves' own expansions (pool src) added to the expansions k.mp of the
// groups' slots (after sep_up).
cudaError_t sep_add(const KP& k, const double2* src, const double2* ph, const MergeGroup* groups, int ngroups,
                    const SepShift* shifts, cudaStream_t st);

// Upward: Hermite blocks in hbuf -> the expansions k.mp of the boxes' slots.
cudaError_t sep_up(const KP& k, const SepDev& S, const double* hbuf, cudaStream_t st, long long& launches);

}  // namespace fgtb
