// The treecode's device tree, shared by its kernels (csrc/fs_tree.cu,
// csrc/fs_treecells.cu).
#pragma once

#include "fs_device.cuh"

namespace fsb {

constexpr int kMaxDegree = 16;
constexpr int kMaxDepth = 60;
constexpr int kFarCap = 256;   // far-list entries per leaf
constexpr int kNearCap = 64;   // near-list entries per leaf

struct TNode {
    double x0, x1, xc;
    int m0, m1;       // inclusive member range in sorted order
    int child0, child1;
    int parent, level;
};

// One evaluation's tree on the device.  meta: [0] nodes, [1] leaves, [2] error
// code, [3] depth.
struct TreeView {
    const TNode* nodes;
    const int *leaves, *meta, *leaf_of;
    const int *far_list, *far_n, *near_list, *near_n;
    const double *mom, *consts;   // cluster moments; cos(k pi/P) and weights
    const double *sx, *lam;       // sorted positions (fmod L) and charges
    const int* sidx;              // sorted slot -> point
    int n, P, cap_leaves;
};

// A near leaf's slots (csrc/fs_treecells.cu).
struct NearSlots {
    int slot, n, c0;  // first slot, slots, first cell
};

// Near and far sums of every point through cells (csrc/fs_treecells.cu).
class TreeCells {
   public:
    // False where the cells do not cover (L, eps).
    bool init(double L, double eps);
    bool ready() const { return plan_.M > 0; }
    // norm * (near + far) at every point through the stage epilogue.
    void eval(const TreeView& T, int max_source, double norm, const Stage& S, cudaStream_t st);

   private:
    CellPlan plan_;
    DevBuf<double> tab_, mom_, loc_, part_, e_;
    DevBuf<NearSlots> near_;
    DevBuf<int2> leaf_steps_, extra_;
    DevBuf<int> leaf_chunk_, arrived_, leaf_c0_, leaf_slot_, slot_leaf_, chunk_leaf_, chunk_c_, count_;
};

}  // namespace fsb
