// Tree far field (farfield_tree.cu): multipole and local expansions between
// separated clusters, point pairs between close cells.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <memory>

#include "engine.h"
#include "tree_plan.h"

namespace eb {

// Expansion orders. The far sum's truncation stays below the rounding of the
// rest: measured against 64-bit sums (random and smooth densities).
#ifndef EB_TREE_ORDER32
#define EB_TREE_ORDER32 14
#endif
#ifndef EB_TREE_ORDER64
#define EB_TREE_ORDER64 28
#endif
constexpr int kTreeOrder32 = EB_TREE_ORDER32;  // mixed applies
constexpr int kTreeOrder64 = EB_TREE_ORDER64;  // FP64 applies
static_assert(kTreeOrder64 <= 30 && kTreeOrder32 <= 30, "one warp lane per degree, 10-bit coefficient positions");
// complex coefficients (m >= 0) of an expansion
__host__ __device__ constexpr int tree_pairs(int order) { return (order + 1) * (order + 2) / 2; }

struct TreeMovesDev {
  const int* tgt;
  const int* ptr;
  const int* src;
};

// Per-mesh view of the kernels (device pointers); a batch passes an array.
struct TreeDesc {
  FarMeshDesc far;           // records and tables of the close pairs
  const dq* pos;             // [ne * Q] (-2 y, |y|^2) relative to the cell centre (FP64)
  const dq* ball;            // [nnodes] centre, radius
  TreeMovesDev up[kTreePasses], m2l, down;
  const char* has_local;     // [nnodes]
  const int4* tasks;
  const int2* entries;
  const int* slot_off;       // [ncells + 1]
  double2* multipole;        // [columns][nnodes][pairs]
  double2* local;
  double* partial;           // [columns][slots][kCell]
  int nnodes, ncells;
  int ntasks, nm2l, nup[kTreePasses];
  int first_col;             // of partial: 1 for a double layer alone (column 0: its zero single layer)
};

// Scratch and descriptor of one variant, made on its first apply and kept.
struct TreeScratch {
  DevBuf multipole, local, partial, desc;
  TreeDesc host;
};

// The close pairs' stream: they run beside the expansions (the FP32 pipe and
// MUFU beside FP64 mma in a mixed apply), forked from and joined to the
// apply's stream, at the least priority so that the shorter kernels of the
// expansions take freed SMs first.
struct TreeSide {
  cudaStream_t st = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  TreeSide() = default;
  TreeSide(const TreeSide&) = delete;
  TreeSide& operator=(const TreeSide&) = delete;
  ~TreeSide();
  int create();  // no-op when made
};

// A mesh's tree, made on the first apply that takes it.
struct TreeMesh {
  bool usable = false;
  TreePlan plan;
  DevBuf lists;  // one allocation
  TreeDesc base; // static pointers
  const int4* fwd_tasks;      // TreePlan::fwd
  const int2* fwd_entries;
  const int* fwd_slot_off;
  TreeSide side;
  std::map<int, std::unique_ptr<TreeScratch>> scratch;
};

// True when mesh m applies this far-field variant through the tree; makes the
// tree (host work and one upload) the first time the rules allow it.
bool tree_eligible(Mesh* m, bool fp32, int nsl, int nd);
// The far field of mesh m: expansions and close pairs into the partial slots
// (A.partial and A.slot_off are set for the finalize).
int tree_far_apply(Mesh* m, bool fp32, int nsl, int nd, ApplyArgs* A, cudaStream_t st);
// Partial slots (summed over the rows, per output).
long long tree_far_slots(const Mesh* m, int nd);

}  // namespace eb
