// Tree far field (farfield_tree.cu): multipole and local expansions between
// separated clusters, point pairs between close cells.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <memory>
#include <mutex>

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

// Operator combinations are (nsl, nd) as elsewhere; this nsl with nd = 0 is the
// P1 single layer (one column of vertex values in ApplyArgs::u, three outputs).
constexpr int kTreeP1 = 12;

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

// Scratch of the potential evaluation.
struct TreePoints {
  DevBuf code, perm, multipole, local, ball, ptr, far, near, part, desc, apart;
};

// Block counts of each kernel over the meshes of a launch and, for more than
// one mesh, the first block of each (device).
struct TreeGrid {
  int nmesh = 1;
  const int *cells = nullptr, *m2l = nullptr, *tasks = nullptr, *up[kTreePasses] = {};
  int ncells = 0, nm2l = 0, ntasks = 0, nup[kTreePasses] = {};
  bool expansions = true;
  int rule = 0;  // points of the triangle rule
};

// A mesh's tree: the plan of a new mesh, the rest with the first apply.
struct TreeMesh {
  bool usable = false;
  TreePlan plan;
  // The lists are made once, by the first descriptor that needs them: of a call
  // on the mesh, or of a batch or solver, which share it between threads.
  std::mutex lists_lock;
  bool lists_ready = false, fwd_ready = false;
  DevBuf lists;  // one allocation
  TreeDesc base; // static pointers
  // close pairs in forward order
  TreeNear fwd;
  DevBuf fwd_lists;
  const int2* children = nullptr;  // of the inner nodes (device)
  const char* formed = nullptr;    // TreePlan::formed (device)
  TreePoints points;
  TreeSide side;
  std::map<int, std::unique_ptr<TreeScratch>> scratch;
};

// The tree of mesh m when its size allows one (host work, done while the GPU
// computes the near field of a new mesh).
void tree_prepare(Mesh* m);
// True when mesh m applies this far-field variant through the tree (the same in
// both precisions but for several double layers).
bool tree_eligible(const Mesh* m, int nsl, int nd, bool fp32 = false);
// The far field of mesh m: expansions and close pairs into the partial slots
// (A.partial and A.slot_off are set for the finalize).
int tree_far_apply(Mesh* m, bool fp32, int nsl, int nd, ApplyArgs* A, cudaStream_t st);
// Partial slots (summed over the rows, per output).
long long tree_far_slots(const Mesh* m, int nsl, int nd);
// Descriptor of mesh m for one variant over the given scratch (tree_scratch_bytes);
// uploads the mesh's lists the first time.
int tree_desc(Mesh* m, bool fp32, int nsl, int nd, void* rec, void* multipole, void* local, double* partial,
              TreeDesc* out);
// Where the finalize reads the sums of descriptor d (of m and this variant).
void tree_finalize_args(const Mesh* m, int nsl, int nd, const TreeDesc& d, ApplyArgs* A);
// Bytes of one of the two expansion buffers, and of the partial slots.
size_t tree_expansion_bytes(const Mesh* m, int order, int cols);
size_t tree_partial_bytes(const Mesh* m, int nsl, int nd);
// The kernels of the meshes of g: descriptors d, arguments one (a single mesh)
// or many (device).
int tree_launch(bool fp32, int nsl, int nd, const TreeDesc* d, const TreeGrid& g, const ApplyArgs& one,
                const ApplyArgs* many, int device, const TreeSide& side, cudaStream_t st);
// Potentials V t - W u at npts points (pts host, d_pts the same on the device)
// through the tree. Waits for the stream.
bool tree_points_eligible(const Mesh* m, bool fp32, int npts);
int tree_evaluate(Mesh* m, bool fp32, int npts, const double* pts, const double* d_pts, const double* d_t,
                  const double* d_u, double* d_out, cudaStream_t st);
// Makes the constant tables that a launch needs (before a stream capture).
int tree_tables(bool fp32, int device);
// Device bytes of the mesh's tree and its single-mesh scratch; gives the
// scratch back (no work on the mesh in flight).
size_t tree_bytes(const Mesh* m);
void tree_release_scratch(Mesh* m);

}  // namespace eb
