// Cluster tree of a mesh's far field (host side): the cells of the sorted
// order are the leaves, the ranges of the bisection the inner nodes.
//
// A pair of nodes is separated when the sum of its radii is below kTreeTheta
// times the distance of its centres. The traversal of the tree against itself
// splits all cell pairs exactly once into separated node pairs (evaluated
// through multipole and local expansions) and close cell pairs (evaluated
// point by point).
#pragma once

#include <utility>
#include <vector>

#include "farfield.cuh"
#include "mesh_host.h"

namespace eb {

// Separation: measured on the perturbed icosphere L5 and a torus, random
// densities, far sum against the whole sum. At 0.5, order 14: 1.9e-10 (SL) and
// 6.8e-9 (DL); order 24: 3.4e-15 and 3.5e-14. A wider ratio trades close cell
// pairs (16 a cell at 0.5, 11 at 0.6) for higher orders (18 at 0.6 for the
// accuracy of 14 at 0.5).
constexpr double kTreeTheta = 0.5;
// Least distance of a node's centre from its descendants' centres, over its radius.
constexpr double kTreeMinStep = 1e-3;
// The upward pass covers three levels of the tree per launch (up to eight
// descendants a node).
constexpr int kTreeLevelsPerPass = 3;
constexpr int kTreePasses = 6;  // enough for 2^18 cells
constexpr int kTreeMaxNodes = 1 << 24;
// Points x triangles from which the potential evaluation takes the tree, and
// least triangles in FP64 (whose point sums are only 1.5 to 3 times dearer
// than in the mixed evaluation, while the moves cost eight times the work).
// Measured, direct -> tree (ms): mixed 5,940 triangles 2,000 points 0.41 -> 0.45,
// 4,000 0.76 -> 0.47; FP64 17,860 x 4,000 1.09 -> 1.11, 8,000 1.97 -> 1.47;
// 3,280 x 100,000 4.34 -> 4.53.
constexpr double kTreePointPairs32 = 2e7, kTreePointPairs64 = 1e8;
constexpr int kTreePointTriangles64 = 5000;
// Separation of a group of points from a node. Potentials in the volume are
// small against the contributions that cancel in them (rough double-layer
// densities above all), so the same orders need smaller ratios than the
// applies. Error against 64-bit sums, 50,000 points inside an icosphere L5
// (the direct sums: 8.3e-8 mixed, 7.1e-16 FP64): at 0.5 1.8e-7 and 1.5e-12, at
// 0.45 2.8e-8 and 5.2e-14, at 0.4 1.5e-15, at 0.35 5.1e-16 in FP64.
constexpr double kTreePointTheta32 = 0.45;
constexpr double kTreePointTheta64 = 0.35;
// Close cell pairs per near task (one warp's work; the diagonal counts): at
// most kTreeNearChunk, fewer while that leaves less than kTreeNearTasks tasks
// (four warps on each of the 592 SM quarters).
constexpr int kTreeNearChunk = 4;
constexpr int kTreeNearTasks = 4 * 592;
// Where single pairs leave less, a pair is cut into up to kTreeNearParts tasks
// of consecutive sources: 820 pairs (1,280 triangles) leave 364 of the 592
// quarters one warp with nothing to hide its latency and give 228 two. FP64,
// one operator at 1,280 triangles: 94 -> 85 us (the near kernel 65 before);
// SL+DL at 512: 96 -> 37, where the ordered-pair kernel takes 69. Up to 2 parts
// are slower below 800 triangles (54 at 512); 8 gain at 128 (25 against 34) but
// give the finalize more slots to add (512: P1 layer 93 against 75; 800 mixed
// 40 against 37).
constexpr int kTreeNearParts = 4;
// A pair's source cell in a list entry, with the part of it: x = cell, the
// part and log2 of the number of parts in the upper bits.
constexpr int kTreePartShift = 25, kTreePartsShift = 28;
// Smaller meshes (cells) have no separated clusters worth an expansion: all
// their cell pairs are close. Up to here the near tasks alone also beat the
// symmetric kernel, whose items (a 128-triangle tile against 8 cells) leave
// SMs idle.
constexpr int kTreeMinCells = 100;
constexpr int kTreeAllCloseCells = 140;
// Expansions moved into node tgt[k] from nodes src[ptr[k] .. ptr[k + 1]). The
// upper 8 bits of a source are the share f / 255 of the degrees that its pair
// needs: an expansion of order p is used up to (p + 1) f / 255 - 1 (rounded
// up). With radii r and distance d the truncation falls as (r / d)^(order + 1),
// so f = ln(kTreeTheta) / ln(r / d) gives every pair the bound of the closest
// ones (0.8 on average: half of the work). Sorted by f, largest first.
struct TreeMoves {
  std::vector<int> tgt, ptr = {0}, src;
};

// Close cell pairs. A task is (cell, first entry, last entry, slot of its
// forward sums), an entry (other cell, slot of the transposed sums or -1); the
// slots of cell c are slot_off[c] .. slot_off[c + 1]), the last one for the
// far sum (if there is one).
struct TreeNear {
  std::vector<int4> tasks;
  std::vector<int2> entries;
  std::vector<int> slot_off;
};

struct TreePlan {
  int ncells = 0, nnodes = 0;  // nodes 0 .. ncells - 1 are the cells
  bool all_close = false;      // no expansions: every cell pair in near
  std::vector<dq> ball;        // centre; radius over the quadrature points
  std::vector<int2> child;     // of node ncells + k
  TreeMoves up[kTreePasses];   // multipoles of descendants into inner nodes
  TreeMoves m2l;               // multipoles of separated nodes into locals
  TreeMoves down;              // locals of the ancestors into every cell
  std::vector<char> has_local; // per node: it is a target of m2l
  std::vector<char> formed;    // per node: the upward passes form its multipole
  std::vector<std::pair<int, int>> near;  // close cells, the earlier one first
  TreeNear sym;  // every unordered pair of cells once
};

// False when more than a third of all cell pairs are close in a mesh of more
// than kTreeAllCloseCells (the tree would not pay): the plan is then incomplete.
bool make_tree_plan(const HostMesh& h, TreePlan* plan);
// Tasks and slots of a plan's close pairs: every unordered pair once (both),
// or every ordered pair.
void make_near_lists(const TreePlan& plan, bool both, TreeNear* out);

}  // namespace eb
