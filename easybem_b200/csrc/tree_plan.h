// Cluster tree of a mesh's far field (host side): the cells of the sorted
// order are the leaves, the ranges of the bisection the inner nodes.
//
// A pair of nodes is separated when its expansions converge fast enough
// (separation_ratio). The traversal of the tree against itself
// splits all cell pairs exactly once into separated node pairs (evaluated
// through multipole and local expansions) and close cell pairs (evaluated
// point by point).
#pragma once

#include <cmath>
#include <utility>
#include <vector>

#include "farfield.cuh"
#include "mesh_host.h"

namespace eb {

// What an expansion of order p leaves out of the sum between two balls falls as
// the (p + 1)-th power of the larger of r_a / (d - r_b) and r_b / (d - r_a)
// (the multipole's sources against the nearest target point, the targets
// against the nearest source), which is the larger ball's ratio. It is below 1
// for balls that do not touch.
__host__ __device__ inline double separation_ratio(double ra, double rb, double dist)
{
  return ra > rb ? ra / (dist - rb) : rb / (dist - ra);
}
// True when that ratio is below q < 1 (d2 = dist^2).
__host__ __device__ inline bool separated(double ra, double rb, double d2, double q)
{
  const double least = ra > rb ? rb + ra / q : ra + rb / q;
  return d2 > least * least;
}
// Degrees that such a pair needs, as f / 255 of those that ratio q needs.
__host__ __device__ inline unsigned degree_share(double ra, double rb, double d2, double q)
{
  const double f = ceil(255.0 * log(q) / log(separation_ratio(ra, rb, sqrt(d2))));
  return f < 1.0 ? 1u : f < 255.0 ? (unsigned)f : 255u;
}
// Closest pairs. Times of the SL+DL apply of a sphere of 81,920 triangles in
// us, mixed / FP64, and errors against FP64 point sums, random densities.
// "sphere": 14,208 triangles refined towards a
// pole by 0.9 per ring, the rows of its smallest quarter (DL; the symmetric
// kernels 1.6e-7 and 1.4e-12 there); "bodies": two spheres of radius 1 and 0.02
// at 0.2, the rows of the small one (3.3e-7 and 7.6e-14):
//   r_a + r_b < 0.5 d   2,128 / 8,720   sphere 2.1e-6, 1.0e-10   bodies 1.2e-6, 3.7e-11
//   0.33                2,264 / 9,380   sphere 5.9e-8, 1.8e-12   bodies 2.4e-7, 9.0e-14
//   0.36                2,075 / 8,575   sphere 8.9e-8, 1.8e-12   bodies 2.4e-7, 9.0e-14
//   0.40                1,810 / 7,485   sphere 4.8e-7, 1.9e-12
// A sum of the radii says little about unequal balls (a coarse cell beside a
// small body, which a cell's radius cannot follow), where its bound is 0.5.
constexpr double kTreeRatio = 0.36;
// Triangles that share a vertex must stay in close cells. With the outermost
// points of the 7-point rule at 0.696 of the way from the centroid to a vertex
// (farther out in the larger rules), a cell's vertices lie within 1.873 of its
// radius over the points, so separated nodes, at least (1 + 1 / ratio) / 2 of
// the sum of their radii apart, have no common one.
static_assert((1.0 + 1.0 / kTreeRatio) / 2.0 > 1.873, "separated nodes share no vertex");
// Least distance of a node's centre from its descendants' centres, over its radius.
constexpr double kTreeMinStep = 1e-3;
// The upward pass covers three levels of the tree per launch (up to eight
// descendants a node).
constexpr int kTreeLevelsPerPass = 3;
constexpr int kTreePasses = 6;  // enough for 2^18 cells
constexpr int kTreeMaxNodes = 1 << 24;
// The potential evaluation takes the tree where points x triangles are at least
// kTreePointPairs + kTreePointTriangles x triangles + kTreePointPoints x points:
// what the direct sums take for a pair goes into each term of the tree's cost,
// the launches, the multipoles of all cells and the groups' moves. Direct ->
// tree in ms, points uniform inside a sphere or torus (points near the surface
// and around it gain from slightly smaller numbers, in the mixed evaluation
// points far away from some 3,000):
//   triangles   mixed                                   FP64
//     5,120     2,000 0.39 -> 0.48, 4,000 0.63 -> 0.49  100,000 6.66 -> 8.38
//     8,192     1,000 0.28 -> 0.50, 2,000 0.49 -> 0.50  16,000 1.75 -> 1.87, 50,000 5.27 -> 4.42
//    20,480     1,000 0.56 -> 0.62, 2,000 0.89 -> 0.64  4,000 1.23 -> 1.52, 8,000 2.26 -> 1.94
//    81,920     500 0.71 -> 1.19, 1,000 1.18 -> 1.21    2,000 2.19 -> 3.13, 4,000 4.68 -> 3.30
//   327,680     500 1.04 -> 3.13, 2,000 2.95 -> 3.07    2,000 8.58 -> 9.22, 4,000 18.6 -> 9.5
constexpr double kTreePointPairs32 = 0.8e7, kTreePointTriangles32 = 900, kTreePointPoints32 = 0;
constexpr double kTreePointPairs64 = 4.3e7, kTreePointTriangles64 = 2000, kTreePointPoints64 = 5200;
// Ratio of a group of points and a node. Potentials in the volume are small
// against the contributions that cancel in them (rough double-layer densities
// above all), so FP64 needs a smaller one than the applies. 50,000 points
// around five meshes (sphere, torus, graded sphere and cube, two bodies of
// size 10 : 1), random densities, against FP64 point sums: mixed 2.6e-8 at 0.36
// (the direct sums 5.2e-8) inside the sphere of 20,480 triangles, 6.0e-6 (9.1e-6)
// at a probe of size 0.001 beside it where the potential nearly cancels, 2.0e-5
// there at 0.38; FP64 2e-15 of the largest potential from 0.21 to 0.32, 5e-14
// at the probe (rounding), times at 0.25, 0.28, 0.30: 8.0, 6.8, 6.1 ms.
constexpr double kTreePointRatio32 = 0.36;
constexpr double kTreePointRatio64 = 0.30;
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
// their cell pairs are close. Host applies in us, SL+DL and SL, of tori of r =
// 0.3 with all pairs close / the tree / the direct default (symmetric mixed,
// ordered FP64):
//   cells   mixed SL+DL    SL             FP64 SL+DL      SL
//      81   163/229/210    107/144/131    329/474/471     189/314/313
//     100   206/199/318    130/147/190    539/459/639     288/383/436
//     133   288/246/321    182/177/193    816/574/1,099   425/464/716
//     169   422/294/434    273/212/278    1,260/759/1,713 677/564/1,117
//     196   546/312/572    353/225/353    1,653/865/2,268 895/584/1,449
constexpr int kTreeMinCells = 100;
// Largest share of close pairs: half (host applies in us, direct default ->
// tree, mixed / FP64 SL+DL: 4,992 triangles graded towards a pole, share 0.36,
// 427 -> 356 and 1,468 -> 813; 20,000 needles, 0.43, 4,680 -> 2,870 and 21.8 ->
// 9.5 ms). Up to kTreeSmallCells a lower one: with all pairs close the single
// layer gains what four columns lose (100 cells: above, and 413/284, 1,019/749).
constexpr double kTreeMaxShare = 0.5, kTreeSmallShare = 0.318;
constexpr int kTreeSmallCells = 140;
// Meshes above that share: up to here the near tasks alone beat the direct
// kernels, whose items (a 128-triangle tile against 8 cells) leave SMs idle, in
// every variant (above; four columns at 169 cells 885 against 897 and 2,213
// against 2,445).
constexpr int kTreeAllCloseCells = 170;
// Four double layers run their close pairs in both orders one by one: with all
// pairs close up to here, then the direct kernels. Host right-hand sides in us,
// all close / direct, mixed and FP64: 10 cells 55/73, 93/136; 40 cells 125/118,
// 198/254; 66 cells 220/206, 423/485; 91 cells 351/346, 789/795; 100 cells
// 413/371, 1,019/929.
constexpr int kTreeForwardCells32 = 32, kTreeForwardCells64 = 90;
// Meshes whose partial slots would pass this in a variant keep the direct
// kernels there (ordinary surfaces take 80 bytes a triangle and column; the
// limit is the symmetric kernels').
constexpr size_t kTreeMaxSlotBytes = (size_t)1 << 35;
// Expansions moved into node tgt[k] from nodes src[ptr[k] .. ptr[k + 1]). The
// upper 8 bits of a source are the share f / 255 of the degrees that its pair
// needs: an expansion of order p is used up to (p + 1) f / 255 - 1 (rounded
// up). With f = ln(kTreeRatio) / ln(ratio) every pair has the bound of the
// closest ones (0.8 on average: half of the work). Sorted by f, largest first.
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
  int forward_slots = 0;  // of the lists of every ordered pair, which are made when a variant needs them
};

// False when more than half of all cell pairs are close in a mesh of more than
// kTreeAllCloseCells (the tree would not pay), or their slots pass
// kTreeMaxSlotBytes in every variant: the plan is then incomplete.
bool make_tree_plan(const HostMesh& h, TreePlan* plan);
// Tasks and slots of a plan's close pairs: every unordered pair once (both),
// or every ordered pair.
void make_near_lists(const TreePlan& plan, bool both, TreeNear* out);

}  // namespace eb
