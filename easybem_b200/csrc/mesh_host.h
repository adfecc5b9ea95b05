// Host-side preparation of one surface mesh for the device apply.
//
// Replaces the reference's host topology (src/meshTopology.cpp:22-261, an
// O(ne * nedges) edge search) and its per-matvec host pair enumeration
// (src/BEM3dLaplaceGPU.cu:1224-1260) with one O(ne log ne) pass at mesh
// creation: triangles are reordered by recursive bisection of their centroids,
// grouped in cells of kCell consecutive triangles (the far-field source
// granularity), and the near pairs (triangles sharing at least one vertex)
// are listed once in CSR form for the Sauter-Schwab correction.
#pragma once

#include <cstdint>
#include <vector>

#include "quadrature.h"

namespace eb {

constexpr int kCell = 32;  // source triangles per cell (shared origin for FP32 coordinates)

struct HostMesh {
  int nv = 0, ne = 0, order = 4, Q = 0;
  Quadrature quad;
  std::vector<double> nodes;  // [nv][3]
  std::vector<int> elems;     // [ne][3], 0-based

  // Sorted order: perm[s] = original index of sorted triangle s; iperm inverse.
  // Recursive bisection across the longest side of the centroids' box, at
  // multiples of kCell (split_cells), so cells and the ranges of the bisection
  // are compact patches. Cells of a Morton curve jump across its faces: on
  // the perturbed icosphere L5 47 cells lay within twice the sum of the radii
  // of a cell, against 16 here.
  std::vector<int> perm, iperm;
  int ncells = 0;
  std::vector<double> cell_ball;  // [ncells][4]: centre and radius of a ball around the cell's vertices
  std::vector<double> cell_rho;   // [ncells]: the ball's radius over the quadrature points only (with the static tables)

  // Target items: a triangle's Q points split into chunks of at most K points.
  int K = 0;        // target points per item (compile-time kernel width)
  int nchunk = 0;   // items per triangle
  int nitems = 0;   // ne * nchunk

  // Near pairs (including coincident), CSR by original test triangle.
  std::vector<int> sl_rowptr, sl_col;  // col = original trial triangle
  std::vector<int> pair_i;             // original test triangle of each pair
  std::vector<int8_t> pair_kind;
  // DL near CSR over vertex columns; entry e = 3*pair + k feeds slot dl_slot_of[e].
  std::vector<int> dl_rowptr, dl_col;
  std::vector<int> dl_contrib_ptr, dl_contrib;  // slot -> entries, ascending

  long long far_quad_pairs = 0;  // regular quadrature-point pairs per apply
  bool topology_on_device = false;  // near-pair lists built by device_topology
};

// Cells of the first half of a range of ncells cells in the bisection.
int split_cells(int ncells);
// Centre and radius of a small ball around the vertices of sorted triangles
// [s0, s1): the box centre, moved towards the farthest vertex four times.
void vertex_ball(const HostMesh& m, int s0, int s1, double* ball);

// Validates and prepares (sorted order, cells, target items and, when
// topology is set, the near-pair CSR through host_topology); returns EB_OK or
// an error status with a message.
int prepare_host_mesh(int nv, const double* nodes, int ne, const int* elems1, int order, HostMesh* m,
                      bool topology = true);

// The near-pair CSR (sl_*, pair_*, dl_*) and far_quad_pairs of a prepared
// mesh, on the host. device_topology (topology.cu) builds the same arrays on
// the GPU for large meshes.
void host_topology(HostMesh* m);

// The same arrays built on the current GPU (topology.cu); *done is false when
// a row has too many candidates and the caller must use host_topology.
int device_topology(HostMesh* m, bool* done);
// Meshes with at least this many triangles use device_topology.
int device_topology_min();

// Target items per triangle and points per item for Q quadrature points.
void target_split(int Q, int* K, int* nchunk);

}  // namespace eb
