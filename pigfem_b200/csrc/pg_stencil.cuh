// pg_stencil.cuh -- neighbourhoods of the structured grids.
//
// The background meshes are the reference's structured grids (Mesh::generate_mesh,
// src/Mesh.cpp:386-604): quads, quads split into two tri3 with the union-jack alternation, hexes
// split into six tet4.  Away from the domain boundary and from cut elements every DOF node of such
// a grid has the same neighbourhood up to its class (the parity of i + j for tri3, a single class
// for quad4 and tet4).  The tables below give, for each class, the neighbour offsets in row order and, for
// each adjacent element, its cell offset, its index within the cell, the row node's local index
// and the neighbour slot of each of its nodes.  They restate the reference's cell-splitting
// tables in row-owner form; the set-up checks every node it sends here against them and sends any
// node that does not match to the general rows.
#pragma once

#include "pg_kernels.cuh"

namespace pgd {

struct Tri3Stencil0 {
  static constexpr int NN = 9, NADJ = 8;
  // neighbour offsets (di, dj, dk) in row (node id) order
  __host__ __device__ static constexpr int off(int s, int d) {
    constexpr int t[NN][3] = {{-1, -1, 0}, {0, -1, 0}, {1, -1, 0}, {-1, 0, 0}, {0, 0, 0}, {1, 0, 0}, {-1, 1, 0}, {0, 1, 0}, {1, 1, 0}};
    return t[s][d];
  }
  // adjacent elements: cell offset (di, dj, dk), element within the cell, local index of the
  // row node, neighbour slot of each element node in connectivity order
  __host__ __device__ static constexpr int ent(int a, int c) {
    constexpr int t[NADJ][8] = {{-1, -1, 0, 0, 2, 0, 1, 4}, {-1, -1, 0, 1, 1, 0, 4, 3}, {0, -1, 0, 0, 2, 1, 2, 4}, {0, -1, 0, 1, 2, 2, 5, 4}, {-1, 0, 0, 0, 1, 3, 4, 6}, {-1, 0, 0, 1, 0, 4, 7, 6}, {0, 0, 0, 0, 0, 4, 5, 8}, {0, 0, 0, 1, 0, 4, 8, 7}};
    return t[a][c];
  }
};
struct Tri3Stencil1 {
  static constexpr int NN = 5, NADJ = 4;
  // neighbour offsets (di, dj, dk) in row (node id) order
  __host__ __device__ static constexpr int off(int s, int d) {
    constexpr int t[NN][3] = {{0, -1, 0}, {-1, 0, 0}, {0, 0, 0}, {1, 0, 0}, {0, 1, 0}};
    return t[s][d];
  }
  // adjacent elements: cell offset (di, dj, dk), element within the cell, local index of the
  // row node, neighbour slot of each element node in connectivity order
  __host__ __device__ static constexpr int ent(int a, int c) {
    constexpr int t[NADJ][8] = {{-1, -1, 0, 1, 1, 0, 2, 1}, {0, -1, 0, 1, 2, 0, 3, 2}, {-1, 0, 0, 0, 1, 1, 2, 4}, {0, 0, 0, 0, 0, 2, 3, 4}};
    return t[a][c];
  }
};
struct Tet4Stencil0 {
  static constexpr int NN = 15, NADJ = 24;
  // neighbour offsets (di, dj, dk) in row (node id) order
  __host__ __device__ static constexpr int off(int s, int d) {
    constexpr int t[NN][3] = {{-1, -1, -1}, {0, -1, -1}, {-1, 0, -1}, {0, 0, -1}, {-1, -1, 0}, {0, -1, 0}, {-1, 0, 0}, {0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {1, 1, 0}, {0, 0, 1}, {1, 0, 1}, {0, 1, 1}, {1, 1, 1}};
    return t[s][d];
  }
  // adjacent elements: cell offset (di, dj, dk), element within the cell, local index of the
  // row node, neighbour slot of each element node in connectivity order
  __host__ __device__ static constexpr int ent(int a, int c) {
    constexpr int t[NADJ][9] = {{-1, -1, -1, 0, 3, 0, 3, 2, 7}, {-1, -1, -1, 1, 3, 0, 2, 6, 7}, {-1, -1, -1, 2, 3, 0, 6, 4, 7}, {-1, -1, -1, 3, 2, 0, 5, 7, 4}, {-1, -1, -1, 4, 2, 1, 5, 7, 0}, {-1, -1, -1, 5, 1, 1, 7, 3, 0}, {0, -1, -1, 1, 2, 1, 3, 7, 8}, {0, -1, -1, 2, 1, 1, 7, 5, 8}, {-1, 0, -1, 3, 1, 2, 7, 9, 6}, {-1, 0, -1, 4, 1, 3, 7, 9, 2}, {0, 0, -1, 2, 2, 3, 9, 7, 10}, {0, 0, -1, 3, 3, 3, 8, 10, 7}, {-1, -1, 0, 0, 1, 4, 7, 6, 11}, {-1, -1, 0, 5, 2, 5, 11, 7, 4}, {0, -1, 0, 0, 2, 5, 8, 7, 12}, {0, -1, 0, 1, 1, 5, 7, 11, 12}, {-1, 0, 0, 4, 0, 7, 11, 13, 6}, {-1, 0, 0, 5, 0, 7, 13, 9, 6}, {0, 0, 0, 0, 0, 7, 10, 9, 14}, {0, 0, 0, 1, 0, 7, 9, 13, 14}, {0, 0, 0, 2, 0, 7, 13, 11, 14}, {0, 0, 0, 3, 0, 7, 12, 14, 11}, {0, 0, 0, 4, 3, 8, 12, 14, 7}, {0, 0, 0, 5, 3, 8, 14, 10, 7}};
    return t[a][c];
  }
};
struct Quad4Stencil0 {
  static constexpr int NN = 9, NADJ = 4;
  __host__ __device__ static constexpr int off(int s, int d) { return Tri3Stencil0::off(s, d); }
  __host__ __device__ static constexpr int ent(int a, int c) {
    constexpr int t[NADJ][9] = {{-1, -1, 0, 0, 2, 0, 1, 4, 3}, {0, -1, 0, 0, 3, 1, 2, 5, 4}, {-1, 0, 0, 0, 1, 3, 4, 7, 6}, {0, 0, 0, 0, 0, 4, 5, 8, 7}};
    return t[a][c];
  }
};

// part = (B_a(:, q))^T D using only the nonzero entries of the isotropic D (the zero terms of the
// reference's SmallStrainKFast contribute exact zeros).
template <int DIM, typename T>
__device__ __forceinline__ void part_iso(const T* d, const T* ga, int q, T* part) {
  if (DIM == 2) {
    if (q == 0) { part[0] = ga[0] * d[0]; part[1] = ga[0] * d[1]; part[2] = ga[1] * d[4]; }
    else        { part[0] = ga[1] * d[2]; part[1] = ga[1] * d[3]; part[2] = ga[0] * d[4]; }
  } else {
    if (q == 0) { part[0] = ga[0] * d[0]; part[1] = ga[0] * d[1]; part[2] = ga[0] * d[2]; part[3] = T(0); part[4] = ga[2] * d[10]; part[5] = ga[1] * d[11]; }
    else if (q == 1) { part[0] = ga[1] * d[3]; part[1] = ga[1] * d[4]; part[2] = ga[1] * d[5]; part[3] = ga[2] * d[9]; part[4] = T(0); part[5] = ga[0] * d[11]; }
    else { part[0] = ga[2] * d[6]; part[1] = ga[2] * d[7]; part[2] = ga[2] * d[8]; part[3] = ga[1] * d[9]; part[4] = ga[0] * d[10]; part[5] = T(0); }
  }
}

// the nonzero entries of an isotropic D (36 entries, row-major) in part_iso's order
template <int DIM, typename T>
__device__ __forceinline__ void iso_from(const T* D, T* d) {
  constexpr int n = (DIM == 2) ? 5 : 12;
  constexpr int i2[5] = {0, 1, 3, 4, 8};
  constexpr int i3[12] = {0, 1, 2, 6, 7, 8, 12, 13, 14, 21, 28, 35};
#pragma unroll
  for (int k = 0; k < n; ++k) d[k] = D[(DIM == 2) ? i2[k] : i3[k]];
}

}  // namespace pgd
