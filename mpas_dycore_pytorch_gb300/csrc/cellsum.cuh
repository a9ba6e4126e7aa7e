// Signed sums of edge values over a cell's edges, sum_j sign_j F[edge_j, k]: the divergence of a
// flux formed once per edge.  The slots (edge row, sign) of the cells a block covers are in
// shared memory; a kernel that needs two sums takes one on the integer pipes (fixdot.cuh) and
// one on the float64 pipe.
#pragma once

#include "common.cuh"

namespace cellsum {

struct Slot {
  uint32_t row, sgn;  // edge, sign bit (bit 31 set: minus)
};

// slots of the cells [c0, c0 + n): N per cell (a cell with more edges uses the mesh arrays)
template <int N>
MPASG_D void load(const mpasg_mesh& m, uint32_t c0, uint32_t n, Slot* tab) {
  for (uint32_t t = threadIdx.x; t < n * N; t += blockDim.x) {
    const uint32_t cl = t / N, j = t - cl * N, c = c0 + cl;
    const size_t o = (size_t)c * m.maxEdges + j;
    tab[t] = (int)j < m.nEdgesOnCell[c]
                 ? Slot{(uint32_t)m.edgesOnCell[o], (uint32_t)__double2hiint(m.edgesOnCell_sign[o]) & 0x80000000u}
                 : Slot{0u, 0u};
  }
}

MPASG_D double flip(double x, uint32_t sgn) {
  return __hiloint2double((int)((uint32_t)__double2hiint(x) ^ sgn), __double2loint(x));
}

// slots in order, in float64 (any number of edges)
MPASG_D double wide(const mpasg_mesh& m, uint32_t c, const double* __restrict__ f, uint32_t pitch, uint32_t k) {
  const size_t o = (size_t)c * m.maxEdges;
  double acc = 0.0;
  for (int j = 0; j < m.nEdgesOnCell[c]; ++j)
    acc = fma(m.edgesOnCell_sign[o + j], f[(size_t)m.edgesOnCell[o + j] * pitch + k], acc);
  return acc;
}

// on the float64 pipe
// (Index: the type of an index into f; size_t where rows times pitch may pass 2^32)
template <int N, typename Index = uint32_t>
MPASG_D double f64(const mpasg_mesh& m, uint32_t c, int n, const Slot* s, const double* __restrict__ f,
                   uint32_t pitch, uint32_t k) {
  if (n > N) return wide(m, c, f, pitch, k);
  double x[N];
#pragma unroll
  for (int j = 0; j < N; ++j) x[j] = j < n ? f[(Index)s[j].row * pitch + k] : 0.0;
  double acc = flip(x[0], s[0].sgn);
#pragma unroll
  for (int j = 1; j < N; ++j)
    if (j < n) acc = acc + flip(x[j], s[j].sgn);
  return acc;
}

// on the integer pipes
template <int N, typename Index = uint32_t>
MPASG_D double fixed(const mpasg_mesh& m, uint32_t c, int n, const Slot* s, const double* __restrict__ f,
                     uint32_t pitch, uint32_t k) {
  if (n > N) return wide(m, c, f, pitch, k);
  double x[N], out;
  uint32_t sgn[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    x[j] = j < n ? f[(Index)s[j].row * pitch + k] : 0.0;
    sgn[j] = s[j].sgn;
  }
  return fx::sum<N>(x, sgn, &out) ? out : wide(m, c, f, pitch, k);
}

// cells a block of consecutive (cell, level) threads covers, at most
inline int max_cells(int levels) { return (kBlock - 1) / levels + 2; }

}  // namespace cellsum
