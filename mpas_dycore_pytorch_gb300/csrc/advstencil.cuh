// The advection stencil of an edge (adv_coefs +/- adv_coefs_3rd over advCellsForEdge) as
// fixed-point weights in shared memory (fixdot.cuh): the tendencies' theta and w fluxes and
// the scalars' edge values read it.
#pragma once

#include "common.cuh"
#include "fixdot.cuh"

namespace adv {

// Table of the edges [e0, e0 + n): per edge N weights for a flux along the edge normal
// (coefs + 3rd), then N for the opposite one (coefs - 3rd), with the cell each gathers.  An edge
// with more than N stencil cells is marked for the float64 sum.
template <int N>
MPASG_D void load(const mpasg_mesh& m, uint32_t e0, uint32_t n, fx::Weight* tab) {
  for (uint32_t t = threadIdx.x; t < n * N; t += blockDim.x) {
    const uint32_t el = t / N, j = t - el * N, e = e0 + el;
    const int nadv = m.nAdvCellsForEdge[e];
    const size_t o = (size_t)e * m.nAdvMax;
    fx::Weight* w = tab + el * (2 * N) + j;
    if ((int)j < nadv && nadv <= N) {
      const int32_t cell = m.advCellsForEdge[o + j];
      w[0] = fx::weight(m.adv_coefs_p[o + j], cell);
      w[N] = fx::weight(m.adv_coefs_m[o + j], cell);
    } else {
      const fx::Weight z{0, 0, nadv > N ? fx::kBadWeight : 0u, nadv > 0 ? m.advCellsForEdge[o] : 0};
      w[0] = z;
      w[N] = z;
    }
  }
}

constexpr size_t kEntryBytes = 2 * sizeof(fx::Weight);  // table bytes per edge and slot

// the same sum in float64, slots in order: q at (cell, k) is q[cell * pitch + k]
MPASG_D double sum(const mpasg_mesh& m, uint32_t e, bool back, const double* __restrict__ q, uint32_t pitch,
                   uint32_t k) {
  const size_t o = (size_t)e * m.nAdvMax;
  const double* cf = (back ? m.adv_coefs_m : m.adv_coefs_p) + o;
  const int32_t* cells = m.advCellsForEdge + o;
  double acc = 0.0;
  for (int a = 0; a < m.nAdvCellsForEdge[e]; ++a) acc = fma(cf[a], q[(size_t)cells[a] * pitch + k], acc);
  return acc;
}

}  // namespace adv
