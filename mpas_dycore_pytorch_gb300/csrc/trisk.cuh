// TRiSK sums over an edge's neighbours, sum_j weightsOnEdge_j F[edgesOnEdge_j, k], on the integer
// pipes (fixdot.cuh): the block's weights in shared memory, converted once per block and edge.
#pragma once

#include "common.cuh"

namespace trisk {

// entries of the edges [e0, e0 + n), N per edge; an edge with more neighbours is marked for the
// float64 sum
template <int N>
MPASG_D void load(const mpasg_mesh& m, uint32_t e0, uint32_t n, fx::Weight* tab) {
  const int me2 = m.maxEdges2;
  for (uint32_t t = threadIdx.x; t < n * N; t += blockDim.x) {
    const uint32_t el = t / N, j = t - el * N, e = e0 + el;
    const int n2 = m.nEdgesOnEdge[e];
    if ((int)j < n2 && n2 <= N) {
      tab[t] = fx::weight(m.weightsOnEdge[e * me2 + j], m.edgesOnEdge[e * me2 + j]);
    } else {
      fx::Weight z{0, 0, n2 > N ? fx::kBadWeight : 0u, n2 > 0 ? m.edgesOnEdge[e * me2] : (int)e};
      tab[t] = z;
    }
  }
}

template <int N>
MPASG_D double sum(const mpasg_mesh& m, const double* __restrict__ field, const fx::Weight* w, uint32_t e, uint32_t k,
                   uint32_t L) {
  double x[N], out;
#pragma unroll
  for (int j = 0; j < N; ++j) x[j] = field[(uint32_t)w[j].row * L + k];
  if (!fx::dot<N>(x, w, &out)) {
    out = 0.0;
    const size_t o = (size_t)e * m.maxEdges2;
    for (int j = 0; j < m.nEdgesOnEdge[e]; ++j)
      out = fma(m.weightsOnEdge[o + j], field[(size_t)m.edgesOnEdge[o + j] * L + k], out);
  }
  return out;
}

}  // namespace trisk
