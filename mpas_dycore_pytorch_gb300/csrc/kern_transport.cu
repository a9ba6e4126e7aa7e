// Flux-form scalar transport: explicit RK stages (mpas_pytorch/dynamics/advance_scalars.py:1272,
// composition :861, Pattern-C edge values dynamics/pattern_c.py:234-305) and the monotone
// flux-corrected final stage (dynamics/advance_scalars_mono.py:3332, tile :1476, neighbour
// bounds autodiff/soft_limiter.py:72).  Scalar fields are (C+1, L, S), edge fluxes (E+1, L, S).
#include <algorithm>
#include <mutex>

#include "advstencil.cuh"
#include "cellsum.cuh"

namespace {

// Every transport kernel is a template on the stencil arithmetic type T (common.cuh).
// In the mixed form the edge values, flux divergences, bounds and limiter factors are
// float32; the density weighting and the stage update of each scalar are float64.

template <typename T>
MPASG_D T mz(T x) { return x > T(0) ? x : T(0); }

// sum_m (adv_coefs + sign(uh) adv_coefs_3rd) q[advCell_m]  for every scalar (mixed form)
template <typename T>
__global__ void k_pattern_c(mpasg_mesh m, FastDiv fl, int S, const double* __restrict__ uh,
                            const double* __restrict__ q, double* __restrict__ out, int times_uh) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nEdges * L) return;
  uint32_t e = fl.div(i), k = i - e * L;
  const int na = m.nAdvMax;
  const int nadv = m.nAdvCellsForEdge[e];
  const T u = cv<T>(uh[i]);
  const double* cf = (u >= T(0) ? m.adv_coefs_p : m.adv_coefs_m) + (size_t)e * na;
  T acc[8];
  for (int s = 0; s < S; ++s) acc[s] = T(0);
  for (int a = 0; a < nadv; ++a) {
    int cell = m.advCellsForEdge[e * na + a];
    T w = cv<T>(cf[a]);
    const double* qc = q + ((size_t)cell * L + k) * S;
    for (int s = 0; s < S; ++s) {
      T t = w * cv<T>(qc[s]);
      acc[s] = (a == 0) ? t : acc[s] + t;
    }
  }
  for (int s = 0; s < S; ++s) out[(size_t)i * S + s] = f64(times_uh ? u * acc[s] : acc[s]);
}

// ---------------------------------------------------------------- float64 form
// A thread takes one (level, scalar) value of a row, so neighbouring threads read neighbouring
// values and a scalar costs no strided pass; the horizontal sums run on the integer pipes
// (fixdot.cuh), comparisons, minima and clamps on the integer side too (each would take a
// float64 slot).
// A launch numbers its (row, value) threads in 32 bits and divides by FastDiv, which holds below
// 2^31: rows that reach it are taken in several launches, each of which gets what it indexes by
// its rows as pointers to its first one (cells_from, edges_from; offsets added in the thread cost
// the explicit stage at 10242 x 41 x 3 2 %).  Gathers over all rows are 64 bits wide.  (A build may
// lower the limit to test the split.)
#ifndef MPASG_MAX_THREADS
#define MPASG_MAX_THREADS (0x7fffffffu - kBlock)
#endif
constexpr uint32_t kMaxThreads = MPASG_MAX_THREADS;

// calls launch(first row, rows) over n rows of `width` threads each
template <typename Launch>
int launch_rows(int n, uint32_t width, Launch launch) {
  const int most = (int)std::min<uint32_t>((uint32_t)n, std::max(1u, kMaxThreads / width));
  for (int first = 0; first < n; first += most) {
    launch((uint32_t)first, (uint32_t)std::min(most, n - first));
    MPASG_LAUNCH_CHECK();
    if (most > n - first) break;  // (first + most may pass the last int)
  }
  return MPASG_OK;
}

// the mesh and the fields the cells' kernels index by cell, from a cell on
mpasg_mesh cells_from(const mpasg_mesh& m, size_t first) {
  mpasg_mesh g = m;
  g.nEdgesOnCell += first;
  g.edgesOnCell += first * m.maxEdges;
  g.edgesOnCell_sign += first * m.maxEdges;
  g.cellsOnCell += first * m.maxEdges;
  g.invAreaCell += first;
  return g;
}
mpasg_fields cells_from(const mpasg_mesh& m, const mpasg_fields& f, int S, size_t first) {
  const size_t L = m.nVertLevels, row = first * L * S;
  mpasg_fields g = f;
  g.wwAvg += first * (L + 1);
  g.rho_zz += first * L;
  g.rho_zz_old_split += first * L;
  g.rho_int += first * L;
  g.wflux += first * (L + 1) * S;
  g.rows += row;
  g.scale_in += row;
  g.scale_out += row;
  g.s_max += row;
  g.s_min += row;
  return g;
}
// the mesh the edges' kernels index by edge, from an edge on
mpasg_mesh edges_from(const mpasg_mesh& m, size_t first) {
  mpasg_mesh g = m;
  g.nAdvCellsForEdge += first;
  g.advCellsForEdge += first * m.nAdvMax;
  g.adv_coefs_p += first * m.nAdvMax;
  g.adv_coefs_m += first * m.nAdvMax;
  g.dvEdge += first;
  g.cellsOnEdge += 2 * first;
  return g;
}

struct TransportScalars {
  double dt, w_old, w_new, f3[4];  // f3: 7 + 3 c, 7 - 3 c, 1 + c, 1 - c of the upwind flux3
};

inline TransportScalars transport_scalars(double dt, double w_old, double w_new, double c) {
  return TransportScalars{dt, w_old, w_new, {7.0 + 3.0 * c, 7.0 - 3.0 * c, 1.0 + c, 1.0 - c}};
}

// Horizontal edge fluxes.  A row of an edge is cut in two halves and a thread takes the same
// place of both: the first half's sum on the integer pipes, the second's on the float64 pipe
// beside it.  Weights are converted once per block and edge.
// MONO: out = the upwind flux of s_old, out2 = dt times the high-order flux minus it;
// else out = the high-order flux.
// 40962 x 55 with 3 tracers, edge values only: 392 -> 363 us; 2562 x 37 with 8: 73 -> 47 us (48
// registers; with the two sums of a thread interleaved instruction by instruction 481 and 62
// us, the registers costing more warps than the overlap inside a warp gives).
template <bool MONO>
MPASG_D void store_edge_flux(const mpasg_mesh& m, uint32_t e, uint32_t row, uint32_t r, double u, double value,
                             double dvdt, double dt, const double* __restrict__ s_old, double* __restrict__ out,
                             double* __restrict__ out2) {
  const size_t o = (size_t)e * row + r;
  const double flux = u * value;
  if (!MONO) {
    out[o] = flux;
    return;
  }
  const int up = m.cellsOnEdge[2 * e + (__double2hiint(u) < 0 ? 1 : 0)];
  const double fup = dvdt * (u * s_old[(size_t)up * row + r]);
  out[o] = fup;
  out2[o] = fma(dt, flux, -fup);
}

template <int N, bool MONO>
__global__ void __launch_bounds__(kBlock, 5) k_edge_flux_fx(mpasg_mesh m, FastDiv fh, FastDiv fs, uint32_t n_all,
                                                         uint32_t half, double dt, const double* __restrict__ uh,
                                                         const double* __restrict__ q,
                                                         const double* __restrict__ s_old, double* __restrict__ out,
                                                         double* __restrict__ out2) {
  extern __shared__ fx::Weight s_w[];
  const uint32_t L = (uint32_t)m.nVertLevels, row = L * fs.d;
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t e0 = fh.div(i0), e1 = fh.div(min(i0 + kBlock, n_all) - 1u);
  adv::load<N>(m, e0, e1 - e0 + 1, s_w);
  __syncthreads();
  if (i >= n_all) return;
  const uint32_t e = fh.div(i), a = i - e * half, b = a + half;
  const fx::Weight* w = s_w + (e - e0) * (2 * N);
  double x[N], acc;
  const double ua = uh[(size_t)e * L + fs.div(a)], dvdt = MONO ? m.dvEdge[e] * dt : 0.0;
  const bool back = __double2hiint(ua) < 0;
  if (back) w += N;
#pragma unroll
  for (int j = 0; j < N; ++j) x[j] = q[(size_t)w[j].row * row + a];
  if (b < row) {
    const double ub = uh[(size_t)e * L + fs.div(b)];
    store_edge_flux<MONO>(m, e, row, b, ub, adv::sum(m, e, __double2hiint(ub) < 0, q, row, b), dvdt, dt, s_old, out,
                          out2);
  }
  if (!fx::dot<N>(x, w, &acc)) acc = adv::sum(m, e, back, q, row, a);
  store_edge_flux<MONO>(m, e, row, a, ua, acc, dvdt, dt, s_old, out, out2);
}

template <bool MONO>
int launch_edge_flux_fx(const mpasg_mesh* m, int S, double dt, const double* uh, const double* q, const double* s_old,
                        double* out, double* out2, cudaStream_t s) {
  const uint32_t half = ((uint32_t)m->nVertLevels * S + 1) / 2;
  // (rows of few values: a block covers many edges, up to 115 KB of them at one value and 14 slots)
  const size_t smem = (size_t)((kBlock - 1) / half + 2) * adv::kEntryBytes;
  const auto run = [&](auto kernel, int slots) -> int {
    if (!allow_smem(kernel, smem * slots)) return MPASG_E_CUDA;
    return launch_rows(m->nEdges, half, [&](uint32_t first, uint32_t n) {
      const size_t L = m->nVertLevels, at = first * L * S;
      kernel<<<nblocks((long long)n * half), kBlock, smem * slots, s>>>(edges_from(*m, first), FastDiv(half), FastDiv(S),
                                                                        n * half, half, dt, uh + first * L, q, s_old,
                                                                        out + at, out2 ? out2 + at : nullptr);
    });
  };
  return m->nAdvMax <= 10 ? run(k_edge_flux_fx<10, MONO>, 10) : run(k_edge_flux_fx<14, MONO>, 14);
}

// the thread's place in a (cell, level, scalar) row
struct CellRow {
  uint32_t c, r, k, s;
};
MPASG_D CellRow cell_row(uint32_t i, uint32_t row, const FastDiv& fr, const FastDiv& fs) {
  CellRow t;
  t.c = fr.div(i);
  t.r = i - t.c * row;
  t.k = fs.div(t.r);
  t.s = t.r - t.k * fs.d;
  return t;
}

// vertical flux at the interface below level k, a linear combination of the column's values
// times the interface velocity: returns the combination (times 12 inside) in *comb and the
// factor 1 or 1/12 that goes with it
MPASG_D double interface_value(const double* __restrict__ q, uint32_t S, double ww, uint32_t k, uint32_t L,
                               const double* fnm, const double* fnp, const double* f3, double* factor) {
  // (the second-order interfaces: the same instructions with other coefficients, a branch of
  // theirs would cost nearly every warp its operations again)
  const bool low = k == 1 || k == L - 1, down = low || __double2hiint(ww) < 0;
  const int s = (int)S;
  const double a = q[down ? 0 : -s], b = q[down ? -s : 0];
  const double a2 = low ? 0.0 : q[down ? s : -2 * s], b2 = low ? 0.0 : q[down ? -2 * s : s];
  *factor = low ? 1.0 : kInv12;
  return fma(low ? fnm[k] : f3[0], a, fma(low ? fnp[k] : f3[1], b, -fma(f3[2], a2, f3[3] * b2)));
}

// explicit stage update: 20 float64 operations a value and one integer sum, about 33 in the
// per-cell loop over the scalars (40962 x 55 x 3: 380 -> 283 us a stage)
template <int N>
__global__ void __launch_bounds__(kBlock, 5) k_scalars_update_fx(mpasg_mesh m, mpasg_fields f, FastDiv fr, FastDiv fs,
                                                              uint32_t n_all, TransportScalars p,
                                                              const double* __restrict__ s_old,
                                                              const double* __restrict__ s_new,
                                                              double* __restrict__ s_out) {
  extern __shared__ cellsum::Slot s_c[];
  __shared__ double s_wd[kBlock];
  const uint32_t L = (uint32_t)m.nVertLevels, S = fs.d, row = L * S;
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t c0 = fr.div(i0), c1 = fr.div(min(i0 + kBlock, n_all) - 1u);
  cellsum::load<N>(m, c0, c1 - c0 + 1, s_c);
  const bool active = i < n_all;
  CellRow t{c0, 0, 0, 0};
  auto flux_at = [&](uint32_t k) {  // at the interface below level k of this thread's column
    if (k == 0 || k >= L) return 0.0;
    const double ww = f.wwAvg[(size_t)t.c * (L + 1) + k];
    double fac;
    const double v = interface_value(s_new + (size_t)t.c * row + k * S + t.s, S, ww, k, L, m.fnm, m.fnp, p.f3, &fac);
    return (ww * fac) * v;
  };
  double lo = 0.0;
  if (active) {
    t = cell_row(i, row, fr, fs);
    lo = flux_at(t.k);
  }
  s_wd[threadIdx.x] = lo;
  __syncthreads();
  if (!active) return;
  const double hi = t.k + 1 >= L ? 0.0 : threadIdx.x + S < kBlock ? s_wd[threadIdx.x + S] : flux_at(t.k + 1);
  const double div = cellsum::fixed<N, size_t>(m, t.c, m.nEdgesOnCell[t.c], s_c + (t.c - c0) * N, f.hflux, row, t.r);
  const size_t ic = (size_t)t.c * L + t.k;
  const double tend = fma(m.rdnw[t.k], lo - hi, -(div * m.invAreaCell[t.c]));
  const double rho_old = f.rho_zz_old_split[ic];
  double rho = f.rho_zz[ic];
  if (p.w_old != 0.0) rho = p.w_old * rho_old + p.w_new * rho;
  s_out[i] = fx::quotient(fma(p.dt, tend, s_old[i] * rho_old), rho);
}

// monotone stage: density at its end
__global__ void k_mono_density_fx(mpasg_mesh m, mpasg_fields f, FastDiv fl, double dt) {
  const uint32_t L = (uint32_t)m.nVertLevels, n_all = (uint32_t)m.nCells * L;
  const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n_all) return;
  const uint32_t c = fl.div(i), k = i - c * L;
  const size_t o = (size_t)c * m.maxEdges, ow = (size_t)c * (L + 1) + k;
  double h = 0.0;
  for (int j = 0; j < m.nEdgesOnCell[c]; ++j)
    h = fma(m.cell_edge_geo[o + j], f.ruAvg[(size_t)m.edgesOnCell[o + j] * L + k], h);
  f.rho_int[i] = f.rho_zz_old_split[i] - dt * fma(m.rdnw[k], f.wwAvg[ow + 1] - f.wwAvg[ow], h);
}

// Monotone stage, per value: local and neighbour bounds, vertical upwind update, vertical parts
// of the limiter scale sums; the high-minus-upwind vertical flux at the interface below the
// level goes to wflux (k >= 1).  The 18 minima and maxima of the bounds are integer comparisons
// (735 -> 273 us at 40962 x 55 x 3, and 40 us for the density).
template <int N>
__global__ void __launch_bounds__(kBlock, 5) k_mono_cells_a_fx(mpasg_mesh m, mpasg_fields f, FastDiv fr, FastDiv fs,
                                                            uint32_t n_all, TransportScalars p,
                                                            const double* __restrict__ so_all,
                                                            const double* __restrict__ so,
                                                            const double* __restrict__ sn) {
  __shared__ double s_wm[kBlock], s_fu[kBlock];
  const uint32_t L = (uint32_t)m.nVertLevels, S = fs.d, row = L * S;
  const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  const bool active = i < n_all;
  CellRow t{0, 0, 0, 0};
  auto fluxes = [&](uint32_t k, double* wm, double* fu) {
    *wm = *fu = 0.0;
    if (k == 0 || k >= L) return;
    const double ww = f.wwAvg[(size_t)t.c * (L + 1) + k], dtw = p.dt * ww;
    const size_t o = (size_t)t.c * row + k * S + t.s;
    double fac;
    const double v = interface_value(sn + o, S, ww, k, L, m.fnm, m.fnp, p.f3, &fac);
    *fu = dtw * so[__double2hiint(ww) < 0 ? o : o - S];
    *wm = fma(dtw * fac, v, -*fu);
  };
  double wm_lo = 0.0, fu_lo = 0.0;
  if (active) {
    t = cell_row(i, row, fr, fs);
    fluxes(t.k, &wm_lo, &fu_lo);
  }
  s_wm[threadIdx.x] = wm_lo;
  s_fu[threadIdx.x] = fu_lo;
  __syncthreads();
  if (!active) return;
  double wm_hi = 0.0, fu_hi = 0.0;
  if (t.k + 1 < L) {
    if (threadIdx.x + S < kBlock) {
      wm_hi = s_wm[threadIdx.x + S];
      fu_hi = s_fu[threadIdx.x + S];
    } else {
      fluxes(t.k + 1, &wm_hi, &fu_hi);
    }
  }
  if (t.k >= 1) f.wflux[((size_t)t.c * (L + 1) + t.k) * S + t.s] = wm_lo;
  // bounds over the column's neighbours and the adjacent cells
  const double here = so[i];
  int64_t kmax = fx::order_key(here), kmin = kmax;
  auto bound = [&](double x) {
    const int64_t q = fx::order_key(x);
    kmax = q > kmax ? q : kmax;
    kmin = q < kmin ? q : kmin;
  };
  if (t.k >= 1) bound(so[i - S]);
  if (t.k + 1 < L) bound(so[i + S]);
  const size_t oc = (size_t)t.c * m.maxEdges;
  const int n = m.nEdgesOnCell[t.c];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if (j < n) {
      const int nb = m.cellsOnCell[oc + j];
      if (nb < m.nCells) bound(so_all[(size_t)nb * row + t.r]);
    }
  }
  for (int j = N; j < n; ++j) {
    const int nb = m.cellsOnCell[oc + j];
    if (nb < m.nCells) bound(so_all[(size_t)nb * row + t.r]);
  }
  double smax = fx::from_order_key(kmax), smin = fx::from_order_key(kmin);
  if (!(fx::is_finite(smax) && fx::is_finite(smin))) {  // a NaN among them: left out, as fmax / fmin do
    smax = smin = here;
    auto wide = [&](double x) {
      smax = fmax(smax, x);
      smin = fmin(smin, x);
    };
    if (t.k >= 1) wide(so[i - S]);
    if (t.k + 1 < L) wide(so[i + S]);
    for (int j = 0; j < n; ++j) {
      const int nb = m.cellsOnCell[oc + j];
      if (nb < m.nCells) wide(so_all[(size_t)nb * row + t.r]);
    }
  }
  const double rd = m.rdnw[t.k];
  f.rows[i] = fma(rd, fu_lo - fu_hi, here * f.rho_zz_old_split[(size_t)t.c * L + t.k]);
  // in and out fluxes of the correction through the level's two interfaces
  f.scale_in[i] = rd * (fx::positive(wm_lo) + fx::positive(-wm_hi));
  f.scale_out[i] = -rd * (fx::positive(wm_hi) + fx::positive(-wm_lo));
  f.s_max[i] = smax;
  f.s_min[i] = smin;
}

// per value: horizontal upwind update and scale sums, then the limiter factors.  Three integer
// sums and 17 float64 operations a value, about 65 with the comparisons and divisions of the
// per-cell loop (913 -> 256 us at 40962 x 55 x 3).
template <int N>
__global__ void __launch_bounds__(kBlock, 5) k_mono_cells_b_fx(mpasg_mesh m, mpasg_fields f, FastDiv fr, FastDiv fs,
                                                            uint32_t n_all) {
  extern __shared__ cellsum::Slot s_c[];
  const uint32_t L = (uint32_t)m.nVertLevels, row = L * fs.d;
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t c0 = fr.div(i0), c1 = fr.div(min(i0 + kBlock, n_all) - 1u);
  cellsum::load<N>(m, c0, c1 - c0 + 1, s_c);
  __syncthreads();
  if (i >= n_all) return;
  const CellRow t = cell_row(i, row, fr, fs);
  const int n = m.nEdgesOnCell[t.c];
  const cellsum::Slot* s = s_c + (t.c - c0) * N;
  const double ia = m.invAreaCell[t.c], rint = f.rho_int[(size_t)t.c * L + t.k];
  const double up = cellsum::fixed<N, size_t>(m, t.c, n, s, f.flux_up, row, t.r);
  double out = 0.0, in = 0.0;
  bool ok = n <= N;
  if (ok) {
    double x[N];
    uint32_t sgn[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      x[j] = j < n ? f.flux_tmp[(size_t)s[j].row * row + t.r] : 0.0;
      sgn[j] = s[j].sgn;
    }
    ok = fx::sum_parts<N>(x, sgn, &out, &in);
  }
  if (!ok) {
    out = in = 0.0;
    const size_t o = (size_t)t.c * m.maxEdges;
    for (int j = 0; j < n; ++j) {
      const double sf = m.edgesOnCell_sign[o + j] * f.flux_tmp[(size_t)m.edgesOnCell[o + j] * row + t.r];
      out = out + mz(sf);
      in = in + mz(-sf);
    }
  }
  const double rows = fma(-ia, up, f.rows[i]), eps = 1.0e-20;
  const double sin_ = fma(ia, in, f.scale_in[i]) + eps, sout = fma(ia, out, -f.scale_out[i]) + eps;
  f.rows[i] = rows;
  f.scale_in[i] = fx::clamp01(fx::quotient(fma(f.s_max[i], rint, -rows), sin_));
  f.scale_out[i] = fx::clamp01(fx::quotient(fma(-f.s_min[i], rint, rows), sout));
}

// per (edge, value): limited horizontal flux (stored in hflux)
__global__ void k_mono_edges_b_fx(mpasg_mesh m, mpasg_fields f, FastDiv fr, uint32_t n_all) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_all) return;
  const uint32_t e = fr.div(i), r = i - e * fr.d;
  const double ft = f.flux_tmp[i];
  const uint32_t back = __double2hiint(ft) < 0 ? 1u : 0u;
  const size_t from = (size_t)m.cellsOnEdge[2 * e + back] * fr.d + r;
  const size_t to = (size_t)m.cellsOnEdge[2 * e + 1 - back] * fr.d + r;
  f.hflux[i] = ft * fx::min_nonneg(f.scale_out[from], f.scale_in[to]);
}

// per value: limited horizontal and vertical fluxes, positivity
template <int N>
__global__ void __launch_bounds__(kBlock, 5) k_mono_cells_c_fx(mpasg_mesh m, mpasg_fields f, FastDiv fr, FastDiv fs,
                                                            uint32_t n_all, double* __restrict__ s_out) {
  extern __shared__ cellsum::Slot s_c[];
  const uint32_t L = (uint32_t)m.nVertLevels, S = fs.d, row = L * S;
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t c0 = fr.div(i0), c1 = fr.div(min(i0 + kBlock, n_all) - 1u);
  cellsum::load<N>(m, c0, c1 - c0 + 1, s_c);
  __syncthreads();
  if (i >= n_all) return;
  const CellRow t = cell_row(i, row, fr, fs);
  const double* wf = f.wflux + ((size_t)t.c * (L + 1) + t.k) * S + t.s;
  auto limited = [&](double wm, uint32_t below, uint32_t above) {  // an upward flux leaves `below`
    const bool down = __double2hiint(wm) < 0;
    return wm * fx::min_nonneg(f.scale_out[down ? above : below], f.scale_in[down ? below : above]);
  };
  const double lo = t.k >= 1 ? limited(wf[0], i - S, i) : 0.0;
  const double hi = t.k + 1 < L ? limited(wf[S], i, i + S) : 0.0;
  const double h = cellsum::fixed<N, size_t>(m, t.c, m.nEdgesOnCell[t.c], s_c + (t.c - c0) * N, f.hflux, row, t.r);
  const double rows = fma(m.rdnw[t.k], lo - hi, fma(-m.invAreaCell[t.c], h, f.rows[i]));
  s_out[i] = fx::positive(fx::quotient(rows, f.rho_int[(size_t)t.c * L + t.k]));
}

template <typename T>
MPASG_D T wdtn_at(const double* sn, const double* ww, int kk, int L, int S, int s, const double* fnm,
                  const double* fnp, T coef3) {
  if (kk <= 0 || kk >= L) return T(0);
  if (kk == 1 || kk == L - 1)
    return cv<T>(ww[kk]) * (cv<T>(fnm[kk]) * cv<T>(sn[kk * S + s]) + cv<T>(fnp[kk]) * cv<T>(sn[(kk - 1) * S + s]));
  return flux3<T>(cv<T>(sn[(kk - 2) * S + s]), cv<T>(sn[(kk - 1) * S + s]), cv<T>(sn[kk * S + s]),
                  cv<T>(sn[(kk + 1) * S + s]), cv<T>(ww[kk]), coef3);
}

// explicit stage update for all scalars at (cell, level) (mixed form)
template <typename T>
__global__ void __launch_bounds__(kBlock) k_scalars_update(mpasg_mesh m, mpasg_fields f, FastDiv fl, int S,
                                                           double dt, double w_old, double w_new, double coef3,
                                                           const double* __restrict__ s_old,
                                                           const double* __restrict__ s_new,
                                                           double* __restrict__ s_out) {
  extern __shared__ __align__(8) unsigned char s_raw[];
  T* s_wdtn = reinterpret_cast<T*>(s_raw);  // [blockDim.x][S]: vertical flux at the interface below
  const int L = m.nVertLevels;
  const T c3 = cv<T>(coef3);
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < (uint32_t)m.nCells * L;
  uint32_t c = 0, k = 0;
  if (active) {
    c = fl.div(i);
    k = i - c * L;
    const double* sn0 = s_new + (size_t)c * L * S;
    const double* ww0 = f.wwAvg + (size_t)c * (L + 1);
    for (int s = 0; s < S; ++s) s_wdtn[threadIdx.x * S + s] = wdtn_at<T>(sn0, ww0, k, L, S, s, m.fnm, m.fnp, c3);
  }
  __syncthreads();
  if (!active) return;
  const int me = m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  T div[8];
  for (int s = 0; s < S; ++s) div[s] = T(0);
  for (int j = 0; j < n; ++j) {
    int e = m.edgesOnCell[c * me + j];
    T w = -cv<T>(m.edgesOnCell_sign[c * me + j]) * cv<T>(f.ruAvg[(size_t)e * L + k]);
    const double* hf = f.hflux + ((size_t)e * L + k) * S;
    for (int s = 0; s < S; ++s) {
      T t = w * cv<T>(hf[s]);
      div[s] = (j == 0) ? t : div[s] + t;
    }
  }
  const T ia = cv<T>(m.invAreaCell[c]);
  const double* sn = s_new + (size_t)c * L * S;
  const double* ww = f.wwAvg + (size_t)c * (L + 1);
  double rho_old = f.rho_zz_old_split[i];
  double rho_i = w_old * rho_old + w_new * f.rho_zz[i];
  double inv = fdiv<T>(1.0, rho_i);
  const bool next_in_block = threadIdx.x + 1 < blockDim.x;
  const T rd = cv<T>(m.rdnw[k]);
  const T dt_t = cv<T>(dt);
  for (int s = 0; s < S; ++s) {
    T tend_col = div[s] * ia + T(0);
    T lo = s_wdtn[threadIdx.x * S + s];
    T hi = (k + 1 >= (uint32_t)L) ? T(0)
           : next_in_block ? s_wdtn[(threadIdx.x + 1) * S + s]
                           : wdtn_at<T>(sn, ww, k + 1, L, S, s, m.fnm, m.fnp, c3);
    T vdiv = rd * (hi - lo);
    s_out[(size_t)i * S + s] = (s_old[(size_t)i * S + s] * rho_old + f64(dt_t * (tend_col - vdiv))) * inv;
  }
}

// ---------------------------------------------------------------- monotone stage, mixed form

// per (cell, level): rho_int, local+neighbour bounds, vertical upwind update,
// vertical parts of the limiter scale sums; stores the high-minus-upwind vertical flux
// at the interface below the level (wflux[c, k, s], k >= 1)
template <typename T>
__global__ void __launch_bounds__(kBlock) k_mono_cells_a(mpasg_mesh m, mpasg_fields f, FastDiv fl, int S,
                                                         double dt, double coef3,
                                                         const double* __restrict__ so_all,
                                                         const double* __restrict__ sn_all) {
  extern __shared__ __align__(8) unsigned char s_raw[];
  T* s_wm = reinterpret_cast<T*>(s_raw);  // [blockDim.x][2 S]: high-minus-upwind and upwind flux below
  const int L = m.nVertLevels;
  const T c3 = cv<T>(coef3);
  const T dt_t = cv<T>(dt);
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < (uint32_t)m.nCells * L;
  uint32_t c = 0, k = 0;
  if (active) {
    c = fl.div(i);
    k = i - c * L;
    const double* so0 = so_all + (size_t)c * L * S;
    const double* sn0 = sn_all + (size_t)c * L * S;
    const double* ww0 = f.wwAvg + (size_t)c * (L + 1);
    for (int s = 0; s < S; ++s) {
      T fup = T(0), wm = T(0);
      if (k >= 1) {
        T wk = cv<T>(ww0[k]);
        fup = dt_t * (wk * cv<T>(wk >= T(0) ? so0[(k - 1) * S + s] : so0[k * S + s]));
        wm = dt_t * wdtn_at<T>(sn0, ww0, k, L, S, s, m.fnm, m.fnp, c3) - fup;
      }
      s_wm[threadIdx.x * 2 * S + s] = wm;
      s_wm[threadIdx.x * 2 * S + S + s] = fup;
    }
  }
  __syncthreads();
  if (!active) return;
  const int me = m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  const T ia = cv<T>(m.invAreaCell[c]);
  // density at the end of the stage
  T hdiv = T(0);
  for (int j = 0; j < n; ++j) {
    int e = m.edgesOnCell[c * me + j];
    T t = (cv<T>(f.ruAvg[(size_t)e * L + k]) * (-cv<T>(m.edgesOnCell_sign[c * me + j]) * cv<T>(m.dvEdge[e]))) * ia;
    hdiv = (j == 0) ? t : hdiv + t;
  }
  const double* ww = f.wwAvg + (size_t)c * (L + 1);
  double rho_old = f.rho_zz_old_split[i];
  const T rd = cv<T>(m.rdnw[k]);
  double rho_int = rho_old + f64(dt_t * (hdiv - rd * (cv<T>(ww[k + 1]) - cv<T>(ww[k]))));
  f.rho_int[i] = rho_int;
  const double* so = so_all + (size_t)c * L * S;
  const double* sn = sn_all + (size_t)c * L * S;
  for (int s = 0; s < S; ++s) {
    T smax, smin;
    if (k == 0) {
      smax = vmax(cv<T>(so[0 * S + s]), cv<T>(so[1 * S + s]));
      smin = vmin(cv<T>(so[0 * S + s]), cv<T>(so[1 * S + s]));
    } else if (k == (uint32_t)L - 1) {
      smax = vmax(cv<T>(so[k * S + s]), cv<T>(so[(k - 1) * S + s]));
      smin = vmin(cv<T>(so[k * S + s]), cv<T>(so[(k - 1) * S + s]));
    } else {
      smax = vmax(vmax(cv<T>(so[(k - 1) * S + s]), cv<T>(so[k * S + s])), cv<T>(so[(k + 1) * S + s]));
      smin = vmin(vmin(cv<T>(so[(k - 1) * S + s]), cv<T>(so[k * S + s])), cv<T>(so[(k + 1) * S + s]));
    }
    // neighbour extrema (first valid neighbour seeds the running bound)
    T nmax = T(0), nmin = T(0);
    bool seen = false;
    for (int j = 0; j < n; ++j) {
      int nb = m.cellsOnCell[c * me + j];
      if (nb >= m.nCells) continue;
      T val = cv<T>(so_all[((size_t)nb * L + k) * S + s]);
      if (!seen) {
        nmax = val;
        nmin = val;
        seen = true;
      } else {
        nmax = vmax(nmax, val);
        nmin = vmin(nmin, val);
      }
    }
    if (seen) {
      smax = vmax(smax, nmax);
      smin = vmin(smin, nmin);
    }
    // vertical high-order and upwind fluxes at the interfaces below (k) and above (k+1)
    T fup_lo = T(0), fup_hi = T(0), wm_lo = T(0), wm_hi = T(0);
    if (k >= 1) {
      wm_lo = s_wm[threadIdx.x * 2 * S + s];
      fup_lo = s_wm[threadIdx.x * 2 * S + S + s];
      f.wflux[((size_t)c * (L + 1) + k) * S + s] = f64(wm_lo);
    }
    if (k + 1 < (uint32_t)L) {
      if (threadIdx.x + 1 < blockDim.x) {
        wm_hi = s_wm[(threadIdx.x + 1) * 2 * S + s];
        fup_hi = s_wm[(threadIdx.x + 1) * 2 * S + S + s];
      } else {
        T wk = cv<T>(ww[k + 1]);
        fup_hi = dt_t * (wk * cv<T>(wk >= T(0) ? so[k * S + s] : so[(k + 1) * S + s]));
        wm_hi = dt_t * wdtn_at<T>(sn, ww, k + 1, L, S, s, m.fnm, m.fnp, c3) - fup_hi;
      }
    }
    double rows = so[k * S + s] * rho_old;
    if (k + 1 < (uint32_t)L) rows = rows - f64(fup_hi * rd);
    if (k >= 1) rows = rows + f64(fup_lo * rd);
    // prev = interface below (0 at the surface), next = interface above (0 at the top)
    T prev = wm_lo, nxt = wm_hi;
    T sin_ = -rd * ((-mz(-nxt)) - mz(prev));
    T sout = -rd * (mz(nxt) - (-mz(-prev)));
    size_t o = (size_t)i * S + s;
    f.rows[o] = rows;
    f.scale_in[o] = f64(sin_);
    f.scale_out[o] = f64(sout);
    f.s_max[o] = f64(smax);
    f.s_min[o] = f64(smin);
  }
}

// per (edge, level): horizontal upwind flux and high-minus-upwind correction flux
template <typename T>
__global__ void k_mono_edges_a(mpasg_mesh m, mpasg_fields f, FastDiv fl, int S, double dt,
                               const double* __restrict__ so_all) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nEdges * L) return;
  uint32_t e = fl.div(i), k = i - e * L;
  int c1 = m.cellsOnEdge[2 * e], c2 = m.cellsOnEdge[2 * e + 1];
  const T u = cv<T>(f.ruAvg[i]);
  int up = u >= T(0) ? c1 : c2;
  const T dt_t = cv<T>(dt);
  const T dvdt = cv<T>(m.dvEdge[e]) * dt_t;
  for (int s = 0; s < S; ++s) {
    size_t o = (size_t)i * S + s;
    T fup = dvdt * (u * cv<T>(so_all[((size_t)up * L + k) * S + s]));
    f.flux_up[o] = f64(fup);
    f.flux_tmp[o] = f64(dt_t * cv<T>(f.hflux[o]) - fup);
  }
}

// per (cell, level): horizontal upwind update and scale sums, then the limiter factors
template <typename T>
__global__ void k_mono_cells_b(mpasg_mesh m, mpasg_fields f, FastDiv fl, int S) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nCells * L) return;
  uint32_t c = fl.div(i), k = i - c * L;
  const int me = m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  const T ia = cv<T>(m.invAreaCell[c]);
  const T eps = T(1.0e-20);
  const double rint = f.rho_int[i];
  for (int s = 0; s < S; ++s) {
    size_t o = (size_t)i * S + s;
    double rows = f.rows[o];
    T sin_ = cv<T>(f.scale_in[o]), sout = cv<T>(f.scale_out[o]);
    T hsum = T(0);
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      T sgn_ = cv<T>(m.edgesOnCell_sign[c * me + j]);
      T sw = sgn_ * ia;
      size_t oe = ((size_t)e * L + k) * S + s;
      hsum = hsum - cv<T>(f.flux_up[oe]) * sw;
      T sf = sgn_ * cv<T>(f.flux_tmp[oe]);
      sout = sout - mz(sf) * ia;
      sin_ = sin_ - (-mz(-sf)) * ia;
    }
    rows = rows + f64(hsum);
    const T rows_t = cv<T>(rows), rint_t = cv<T>(rint);
    T a = (cv<T>(f.s_max[o]) * rint_t - rows_t) / (sin_ + eps);
    T b = (cv<T>(f.s_min[o]) * rint_t - rows_t) / (sout - eps);
    f.rows[o] = rows;
    f.scale_in[o] = f64(vmin(vmax(a, T(0)), T(1)));
    f.scale_out[o] = f64(vmin(vmax(b, T(0)), T(1)));
  }
}

// per (edge, level): limited horizontal flux (stored in hflux)
template <typename T>
__global__ void k_mono_edges_b(mpasg_mesh m, mpasg_fields f, FastDiv fl, int S) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nEdges * L) return;
  uint32_t e = fl.div(i), k = i - e * L;
  int c1 = m.cellsOnEdge[2 * e], c2 = m.cellsOnEdge[2 * e + 1];
  for (int s = 0; s < S; ++s) {
    size_t o = (size_t)i * S + s;
    size_t o1 = ((size_t)c1 * L + k) * S + s, o2 = ((size_t)c2 * L + k) * S + s;
    T ft = cv<T>(f.flux_tmp[o]);
    T lim = ft >= T(0) ? vmin(cv<T>(f.scale_out[o1]), cv<T>(f.scale_in[o2]))
                       : vmin(cv<T>(f.scale_in[o1]), cv<T>(f.scale_out[o2]));
    f.hflux[o] = f64(ft * lim);
  }
}

// per (cell, level): apply limited horizontal and vertical fluxes, positivity
template <typename T>
__global__ void k_mono_cells_c(mpasg_mesh m, mpasg_fields f, FastDiv fl, int S, double* __restrict__ s_out) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nCells * L) return;
  uint32_t c = fl.div(i), k = i - c * L;
  const int me = m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  const T ia = cv<T>(m.invAreaCell[c]);
  const double rint = f.rho_int[i];
  const double inv_rint = fdiv<T>(1.0, rint);  // one reciprocal for every scalar of the cell-level
  const size_t oc = (size_t)c * L;
  for (int s = 0; s < S; ++s) {
    size_t o = (size_t)i * S + s;
    // limited vertical fluxes at the interfaces below (k) and above (k+1)
    T wl_lo = T(0), wl_hi = T(0);
    if (k >= 1) {
      T wm = cv<T>(f.wflux[((size_t)c * (L + 1) + k) * S + s]);
      T lim = wm >= T(0) ? vmin(cv<T>(f.scale_out[(oc + k - 1) * S + s]), cv<T>(f.scale_in[(oc + k) * S + s]))
                         : vmin(cv<T>(f.scale_out[(oc + k) * S + s]), cv<T>(f.scale_in[(oc + k - 1) * S + s]));
      wl_lo = wm * lim;
    }
    if (k + 1 < (uint32_t)L) {
      T wm = cv<T>(f.wflux[((size_t)c * (L + 1) + k + 1) * S + s]);
      T lim = wm >= T(0) ? vmin(cv<T>(f.scale_out[(oc + k) * S + s]), cv<T>(f.scale_in[(oc + k + 1) * S + s]))
                         : vmin(cv<T>(f.scale_out[(oc + k + 1) * S + s]), cv<T>(f.scale_in[(oc + k) * S + s]));
      wl_hi = wm * lim;
    }
    double rows = f.rows[o];
    T hsum = T(0);
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      T sw = cv<T>(m.edgesOnCell_sign[c * me + j]) * ia;
      hsum = hsum - cv<T>(f.hflux[((size_t)e * L + k) * S + s]) * sw;
    }
    rows = rows + f64(hsum);
    double st2 = (rows - f64(cv<T>(m.rdnw[k]) * (wl_hi - wl_lo))) * inv_rint;
    s_out[o] = st2 > 0.0 ? st2 : 0.0;
  }
}

}  // namespace

static void time_weights(int advance_density, int rk_step, int order, double* w_old, double* w_new) {
  double wn;
  if (advance_density == 0) wn = 1.0;
  else if (rk_step == 1 && order == 3) wn = 1.0 / 3.0;
  else if ((rk_step == 1 && order == 2) || rk_step == 2) wn = 1.0 / 2.0;
  else wn = 1.0;
  *w_new = wn;
  *w_old = 1.0 - wn;
}

namespace {

// Launches of the float64 form for cells of at most 6 edges (N = 6) or 8; cells with more
// take the sums' float64 loops.
template <int N>
int launch_scalars_fx(const mpasg_mesh* m, const mpasg_fields& g, const TransportScalars& p, int S, cudaStream_t s) {
  const int L = m->nVertLevels, row = L * S;
  const int rc = launch_edge_flux_fx<false>(m, S, 0.0, g.ruAvg, g.scalars_a, nullptr, g.hflux, nullptr, s);
  if (rc != MPASG_OK) return rc;
  const size_t smem = cellsum::max_cells(row) * N * sizeof(cellsum::Slot);
  return launch_rows(m->nCells, row, [&](uint32_t first, uint32_t n) {
    const size_t at = (size_t)first * row;
    k_scalars_update_fx<N><<<nblocks((long long)n * row), kBlock, smem, s>>>(
        cells_from(*m, first), cells_from(*m, g, S, first), FastDiv(row), FastDiv(S), n * row, p, g.scalars_init + at,
        g.scalars_a + at, g.scalars_b + at);
  });
}

template <int N>
int launch_scalars_mono_fx(const mpasg_mesh* m, const mpasg_fields* f, const TransportScalars& p, int S,
                           cudaStream_t s) {
  const int L = m->nVertLevels, row = L * S;
  const FastDiv fr(row), fs(S);
  const size_t smem = cellsum::max_cells(row) * N * sizeof(cellsum::Slot);
  int rc = launch_edge_flux_fx<true>(m, S, p.dt, f->ruAvg, f->scalars_a, f->scalars_init, f->flux_up, f->flux_tmp, s);
  if (rc != MPASG_OK) return rc;
  k_mono_density_fx<<<nblocks((long long)m->nCells * L), kBlock, 0, s>>>(*m, *f, FastDiv(L), p.dt);
  MPASG_LAUNCH_CHECK();
  rc = launch_rows(m->nCells, row, [&](uint32_t first, uint32_t n) {
    const size_t at = (size_t)first * row;
    k_mono_cells_a_fx<N><<<nblocks((long long)n * row), kBlock, 0, s>>>(
        cells_from(*m, first), cells_from(*m, *f, S, first), fr, fs, n * row, p, f->scalars_init, f->scalars_init + at,
        f->scalars_a + at);
  });
  if (rc != MPASG_OK) return rc;
  rc = launch_rows(m->nCells, row, [&](uint32_t first, uint32_t n) {
    k_mono_cells_b_fx<N><<<nblocks((long long)n * row), kBlock, smem, s>>>(
        cells_from(*m, first), cells_from(*m, *f, S, first), fr, fs, n * row);
  });
  if (rc != MPASG_OK) return rc;
  rc = launch_rows(m->nEdges, row, [&](uint32_t first, uint32_t n) {
    mpasg_fields g = *f;
    g.flux_tmp += (size_t)first * row;
    g.hflux += (size_t)first * row;
    k_mono_edges_b_fx<<<nblocks((long long)n * row), kBlock, 0, s>>>(edges_from(*m, first), g, fr, n * row);
  });
  if (rc != MPASG_OK) return rc;
  return launch_rows(m->nCells, row, [&](uint32_t first, uint32_t n) {
    k_mono_cells_c_fx<N><<<nblocks((long long)n * row), kBlock, smem, s>>>(
        cells_from(*m, first), cells_from(*m, *f, S, first), fr, fs, n * row, f->scalars_b + (size_t)first * row);
  });
}

// One explicit RK transport stage with the edge values (mixed form) or fluxes in `hflux` (f->hflux
// or the library-owned scratch): scalars_init, scalars_a -> scalars_b.
int launch_scalars(const mpasg_mesh* m, const mpasg_config* c, const mpasg_fields* f, double* hflux, int rk_step,
                   double dt_stage, cudaStream_t s) {
  const int L = m->nVertLevels, S = c->num_scalars;
  mpasg_fields g = *f;
  g.hflux = hflux;
  // density weights: advanced with the stage in the split transport loop; the stage's
  // new density in the coupled mode (one dynamics substep, time_integration.py:7930-8200)
  double w_old, w_new;
  time_weights(c->dynamics_split_steps > 1 ? 1 : 0, rk_step, c->time_integration_order, &w_old, &w_new);
  if (c->precision != MPASG_PRECISION_MIXED) {
    const TransportScalars p = transport_scalars(dt_stage, w_old, w_new, c->coef_3rd_order);
    return m->maxEdges <= 6 ? launch_scalars_fx<6>(m, g, p, S, s) : launch_scalars_fx<8>(m, g, p, S, s);
  }
  using T = float;
  FastDiv fl(L);
  k_pattern_c<T><<<nblocks((long long)m->nEdges * L), kBlock, 0, s>>>(*m, fl, S, g.ruAvg, g.scalars_a, hflux, 0);
  MPASG_LAUNCH_CHECK();
  k_scalars_update<T><<<nblocks((long long)m->nCells * L), kBlock, kBlock * S * sizeof(T), s>>>(
      *m, g, fl, S, dt_stage, w_old, w_new, c->coef_3rd_order, g.scalars_init, g.scalars_a, g.scalars_b);
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

int launch_scalars_mono(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f, double dt_stage,
                        cudaStream_t s) {
  const int L = m->nVertLevels, S = c->num_scalars;
  if (c->precision != MPASG_PRECISION_MIXED) {
    const TransportScalars p = transport_scalars(dt_stage, 0.0, 1.0, c->coef_3rd_order);
    return m->maxEdges <= 6 ? launch_scalars_mono_fx<6>(m, f, p, S, s) : launch_scalars_mono_fx<8>(m, f, p, S, s);
  }
  using T = float;
  FastDiv fl(L);
  const long long nel = (long long)m->nEdges * L, ncl = (long long)m->nCells * L;
  k_pattern_c<T><<<nblocks(nel), kBlock, 0, s>>>(*m, fl, S, f->ruAvg, f->scalars_a, f->hflux, 1);
  MPASG_LAUNCH_CHECK();
  k_mono_cells_a<T><<<nblocks(ncl), kBlock, kBlock * 2 * S * sizeof(T), s>>>(*m, *f, fl, S, dt_stage,
                                                                          c->coef_3rd_order, f->scalars_init,
                                                                          f->scalars_a);
  MPASG_LAUNCH_CHECK();
  k_mono_edges_a<T><<<nblocks(nel), kBlock, 0, s>>>(*m, *f, fl, S, dt_stage, f->scalars_init);
  MPASG_LAUNCH_CHECK();
  k_mono_cells_b<T><<<nblocks(ncl), kBlock, 0, s>>>(*m, *f, fl, S);
  MPASG_LAUNCH_CHECK();
  k_mono_edges_b<T><<<nblocks(nel), kBlock, 0, s>>>(*m, *f, fl, S);
  MPASG_LAUNCH_CHECK();
  k_mono_cells_c<T><<<nblocks(ncl), kBlock, 0, s>>>(*m, *f, fl, S, f->scalars_b);
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

}  // namespace

extern "C" int mpasg_advance_scalars(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f, int rk_step,
                                     double dt_stage, void* stream) {
  if (!m || !c || !f || c->num_scalars < 1 || c->num_scalars > 8) return MPASG_E_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  return launch_scalars(m, c, f, f->hflux, rk_step, dt_stage, s);
}

extern "C" int mpasg_advance_scalars_mono(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f,
                                          double dt_stage, void* stream) {
  if (!m || !c || !f || c->num_scalars < 1 || c->num_scalars > 8) return MPASG_E_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  return launch_scalars_mono(m, c, f, dt_stage, s);
}

// ---------------------------------------------------------------- library-owned scratch
// Edge values of mpasg_advance_scalars_static live here instead of in f->hflux.
static __device__ __align__(256) double g_static_hflux[MPASG_STATIC_SCRATCH_DOUBLES];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mutex;
double* g_static_ptr[kMaxDevices] = {};

// Device address of g_static_hflux on the current device, looked up once per device.
// The cached address belongs to the device's primary context: it stays valid for the life
// of the process unless that context is destroyed (cudaDeviceReset), after which a caller
// must not use this entry point on that device again.  A failed lookup clears CUDA's
// sticky last-error state, so it is not reported again by a later, unrelated launch check.
int static_scratch(double** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return MPASG_E_CUDA;
  }
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (!g_static_ptr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_static_hflux) != cudaSuccess || !p) {
      cudaGetLastError();
      return MPASG_E_CUDA;
    }
    g_static_ptr[dev] = static_cast<double*>(p);
  }
  *out = g_static_ptr[dev];
  return MPASG_OK;
}
}  // namespace

extern "C" int mpasg_advance_scalars_static(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f,
                                            int rk_step, double dt_stage, void* stream) {
  if (!m || !c || !f || c->num_scalars < 1 || c->num_scalars > 8) return MPASG_E_ARG;
  if (m->nEdges < 0 || m->nCells < 0 || m->nVertLevels < 1) return MPASG_E_ARG;
  const long long need = (long long)m->nEdges * m->nVertLevels * c->num_scalars;
  if (need > MPASG_STATIC_SCRATCH_DOUBLES) return MPASG_E_SCRATCH;
  double* scratch = nullptr;
  const int rc = static_scratch(&scratch);
  if (rc != MPASG_OK) return rc;
  cudaStream_t s = (cudaStream_t)stream;  // the caller's struct is left as it is
  return launch_scalars(m, c, f, scratch, rk_step, dt_stage, s);
}
