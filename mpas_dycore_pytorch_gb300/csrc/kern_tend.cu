// Large-step tendencies (the reference's atm_compute_dyn_tend_work,
// mpas_pytorch/dynamics/dyn_tend.py:10836, canonical composition :9390).
//
//   k_tend_cells_a   h_divergence (+ rk 1: Smagorinsky kdiff, tend_rho, dpdz)   sections :9925-9992
//   k_tend_u         u tendency: vertical transport, PV flux, KE gradient, divergence
//                    coupling (+ rk 1: pressure gradient and del2 mixing)        :9993-10315
//   k_del4_vertex / k_del4_cell / k_tend_u_finish   del4 filter and vertical mixing of u
//                    (rk 1)                                                      :10075-10315
//   k_mix_cells_a / k_mix_cells_b   w and theta del2 / del4 mixing (rk 1)       :10355, :10544
//   k_adv_edges      horizontal advective fluxes of w and theta, once per edge    :10316, :10442
//   k_tend_w_theta   w and theta flux divergence, vertical fluxes, buoyancy,
//                    diabatic term                                                :10386, :10679
//
// Kernels are templates on the stencil arithmetic type T (common.cuh), double for the float64
// form, or have a float64 version of their own (_fx, k_mix_edges_* and k_mix_cells), whose
// stencil sums run in fixed point on the integer pipes; float for the mixed form, which reads the float32 copies of the
// geometry and of u, w, rw, pv_edge (fp<T> / G) and float64 fields through cv<T>.
#include <cmath>

#include "common.cuh"
#include "advstencil.cuh"
#include "branches.cuh"
#include "cellsum.cuh"
#include "trisk.cuh"

namespace {

struct TendScalars {
  double inv_dt, c_s_len2, kdiff_cap, h_mom_visc4, h_theta_visc4, del4u_div, coef3, visc2;
  double cam_base, v_mom, v_theta;  // CAM damping base, vertical mixing coefficients (0: off)
  double ray_coef;                  // 1 / (levels * timescale): Rayleigh damping of u
  int rk_step, smag, del4;
  int ncam;   // CAM damping levels (0: off)
  int ray_n;  // Rayleigh-damped top levels of u (0: off)
  int mix_pert;  // vertical mixing of the perturbation from the initial profiles
  double f3[4];  // flux3 with coef3 by upwind side: 7 + 3 c, 7 - 3 c, 1 + c, 1 - c
  double first_dts;    // > 0: the kernel that completes tend_u also starts the acoustic substeps
  double* first_flux;  // ru_p theta of their first edge update (TendFusion)
  int smlstep;       // k_tend_w_theta also forms tend_rw
  int v_current;     // v already holds the TRiSK sum of u
  int defer;  // k_tend_u leaves tend_u_euler to k_tend_u_finish (del4 and / or vertical mixing)
};

// CAM-style damping of the top ncam levels (dyn_tend.py:3434-3456): kdiff raised to
// base * (1 - (L - (k + 1)) / ncam), base = 4 * 2.0833 * len_disp * mpas_cam_coef
MPASG_D double cam_kdiff(double kd, const TendScalars& p, uint32_t k, int L) {
  const double factor = 1.0 - (double)(L - (int)(k + 1)) / (double)p.ncam;
  return fmax(kd, p.cam_base * factor);
}

// tend_u is complete: stored, and the first acoustic substep's edge update made from it
// (k_acoustic_edges with small_step 1)
template <typename T>
MPASG_D void complete_tend_u(const mpasg_fields& f, size_t i, T tu, const TendScalars& p) {
  const double stored = f64(tu);
  f.tend_u[i] = stored;
  if (p.first_dts > 0.0) {
    // of the stored value: a float32 beyond the normal range does not come back from it as it was
    const double rup = f64(cv<T>(p.first_dts) * cv<T>(stored));
    f.ru_p[i] = rup;
    f.ruAvg[i] = rup;
    if (sizeof(T) == sizeof(double)) p.first_flux[i] = rup * f.theta_edge_save[i];
  }
}

template <typename T, bool CAM = false>
__global__ void k_tend_cells_a(mpasg_mesh m, mpasg_fields f, FastDiv fl, TendScalars p) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nCells * L) return;
  uint32_t c = fl.div(i), k = i - c * L;
  const int me = m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  // the mass-flux divergence cancels strongly: float64 in both forms
  double hdiv = 0.0;
  for (int j = 0; j < n; ++j) {
    int e = m.edgesOnCell[c * me + j];
    const double ru = f.ru[(size_t)e * L + k], sdv = m.cell_edge_sdv[c * me + j];  // sign * dvEdge
    if constexpr (sizeof(T) == sizeof(double)) {
      hdiv = fma(sdv, ru, hdiv);
    } else {
      double t = sdv * ru;
      hdiv = (j == 0) ? t : hdiv + t;
    }
  }
  hdiv = hdiv * m.invAreaCell[c];
  f.h_divergence[i] = hdiv;
  if (p.rk_step != 1) return;
  const size_t ow = (size_t)c * (L + 1) + k;
  f.tend_rho[i] = -hdiv - m.rdzw[k] * (f.rw[ow + 1] - f.rw[ow]);
  // dpdz nearly balances the vertical pressure gradient (k_tend_w_theta): float64
  double q = f.qtot[i];
  f.dpdz[i] = -kGravity * (m.rho_base[i] * q + f.rr_save[i] * (1.0 + q));
  if (p.smag) {
    const T* defc_a = G(defc_a);
    const T* defc_b = G(defc_b);
    const T* u = fp<T>(f.u, f.u_f32);
    T dd = T(0), dof = T(0);
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      T ca = defc_a[c * me + j], cb = defc_b[c * me + j];
      T ue = u[(size_t)e * L + k], ve = cv<T>(f.v[(size_t)e * L + k]);
      T ndd = (dd + ca * ue) - cb * ve;
      T ndo = (dof + cb * ue) + ca * ve;
      dd = ndd;
      dof = ndo;
    }
    double kd;
    if constexpr (sizeof(T) == sizeof(double))
      kd = fx::min_nonneg(p.c_s_len2 * sqrt(dd * dd + dof * dof), p.kdiff_cap);
    else
      kd = f64(vmin(cv<T>(p.c_s_len2) * vsqrt(dd * dd + dof * dof), cv<T>(p.kdiff_cap)));
    if (CAM && (int)k >= L - p.ncam) kd = cam_kdiff(kd, p, k, L);
    f.kdiff[i] = kd;
  } else {  // 2d_fixed: the theta del2 coefficient everywhere
    f.kdiff[i] = (CAM && (int)k >= L - p.ncam) ? cam_kdiff(p.visc2, p, k, L) : p.visc2;
  }
}

// k_tend_cells_a in float64 with the three stencil sums (mass-flux divergence, the two
// deformations) on the integer pipes: 36 of its ~60 operations a level, of which it kept the
// float64 pipe 87 % busy; 189 -> 152 us at 40962 x 55.
// Block table, a cell: 6 divergence weights, then (Smagorinsky) 12 of the deformation a u - b v
// and 12 of b u + a v.
constexpr int kDefW = 30;

template <bool CAM>
__global__ void __launch_bounds__(kBlock, 5) k_tend_cells_fx(mpasg_mesh m, mpasg_fields f, FastDiv fl, TendScalars p) {
  extern __shared__ fx::Weight s_w[];
  const uint32_t L = (uint32_t)m.nVertLevels, n_all = (uint32_t)m.nCells * L;
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t c0 = fl.div(i0), nc = fl.div(min(i0 + kBlock, n_all) - 1u) - c0 + 1;
  const bool def = p.smag && p.rk_step == 1;
  for (uint32_t t = threadIdx.x; t < nc * 6; t += kBlock) {
    const uint32_t cl = t / 6, j = t - cl * 6, c = c0 + cl;
    const size_t o = (size_t)c * m.maxEdges;
    const int n = m.nEdgesOnCell[c], e = n > 0 ? m.edgesOnCell[o + ((int)j < n ? j : 0)] : 0;
    const auto w = [&](double x) { return (int)j < n ? fx::weight(x, e) : fx::Weight{0, 0, 0u, e}; };
    const size_t q = (int)j < n ? o + j : o;
    fx::Weight* tab = s_w + cl * kDefW + j;
    tab[0] = w(m.cell_edge_sdv[q]);
    if (def) {
      const double a = m.defc_a[q], b = m.defc_b[q];
      tab[6] = w(a);
      tab[12] = w(-b);
      tab[18] = w(b);
      tab[24] = w(a);
    }
  }
  __syncthreads();
  if (i >= n_all) return;
  const uint32_t c = fl.div(i), k = i - c * L;
  const fx::Weight* w = s_w + (c - c0) * kDefW;
  const size_t o = (size_t)c * m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  double ru[6], hdiv;
#pragma unroll
  for (int j = 0; j < 6; ++j) ru[j] = f.ru[(uint32_t)w[j].row * L + k];
  if (!fx::dot<6>(ru, w, &hdiv)) {
    hdiv = 0.0;
    for (int j = 0; j < n; ++j) hdiv = fma(m.cell_edge_sdv[o + j], f.ru[(size_t)m.edgesOnCell[o + j] * L + k], hdiv);
  }
  hdiv = hdiv * m.invAreaCell[c];
  f.h_divergence[i] = hdiv;
  if (p.rk_step != 1) return;
  const size_t ow = (size_t)c * (L + 1) + k;
  f.tend_rho[i] = -hdiv - m.rdzw[k] * (f.rw[ow + 1] - f.rw[ow]);
  const double q = f.qtot[i];
  f.dpdz[i] = -kGravity * (m.rho_base[i] * q + f.rr_save[i] * (1.0 + q));
  double kd = p.visc2;  // 2d_fixed: the theta del2 coefficient everywhere
  if (p.smag) {
    double x[12];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const uint32_t e = (uint32_t)w[j].row * L + k;
      x[j] = f.u[e];
      x[6 + j] = f.v[e];
    }
    double dd, dof;
    const bool ok = fx::dot<12>(x, w + 6, &dd);
    if (!(fx::dot<12>(x, w + 18, &dof) && ok)) {
      dd = dof = 0.0;
      for (int j = 0; j < n; ++j) {
        const size_t e = (size_t)m.edgesOnCell[o + j] * L + k;
        const double a = m.defc_a[o + j], b = m.defc_b[o + j];
        dd = fma(-b, f.v[e], fma(a, f.u[e], dd));
        dof = fma(a, f.v[e], fma(b, f.u[e], dof));
      }
    }
    kd = fx::min_nonneg(p.c_s_len2 * sqrt(dd * dd + dof * dof), p.kdiff_cap);
  }
  if (CAM && (int)k >= (int)L - p.ncam) kd = cam_kdiff(kd, p, k, (int)L);
  f.kdiff[i] = kd;
}

// Rayleigh damping of u on the top ray_n levels (dyn_tend.py:2956-2990), every RK stage:
// tend_u - rho_edge u ((k + 1) - k0) / (ray_n timescale), k0 = L - ray_n
template <typename T>
MPASG_D T rayleigh_u(T tu, T rho_e, T u_k, int k, int L, const TendScalars& p) {
  const int k0 = L - p.ray_n;
  if (p.ray_n <= 0 || k < k0) return tu;
  const double damp = (((double)k + 1.0) - (double)k0) * p.ray_coef;
  return tu - rho_e * u_k * cv<T>(damp);
}

template <typename T>
MPASG_D T wduz_at(const T* __restrict__ u, T rwe, int kk, int L, const T* fzm, const T* fzp) {
  if (kk <= 0 || kk >= L) return T(0);
  if (kk == 1 || kk == L - 1) return rwe * (fzm[kk] * u[kk] + fzp[kk] * u[kk - 1]);
  return flux3<T>(u[kk - 2], u[kk - 1], u[kk], u[kk + 1], rwe, T(1));
}

// pv_edge * u at every edge level, the neighbour factor of the float64 PV flux sum (below),
// stored in ke_edge (the diagnostics' edge kinetic-energy scratch).  Inside a step the
// diagnostics form it (k_diag_edges_b); this kernel serves the first stage and the stage entry
// point
__global__ void k_pvu(mpasg_fields f, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) f.ke_edge[i] = f.pv_edge[i] * f.u[i];
}

// The mixed form's u tendency (T = float; the float64 form's is k_tend_u_fx).
// RAY: Rayleigh damping of u compiled in (a run-time test would cost work in every thread
// of the hot kernel once the compiler predicates it)
template <typename T, bool RAY = false>
__global__ void __launch_bounds__(kBlock) k_tend_u(mpasg_mesh m, mpasg_fields f, FastDiv fl, TendScalars p) {
  __shared__ T s_wd[kBlock];
  const int L = m.nVertLevels;
  const uint32_t n_all = (uint32_t)m.nEdges * L;
  const T* u = fp<T>(f.u, f.u_f32);
  const T* rw = fp<T>(f.rw, f.rw_f32);
  const T* fzm = G(fzm);
  const T* fzp = G(fzp);
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < n_all;
  uint32_t e = 0, k = 0;
  int c1 = 0, c2 = 0;
  const T* ue = u;
  T wd_k = T(0);
  if (active) {
    e = fl.div(i);
    k = i - e * L;
    c1 = m.cellsOnEdge[2 * e];
    c2 = m.cellsOnEdge[2 * e + 1];
    ue = u + (size_t)e * L;
    T rwe_k = T(0.5) * (rw[(size_t)c1 * (L + 1) + k] + rw[(size_t)c2 * (L + 1) + k]);
    wd_k = wduz_at<T>(ue, rwe_k, k, L, fzm, fzp);
  }
  s_wd[threadIdx.x] = wd_k;  // vertical flux at the interface below level k
  __syncthreads();
  if (!active) return;
  T wd_k1;
  if (k + 1 >= (uint32_t)L) {
    wd_k1 = T(0);
  } else if (threadIdx.x + 1 < blockDim.x) {
    wd_k1 = s_wd[threadIdx.x + 1];  // same edge, next level
  } else {
    T rwe_k1 = T(0.5) * (rw[(size_t)c1 * (L + 1) + k + 1] + rw[(size_t)c2 * (L + 1) + k + 1]);
    wd_k1 = wduz_at<T>(ue, rwe_k1, k + 1, L, fzm, fzp);
  }
  T tu = -G(rdzw)[k] * (wd_k1 - wd_k);
  // nonlinear Coriolis / PV flux over the TRiSK stencil, sum_j w_j u_j 0.5 (pv_self + pv_j)
  // over the slots in order, the exact power-of-two factor 0.5 applied once to the sum
  const int n2 = m.nEdgesOnEdge[e];
  const int me2 = m.maxEdges2;
  const T* pv = fp<T>(f.pv_edge, f.pv_edge_f32);
  const T* woe = G(weightsOnEdge);
  const T pv_self = pv[i];
  T q = T(0);
  for (int j = 0; j < n2; ++j) {
    int eo = m.edgesOnEdge[e * me2 + j];
    T t = (woe[e * me2 + j] * u[(size_t)eo * L + k]) * (pv_self + pv[(size_t)eo * L + k]);
    q = (j == 0) ? t : q + t;
  }
  q = T(0.5) * q;
  const size_t i1 = (size_t)c1 * L + k, i2 = (size_t)c2 * L + k;
  const T inv_dc = G(invDcEdge)[e];
  const T rho_e = cv<T>(f.h_edge[i]);
  tu = tu + rho_e * (q - dif<T>(f.ke[i2], f.ke[i1]) * inv_dc) -
       ue[k] * T(0.5) * (cv<T>(f.h_divergence[i1]) + cv<T>(f.h_divergence[i2]));
  if (RAY) tu = rayleigh_u<T>(tu, rho_e, ue[k], (int)k, L, p);
  if (p.rk_step == 1) {
    const T* zz = G(zz);
    T teu = -cv<T>(f.cqu_e[i]) * (div_or_one<T>(dif<T>(f.pressure_p[i2], f.pressure_p[i1]) * inv_dc,
                                                T(0.5) * (zz[i2] + zz[i1])) -
                                  T(0.5) * G(zxu)[i] * (cv<T>(f.dpdz[i1]) + cv<T>(f.dpdz[i2])));
    int v1 = m.verticesOnEdge[2 * e], v2 = m.verticesOnEdge[2 * e + 1];
    T r_dv = vmin(G(invDvEdge)[e], T(4) * inv_dc);
    T u_diff = (cv<T>(f.divergence[i2]) - cv<T>(f.divergence[i1])) * inv_dc -
               (cv<T>(f.vorticity[(size_t)v2 * L + k]) - cv<T>(f.vorticity[(size_t)v1 * L + k])) * r_dv;
    f.delsq_u[i] = f64(u_diff);
    T kdiffu = T(0.5) * (cv<T>(f.kdiff[i1]) + cv<T>(f.kdiff[i2]));
    teu = teu + rho_e * kdiffu * u_diff * G(meshScalingDel2)[e];
    f.tend_u_euler[i] = f64(teu);
    if (p.defer) f.tend_u[i] = f64(tu);
    else complete_tend_u(f, i, tu + teu, p);
  } else {
    complete_tend_u(f, i, tu + cv<T>(f.tend_u_euler[i]), p);
  }
}

// k_tend_u with V consecutive levels per thread (a tile of the autotuner): the edge's
// connectivity and TRiSK weights are loaded once for V levels, the V neighbour gathers
// are independent, and the interface fluxes at k0 .. k0+V are computed in-thread (the
// top one again by the next chunk).  Per level, the same expressions in the same order as
// k_tend_u; the compiler may fuse multiply-adds differently in the two kernels, so the
// tiles agree to the rounding of one FMA (last bit).  Mixed form only: k_tend_u_fx has one
// tile.
template <typename T, int V, bool RAY = false>
__global__ void __launch_bounds__(kBlock) k_tend_u_chunk(mpasg_mesh m, mpasg_fields f, FastDiv flc, int nchunk,
                                                         TendScalars p) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nEdges * (uint32_t)nchunk) return;
  const uint32_t e = flc.div(i);
  const int k0 = (int)(i - e * (uint32_t)nchunk) * V;
  const T* u = fp<T>(f.u, f.u_f32);
  const T* rw = fp<T>(f.rw, f.rw_f32);
  const T* fzm = G(fzm);
  const T* fzp = G(fzp);
  const int c1 = m.cellsOnEdge[2 * e], c2 = m.cellsOnEdge[2 * e + 1];
  const T* ue = u + (size_t)e * L;
  T wd[V + 1];
#pragma unroll
  for (int v = 0; v <= V; ++v) {
    const int kk = k0 + v;
    wd[v] = T(0);
    if (kk < L) {
      T rwe = T(0.5) * (rw[(size_t)c1 * (L + 1) + kk] + rw[(size_t)c2 * (L + 1) + kk]);
      wd[v] = wduz_at<T>(ue, rwe, kk, L, fzm, fzp);
    }
  }
  const int n2 = m.nEdgesOnEdge[e];
  const int me2 = m.maxEdges2;
  const T* pv = fp<T>(f.pv_edge, f.pv_edge_f32);
  const T* woe = G(weightsOnEdge);
  T pv_self[V], sa[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    pv_self[v] = (k0 + v < L) ? pv[(size_t)e * L + k0 + v] : T(0);
    sa[v] = T(0);
  }
  for (int j = 0; j < n2; ++j) {
    const int eo = m.edgesOnEdge[e * me2 + j];
    const T w = woe[e * me2 + j];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (k0 + v < L) {
        const size_t oo = (size_t)eo * L + k0 + v;
        const T t = (w * u[oo]) * (pv_self[v] + pv[oo]);
        sa[v] = (j == 0) ? t : sa[v] + t;
      }
    }
  }
  const T inv_dc = G(invDcEdge)[e];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int k = k0 + v;
    if (k >= L) break;
    const size_t ie = (size_t)e * L + k;
    T tu = -G(rdzw)[k] * ((k + 1 >= L ? T(0) : wd[v + 1]) - wd[v]);
    const T qv = T(0.5) * sa[v];
    const size_t i1 = (size_t)c1 * L + k, i2 = (size_t)c2 * L + k;
    const T rho_e = cv<T>(f.h_edge[ie]);
    tu = tu + rho_e * (qv - dif<T>(f.ke[i2], f.ke[i1]) * inv_dc) -
         ue[k] * T(0.5) * (cv<T>(f.h_divergence[i1]) + cv<T>(f.h_divergence[i2]));
    if (RAY) tu = rayleigh_u<T>(tu, rho_e, ue[k], k, L, p);
    if (p.rk_step == 1) {
      const T* zz = G(zz);
      T teu = -cv<T>(f.cqu_e[ie]) * (div_or_one<T>(dif<T>(f.pressure_p[i2], f.pressure_p[i1]) * inv_dc,
                                                   T(0.5) * (zz[i2] + zz[i1])) -
                                     T(0.5) * G(zxu)[ie] * (cv<T>(f.dpdz[i1]) + cv<T>(f.dpdz[i2])));
      int v1 = m.verticesOnEdge[2 * e], v2 = m.verticesOnEdge[2 * e + 1];
      T r_dv = vmin(G(invDvEdge)[e], T(4) * inv_dc);
      T u_diff = (cv<T>(f.divergence[i2]) - cv<T>(f.divergence[i1])) * inv_dc -
                 (cv<T>(f.vorticity[(size_t)v2 * L + k]) - cv<T>(f.vorticity[(size_t)v1 * L + k])) * r_dv;
      f.delsq_u[ie] = f64(u_diff);
      T kdiffu = T(0.5) * (cv<T>(f.kdiff[i1]) + cv<T>(f.kdiff[i2]));
      teu = teu + rho_e * kdiffu * u_diff * G(meshScalingDel2)[e];
      f.tend_u_euler[ie] = f64(teu);
      if (p.defer) f.tend_u[ie] = f64(tu);
      else complete_tend_u(f, ie, tu + teu, p);
    } else {
      complete_tend_u(f, ie, tu + cv<T>(f.tend_u_euler[ie]), p);
    }
  }
}

// ---------------------------------------------------------------- u tendency, float64 form
// The PV flux sums of k_tend_u on the integer pipes (fixdot.cuh): sum_j w_j u_j and
// sum_j w_j (pv u)_j over the TRiSK stencil were 20 of the ~44 float64 operations an edge level
// issued on the pipe that bounded the kernel (82 % active, 14 % of the issue slots used).
// 40962 x 55, a later RK stage: 628 us in float64, 378 us here with the first acoustic edge
// update (one of the sums in float64: 23 us more), the first stage 970 -> 434 us.  48 registers
// (5 blocks an SM): 346 us in a tuning loop against 593 us at 80 registers, 362 at 64 and 361 at
// 40, the latency of 22 warps an SM being what held the 80-register build; at 48 it spills 216
// bytes of stores and 204 of loads a thread (14 slots: 492 and 504).  The float64 pipe
// is now 74 % busy with ~21 operations an edge level, the issue slots 32 % (10242 x 41).
// The block converts the weights of the 5-7 edges it covers once, into shared memory
// (with the neighbour rows), so a term costs its thread one 16-byte broadcast and one gather.
// The upwind combination of flux3 with coefficient 1 is a three-point formula,
//   12 flux = (rw1 + rw2) (2 a + 5 b - c),  a / b downwind / upwind of the interface, c behind b,
// so the vertical flux takes 4 float64 operations instead of 11.
// N: slots a thread sums (unused slots hold zero weights); an edge with more than N
// neighbours, and a sum the fixed-point format refuses, are summed in float64.

// 12 times the vertical flux of u at interface kk; rw2 = rw1 + rw2 of the edge's two cells.  The
// second-order interfaces 1 and L-1 take the same instructions with other coefficients: as a
// branch of their own they cost nearly every warp its operations again.
MPASG_D double wduz12_at(const double* __restrict__ u, double rw2, int kk, int L, const double* fzm,
                         const double* fzp) {
  if (kk <= 0 || kk >= L) return 0.0;
  const bool low = kk == 1 || kk == L - 1, down = !low && __double2hiint(rw2) < 0;
  const double a = u[down || low ? kk - 1 : kk], b = u[down || low ? kk : kk - 1];
  const double c = low ? 0.0 : u[down ? kk + 1 : kk - 2];
  const double f = fma(low ? fzp[kk] : 2.0, a, fma(low ? fzm[kk] : 5.0, b, -c));
  return (low ? 6.0 * rw2 : rw2) * f;
}

// Per-edge constants of the u tendency, formed once per block and edge
struct EdgeConst {
  double inv_dc, inv_dc2;  // 1 / dc and 2 / dc
  double r_dv, half_ms2;   // rk 1: min(1 / dv, 4 / dc), meshScalingDel2 / 2
};

MPASG_D void load_edge_const(const mpasg_mesh& m, uint32_t e0, uint32_t n, EdgeConst* ec) {
  for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) {
    const double idc = m.invDcEdge[e0 + t];
    ec[t] = EdgeConst{idc, idc + idc, fmin(m.invDvEdge[e0 + t], 4.0 * idc), 0.5 * m.meshScalingDel2[e0 + t]};
  }
}

template <int N, bool RAY = false>
__global__ void __launch_bounds__(kBlock, 5) k_tend_u_fx(mpasg_mesh m, mpasg_fields f, FastDiv fl, TendScalars p) {
  extern __shared__ fx::Weight s_w[];
  __shared__ double s_wd[kBlock];
  const uint32_t L = (uint32_t)m.nVertLevels;
  const uint32_t n_all = (uint32_t)m.nEdges * L;
  const double* __restrict__ u = f.u;
  const double* __restrict__ rw = f.rw;
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t e0 = fl.div(i0), e1 = fl.div(min(i0 + kBlock, n_all) - 1u);
  EdgeConst* s_e = reinterpret_cast<EdgeConst*>(s_w + (e1 - e0 + 1) * N);
  trisk::load<N>(m, e0, e1 - e0 + 1, s_w);
  load_edge_const(m, e0, e1 - e0 + 1, s_e);
  const bool active = i < n_all;
  uint32_t e = e0, k = 0;
  int c1 = 0, c2 = 0;
  const double* ue = u;
  double wd_k = 0.0;
  if (active) {
    e = fl.div(i);
    k = i - e * L;
    c1 = m.cellsOnEdge[2 * e];
    c2 = m.cellsOnEdge[2 * e + 1];
    ue = u + (size_t)e * L;
    wd_k = wduz12_at(ue, rw[(size_t)c1 * (L + 1) + k] + rw[(size_t)c2 * (L + 1) + k], k, L, m.fzm, m.fzp);
  }
  s_wd[threadIdx.x] = wd_k;  // vertical flux at the interface below level k
  __syncthreads();
  if (!active) return;
  double wd_k1 = 0.0;
  if (k + 1 < L)
    wd_k1 = threadIdx.x + 1 < kBlock
                ? s_wd[threadIdx.x + 1]  // same edge, next level
                : wduz12_at(ue, rw[(size_t)c1 * (L + 1) + k + 1] + rw[(size_t)c2 * (L + 1) + k + 1], k + 1, L, m.fzm,
                            m.fzp);
  const fx::Weight* w = s_w + (e - e0) * N;
  const EdgeConst ec = s_e[e - e0];
  const double sa = p.v_current ? f.v[i] : trisk::sum<N>(m, u, w, e, k, L);
  const double sb = trisk::sum<N>(m, f.ke_edge, w, e, k, L);  // pv u
  const size_t i1 = (size_t)c1 * L + k, i2 = (size_t)c2 * L + k;
  const double rho_e = f.h_edge[i], u_k = ue[k];
  const double pv = fma(f.pv_edge[i], sa, sb);  // twice the PV flux
  // 0.5 (rho_e (pv - 2 dke / dc) - u (hdiv_1 + hdiv_2)), the exact factors of two outside
  const double g = fma(f.ke[i1] - f.ke[i2], ec.inv_dc2, pv);
  const double br = fma(rho_e, g, -(u_k * (f.h_divergence[i1] + f.h_divergence[i2])));
  double tu = fma(0.5, br, (m.rdzw[k] * kInv12) * (wd_k - wd_k1));
  if (RAY) tu = rayleigh_u<double>(tu, rho_e, u_k, (int)k, (int)L, p);
  if (p.rk_step == 1) {
    double grad = (f.pressure_p[i2] - f.pressure_p[i1]) * ec.inv_dc;
    const double z2 = m.zz[i2] + m.zz[i1];
    if (!fx::is_two(z2)) grad = grad / (0.5 * z2);
    if (!m.flatTerrain) grad = fma(-0.5 * m.zxu[i], f.dpdz[i1] + f.dpdz[i2], grad);
    const int v1 = m.verticesOnEdge[2 * e], v2 = m.verticesOnEdge[2 * e + 1];
    const double u_diff = (f.divergence[i2] - f.divergence[i1]) * ec.inv_dc -
                          (f.vorticity[(size_t)v2 * L + k] - f.vorticity[(size_t)v1 * L + k]) * ec.r_dv;
    f.delsq_u[i] = u_diff;
    const double mix = (rho_e * (f.kdiff[i1] + f.kdiff[i2])) * (u_diff * ec.half_ms2);
    const double teu = fma(-f.cqu_e[i], grad, mix);
    f.tend_u_euler[i] = teu;
    if (p.defer) f.tend_u[i] = tu;
    else complete_tend_u(f, i, tu + teu, p);
  } else {
    complete_tend_u(f, i, tu + f.tend_u_euler[i], p);
  }
}

template <bool RAY>
void launch_tend_u_fx(const mpasg_mesh* m, const mpasg_fields* f, const TendScalars& p, cudaStream_t s) {
  const int L = m->nVertLevels;
  const int nb = nblocks((long long)m->nEdges * L), ne = (kBlock - 1) / L + 2;
  if (m->maxEdges2 <= 10)
    k_tend_u_fx<10, RAY><<<nb, kBlock, ne * (10 * sizeof(fx::Weight) + sizeof(EdgeConst)), s>>>(*m, *f, FastDiv(L), p);
  else
    k_tend_u_fx<14, RAY><<<nb, kBlock, ne * (14 * sizeof(fx::Weight) + sizeof(EdgeConst)), s>>>(*m, *f, FastDiv(L), p);
}

// The del4 filter's curl and divergence of delsq_u.  In float64 the geometry is one table value a
// slot (three operations a slot otherwise, on the pipe that bounds these kernels): 40962 x 55
// 97 -> 43 us and 87 -> 43 us.
template <typename T>
__global__ void k_del4_vertex(mpasg_mesh m, mpasg_fields f, FastDiv fl) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nVertices * L) return;
  uint32_t v = fl.div(i), k = i - v * L;
  const int vd = m.vertexDegree;
  const T* iat = G(invAreaTriangle);
  const T* dc = G(dcEdge);
  const T* sg = G(edgesOnVertex_sign);
  T acc = T(0);
  if constexpr (sizeof(T) == sizeof(double)) {
    for (int j = 0; j < vd; ++j)
      acc = fma(m.vertex_edge_sdc[v * vd + j], f.delsq_u[(size_t)m.edgesOnVertex[v * vd + j] * L + k], acc);
    f.delsq_vort[i] = iat[v] * acc;
    return;
  }
  for (int j = 0; j < vd; ++j) {
    int e = m.edgesOnVertex[v * vd + j];
    T es = iat[v] * dc[e] * sg[v * vd + j];
    T t = es * cv<T>(f.delsq_u[(size_t)e * L + k]);
    acc = (j == 0) ? t : acc + t;
  }
  f.delsq_vort[i] = f64(acc);
}

template <typename T>
__global__ void k_del4_cell(mpasg_mesh m, mpasg_fields f, FastDiv fl) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nCells * L) return;
  uint32_t c = fl.div(i), k = i - c * L;
  const int me = m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  const T* ia = G(invAreaCell);
  const T* dv = G(dvEdge);
  const T* sg = G(edgesOnCell_sign);
  T acc = T(0);
  if constexpr (sizeof(T) == sizeof(double)) {
    for (int j = 0; j < n; ++j)
      acc = fma(m.cell_edge_geo[c * me + j], f.delsq_u[(size_t)m.edgesOnCell[c * me + j] * L + k], acc);
    f.delsq_div[i] = acc;
    return;
  }
  for (int j = 0; j < n; ++j) {
    int e = m.edgesOnCell[c * me + j];
    T es = ia[c] * dv[e] * sg[c * me + j];
    T t = es * cv<T>(f.delsq_u[(size_t)e * L + k]);
    acc = (j == 0) ? t : acc + t;
  }
  f.delsq_div[i] = f64(acc);
}

// rk 1 completion of the u tendency when k_tend_u deferred it: del4 filter (if enabled),
// then vertical mixing of u (dyn_tend.py:2730-2780; full state, interior levels, heights
// of the edge's interfaces as the mean of its two cells), then tend_u += tend_u_euler
// In float64 the filter's factors are formed once per block and edge: 40962 x 55 211 -> 184 us.
struct Del4Edge {
  double r_dc, r_dv;
};

template <typename T>
__global__ void __launch_bounds__(kBlock) k_tend_u_finish(mpasg_mesh m, mpasg_fields f, FastDiv fl, TendScalars p) {
  extern __shared__ Del4Edge s_d4[];
  const int L = m.nVertLevels;
  const uint32_t n_all = (uint32_t)m.nEdges * L, i0 = blockIdx.x * kBlock, e0 = fl.div(i0);
  if (sizeof(T) == sizeof(double) && p.del4) {
    const uint32_t ne = fl.div(min(i0 + kBlock, n_all) - 1u) - e0 + 1;
    for (uint32_t t = threadIdx.x; t < ne; t += kBlock) {
      const double mix = m.meshScalingDel4[e0 + t] * p.h_mom_visc4, idc = m.invDcEdge[e0 + t];
      s_d4[t] = Del4Edge{mix * p.del4u_div * idc, mix * fmin(m.invDvEdge[e0 + t], 4.0 * idc)};
    }
    __syncthreads();
  }
  uint32_t i = i0 + threadIdx.x;
  if (i >= n_all) return;
  uint32_t e = fl.div(i), k = i - e * L;
  const int c1 = m.cellsOnEdge[2 * e], c2 = m.cellsOnEdge[2 * e + 1];
  T teu = cv<T>(f.tend_u_euler[i]);
  if (p.del4) {
    const int v1 = m.verticesOnEdge[2 * e], v2 = m.verticesOnEdge[2 * e + 1];
    T r_dc4, r_dv4;
    if constexpr (sizeof(T) == sizeof(double)) {
      const Del4Edge d = s_d4[e - e0];
      r_dc4 = d.r_dc;
      r_dv4 = d.r_dv;
    } else {
      const T inv_dc = G(invDcEdge)[e];
      T u_mix = G(meshScalingDel4)[e] * cv<T>(p.h_mom_visc4);
      r_dc4 = u_mix * cv<T>(p.del4u_div) * inv_dc;
      r_dv4 = u_mix * vmin(G(invDvEdge)[e], T(4) * inv_dc);
    }
    T u_diff4 = (cv<T>(f.delsq_div[(size_t)c2 * L + k]) - cv<T>(f.delsq_div[(size_t)c1 * L + k])) * r_dc4 -
                (cv<T>(f.delsq_vort[(size_t)v2 * L + k]) - cv<T>(f.delsq_vort[(size_t)v1 * L + k])) * r_dv4;
    teu = teu - cv<T>(f.h_edge[i]) * u_diff4;
  }
  if (p.v_mom > 0.0 && k >= 1 && k + 1 < (uint32_t)L) {
    const double* z1p = m.zgrid + (size_t)c1 * (L + 1);
    const double* z2p = m.zgrid + (size_t)c2 * (L + 1);
    const double za = 0.5 * (z1p[k - 1] + z2p[k - 1]), zb = 0.5 * (z1p[k] + z2p[k]);
    const double zc = 0.5 * (z1p[k + 1] + z2p[k + 1]), zd = 0.5 * (z1p[k + 2] + z2p[k + 2]);
    const double zm = 0.5 * (za + zb), z0 = 0.5 * (zb + zc), zp = 0.5 * (zc + zd);
    const double* u = f.u + (size_t)e * L;
    double um = u[k - 1], u0 = u[k], up = u[k + 1];
    if (p.mix_pert) {  // perturbation from the initial profile along the edge normal
      const double ca = cos(m.angleEdge[e]), sa = sin(m.angleEdge[e]);
      um = um - m.u_init[k - 1] * ca - m.v_init[k - 1] * sa;
      u0 = u0 - m.u_init[k] * ca - m.v_init[k] * sa;
      up = up - m.u_init[k + 1] * ca - m.v_init[k + 1] * sa;
    }
    const T d_up = dif<T>(up, u0) / cv<T>(zp - z0);
    const T d_dn = dif<T>(u0, um) / cv<T>(z0 - zm);
    teu = teu + cv<T>(f.h_edge[i]) * cv<T>(p.v_mom) * (d_up - d_dn) / cv<T>(0.5 * (zp - zm));
  }
  f.tend_u_euler[i] = f64(teu);
  complete_tend_u(f, i, cv<T>(f.tend_u[i]) + teu, p);
}

// vertical mixing of w at interface k, 1 <= k <= L-1 (dyn_tend.py:4636-4648, rk 1)
MPASG_D double w_vmix(const mpasg_mesh& m, const mpasg_fields& f, size_t oc, size_t ow, uint32_t k, double v) {
  const double rho_half = 0.5 * (f.rho_zz[oc + k] + f.rho_zz[oc + k - 1]);
  const double w_up = (f.w[ow + k + 1] - f.w[ow + k]) * m.rdzw[k];
  const double w_down = (f.w[ow + k] - f.w[ow + k - 1]) * m.rdzw[k - 1];
  return v * rho_half * (w_up - w_down) * m.rdzu[k];
}

// vertical mixing of theta at level k, 1 <= k <= L-2 (dyn_tend.py:5064-5100, rk 1;
// Prandtl factor 1)
MPASG_D double theta_vmix(const mpasg_mesh& m, const mpasg_fields& f, uint32_t c, uint32_t k, int L, double v,
                          int mix_pert) {
  const double* zg = m.zgrid + (size_t)c * (L + 1);
  const double zm = 0.5 * (zg[k - 1] + zg[k]), z0 = 0.5 * (zg[k] + zg[k + 1]), zp = 0.5 * (zg[k + 1] + zg[k + 2]);
  const double* th = f.theta_m + (size_t)c * L;
  double tm = th[k - 1], t0 = th[k], tp = th[k + 1];
  if (mix_pert) {  // perturbation from the initial profile
    const double* ti = m.t_init + (size_t)c * L;
    tm = tm - ti[k - 1];
    t0 = t0 - ti[k];
    tp = tp - ti[k + 1];
  }
  const double diff = (tp - t0) / (zp - z0) - (t0 - tm) / (z0 - zm);
  return v * 1.0 * f.rho_zz[(size_t)c * L + k] * diff / (0.5 * (zp - zm));
}

// ---------------------------------------------------------------- w / theta mixing, float64 form
// The fluxes are formed once per edge instead of once per adjacent cell, the cells only sum
// them (cellsum.cuh):
//   k_mix_edges_a  F_w = (rho_k + rho_km1) dw dv/dc,  F_t = rho dtheta dv/dc   (flux_w_e, flux_th_e)
//   k_mix_cells    their divergences: 2 delsq_w, delsq_theta                  (del4 on only)
//   k_mix_edges_b  the del2 fluxes with the eddy viscosity, minus the del4 fluxes, in place
//   k_mix_cells    their divergences: tend_w_euler, tend_theta_euler
// 8 + 12 float64 operations an edge level and 8 a cell level and pass instead of 193 a cell level; the
// four kernels take 1.16 ms a step at 40962 x 55, the two cell kernels before them 2.44 ms.
struct MixEdge {
  double dvdc;      // dvEdge / dcEdge
  double k_w, k_t;  // meshScalingDel2 / 8 and / 2
  double d4_w, d4_t;  // meshScalingDel4 times the del4 viscosity times dv / dc
};

MPASG_D void load_mix(const mpasg_mesh& m, const TendScalars& p, uint32_t e0, uint32_t n, MixEdge* tab) {
  for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) {
    const uint32_t e = e0 + t;
    const double dvdc = m.dvEdge[e] * m.invDcEdge[e], ms2 = m.meshScalingDel2[e], ms4 = m.meshScalingDel4[e];
    tab[t] = MixEdge{dvdc, 0.125 * ms2, 0.5 * ms2, ms4 * p.h_mom_visc4 * dvdc, ms4 * p.h_theta_visc4 * dvdc};
  }
}

__global__ void __launch_bounds__(kBlock) k_mix_edges_a(mpasg_mesh m, mpasg_fields f, FastDiv fl, TendScalars p) {
  extern __shared__ MixEdge s_m[];
  const uint32_t L = (uint32_t)m.nVertLevels, n_all = (uint32_t)m.nEdges * L;
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t e0 = fl.div(i0), e1 = fl.div(min(i0 + kBlock, n_all) - 1u);
  load_mix(m, p, e0, e1 - e0 + 1, s_m);
  __syncthreads();
  if (i >= n_all) return;
  const uint32_t e = fl.div(i), k = i - e * L;
  const size_t c1 = (size_t)m.cellsOnEdge[2 * e], c2 = (size_t)m.cellsOnEdge[2 * e + 1];
  const double dvdc = s_m[e - e0].dvdc, h = f.h_edge[i];
  f.flux_th_e[i] = (h * dvdc) * (f.theta_m[c2 * L + k] - f.theta_m[c1 * L + k]);
  if (k >= 1)
    f.flux_w_e[i] = ((h + f.h_edge[i - 1]) * dvdc) * (f.w[c2 * (L + 1) + k] - f.w[c1 * (L + 1) + k]);
}

template <bool DEL4>
__global__ void __launch_bounds__(kBlock) k_mix_edges_b(mpasg_mesh m, mpasg_fields f, FastDiv fl, TendScalars p) {
  extern __shared__ MixEdge s_m[];
  __shared__ double s_k[kBlock];
  const uint32_t L = (uint32_t)m.nVertLevels, n_all = (uint32_t)m.nEdges * L;
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t e0 = fl.div(i0), e1 = fl.div(min(i0 + kBlock, n_all) - 1u);
  load_mix(m, p, e0, e1 - e0 + 1, s_m);
  uint32_t e = e0, k = 0;
  size_t c1 = 0, c2 = 0;
  double kd = 0.0;
  if (i < n_all) {
    e = fl.div(i);
    k = i - e * L;
    c1 = (size_t)m.cellsOnEdge[2 * e];
    c2 = (size_t)m.cellsOnEdge[2 * e + 1];
    kd = f.kdiff[c1 * L + k] + f.kdiff[c2 * L + k];
  }
  s_k[threadIdx.x] = kd;
  __syncthreads();
  if (i >= n_all) return;
  const MixEdge me = s_m[e - e0];
  double ft = f.flux_th_e[i] * (kd * me.k_t);
  if (DEL4) ft = fma(-me.d4_t, f.delsq_theta[c2 * L + k] - f.delsq_theta[c1 * L + k], ft);
  f.flux_th_e[i] = ft;
  if (k >= 1) {
    const double km = threadIdx.x >= 1 ? s_k[threadIdx.x - 1] : f.kdiff[c1 * L + k - 1] + f.kdiff[c2 * L + k - 1];
    double fw = f.flux_w_e[i] * ((kd + km) * me.k_w);
    // (delsq_w holds the del2 of w; at the ends of the column no w equation, the sums skip them)
    if (DEL4) fw = fma(-me.d4_w, f.delsq_w[c2 * (L + 1) + k] - f.delsq_w[c1 * (L + 1) + k], fw);
    f.flux_w_e[i] = fw;
  }
}

// divergences of flux_w_e (w levels 1..L-1, zero at the ends) and flux_th_e; `half`: the del2
// pass, whose F_w is twice the flux
template <int N>
__global__ void __launch_bounds__(kBlock, 5) k_mix_cells(mpasg_mesh m, mpasg_fields f, FastDiv fl1, int half,
                                                      double* __restrict__ div_w, double* __restrict__ div_t) {
  extern __shared__ cellsum::Slot s_c[];
  const uint32_t L = (uint32_t)m.nVertLevels, n_all = (uint32_t)m.nCells * (L + 1);
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t c0 = fl1.div(i0), c1 = fl1.div(min(i0 + kBlock, n_all) - 1u);
  cellsum::load<N>(m, c0, c1 - c0 + 1, s_c);
  __syncthreads();
  if (i >= n_all) return;
  const uint32_t c = fl1.div(i), k = i - c * (L + 1);
  const int n = m.nEdgesOnCell[c];
  const cellsum::Slot* s = s_c + (c - c0) * N;
  const double ia = m.invAreaCell[c];
  if (k < L) div_t[(size_t)c * L + k] = ia * cellsum::f64<N>(m, c, n, s, f.flux_th_e, L, k);
  double dw = 0.0;
  if (k >= 1 && k < L) {
    dw = ia * cellsum::fixed<N>(m, c, n, s, f.flux_w_e, L, k);
    if (half) dw = 0.5 * dw;
  }
  div_w[i] = dw;
}

int launch_mix_fx(const mpasg_mesh* m, const mpasg_fields* f, const TendScalars& p, cudaStream_t s) {
  const int L = m->nVertLevels;
  const int ne = nblocks((long long)m->nEdges * L), nc = nblocks((long long)m->nCells * (L + 1));
  const size_t se = cellsum::max_cells(L) * sizeof(MixEdge);
  const bool narrow = m->maxEdges <= 6, del4 = p.h_mom_visc4 > 0.0 || p.h_theta_visc4 > 0.0;
  const size_t sc = cellsum::max_cells(L + 1) * (narrow ? 6 : 8) * sizeof(cellsum::Slot);
  TendScalars q = p;
  if (!(p.h_mom_visc4 > 0.0)) q.h_mom_visc4 = 0.0;
  if (!(p.h_theta_visc4 > 0.0)) q.h_theta_visc4 = 0.0;
  auto cells = [&](int half, double* w, double* t) {
    if (narrow) k_mix_cells<6><<<nc, kBlock, sc, s>>>(*m, *f, FastDiv(L + 1), half, w, t);
    else k_mix_cells<8><<<nc, kBlock, sc, s>>>(*m, *f, FastDiv(L + 1), half, w, t);
  };
  k_mix_edges_a<<<ne, kBlock, se, s>>>(*m, *f, FastDiv(L), q);
  MPASG_LAUNCH_CHECK();
  if (del4) {
    cells(1, f->delsq_w, f->delsq_theta);
    MPASG_LAUNCH_CHECK();
    k_mix_edges_b<true><<<ne, kBlock, se, s>>>(*m, *f, FastDiv(L), q);
  } else {
    k_mix_edges_b<false><<<ne, kBlock, se, s>>>(*m, *f, FastDiv(L), q);
  }
  MPASG_LAUNCH_CHECK();
  cells(0, f->tend_w_euler, f->tend_theta_euler);
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

// w / theta del2 mixing and the del2 fields for del4 (rk 1), mixed form; index space (C, L+1)
template <typename T>
__global__ void k_mix_cells_a(mpasg_mesh m, mpasg_fields f, FastDiv fl1) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nCells * (L + 1)) return;
  uint32_t c = fl1.div(i), k = i - c * (L + 1);
  const int me = m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  const T ia = G(invAreaCell)[c];
  const T* sg = G(edgesOnCell_sign);
  const T* dv = G(dvEdge);
  const T* idc = G(invDcEdge);
  const T* msd2 = G(meshScalingDel2);
  if (k >= 1 && k < (uint32_t)L) {  // w
    const T* w = fp<T>(f.w, f.w_f32);
    T dw = T(0), tw = T(0);
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      int ec1 = m.cellsOnEdge[2 * e], ec2 = m.cellsOnEdge[2 * e + 1];
      T es = T(0.5) * ia * sg[c * me + j] * dv[e] * idc[e];
      T flux = es * (cv<T>(f.h_edge[(size_t)e * L + k]) + cv<T>(f.h_edge[(size_t)e * L + k - 1])) *
               (w[(size_t)ec2 * (L + 1) + k] - w[(size_t)ec1 * (L + 1) + k]);
      dw = dw + flux;
      flux = flux * msd2[e] * T(0.25) *
             (cv<T>(f.kdiff[(size_t)ec1 * L + k]) + cv<T>(f.kdiff[(size_t)ec2 * L + k]) +
              cv<T>(f.kdiff[(size_t)ec1 * L + k - 1]) + cv<T>(f.kdiff[(size_t)ec2 * L + k - 1]));
      tw = tw + flux;
    }
    f.delsq_w[i] = f64(dw);
    f.tend_w_euler[i] = f64(tw);
  } else {
    f.delsq_w[i] = 0.0;
    f.tend_w_euler[i] = 0.0;
  }
  if (k < (uint32_t)L) {  // theta
    const size_t o = (size_t)c * L + k;
    T dt_ = T(0), tt = T(0);
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      int ec1 = m.cellsOnEdge[2 * e], ec2 = m.cellsOnEdge[2 * e + 1];
      T es = ia * sg[c * me + j] * dv[e] * idc[e];
      T pr = T(1) * msd2[e];
      T flux = es * dif<T>(f.theta_m[(size_t)ec2 * L + k], f.theta_m[(size_t)ec1 * L + k]) *
               cv<T>(f.h_edge[(size_t)e * L + k]);
      dt_ = dt_ + flux;
      flux = flux * T(0.5) * (cv<T>(f.kdiff[(size_t)ec1 * L + k]) + cv<T>(f.kdiff[(size_t)ec2 * L + k])) * pr;
      tt = tt + flux;
    }
    f.delsq_theta[o] = f64(dt_);
    f.tend_theta_euler[o] = f64(tt);
  }
}

// del4 parts of w / theta mixing (rk 1), mixed form
template <typename T>
__global__ void k_mix_cells_b(mpasg_mesh m, mpasg_fields f, FastDiv fl1, TendScalars p) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nCells * (L + 1)) return;
  uint32_t c = fl1.div(i), k = i - c * (L + 1);
  const int me = m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  const T ia = G(invAreaCell)[c];
  const T* sg = G(edgesOnCell_sign);
  const T* dv = G(dvEdge);
  const T* idc = G(invDcEdge);
  const T* msd4 = G(meshScalingDel4);
  if (k >= 1 && k < (uint32_t)L) {
    T tw = cv<T>(f.tend_w_euler[i]);
    const T hm = cv<T>(p.h_mom_visc4) * ia;
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      int ec1 = m.cellsOnEdge[2 * e], ec2 = m.cellsOnEdge[2 * e + 1];
      T es = msd4[e] * hm * dv[e] * sg[c * me + j] * idc[e];
      tw = tw - es * (cv<T>(f.delsq_w[(size_t)ec2 * (L + 1) + k]) - cv<T>(f.delsq_w[(size_t)ec1 * (L + 1) + k]));
    }
    f.tend_w_euler[i] = f64(tw);
  }
  if (k < (uint32_t)L) {
    const size_t o = (size_t)c * L + k;
    T tt = cv<T>(f.tend_theta_euler[o]);
    const T ht = cv<T>(p.h_theta_visc4) * T(1) * ia;
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      int ec1 = m.cellsOnEdge[2 * e], ec2 = m.cellsOnEdge[2 * e + 1];
      T es = msd4[e] * ht * dv[e] * sg[c * me + j] * idc[e];
      tt = tt - es * (cv<T>(f.delsq_theta[(size_t)ec2 * L + k]) - cv<T>(f.delsq_theta[(size_t)ec1 * L + k]));
    }
    f.tend_theta_euler[o] = f64(tt);
  }
}

template <typename T>
MPASG_D T wdwz_at(const T* w, const T* rw, int kk, int L) {
  if (kk <= 0 || kk >= L) return T(0);
  if (kk == 1 || kk == L - 1) return T(0.25) * (rw[kk] + rw[kk - 1]) * (w[kk] + w[kk - 1]);
  return flux3<T>(w[kk - 2], w[kk - 1], w[kk], w[kk + 1], T(0.5) * (rw[kk] + rw[kk - 1]), T(1));
}

// vertical theta flux at interface kk: th / ths are theta_m / theta_m_save (float64 form)
// or their deviations from the reference profile (mixed form); rw_t is rw as the stencil
// type, rw / rws the float64 rw and rw_save
template <typename T>
MPASG_D T wdtz_at(const T* th, const T* ths, const T* rw_t, const double* rw, const double* rws, int kk, int L,
                  const T* fzm, const T* fzp, T coef3) {
  if (kk <= 0 || kk >= L) return T(0);
  const T fm = fzm[kk], fp = fzp[kk];
  if (kk == L - 1 && kk != 1) return cv<T>(rws[kk]) * (fm * th[kk] + fp * th[kk - 1]);
  T v;
  if (kk == 1)
    v = rw_t[kk] * (fm * th[kk] + fp * th[kk - 1]);
  else
    v = flux3<T>(th[kk - 2], th[kk - 1], th[kk], th[kk + 1], rw_t[kk], coef3);
  return v + dif<T>(rws[kk], rw[kk]) * (fm * ths[kk] + fp * ths[kk - 1]);
}

// Edge-side horizontal advective fluxes of w and theta_m, computed once per edge:
// flux_w_e[e,k] = ru_w * sum_a (adv_coefs +/- adv_coefs_3rd)_a w[advCell_a, k] (w levels 1..L-1)
// flux_th_e[e,k] = ru * sum_a (...)_a theta_m[advCell_a, k] (mass levels 0..L-1).
// The cell sums then apply edgesOnCell_sign (an exact +/-1 factor), which reproduces
// the reference's per-slot (sign * ru) * flux products bit for bit.  The mixed form
// advects the deviation theta_m - ref_theta (its reference part is added in float64 by
// k_tend_w_theta_mixed) and stores float32 fluxes.
template <typename T>
__global__ void k_adv_edges(mpasg_mesh m, mpasg_fields f, FastDiv fl) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nEdges * L) return;
  uint32_t e = fl.div(i), k = i - e * L;
  const int na = m.nAdvMax;
  const int nadv = m.nAdvCellsForEdge[e];
  const int32_t* cells = m.advCellsForEdge + (size_t)e * na;
  const T* cfp = G(adv_coefs_p) + (size_t)e * na;
  const T* cfm = G(adv_coefs_m) + (size_t)e * na;
  const T rue = cv<T>(f.ru[i]);
  {
    const T* th = fp<T>(f.theta_m, f.theta_dev);
    const T* cf = rue >= T(0) ? cfp : cfm;
    T acc = T(0);
    for (int a = 0; a < nadv; ++a) {
      T t = cf[a] * th[(size_t)cells[a] * L + k];
      acc = (a == 0) ? t : acc + t;
    }
    fpw<T>(f.flux_th_e, f.flux_th_e_f32)[i] = rue * acc;
  }
  if (k >= 1) {
    const T* w = fp<T>(f.w, f.w_f32);
    T ru_w = G(fzm)[k] * rue + G(fzp)[k] * cv<T>(f.ru[i - 1]);
    const T* cf = ru_w >= T(0) ? cfp : cfm;
    T acc = T(0);
    for (int a = 0; a < nadv; ++a) {
      T t = cf[a] * w[(size_t)cells[a] * (L + 1) + k];
      acc = (a == 0) ? t : acc + t;
    }
    fpw<T>(f.flux_w_e, f.flux_w_e_f32)[i] = ru_w * acc;
  }
}

// The float64 form: the theta sum on the integer pipes, the w sum on the float64 pipe, so
// that both are busy (two sums of ~10 terms are all this kernel does; both in float64 bound it
// at 82 % of that pipe).  40962 x 55: 374 us in float64 alone, 271 us with both sums
// on the integer side, 216 us with one each.
template <int N, bool PERT>
__global__ void __launch_bounds__(kBlock, 6) k_adv_edges_fx(mpasg_mesh m, mpasg_fields f, FastDiv fl) {
  extern __shared__ fx::Weight s_w[];
  const uint32_t L = (uint32_t)m.nVertLevels;
  const uint32_t n_all = (uint32_t)m.nEdges * L;
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t e0 = fl.div(i0), e1 = fl.div(min(i0 + kBlock, n_all) - 1u);
  adv::load<N>(m, e0, e1 - e0 + 1, s_w);
  __syncthreads();
  if (i >= n_all) return;
  const uint32_t e = fl.div(i), k = i - e * L;
  const double rue = f.ru[i];
  const bool back = __double2hiint(rue) < 0;
  const fx::Weight* w = s_w + (e - e0) * (2 * N) + (back ? N : 0);
  double x[N], th;
#pragma unroll
  for (int j = 0; j < N; ++j) x[j] = f.theta_m[(uint32_t)w[j].row * L + k];
  if (!fx::dot<N>(x, w, &th)) th = adv::sum(m, e, back, f.theta_m, L, k);
  double ft = rue * th;
  // later RK stages: the mass flux already applied, dv (ru_save - ru) theta_save, once per edge
  // (k_tend_w_theta summed it over every cell's slots: 18 operations a cell level, 9 here)
  if (PERT) ft = fma(m.dvEdge[e] * (f.ru_save[i] - rue), f.theta_edge_save[i], ft);
  f.flux_th_e[i] = ft;
  if (k >= 1) {
    const double ru_w = fma(m.fzm[k], rue, m.fzp[k] * f.ru[i - 1]);
    f.flux_w_e[i] = ru_w * adv::sum(m, e, __double2hiint(ru_w) < 0, f.w, L + 1, k);
  }
}

// Vertical fluxes of the float64 form at interface kk, the upwind combination of flux3 taken
// out (as in wduz12_at): of w (coefficient 1, times 12) and of theta (coefficient c,
//   12 flux = rw ((7 + 3c) a + (7 - 3c) b - (1 + c) a' - (1 - c) b'),  a upwind, a' behind it)
// (the second-order interfaces: the same instructions with other coefficients, as above)
MPASG_D double wdwz12_at(const double* __restrict__ w, const double* __restrict__ rw, int kk, int L) {
  if (kk <= 0 || kk >= L) return 0.0;
  const double rw2 = rw[kk] + rw[kk - 1];
  const bool low = kk == 1 || kk == L - 1, down = __double2hiint(rw2) < 0;
  const double a = w[down ? kk - 1 : kk], b = w[down ? kk : kk - 1];
  const double c = low ? 0.0 : w[down ? kk + 1 : kk - 2];
  return rw2 * fma(low ? 3.0 : 2.0, a, fma(low ? 3.0 : 5.0, b, -c));
}

MPASG_D double wdtz_fx_at(const double* __restrict__ th, const double* __restrict__ ths,
                          const double* __restrict__ rw, const double* __restrict__ rws, int kk, int L,
                          const double* fzm, const double* fzp, const TendScalars& p) {
  if (kk <= 0 || kk >= L) return 0.0;
  const double fm = fzm[kk], fp = fzp[kk], r = rw[kk], rs = rws[kk];
  const bool top = kk == L - 1 && kk != 1, low = top || kk == 1;  // top: of theta_m by rw_save alone
  const bool down = low || __double2hiint(r) < 0;
  const double a = th[down ? kk : kk - 1], b = th[down ? kk - 1 : kk];
  const double a2 = low ? 0.0 : th[down ? kk + 1 : kk - 2], b2 = low ? 0.0 : th[down ? kk - 2 : kk + 1];
  const double v = fma(low ? fm : p.f3[0], a, fma(low ? fp : p.f3[1], b, -fma(p.f3[2], a2, p.f3[3] * b2)));
  const double r12 = r * kInv12, dr = rs - r;
  return fma(top ? 0.0 : dr, fma(fm, ths[kk], fp * ths[kk - 1]), (top ? rs : low ? r : r12) * v);
}

// w and theta tendencies (float64 form); index space (C, L+1).  Bound by the float64 pipe: 89
// operations a level before (369 us at 40962 x 55), about 40 with the upwind vertical fluxes,
// the perturbation flux on the edges (k_adv_edges_fx, 216 -> 243 us for it), both divergences
// on the integer pipes and the quotient of fastdiv64.cuh (161 us, the first stage 184).
template <int N>
__global__ void __launch_bounds__(kBlock, 5) k_tend_w_theta(mpasg_mesh m, mpasg_fields f, FastDiv fl1, TendScalars p) {
  extern __shared__ cellsum::Slot s_c[];
  __shared__ double s_wd[kBlock], s_wt[kBlock];
  const uint32_t L = (uint32_t)m.nVertLevels;
  const uint32_t n_all = (uint32_t)m.nCells * (L + 1);
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t c0 = fl1.div(i0), c1 = fl1.div(min(i0 + kBlock, n_all) - 1u);
  cellsum::load<N>(m, c0, c1 - c0 + 1, s_c);
  const bool active = i < n_all;
  uint32_t c = c0, k = 0;
  double wd_k = 0.0, wt_k = 0.0;
  auto wd_at = [&](uint32_t kk) {
    const size_t ow = (size_t)c * (L + 1);
    return wdwz12_at(f.w + ow, f.rw + ow, kk, L);
  };
  auto wt_at = [&](uint32_t kk) {
    const size_t ow = (size_t)c * (L + 1), oc = (size_t)c * L;
    return wdtz_fx_at(f.theta_m + oc, f.theta_m_save + oc, f.rw + ow, f.rw_save + ow, kk, L, m.fzm, m.fzp, p);
  };
  if (active) {
    c = fl1.div(i);
    k = i - c * (L + 1);
    wd_k = wd_at(k);
    wt_k = wt_at(k);
  }
  s_wd[threadIdx.x] = wd_k;  // interface fluxes owned by this level
  s_wt[threadIdx.x] = wt_k;
  __syncthreads();
  if (!active) return;
  double wd_k1 = 0.0, wt_k1 = 0.0;
  if (k < L) {
    wd_k1 = threadIdx.x + 1 < kBlock ? s_wd[threadIdx.x + 1] : wd_at(k + 1);
    wt_k1 = threadIdx.x + 1 < kBlock ? s_wt[threadIdx.x + 1] : wt_at(k + 1);
  }
  const int n = m.nEdgesOnCell[c];
  const cellsum::Slot* s = s_c + (c - c0) * N;
  const double ia = m.invAreaCell[c];
  const size_t oc = (size_t)c * L, ow = (size_t)c * (L + 1);
  if (k >= 1 && k < L) {
    const double rdzu = m.rdzu[k];
    const double tw = fma(-ia, cellsum::fixed<N>(m, c, n, s, f.flux_w_e, L, k), (rdzu * kInv12) * (wd_k - wd_k1));
    double teu = f.tend_w_euler[i];
    if (p.rk_step == 1) {
      // vertical pressure gradient minus buoyancy: a near-hydrostatic residual
      const double res = rdzu * (f.pressure_p[oc + k] - f.pressure_p[oc + k - 1]) -
                         (m.fzm[k] * f.dpdz[oc + k] + m.fzp[k] * f.dpdz[oc + k - 1]);
      teu = teu - f.cqw[ow + k] * res;
      if (p.v_mom > 0.0) teu = teu + w_vmix(m, f, oc, ow, k, p.v_mom);
      f.tend_w_euler[i] = teu;
    }
    f.tend_w[i] = tw + teu;
    // flat terrain: the small-step w tendency has no slope fluxes
    if (p.smlstep) f.tend_rw[i] = fma(m.fzm[k], m.zz[oc + k], m.fzp[k] * m.zz[oc + k - 1]) * (tw + teu);
  } else {
    f.tend_w[i] = 0.0;
    if (p.smlstep) f.tend_rw[i] = 0.0;
  }
  if (k < L) {
    const size_t o = oc + k;
    double tt = fma(-ia, cellsum::fixed<N>(m, c, n, s, f.flux_th_e, L, k), m.rdzw[k] * (wt_k - wt_k1));
    const double rz = f.rho_zz[o];
    // unfused: the difference cancels strongly (as rounded by the reference)
    f.rthdynten[o] = fx::quotient(sub_rn(tt, mul_rn(f.tend_rho[o], f.theta_m[o])), rz);
    tt = tt + rz * f.rt_diabatic_tend[o];
    double tte = f.tend_theta_euler[o];
    if (p.rk_step == 1 && p.v_theta > 0.0 && k >= 1 && k + 1 < L) {
      tte = tte + theta_vmix(m, f, c, k, L, p.v_theta, p.mix_pert);
      f.tend_theta_euler[o] = tte;
    }
    f.tend_theta[o] = tt + tte;
  }
}

// ---------------------------------------------------------------- mixed form, theta split
// theta = ref_theta(k) + theta'.  The flux divergences of theta cancel to a few parts in
// 10^3 of their terms (theta ~ 300 K), too few digits are left in float32; the deviation
// theta' (a few K) is advected in float32 and the reference part, which reduces to
// per-level profile weights times float64 mass fluxes, is added in float64.
__global__ void k_theta_dev(mpasg_mesh m, mpasg_fields f, FastDiv fl) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nCells * L) return;
  uint32_t c = fl.div(i), k = i - c * L;
  (void)c;
  const double r = m.ref_theta[k];
  f.theta_dev[i] = d2f_bits(f.theta_m[i] - r);
  f.theta_save_dev[i] = d2f_bits(f.theta_m_save[i] - r);
}

// float64 vertical flux of the reference profile at interface kk (the reference part of
// wdtz_at: flux3 and second-order interpolations are linear in theta)
MPASG_D double ref_wflux(const mpasg_mesh& m, double rw, double rws, int kk, int L, double coef3) {
  if (kk <= 0 || kk >= L) return 0.0;
  const double w2 = m.ref_theta_w2[kk];
  if (kk == L - 1 && kk != 1) return rws * w2;
  if (kk == 1) return rw * w2 + (rws - rw) * w2;
  return rw * m.ref_theta_w4[kk] + coef3 * fabs(rw) * m.ref_theta_w3[kk] + (rws - rw) * w2;
}

__global__ void __launch_bounds__(kBlock) k_tend_w_theta_mixed(mpasg_mesh m, mpasg_fields f, FastDiv fl1,
                                                               TendScalars p) {
  using T = float;
  __shared__ T s_wd[kBlock], s_wt[kBlock];
  __shared__ double s_wr[kBlock];
  const int L = m.nVertLevels;
  const uint32_t n_all = (uint32_t)m.nCells * (L + 1);
  const T* w = f.w_f32;
  const T* rw = f.rw_f32;
  const T* fzm = m.fzm_f32;
  const T* fzp = m.fzp_f32;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < n_all;
  uint32_t c = 0, k = 0;
  T wd_k = T(0), wt_k = T(0);
  double wr_k = 0.0;
  const T coef3 = cv<T>(p.coef3);
  if (active) {
    c = fl1.div(i);
    k = i - c * (L + 1);
    const size_t ow0 = (size_t)c * (L + 1), oc0 = (size_t)c * L;
    wd_k = wdwz_at<T>(w + ow0, rw + ow0, k, L);
    wt_k = wdtz_at<T>(f.theta_dev + oc0, f.theta_save_dev + oc0, rw + ow0, f.rw + ow0, f.rw_save + ow0, k, L, fzm,
                      fzp, coef3);
    if (k < (uint32_t)L) wr_k = ref_wflux(m, f.rw[ow0 + k], f.rw_save[ow0 + k], k, L, p.coef3);
  }
  s_wd[threadIdx.x] = wd_k;
  s_wt[threadIdx.x] = wt_k;
  s_wr[threadIdx.x] = wr_k;
  __syncthreads();
  if (!active) return;
  T wd_k1 = T(0), wt_k1 = T(0);
  double wr_k1 = 0.0;
  if (k < (uint32_t)L) {
    if (threadIdx.x + 1 < blockDim.x) {
      wd_k1 = s_wd[threadIdx.x + 1];
      wt_k1 = s_wt[threadIdx.x + 1];
      wr_k1 = s_wr[threadIdx.x + 1];
    } else {
      const size_t ow0 = (size_t)c * (L + 1), oc0 = (size_t)c * L;
      wd_k1 = wdwz_at<T>(w + ow0, rw + ow0, k + 1, L);
      wt_k1 = wdtz_at<T>(f.theta_dev + oc0, f.theta_save_dev + oc0, rw + ow0, f.rw + ow0, f.rw_save + ow0, k + 1,
                         L, fzm, fzp, coef3);
      wr_k1 = ref_wflux(m, f.rw[ow0 + k + 1], f.rw_save[ow0 + k + 1], k + 1, L, p.coef3);
    }
  }
  const int me = m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  const T ia = m.invAreaCell_f32[c];
  const T* sg = m.edgesOnCell_sign_f32;
  const size_t oc = (size_t)c * L;
  const size_t ow = (size_t)c * (L + 1);
  if (k >= 1 && k < (uint32_t)L) {
    T tw = T(0);
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      tw = tw - sg[c * me + j] * f.flux_w_e_f32[(size_t)e * L + k];
    }
    tw = tw * ia - m.rdzu_f32[k] * (wd_k1 - wd_k);
    T teu = cv<T>(f.tend_w_euler[i]);
    if (p.rk_step == 1) {
      const double res = m.rdzu[k] * (f.pressure_p[oc + k] - f.pressure_p[oc + k - 1]) -
                         (m.fzm[k] * f.dpdz[oc + k] + m.fzp[k] * f.dpdz[oc + k - 1]);
      teu = teu - cv<T>(f.cqw[ow + k]) * cv<T>(res);
      if (p.v_mom > 0.0) teu = teu + cv<T>(w_vmix(m, f, oc, ow, k, p.v_mom));
      f.tend_w_euler[i] = f64(teu);
    }
    const double w_tend = f64(tw + teu);
    f.tend_w[i] = w_tend;
    if (p.smlstep) {  // as k_smlstep_pert over flat terrain
      const T fzm_t = cv<T>(m.fzm[k]), fzp_t = cv<T>(m.fzp[k]);
      f.tend_rw[i] = f64((fzm_t * cv<T>(m.zz[oc + k]) + fzp_t * cv<T>(m.zz[oc + k - 1])) * cv<T>(w_tend));
    }
  } else {
    f.tend_w[i] = 0.0;
    if (p.smlstep) f.tend_rw[i] = 0.0;
  }
  if (k < (uint32_t)L) {
    const size_t o = oc + k;
    const double rt = m.ref_theta[k];
    T tt = T(0);
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      T x = -(sg[c * me + j] * f.flux_th_e_f32[(size_t)e * L + k]);
      tt = (j == 0) ? x : tt + x;
    }
    // reference part of the horizontal flux divergence: the adv_coefs of an edge sum to
    // its dvEdge (to 1e-11), so it is ref_theta times the float64 mass-flux divergence
    double tmean = -rt * f.h_divergence[o];
    if (p.rk_step > 1) {
      double dsum = 0.0;
      for (int j = 0; j < n; ++j) {
        int e = m.edgesOnCell[c * me + j];
        int ec1 = m.cellsOnEdge[2 * e], ec2 = m.cellsOnEdge[2 * e + 1];
        const double wgt = m.cell_edge_sdv[c * me + j];  // sign * dvEdge (mesh table)
        const double dru = f.ru_save[(size_t)e * L + k] - f.ru[(size_t)e * L + k];
        dsum = dsum + wgt * dru;
        T flux = cv<T>(wgt) * cv<T>(dru) * T(0.5) *
                 (f.theta_save_dev[(size_t)ec2 * L + k] + f.theta_save_dev[(size_t)ec1 * L + k]);
        tt = tt - flux;
      }
      tmean = tmean - rt * dsum * m.invAreaCell[c];
    }
    tt = tt * ia - m.rdzw_f32[k] * (wt_k1 - wt_k);
    tmean = tmean - m.rdzw[k] * (wr_k1 - wr_k);
    const double ttot = f64(tt) + tmean;
    const double rz = f.rho_zz[o];
    // (a diagnostic for physics coupling: the cancelling difference in float64, the
    // quotient in float32)
    f.rthdynten[o] = f64(cv<T>(ttot - f.tend_rho[o] * f.theta_m[o]) / cv<T>(rz));
    double tte = f.tend_theta_euler[o];
    if (p.rk_step == 1 && p.v_theta > 0.0 && k >= 1 && k + 1 < (uint32_t)L) {
      tte = tte + theta_vmix(m, f, c, k, L, p.v_theta, p.mix_pert);
      f.tend_theta_euler[o] = tte;
    }
    f.tend_theta[o] = ttot + rz * f.rt_diabatic_tend[o] + tte;
  }
}

MPASG_HD int tile_levels(int code) { return code == 2 ? 2 : code == 4 ? 4 : 1; }

template <typename T>
int launch_dyn_tend(const mpasg_mesh* m, mpasg_fields* f, const TendScalars& p, int rk_step, cudaStream_t s,
                    int c_tile, bool hdiv_current) {
  const int L = m->nVertLevels;
  const long long ncl = (long long)m->nCells * L, nel = (long long)m->nEdges * L;
  const long long ncw = (long long)m->nCells * (L + 1), nvl = (long long)m->nVertices * L;
  FastDiv fl(L), fl1(L + 1);
  if (rk_step == 1 || !hdiv_current) {
    const bool cam = p.ncam > 0 && rk_step == 1;
    if (sizeof(T) == sizeof(double) && m->maxEdges <= 6) {
      const size_t sd = cellsum::max_cells(L) * kDefW * sizeof(fx::Weight);
      if (cam) k_tend_cells_fx<true><<<nblocks(ncl), kBlock, sd, s>>>(*m, *f, fl, p);
      else k_tend_cells_fx<false><<<nblocks(ncl), kBlock, sd, s>>>(*m, *f, fl, p);
    } else if (cam) {
      k_tend_cells_a<T, true><<<nblocks(ncl), kBlock, 0, s>>>(*m, *f, fl, p);
    } else {
      k_tend_cells_a<T><<<nblocks(ncl), kBlock, 0, s>>>(*m, *f, fl, p);
    }
    MPASG_LAUNCH_CHECK();
  }
  GraphBranches branches(s);  // u beside w and theta
  const bool ray = p.ray_n > 0;
  if constexpr (sizeof(T) == sizeof(double)) {
    if (ray) launch_tend_u_fx<true>(m, f, p, s);
    else launch_tend_u_fx<false>(m, f, p, s);
  } else {
    const int vt = tile_levels(c_tile);  // levels per thread of k_tend_u (autotuner choice)
    const int nchunk = (L + vt - 1) / vt;
    const long long nth = (long long)m->nEdges * nchunk;
    if (vt == 1) {
      if (ray) k_tend_u<T, true><<<nblocks(nel), kBlock, 0, s>>>(*m, *f, fl, p);
      else k_tend_u<T><<<nblocks(nel), kBlock, 0, s>>>(*m, *f, fl, p);
    } else if (vt == 2) {
      if (ray) k_tend_u_chunk<T, 2, true><<<nblocks(nth), kBlock, 0, s>>>(*m, *f, FastDiv(nchunk), nchunk, p);
      else k_tend_u_chunk<T, 2><<<nblocks(nth), kBlock, 0, s>>>(*m, *f, FastDiv(nchunk), nchunk, p);
    } else {
      if (ray) k_tend_u_chunk<T, 4, true><<<nblocks(nth), kBlock, 0, s>>>(*m, *f, FastDiv(nchunk), nchunk, p);
      else k_tend_u_chunk<T, 4><<<nblocks(nth), kBlock, 0, s>>>(*m, *f, FastDiv(nchunk), nchunk, p);
    }
  }
  MPASG_LAUNCH_CHECK();
  if (rk_step == 1) {
    if (p.del4) {
      k_del4_vertex<T><<<nblocks(nvl), kBlock, 0, s>>>(*m, *f, fl);
      MPASG_LAUNCH_CHECK();
      k_del4_cell<T><<<nblocks(ncl), kBlock, 0, s>>>(*m, *f, fl);
      MPASG_LAUNCH_CHECK();
    }
    if (p.defer) {
      const size_t sd = sizeof(T) == sizeof(double) ? cellsum::max_cells(L) * sizeof(Del4Edge) : 0;
      k_tend_u_finish<T><<<nblocks(nel), kBlock, sd, s>>>(*m, *f, fl, p);
      MPASG_LAUNCH_CHECK();
    }
  }
  if (const int rc = branches.next(); rc != MPASG_OK) return rc;
  if (sizeof(T) != sizeof(double)) {
    k_theta_dev<<<nblocks(ncl), kBlock, 0, s>>>(*m, *f, fl);
    MPASG_LAUNCH_CHECK();
  }
  if (rk_step == 1) {
    if constexpr (sizeof(T) == sizeof(double)) {
      const int rc = launch_mix_fx(m, f, p, s);
      if (rc != MPASG_OK) return rc;
    } else {
      k_mix_cells_a<T><<<nblocks(ncw), kBlock, 0, s>>>(*m, *f, fl1);
      MPASG_LAUNCH_CHECK();
      if (p.h_mom_visc4 > 0.0 || p.h_theta_visc4 > 0.0) {
        TendScalars q = p;
        if (!(p.h_mom_visc4 > 0.0)) q.h_mom_visc4 = 0.0;
        k_mix_cells_b<T><<<nblocks(ncw), kBlock, 0, s>>>(*m, *f, fl1, q);
        MPASG_LAUNCH_CHECK();
      }
    }
  }
  if constexpr (sizeof(T) == sizeof(double)) {
    const size_t smem = (size_t)((kBlock - 1) / L + 2) * adv::kEntryBytes;
    const int nb = nblocks(nel);
    const bool narrow = m->nAdvMax <= 10, pert = rk_step > 1;
    if (narrow && pert) k_adv_edges_fx<10, true><<<nb, kBlock, smem * 10, s>>>(*m, *f, fl);
    else if (narrow) k_adv_edges_fx<10, false><<<nb, kBlock, smem * 10, s>>>(*m, *f, fl);
    else if (pert) k_adv_edges_fx<14, true><<<nb, kBlock, smem * 14, s>>>(*m, *f, fl);
    else k_adv_edges_fx<14, false><<<nb, kBlock, smem * 14, s>>>(*m, *f, fl);
  } else {
    k_adv_edges<T><<<nblocks(nel), kBlock, 0, s>>>(*m, *f, fl);
  }
  MPASG_LAUNCH_CHECK();
  if (sizeof(T) == sizeof(double)) {
    const size_t sc = cellsum::max_cells(L + 1) * sizeof(cellsum::Slot);
    if (m->maxEdges <= 6) k_tend_w_theta<6><<<nblocks(ncw), kBlock, sc * 6, s>>>(*m, *f, fl1, p);
    else k_tend_w_theta<8><<<nblocks(ncw), kBlock, sc * 8, s>>>(*m, *f, fl1, p);
  } else
    k_tend_w_theta_mixed<<<nblocks(ncw), kBlock, 0, s>>>(*m, *f, fl1, p);
  MPASG_LAUNCH_CHECK();
  return branches.join();
}

}  // namespace

int mpasgi_theta_dev(const mpasg_mesh* m, mpasg_fields* f, cudaStream_t s) {
  const int L = m->nVertLevels;
  k_theta_dev<<<nblocks((long long)m->nCells * L), kBlock, 0, s>>>(*m, *f, FastDiv(L));
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

int mpasgi_pvu(const mpasg_mesh* m, mpasg_fields* f, cudaStream_t s) {
  const long long n = (long long)m->nEdges * m->nVertLevels;
  k_pvu<<<nblocks(n), kBlock, 0, s>>>(*f, n);
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

extern "C" int mpasg_dyn_tend(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f, int rk_step,
                              void* stream) {
  return mpasgi_dyn_tend(m, c, f, rk_step, (cudaStream_t)stream, false);
}

int mpasgi_dyn_tend(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f, int rk_step, cudaStream_t s,
                    bool copies_current, const TendFusion& fuse) {
  if (!m || !c || !f || rk_step < 1 || rk_step > 3) return MPASG_E_ARG;
  if (!copies_current && c->precision != MPASG_PRECISION_MIXED) {
    int rc = mpasgi_pvu(m, f, s);
    if (rc == MPASG_OK && rk_step > 1) rc = mpasgi_theta_edge(m, f, false, s);  // the edge mean of theta_m_save
    if (rc != MPASG_OK) return rc;
  }
  if (m->nVertLevels < 4) return MPASG_E_ARG;
  if (c->precision != MPASG_PRECISION_FLOAT64 && c->precision != MPASG_PRECISION_MIXED) return MPASG_E_ARG;
  TendScalars p;
  p.inv_dt = 1.0 / c->dt;
  double cl = c->c_s * c->len_disp;
  p.c_s_len2 = cl * cl;
  p.kdiff_cap = (0.01 * (c->len_disp * c->len_disp)) * p.inv_dt;
  p.smag = c->horiz_mixing_smagorinsky;
  if (p.smag) {
    p.h_mom_visc4 = c->visc4_2dsmag * std::pow(c->len_disp, 3.0);  // correctly rounded, as len**3
    p.h_theta_visc4 = p.h_mom_visc4;
  } else {
    p.h_mom_visc4 = c->h_mom_eddy_visc4;
    p.h_theta_visc4 = c->h_theta_eddy_visc4;
  }
  p.visc2 = p.smag ? 0.0 : c->h_theta_eddy_visc2;
  p.del4u_div = c->del4u_div_factor;
  p.coef3 = c->coef_3rd_order;
  p.f3[0] = 7.0 + 3.0 * p.coef3;
  p.f3[1] = 7.0 - 3.0 * p.coef3;
  p.f3[2] = 1.0 + p.coef3;
  p.f3[3] = 1.0 - p.coef3;
  p.rk_step = rk_step;
  p.first_dts = fuse.first_dts;
  p.first_flux = fuse.first_flux;
  p.smlstep = fuse.smlstep ? 1 : 0;
  p.v_current = fuse.v_current ? 1 : 0;
  p.del4 = (p.h_mom_visc4 > 0.0) ? 1 : 0;
  if (c->number_cam_damping_levels > m->nVertLevels) return MPASG_E_ARG;
  p.ncam = (c->mpas_cam_coef > 0.0 && c->number_cam_damping_levels > 0) ? c->number_cam_damping_levels : 0;
  p.cam_base = 4.0 * 2.0833 * c->len_disp * c->mpas_cam_coef;
  p.v_mom = c->v_mom_eddy_visc2 > 0.0 ? c->v_mom_eddy_visc2 : 0.0;
  p.v_theta = c->v_theta_eddy_visc2 > 0.0 ? c->v_theta_eddy_visc2 : 0.0;
  p.defer = (p.del4 || p.v_mom > 0.0) ? 1 : 0;
  if (p.v_mom > 0.0 || p.v_theta > 0.0) {
    if (!m->zgrid) return MPASG_E_ARG;
  }
  p.mix_pert = c->mix_perturbation ? 1 : 0;
  if (p.mix_pert && (p.v_mom > 0.0 || p.v_theta > 0.0) && (!m->u_init || !m->v_init || !m->angleEdge || !m->t_init))
    return MPASG_E_ARG;
  p.ray_n = c->rayleigh_damp_u_levels;
  if (p.ray_n > m->nVertLevels || p.ray_n < 0) return MPASG_E_ARG;
  p.ray_coef = p.ray_n > 0 ? 1.0 / ((double)p.ray_n * (c->rayleigh_damp_u_timescale_days * 86400.0)) : 0.0;
  if (c->precision == MPASG_PRECISION_MIXED) {
    if (!copies_current) {
      const int rc = mpasgi_pack_f32(m, f, s);
      if (rc != MPASG_OK) return rc;
    }
    return launch_dyn_tend<float>(m, f, p, rk_step, s, c->tile_tend_u, fuse.hdiv_current);
  }
  return launch_dyn_tend<double>(m, f, p, rk_step, s, c->tile_tend_u, fuse.hdiv_current);
}

// Autotuner: times the u-tendency kernel with 1, 2 and 4 levels per thread on the current
// state (rk-2 form, 3 launches each after one warm-up) and keeps the fastest in
// c->tile_tend_u.  The float64 form has one tile: it is timed once and kept, its time reported
// for all three.  Host-synchronising: call it outside stream capture.  The kernels only write
// their outputs (tend_u, ...) and the ke_edge scratch, so the state is unchanged.
extern "C" int mpasg_autotune(const mpasg_mesh* m, mpasg_config* c, mpasg_fields* f, float* times_ms,
                              void* stream) {
  if (!m || !c || !f) return MPASG_E_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const bool mixed = c->precision == MPASG_PRECISION_MIXED;
  if (mixed) {
    const int rc = mpasgi_pack_f32(m, f, s);
    if (rc != MPASG_OK) return rc;
  }
  TendScalars p{};
  p.rk_step = 2;
  p.coef3 = c->coef_3rd_order;
  const int L = m->nVertLevels;
  const long long nel = (long long)m->nEdges * L;
  cudaEvent_t a, b;
  if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) return MPASG_E_CUDA;
  if (!mixed) {
    k_pvu<<<nblocks(nel), kBlock, 0, s>>>(*f, nel);
    mpasg_count_launch();
    if (cudaGetLastError() != cudaSuccess) return MPASG_E_LAUNCH;
  }
  const int tiles[3] = {1, 2, 4};
  float best = 1e30f;
  int best_tile = 1;
  int rc = MPASG_OK;
  for (int t = 0; t < 3 && rc == MPASG_OK; ++t) {
    if (!mixed && t > 0) {
      if (times_ms) times_ms[t] = times_ms[0];
      continue;
    }
    const int vt = tiles[t];
    const int nchunk = (L + vt - 1) / vt;
    const long long nth = (long long)m->nEdges * nchunk;
    float ms = 0.0f;
    for (int rep = 0; rep < 4; ++rep) {
      if (rep == 1) cudaEventRecord(a, s);
      if (!mixed) launch_tend_u_fx<false>(m, f, p, s);
      else if (vt == 1) k_tend_u<float><<<nblocks(nel), kBlock, 0, s>>>(*m, *f, FastDiv(L), p);
      else if (vt == 2) k_tend_u_chunk<float, 2><<<nblocks(nth), kBlock, 0, s>>>(*m, *f, FastDiv(nchunk), nchunk, p);
      else k_tend_u_chunk<float, 4><<<nblocks(nth), kBlock, 0, s>>>(*m, *f, FastDiv(nchunk), nchunk, p);
      mpasg_count_launch();
      if (cudaGetLastError() != cudaSuccess) rc = MPASG_E_LAUNCH;
    }
    cudaEventRecord(b, s);
    if (cudaEventSynchronize(b) != cudaSuccess || cudaEventElapsedTime(&ms, a, b) != cudaSuccess) rc = MPASG_E_CUDA;
    ms /= 3.0f;
    if (times_ms) times_ms[t] = ms;
    if (rc == MPASG_OK && ms < best) {
      best = ms;
      best_tile = vt;
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (rc == MPASG_OK) c->tile_tend_u = best_tile;
  return rc;
}
