// Column-oriented stages: moist coefficients, vertical implicit coefficients, the
// acoustic substep (edge pressure-gradient update + per-column implicit solve),
// divergence damping, small-step perturbation and large-step recovery.
//
// Each kernel restates the reference stage's float64 arithmetic in the same operation
// order (mpas_pytorch/dynamics/*.py, cited per kernel); slot sums run in connectivity
// slot order, left to right, so results are deterministic and need no atomics.
#include "common.cuh"
#include "columns.cuh"
#include "pow_exner_fx.cuh"

namespace {

// ---------------------------------------------------------------- moist coefficients
// dynamics/moist_coefficients.py:124
__global__ void k_moist_cells(int nc, int L, int S, int ms, int me, const double* __restrict__ sc,
                              double* __restrict__ qtot, double* __restrict__ cqw) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  double qprev = 0.0;
  for (int k = 0; k < L; ++k) {
    double q = 0.0;
    for (int s = ms - 1; s < me; ++s) q = q + sc[((size_t)c * L + k) * S + s];
    qtot[(size_t)c * L + k] = q;
    double w;
    if (k == 0) w = 0.0;
    else w = (me >= ms) ? 1.0 / (1.0 + 0.5 * (q + qprev)) : 1.0;
    cqw[(size_t)c * (L + 1) + k] = w;
    qprev = q;
  }
  cqw[(size_t)c * (L + 1) + L] = 0.0;
}

__global__ void k_moist_edges(int ne, int L, FastDiv fl, int ms, int me, const int32_t* __restrict__ coe,
                              const double* __restrict__ qtot, double* __restrict__ cqu) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)ne * L) return;
  uint32_t e = fl.div(i), k = i - e * L;
  if (me >= ms) {
    int c1 = coe[2 * e], c2 = coe[2 * e + 1];
    cqu[i] = 1.0 / (1.0 + 0.5 * (qtot[(size_t)c1 * L + k] + qtot[(size_t)c2 * L + k]));
  } else {
    cqu[i] = 1.0;
  }
}

// ---------------------------------------------------------------- vertical implicit coefficients
// dynamics/vert_imp_coefs.py:188 (coefficients :343-446, Thomas factor :100-121).
// k_vimp_columns builds every level's coefficients and tridiagonal diagonals in parallel
// and runs the sequential Thomas factorisation, one thread per column, on columns held in
// shared memory; k_vimp_coefs and k_vimp_factor do the same through memory for columns
// too high for it.
struct VimpLevel {
  double cofwt, coftz;
};

// Products of the stage's scalars, formed once on the host (a thread would spend float64
// operations on each): the reference's leading factors in its own association.
struct VimpScalars {
  double dtseps;  // 0.5 dts (1 + epssm)
  double cw;      // 0.5 dtseps R/cv
  double cg;      // 0.5 dtseps g
  double c2;      // dtseps cp R/cv
  double cm;      // mixed form: dtseps (0.5 R/cv g)
  double cwg;     // cw g
};
inline VimpScalars vimp_scalars(double dts, double epssm) {
  const double rcv = kRgas / (kCp - kRgas);
  VimpScalars p;
  p.dtseps = 0.5 * dts * (1.0 + epssm);
  p.cw = 0.5 * p.dtseps * rcv;
  p.cg = 0.5 * p.dtseps * kGravity;
  p.c2 = p.dtseps * (kCp * rcv);
  p.cm = p.dtseps * (0.5 * rcv * kGravity);
  p.cwg = p.cw * kGravity;
  return p;
}

// (float64 in both forms; T selects the division: the rounded quotient in the float64 form,
// Newton reciprocal in the mixed form)
template <typename T>
MPASG_D VimpLevel vimp_level(const mpasg_mesh& m, const mpasg_fields& f, size_t o, int k, const VimpScalars& s) {
  VimpLevel v;
  double zz = m.zz[o + k], p = f.exner[o + k];
  double rb = m.rho_base[o + k], rtb = f.rtheta_base[o + k], pb = f.exner_base[o + k];
  double rt = f.rtheta_p[o + k], q = f.qtot[o + k];
  const bool dry = fx::is_zero(q);  // x / (1 + q) is x itself: the division is skipped, not changed
  if (sizeof(T) == sizeof(double)) {
    const double x = (fx::is_one(zz) ? s.cwg : s.cw * zz * kGravity) * rb;
    v.cofwt = fdiv<T>((dry ? x : fdiv<T>(x, 1.0 + q)) * p, (rtb + rt) * pb);
  } else {  // constants folded into one factor
    const double x = s.cm * zz * rb;
    v.cofwt = (dry ? x : fdiv<T>(x, 1.0 + q)) * p * rcp_nr((rtb + rt) * pb);
  }
  v.coftz = (k == 0) ? 0.0 : s.dtseps * (m.fzm[k] * f.theta_m[o + k] + m.fzp[k] * f.theta_m[o + k - 1]);
  return v;
}

// An inner level's cofwr and cofwz and its row of the tridiagonal matrix, from the level
// itself and its neighbours below (lo) and above (coftz only).
struct VimpRow {
  double a, b, c;
};

// What depends on the level alone, for a level over flat terrain (zz exactly 1 here and
// below): the values the expressions of vimp_row round to, formed once per block.
struct VimpFlat {
  double rz, rz_lo, drz;  // dts (1 + epssm) / 2 rdzw at k and k-1, and their difference
  double cofwr, cz, sum;  // cg z, c2 z rdzu, rdzw_k + rdzw_km1
};
MPASG_D VimpFlat vimp_flat(const mpasg_mesh& m, uint32_t k, const VimpScalars& s) {
  VimpFlat t;
  const double z = m.fzm[k] + m.fzp[k], rz = m.rdzw[k], rzm = m.rdzw[k - 1];
  t.rz = s.dtseps * rz;
  t.rz_lo = s.dtseps * rzm;
  t.drz = t.rz - t.rz_lo;
  t.cofwr = s.cg * z;
  t.cz = s.c2 * z * m.rdzu[k];
  t.sum = rz + rzm;
  return t;
}

template <typename T>
MPASG_D VimpRow vimp_row(const mpasg_mesh& m, const mpasg_fields& f, size_t o, size_t ow, uint32_t k,
                         const VimpLevel& at, const VimpLevel& lo, double ct_kp1, const VimpScalars& s,
                         const VimpFlat* flat = nullptr) {
  const double zz = m.zz[o + k], zzm = m.zz[o + k - 1];
  const double fzm = m.fzm[k], fzp = m.fzp[k];
  const double p_i = fzm * f.exner[o + k] + fzp * f.exner[o + k - 1];
  const double ct_km1 = lo.coftz, ct_k = at.coftz;
  const double cw_k = at.cofwt, cw_km1 = lo.cofwt;
  const double rdzw_k = m.rdzw[k], rdzw_km1 = m.rdzw[k - 1];
  // the reference's coefficients (vert_imp_coefs.py:388-428) with their common factors taken out
  const double tm = ct_km1 * rdzw_km1, tp = ct_kp1 * rdzw_k;
  VimpRow r;
  if constexpr (sizeof(T) == sizeof(double)) {
    const bool one = flat && fx::is_one(zz) && fx::is_one(zzm);
    VimpFlat t;
    if (one) {
      t = flat[k];
    } else {
      const double z_i = fma(fzm, zz, fzp * zzm);
      t.rz = s.dtseps * rdzw_k;
      t.rz_lo = s.dtseps * rdzw_km1;
      t.drz = t.rz - t.rz_lo;
      t.cofwr = s.cg * z_i;
      t.cz = s.c2 * z_i * m.rdzu[k];
      t.sum = fma(rdzw_k, zz, rdzw_km1 * zzm);
    }
    const double cqw = f.cqw[ow + k];
    const double cofwz = (fx::is_one(cqw) ? t.cz : t.cz * cqw) * p_i;
    f.cofwr[o + k] = t.cofwr;
    f.cofwz[o + k] = cofwz;
    const double wlo = one ? cofwz + cw_km1 : fma(cofwz, zzm, cw_km1), wk = one ? cofwz : cofwz * zz;
    r.a = fma(t.cofwr, t.rz_lo, -(tm * wlo));
    r.b = fma(t.cofwr, t.drz, fma(ct_k, fma(cofwz, t.sum, -fma(cw_k, rdzw_k, -(cw_km1 * rdzw_km1))), 1.0));
    r.c = fma(cw_k, tp, -fma(wk, tp, t.cofwr * t.rz));
  } else {
    const double z_i = fzm * zz + fzp * zzm;
    const double cofwr = s.cg * z_i;
    const double cofwz = s.c2 * z_i * m.rdzu[k] * f.cqw[ow + k] * p_i;
    f.cofwr[o + k] = cofwr;
    f.cofwz[o + k] = cofwz;
    const double cofrz_k = s.dtseps * rdzw_k, cofrz_km1 = s.dtseps * rdzw_km1;
    r.a = cofwr * cofrz_km1 - tm * (cofwz * zzm + cw_km1);
    r.b = 1.0 + ct_k * (cofwz * (rdzw_k * zz + rdzw_km1 * zzm) - (cw_k * rdzw_k - cw_km1 * rdzw_km1)) +
          cofwr * (cofrz_k - cofrz_km1);
    r.c = tp * (cw_k - cofwz * zz) - cofwr * cofrz_k;
  }
  return r;
}

// Bound by the float64 pipe: 63 operations a level with two divisions in the reference's
// expressions, 40 with the scalars' products formed on the host, the quotient of
// fastdiv64.cuh and the common factors taken out of the diagonals (fewer roundings each):
// 263 -> 193 us at 40962 x 55 before the factorisation joined it (k_vimp_columns).
template <typename T>
__global__ void __launch_bounds__(kBlock) k_vimp_coefs(mpasg_mesh m, mpasg_fields f, FastDiv fl, VimpScalars s) {
  __shared__ double s_cw[kBlock], s_ct[kBlock];
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < (uint32_t)m.nCells * L;
  uint32_t c = 0, k = 0;
  size_t o = 0, ow = 0;
  VimpLevel me_{0.0, 0.0};
  if (active) {
    c = fl.div(i);
    k = i - c * L;
    o = (size_t)c * L;
    ow = (size_t)c * (L + 1);
    me_ = vimp_level<T>(m, f, o, k, s);
    if (c == 0) f.cofrz[k] = s.dtseps * m.rdzw[k];
  }
  s_cw[threadIdx.x] = me_.cofwt;
  s_ct[threadIdx.x] = me_.coftz;
  __syncthreads();
  if (!active) return;
  f.cofwt[o + k] = me_.cofwt;
  f.coftz[ow + k] = me_.coftz;
  if (k == 0) {
    f.cofwr[o] = 0.0;
    f.cofwz[o] = 0.0;
    f.coftz[ow + L] = 0.0;
    f.a_tri[o] = 0.0;
    f.b_tri[o] = 1.0;
    f.c_tri[o] = 0.0;
    return;
  }
  // neighbour levels (k-1 below, k+1 above) from shared memory or recomputed at block edges
  VimpLevel lo = (threadIdx.x >= 1) ? VimpLevel{s_cw[threadIdx.x - 1], s_ct[threadIdx.x - 1]}
                                    : vimp_level<T>(m, f, o, k - 1, s);
  double ct_kp1 = 0.0;
  if (k + 1 < (uint32_t)L)
    ct_kp1 = (threadIdx.x + 1 < blockDim.x) ? s_ct[threadIdx.x + 1] : vimp_level<T>(m, f, o, k + 1, s).coftz;
  const VimpRow r = vimp_row<T>(m, f, o, ow, k, me_, lo, ct_kp1, s);
  f.a_tri[o + k] = r.a;
  f.b_tri[o + k] = r.b;
  f.c_tri[o + k] = r.c;
}

// One column's Thomas factors over rows `pitch` apart (al may be b, gm may be c)
template <typename T>
MPASG_D void factor_column(const double* a, const double* b, const double* c, double* al, double* gm, uint32_t L,
                           uint32_t pitch) {
  double gam = 0.0;
  al[0] = 0.0;
  gm[0] = 0.0;
  for (uint32_t k = 1, q = pitch; k < L; ++k, q += pitch) {
    const double alpha = recip<T>(b[q] - a[q] * gam);
    gam = c[q] * alpha;
    al[q] = alpha;
    gm[q] = gam;
  }
}

// Coefficients and factorisation of `cols` columns in one launch, what passes between them in
// shared memory ([level][column], odd pitch).  In place of two launches, each a few waves of
// latency on a small mesh: a step of 162 columns x 12 levels 664 -> 640 us, 2562 x 26 1359 ->
// 1334, 40962 x 55 25.58 -> 25.37 ms (mixed form 17.61 -> 17.27).
// SHARED: the levels' cofwt and coftz wait for their neighbours in shared memory too; without it
// the neighbours are read back from memory and an SM holds five blocks of 27 columns of 55
// levels instead of three: 255 -> 228 us at 40962 x 55 (step 22.82 -> 22.72 ms).  Where five fit
// all the same, memory only adds latency (step at 2562 x 26 1071 -> 1096 us).
template <typename T, bool SHARED>
__global__ void __launch_bounds__(kBlock) k_vimp_columns(mpasg_mesh m, mpasg_fields f, FastDiv fl, int cols,
                                                         VimpScalars s) {
  extern __shared__ double s_col[];
  const uint32_t L = (uint32_t)m.nVertLevels, pitch = (uint32_t)cols | 1u, nlp = L * pitch;
  double* sa = s_col;  // L x pitch each
  double* sb = sa + nlp;
  double* sc = sb + nlp;
  double* s_cw = sc + nlp;  // SHARED
  double* s_ct = s_cw + nlp;
  VimpFlat* s_flat = reinterpret_cast<VimpFlat*>(SHARED ? s_ct + nlp : s_cw);
  const uint32_t c0 = blockIdx.x * (uint32_t)cols, ncol = min((uint32_t)cols, (uint32_t)m.nCells - c0), nl = ncol * L;
  const size_t o0 = (size_t)c0 * L, ow0 = o0 + c0;
  if (sizeof(T) == sizeof(double))
    for (uint32_t k = 1 + threadIdx.x; k < L; k += kBlock) s_flat[k] = vimp_flat(m, k, s);
  for (uint32_t i = threadIdx.x; i < nl; i += kBlock) {
    const uint32_t col = fl.div(i), k = i - col * L, q = k * pitch + col;
    const VimpLevel v = vimp_level<T>(m, f, o0 + col * L, k, s);
    if (c0 + col == 0) f.cofrz[k] = s.dtseps * m.rdzw[k];
    if (SHARED) {
      s_cw[q] = v.cofwt;
      s_ct[q] = v.coftz;
    }
    f.cofwt[o0 + i] = v.cofwt;
    f.coftz[ow0 + i + col] = v.coftz;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nl; i += kBlock) {
    const uint32_t col = fl.div(i), k = i - col * L, q = k * pitch + col;
    VimpRow r{0.0, 1.0, 0.0};
    if (k == 0) {
      f.cofwr[o0 + i] = 0.0;
      f.cofwz[o0 + i] = 0.0;
      f.coftz[ow0 + i + col + L] = 0.0;
    } else {
      const double* cw = SHARED ? s_cw + q : f.cofwt + o0 + i;
      const double* ct = SHARED ? s_ct + q : f.coftz + ow0 + i + col;
      const int below = SHARED ? -(int)pitch : -1;
      r = vimp_row<T>(m, f, o0 + col * L, ow0 + col * (L + 1), k, VimpLevel{cw[0], ct[0]},
                      VimpLevel{cw[below], ct[below]}, k + 1 < L ? ct[-below] : 0.0, s, s_flat);
    }
    f.a_tri[o0 + i] = sa[q] = r.a;
    f.b_tri[o0 + i] = sb[q] = r.b;
    f.c_tri[o0 + i] = sc[q] = r.c;
  }
  __syncthreads();
  if (threadIdx.x < ncol) {
    const uint32_t t = threadIdx.x;
    factor_column<T>(sa + t, sb + t, sc + t, sb + t, sc + t, L, pitch);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nl; i += kBlock) {
    const uint32_t col = fl.div(i), k = i - col * L, q = k * pitch + col;
    f.alpha_tri[o0 + i] = sb[q];
    f.gamma_tri[o0 + i] = sc[q];
    if (sizeof(T) != sizeof(double) && k > 0) f.tri_m[o0 + i] = -(sb[q] * sa[q]);
  }
}

size_t vimp_columns_smem_bytes(int L, int cols, bool shared) {
  return (size_t)L * ((shared ? 5 : 3) * (cols | 1) * sizeof(double) + sizeof(VimpFlat));
}

template <typename T>
__global__ void k_vimp_factor(mpasg_mesh m, mpasg_fields f) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nCells) return;
  const int L = m.nVertLevels;
  const size_t o = (size_t)c * L;
  factor_column<T>(f.a_tri + o, f.b_tri + o, f.c_tri + o, f.alpha_tri + o, f.gamma_tri + o, L, 1);
  if (sizeof(T) != sizeof(double))
    for (int k = 1; k < L; ++k) f.tri_m[o + k] = -(f.alpha_tri[o + k] * f.a_tri[o + k]);
}

// ---------------------------------------------------------------- acoustic substep, edges
// dynamics/acoustic_step.py:576 (_acoustic_step_horizontal_momentum_update)
// The increment dts (tend_u - pgrad) is formed in the stencil type T; ru_p and ruAvg
// accumulate in float64.
// ru_p after the divergence damping of a substep (dynamics/divergence_damping.py:187-299; the
// increment in the stencil type T, ru_p accumulated in float64).  The fused and the separate
// kernels share this and the explicit multiply-adds below, so a taped step, which runs the
// stages one by one, repeats a step to the bit.
// FROM_ZERO: rtheta_pp_old is zero (the first substep's), so rtheta_pp is the change itself.
template <typename T, bool FROM_ZERO = false>
MPASG_D double damped_ru_p(const mpasg_fields& f, uint32_t i, size_t i1, size_t i2, double coef) {
  // substep change: float64 difference
  T d1 = FROM_ZERO ? -cv<T>(f.rtheta_pp[i1]) : -dif<T>(f.rtheta_pp[i1], f.rtheta_pp_old[i1]);
  T d2 = FROM_ZERO ? -cv<T>(f.rtheta_pp[i2]) : -dif<T>(f.rtheta_pp[i2], f.rtheta_pp_old[i2]);
  // / (theta_m_save_1 + theta_m_save_2) as a product with the reciprocal formed once per
  // dynamics substep (k_theta_edge); within one rounding of the quotient
  if constexpr (sizeof(T) == sizeof(double)) return fma(coef * (d2 - d1), f.theta_edge_rsum[i], f.ru_p[i]);
  return f.ru_p[i] + f64(cv<T>(coef) * (d2 - d1) * cv<T>(f.theta_edge_rsum[i]));
}

// DAMP (small_step > 1): the previous substep's divergence damping first
// (the second substep's: FROM_ZERO)
template <typename T, bool DAMP, bool FROM_ZERO = false>
__global__ void k_acoustic_edges(mpasg_mesh m, mpasg_fields f, FastDiv fl, int small_step,
                                 double dts, double c2, double damp_coef) {  // float64: c2 halved
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nEdges * L) return;
  uint32_t e = fl.div(i), k = i - e * L;
  constexpr bool kDouble = sizeof(T) == sizeof(double);
  double rup;
  if (small_step != 1) {
    int c1 = m.cellsOnEdge[2 * e], c2i = m.cellsOnEdge[2 * e + 1];
    size_t i1 = (size_t)c1 * L + k, i2 = (size_t)c2i * L + k;
    T pgrad = cv<T>(f.rtheta_pp[i2]) - cv<T>(f.rtheta_pp[i1]);
    if (!kDouble) pgrad = pgrad * cv<T>(m.invDcEdge[e]);
    const T z2 = cv<T>(m.zz[i2]) + cv<T>(m.zz[i1]);
    if (!is_two(z2)) pgrad = pgrad / (T(0.5) * z2);
    if constexpr (kDouble) {
      const double cqu = f.cqu_e[i];
      pgrad = pgrad * (f.exner[i1] + f.exner[i2]) * (c2 * m.invDcEdge[e]);
      if (!fx::is_one(cqu)) pgrad = cqu * pgrad;
      if (!m.flatTerrain)  // no slope: adds an exact zero
        pgrad = pgrad + 0.5 * m.zxu[i] * kGravity * (f.rho_pp[i1] + f.rho_pp[i2]);
    } else {
      // the product is rounded once, with the slope term where there is one, on every route:
      // float32 stencils carry a last bit of it to the seventh digit of a step
      const float a = cv<float>(f.cqu_e[i]) * (0.5f * cv<float>(c2)) * (cv<float>(f.exner[i1]) + cv<float>(f.exner[i2]));
      if (m.flatTerrain) {
        pgrad = __fmul_rn(a, pgrad);
      } else {
        const float slope = 0.5f * cv<float>(m.zxu[i]) * float(kGravity);
        pgrad = __fmaf_rn(a, pgrad, __fmul_rn(slope, cv<float>(f.rho_pp[i1]) + cv<float>(f.rho_pp[i2])));
      }
    }
    const double before = DAMP ? damped_ru_p<T, FROM_ZERO>(f, i, i1, i2, damp_coef) : f.ru_p[i];
    if constexpr (kDouble) rup = fma(dts, f.tend_u[i] - pgrad, before);
    else rup = before + f64(cv<T>(dts) * (cv<T>(f.tend_u[i]) - pgrad));
    f.ruAvg[i] = f.ruAvg[i] + rup;
  } else {
    rup = f64(cv<T>(dts) * cv<T>(f.tend_u[i]));
    f.ruAvg[i] = rup;
  }
  f.ru_p[i] = rup;
  // the theta flux of both adjacent cells' sums, once per edge (ke_edge: scratch here)
  if (kDouble) f.ke_edge[i] = rup * f.theta_edge_save[i];
}

// ---------------------------------------------------------------- acoustic substep, columns
// dynamics/acoustic_step.py:456 (cell flux sums), :675 (RHS), :772 (Thomas solve,
// implicit Rayleigh damping, post-solve rho_pp / rtheta_pp); Thomas sweeps from
// autodiff/tridiagonal_solve.py:56-63.  One launch (k_ac_columns, k_ac_columns_mixed), or in
// float64 three, for the forward mode and for columns too high for shared memory: k_ac_prep
// (every level in parallel: flux sums, rs / ts, tridiagonal right-hand side), k_ac_thomas (one
// thread per column: forward elimination and back substitution only) and k_ac_post (every
// level in parallel: Rayleigh damping, ww accumulation, rho_pp / rtheta_pp update).

// edge mean of theta_m_save, 0.5 (theta_2 + theta_1), the value the acoustic right-hand
// side takes per edge, and the reciprocal of the sum that divergence damping divides by
// (theta_m_save only changes at the dynamics substep boundaries)
// MIXED: the mixed form's divergence damping reads the reciprocal as float32, so it is
// the float32 reciprocal of the float32 sum (no float64 division)
template <bool MIXED>
__global__ void k_theta_edge(mpasg_mesh m, mpasg_fields f, FastDiv fl) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nEdges * L) return;
  uint32_t e = fl.div(i), k = i - e * L;
  const int c1 = m.cellsOnEdge[2 * e], c2 = m.cellsOnEdge[2 * e + 1];
  const double sum = f.theta_m_save[(size_t)c2 * L + k] + f.theta_m_save[(size_t)c1 * L + k];
  f.theta_edge_save[i] = 0.5 * sum;
  // divergence damping multiplies instead of dividing
  f.theta_edge_rsum[i] = MIXED ? f2d_bits(1.0f / d2f_bits(sum)) : fx::rcp(sum);
}

// Right-hand sides of the float64 form.  With S1 = sum_j geo_j ru_p_j, S2 = sum_j geo_j (ru_p
// theta)_j over a cell's edges (geo = sign dvEdge / areaCell),
//   rs = rho_pp + dts (tend_rho - S1) - resm cofrz d(rw_p),       R = rs + resm rho_pp
//   ts = rtheta_pp + dts (tend_theta - S2) - resm rdzw d(coftz rw_p),  P = ts + resm rtheta_pp
//   x  = rw_p + dts tend_rw - cofwz (zz_k P_k - zz_km1 P_km1) - cofwr (R_k + R_km1)
//        + cofwt_k P_k + cofwt_km1 P_km1
// Bound by the float64 pipe (63 operations a level, 268 us at 40962 x 55).  S1, and S2 over
// products formed once per edge, are formed on the integer pipes (fixdot.cuh), and the first
// substep, whose perturbations are all zero, has its own instance: 22 operations a level, 11 in
// the first substep.
struct AcLevel {
  double rs, ts, R, P;
};

template <int N, bool FIRST>
MPASG_D AcLevel ac_level(const mpasg_mesh& m, const mpasg_fields& f, const fx::Weight* w, uint32_t c, uint32_t k,
                         double dts, double resm) {
  const uint32_t L = (uint32_t)m.nVertLevels;
  const size_t g = (size_t)c * m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  const auto flux = [&](const double* __restrict__ q) {
    double x[N], sum;
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = q[(uint32_t)w[j].row * L + k];
    if (!fx::dot<N>(x, w, &sum)) {
      sum = 0.0;
      for (int j = 0; j < n; ++j) sum = fma(m.cell_edge_geo[g + j], q[(size_t)m.edgesOnCell[g + j] * L + k], sum);
    }
    return sum;
  };
  const double s1 = flux(f.ru_p), s2 = flux(f.ke_edge);
  const size_t o = (size_t)c * L + k, ow = (size_t)c * (L + 1) + k;
  AcLevel a;
  if (FIRST) {
    a.R = a.rs = dts * (f.tend_rho[o] - s1);
    a.P = a.ts = dts * (f.tend_theta[o] - s2);
  } else {
    const double rho_in = f.rho_pp[o], rt_in = f.rtheta_pp[o], w0 = f.rw_p[ow], w1 = f.rw_p[ow + 1];
    a.rs = fma(-(resm * f.cofrz[k]), w1 - w0, fma(dts, f.tend_rho[o] - s1, rho_in));
    a.ts = fma(-(resm * m.rdzw[k]), fma(f.coftz[ow + 1], w1, -(f.coftz[ow] * w0)),
               fma(dts, f.tend_theta[o] - s2, rt_in));
    a.R = fma(resm, rho_in, a.rs);
    a.P = fma(resm, rt_in, a.ts);
  }
  return a;
}

// the tridiagonal right-hand side of an inner level
template <bool FIRST>
MPASG_D double ac_rhs(const mpasg_mesh& m, const mpasg_fields& f, size_t o, size_t ow, double rwp, double R, double P,
                      double R_lo, double P_lo, double dts) {
  double x = FIRST ? dts * f.tend_rw[ow] : fma(dts, f.tend_rw[ow], rwp);
  x = fma(-f.cofwz[o], fma(m.zz[o], P, -(m.zz[o - 1] * P_lo)), x);
  x = fma(-f.cofwr[o], R + R_lo, x);
  return fma(f.cofwt[o - 1], P_lo, fma(f.cofwt[o], P, x));
}

// rho_pp and rtheta_pp from the solution above and below a level; returns rho_pp
MPASG_D double ac_level_out(const mpasg_mesh& m, const mpasg_fields& f, size_t o, size_t ow, uint32_t k, double rs,
                            double ts, double xr, double xr1) {
  const double rho = fma(-f.cofrz[k], xr1 - xr, rs);
  f.rho_pp[o] = rho;
  f.rtheta_pp[o] = fma(-m.rdzw[k], fma(f.coftz[ow + 1], xr1, -(f.coftz[ow] * xr)), ts);
  return rho;
}

// rho_p and rho_zz after a stage's last substep; returns rho_zz
MPASG_D double recover_rho(const mpasg_mesh& m, const mpasg_fields& f, size_t o, double rho_pp) {
  const double rho_p = f.rho_p_save[o] + rho_pp;
  const double rho_zz = rho_p + m.rho_base[o];
  f.rho_p[o] = rho_p;
  f.rho_zz[o] = rho_zz;
  return rho_zz;
}

template <int N, bool FIRST>
__global__ void __launch_bounds__(kBlock, 5) k_ac_prep(mpasg_mesh m, mpasg_fields f, FastDiv fl1, double dts,
                                                    double ww_lo, double resm) {
  extern __shared__ fx::Weight s_w[];
  __shared__ double s_R[kBlock], s_P[kBlock];
  const uint32_t L = (uint32_t)m.nVertLevels;
  const uint32_t n_all = (uint32_t)m.nCells * (L + 1);
  const uint32_t i0 = blockIdx.x * kBlock, i = i0 + threadIdx.x;
  const uint32_t c0 = fl1.div(i0), c1 = fl1.div(min(i0 + kBlock, n_all) - 1u);
  for (uint32_t t = threadIdx.x; t < (c1 - c0 + 1) * N; t += kBlock) {
    const uint32_t cl = t / N, j = t - cl * N, c = c0 + cl;
    const size_t g = (size_t)c * m.maxEdges;
    const int n = m.nEdgesOnCell[c];
    s_w[t] = ((int)j < n && n <= N) ? fx::weight(m.cell_edge_geo[g + j], m.edgesOnCell[g + j])
                                    : fx::Weight{0, 0, n > N ? fx::kBadWeight : 0u, n > 0 ? m.edgesOnCell[g] : 0};
  }
  __syncthreads();
  const bool active = i < n_all;
  uint32_t c = c0, k = 0;
  AcLevel lv{0.0, 0.0, 0.0, 0.0};
  if (active) {
    c = fl1.div(i);
    k = i - c * (L + 1);
    if (k < L) lv = ac_level<N, FIRST>(m, f, s_w + (c - c0) * N, c, k, dts, resm);
  }
  s_R[threadIdx.x] = lv.R;
  s_P[threadIdx.x] = lv.P;
  __syncthreads();
  if (!active) return;
  const size_t o = (size_t)c * L, ow = (size_t)c * (L + 1);
  if (k < L) {
    f.ac_rs[o + k] = lv.rs;
    f.ac_ts[o + k] = lv.ts;
    f.rtheta_pp_old[o + k] = FIRST ? 0.0 : f.rtheta_pp[o + k];
  }
  const double rwp_k = FIRST ? 0.0 : f.rw_p[ow + k];
  if (k == 0 || k == L) {  // boundary values pass through the solve unchanged
    f.ac_x[ow + k] = rwp_k;
    if (FIRST) f.wwAvg[ow + k] = 0.0;
    return;
  }
  double R_lo, P_lo;
  if (threadIdx.x >= 1) {
    R_lo = s_R[threadIdx.x - 1];
    P_lo = s_P[threadIdx.x - 1];
  } else {
    const AcLevel lo = ac_level<N, FIRST>(m, f, s_w + (c - c0) * N, c, k - 1, dts, resm);
    R_lo = lo.R;
    P_lo = lo.P;
  }
  f.wwAvg[ow + k] = FIRST ? 0.0 : fma(ww_lo, rwp_k, f.wwAvg[ow + k]);
  f.ac_x[ow + k] = ac_rhs<FIRST>(m, f, o + k, ow + k, rwp_k, lv.R, lv.P, R_lo, P_lo, dts);
}

int launch_ac_prep(const mpasg_mesh* m, const mpasg_fields* f, int small_step, double dts, double epssm, double resm,
                   cudaStream_t s) {
  const int L = m->nVertLevels, nb = nblocks((long long)m->nCells * (L + 1)), nc = (kBlock - 1) / (L + 1) + 2;
  const double ww_lo = 0.5 * (1.0 - epssm);
  const FastDiv fl1(L + 1);
  const bool first = small_step == 1, narrow = m->maxEdges <= 6;
  const size_t smem = nc * (narrow ? 6 : 10) * sizeof(fx::Weight);
  if (narrow && first) k_ac_prep<6, true><<<nb, kBlock, smem, s>>>(*m, *f, fl1, dts, ww_lo, resm);
  else if (narrow) k_ac_prep<6, false><<<nb, kBlock, smem, s>>>(*m, *f, fl1, dts, ww_lo, resm);
  else if (first) k_ac_prep<10, true><<<nb, kBlock, smem, s>>>(*m, *f, fl1, dts, ww_lo, resm);
  else k_ac_prep<10, false><<<nb, kBlock, smem, s>>>(*m, *f, fl1, dts, ww_lo, resm);
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

// One column's sweeps over rows `pitch` apart; the next level's operands are read ahead of
// the serial chain.  MIXED: `a` holds -alpha a, one multiply-add a level in the chain
// (alpha x does not depend on it and issues ahead).
template <bool MIXED = false>
MPASG_D void thomas_column(double* x, const double* a, const double* al, const double* g, uint32_t L, uint32_t pitch) {
  const uint32_t q1 = L > 1 ? pitch : 0;
  double xp = x[0], xk = x[q1], ak = a[q1], alk = al[q1];
  for (uint32_t k = 1, q = pitch; k < L; ++k, q += pitch) {
    const uint32_t qn = k + 1 < L ? q + pitch : q;
    const double xn = x[qn], an = a[qn], aln = al[qn];
    xp = MIXED ? fma(ak, xp, alk * xk) : fma(-ak, xp, xk) * alk;
    x[q] = xp;
    xk = xn;
    ak = an;
    alk = aln;
  }
  uint32_t q = (L - 1) * pitch;
  double xn = x[q + pitch], gk = g[q];
  xk = x[q];
  for (uint32_t k = L; k-- > 0;) {
    const uint32_t qn = k > 0 ? q - pitch : q;
    const double xl = x[qn], gl = g[qn];
    xn = fma(-gk, xn, xk);
    x[q] = xn;
    xk = xl;
    gk = gl;
    q = qn;
  }
}

__global__ void k_ac_thomas(mpasg_mesh m, mpasg_fields f) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nCells) return;
  const int L = m.nVertLevels;
  const size_t o = (size_t)c * L;
  const size_t ow = (size_t)c * (L + 1);
  thomas_column(f.ac_x + ow, f.a_tri + o, f.alpha_tri + o, f.gamma_tri + o, L, 1);
}

// ---------------------------------------------------------------- acoustic columns, mixed form
// The acoustic perturbations (rho_pp, rtheta_pp, rw_p, ru_p) are within-stage increments
// without a large mean; the mixed form forms their right-hand sides and post-solve
// increments in float32 and accumulates them in float64 (ac_rs, ac_ts, ac_x, rho_pp,
// rtheta_pp, wwAvg); the tridiagonal solve stays float64.  theta at the edges is split
// into the reference profile and the float32 deviation (theta_save_dev).
struct alignas(16) AcLevelF {
  float drs, dts, rho_in, rt_in;  // float32 increments of rs / ts, and the inputs
};

MPASG_D AcLevelF ac_level_mixed(const mpasg_mesh& m, const mpasg_fields& f, int c, int k, bool first, float dts,
                                float resm, double* rs64, double* ts64) {
  const int L = m.nVertLevels;
  const int me = m.maxEdges;
  const int n = m.nEdgesOnCell[c];
  const float ia = m.invAreaCell_f32[c];
  float rs = 0.0f, tsd = 0.0f;
  for (int j = 0; j < n; ++j) {
    int e = m.edgesOnCell[c * me + j];
    const float wgt = m.edgesOnCell_sign_f32[c * me + j] * m.dvEdge_f32[e];
    const float flux = dts * wgt * cv<float>(f.ru_p[(size_t)e * L + k]) * ia;
    int c1 = m.cellsOnEdge[2 * e], c2 = m.cellsOnEdge[2 * e + 1];
    const float th_e = 0.5f * (f.theta_save_dev[(size_t)c2 * L + k] + f.theta_save_dev[(size_t)c1 * L + k]);
    rs = rs - flux;
    tsd = tsd - flux * th_e;
  }
  const float ts = cv<float>(m.ref_theta[k]) * rs + tsd;  // sum_j -flux_j (ref + theta'_j)
  const size_t o = (size_t)c * L + k;
  const size_t ow = (size_t)c * (L + 1) + k;
  AcLevelF a;
  const double rho_in = first ? 0.0 : f.rho_pp[o];
  const double rt_in = first ? 0.0 : f.rtheta_pp[o];
  a.rho_in = cv<float>(rho_in);
  a.rt_in = cv<float>(rt_in);
  const float rwp_k = first ? 0.0f : cv<float>(f.rw_p[ow]);
  const float rwp_k1 = first ? 0.0f : cv<float>(f.rw_p[ow + 1]);
  a.drs = dts * cv<float>(f.tend_rho[o]) + rs - cv<float>(f.cofrz[k]) * resm * (rwp_k1 - rwp_k);
  a.dts = dts * cv<float>(f.tend_theta[o]) + ts -
          resm * m.rdzw_f32[k] * (cv<float>(f.coftz[ow + 1]) * rwp_k1 - cv<float>(f.coftz[ow]) * rwp_k);
  *rs64 = rho_in + f64(a.drs);
  *ts64 = rt_in + f64(a.dts);
  return a;
}

// the tridiagonal right-hand side's float32 increment at an inner level
MPASG_D float ac_rhs_mixed(const mpasg_mesh& m, const mpasg_fields& f, size_t o, size_t ow, uint32_t k,
                           const AcLevelF& lv, const AcLevelF& lo, float dts, float resm) {
  const float zz_k = m.zz_f32[o + k], zz_km1 = m.zz_f32[o + k - 1];
  const float cw_k = cv<float>(f.cofwt[o + k]), cw_km1 = cv<float>(f.cofwt[o + k - 1]);
  const float ts_k = lv.rt_in + lv.dts, ts_km1 = lo.rt_in + lo.dts;
  const float rs_k = lv.rho_in + lv.drs, rs_km1 = lo.rho_in + lo.drs;
  return dts * cv<float>(f.tend_rw[ow + k]) -
         cv<float>(f.cofwz[o + k]) *
             ((zz_k * ts_k - zz_km1 * ts_km1) + resm * (zz_k * lv.rt_in - zz_km1 * lo.rt_in)) -
         cv<float>(f.cofwr[o + k]) * ((rs_k + rs_km1) + resm * (lv.rho_in + lo.rho_in)) +
         cw_k * (ts_k + resm * lv.rt_in) + cw_km1 * (ts_km1 + resm * lo.rt_in);
}

// Rayleigh damping of the solution (float64); levels without damping pass through
MPASG_D double ac_damped_mixed(const mpasg_mesh& m, const mpasg_fields& f, size_t o, size_t ow, int k, int L,
                               double x, double dts) {
  if (k == 0 || k == L) return x;
  const double dss = m.dss[o + k];
  if (dss == 0.0) return x;
  double fzm = m.fzm[k], fzp = m.fzp[k];
  double zz_i = fzm * m.zz[o + k] + fzp * m.zz[o + k - 1];
  double rho_i = fzm * f.rho_zz[o + k] + fzp * f.rho_zz[o + k - 1];
  double rw_delta = f.rw_save[ow + k] - f.rw[ow + k];
  double num = x + rw_delta - dts * dss * zz_i * rho_i * f.w[ow + k];
  return fdiv<float>(num, 1.0 + dts * dss) - rw_delta;
}

// rho_pp and rtheta_pp from the solution above and below a level; returns rho_pp
MPASG_D double ac_level_out_mixed(const mpasg_mesh& m, const mpasg_fields& f, size_t o, size_t ow, uint32_t k,
                                  double rs, double ts, double xr, double xr1) {
  const float x0 = cv<float>(xr), x1 = cv<float>(xr1);
  const double rho = rs - f64(cv<float>(f.cofrz[k]) * dif<float>(xr1, xr));
  f.rho_pp[o] = rho;
  f.rtheta_pp[o] = ts - f64(m.rdzw_f32[k] * (cv<float>(f.coftz[ow + 1]) * x1 - cv<float>(f.coftz[ow]) * x0));
  return rho;
}

// The same sweeps with the columns staged through shared memory: one warp solves 32
// columns; the block's x, a, alpha and gamma are loaded and stored with coalesced
// accesses (consecutive threads read consecutive levels of a column) into a [level][33]
// layout, so the sequential sweeps read shared memory instead of waiting on one global
// load per level.  The staging runs on all kThomasThreads threads (4 warps, 4x the loads
// in flight: the copy, not the sweep, bounded the one-warp version), the sweeps on the
// first warp.  Same arithmetic as k_ac_thomas.
constexpr int kThomasCols = 32;
constexpr int kThomasPitch = kThomasCols + 1;
constexpr int kThomasThreads = 128;

__global__ void __launch_bounds__(kThomasThreads) k_ac_thomas_staged(mpasg_mesh m, mpasg_fields f, FastDiv fl,
                                                                     FastDiv fl1) {
  extern __shared__ double s_col[];
  const int L = m.nVertLevels;
  double* sx = s_col;                              // (L+1) x pitch
  double* sa = sx + (size_t)(L + 1) * kThomasPitch;  // L x pitch each
  double* sal = sa + (size_t)L * kThomasPitch;
  double* sg = sal + (size_t)L * kThomasPitch;
  const int c0 = blockIdx.x * kThomasCols;
  const int ncol = min(kThomasCols, m.nCells - c0);
  const int t = threadIdx.x;
  const uint32_t nw = (uint32_t)ncol * (L + 1), nl = (uint32_t)ncol * L;
  const double* gx = f.ac_x + (size_t)c0 * (L + 1);
  const size_t o0 = (size_t)c0 * L;
  for (uint32_t idx = t; idx < nw; idx += kThomasThreads) {
    uint32_t col = fl1.div(idx), k = idx - col * (L + 1);
    sx[k * kThomasPitch + col] = gx[idx];
  }
  for (uint32_t idx = t; idx < nl; idx += kThomasThreads) {
    uint32_t col = fl.div(idx), k = idx - col * L;
    sa[k * kThomasPitch + col] = f.a_tri[o0 + idx];
    sal[k * kThomasPitch + col] = f.alpha_tri[o0 + idx];
    sg[k * kThomasPitch + col] = f.gamma_tri[o0 + idx];
  }
  __syncthreads();
  if (t < ncol) thomas_column(sx + t, sa + t, sal + t, sg + t, L, kThomasPitch);
  __syncthreads();
  double* gxo = f.ac_x + (size_t)c0 * (L + 1);
  for (uint32_t idx = t; idx < nw; idx += kThomasThreads) {
    uint32_t col = fl1.div(idx), k = idx - col * (L + 1);
    gxo[idx] = sx[k * kThomasPitch + col];
  }
}

// tri_m = -alpha_tri * a_tri (the mixed forward-sweep factor) from the stored factors
__global__ void k_tri_m(long long n, const double* __restrict__ a, const double* __restrict__ al,
                        double* __restrict__ tm) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) tm[i] = -(al[i] * a[i]);
}

size_t thomas_smem_bytes(int L) { return (size_t)(4 * L + 1) * kThomasPitch * sizeof(double); }

// Rayleigh damping of the solution, (x + d - dts dss zz rho w) / (1 + dts dss) - d with d =
// rw_save - rw; a level without damping keeps x ((x + d) - d without its two roundings)
MPASG_D double ac_damped(const mpasg_mesh& m, const mpasg_fields& f, size_t o, size_t ow, int k, int L, double x,
                         double dts) {
  if (k == 0 || k == L) return x;
  const double dss = m.dss[o + k];
  if (fx::is_zero(dss)) return x;
  const double fzm = m.fzm[k], fzp = m.fzp[k];
  const double zz_i = fzm * m.zz[o + k] + fzp * m.zz[o + k - 1];
  const double rho_i = fzm * f.rho_zz[o + k] + fzp * f.rho_zz[o + k - 1];
  const double rw_delta = f.rw_save[ow + k] - f.rw[ow + k], damp = dts * dss;
  const double num = x + rw_delta - damp * zz_i * rho_i * f.w[ow + k];
  return fx::quotient(num, 1.0 + damp) - rw_delta;
}

// ww_hi: 0.5 (1 + epssm)
__global__ void __launch_bounds__(kBlock) k_ac_post(mpasg_mesh m, mpasg_fields f, FastDiv fl1, double dts,
                                                    double ww_hi) {
  __shared__ double s_xr[kBlock];
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < (uint32_t)m.nCells * (L + 1);
  uint32_t c = 0, k = 0;
  size_t o = 0, ow = 0;
  double xr = 0.0;
  if (active) {
    c = fl1.div(i);
    k = i - c * (L + 1);
    o = (size_t)c * L;
    ow = (size_t)c * (L + 1);
    xr = ac_damped(m, f, o, ow, k, L, f.ac_x[ow + k], dts);
  }
  s_xr[threadIdx.x] = xr;
  __syncthreads();
  if (!active) return;
  f.rw_p[ow + k] = xr;
  if (k >= 1 && k < (uint32_t)L) f.wwAvg[ow + k] = fma(ww_hi, xr, f.wwAvg[ow + k]);
  if (k == (uint32_t)L) return;
  double xr1 = (threadIdx.x + 1 < blockDim.x) ? s_xr[threadIdx.x + 1]
                                              : ac_damped(m, f, o, ow, k + 1, L, f.ac_x[ow + k + 1], dts);
  ac_level_out(m, f, o + k, ow + k, k, f.ac_rs[o + k], f.ac_ts[o + k], xr, xr1);
}

// The float64 substep's columns in one launch: right-hand sides, solve and update of `cols`
// columns a block, with what passes between them in shared memory in a [level][column]
// layout (pitch odd: no bank conflicts).  The three kernels, which the forward mode still
// runs apart, write and read five arrays of a level between them, wait for memory at each
// start and leave the chip idle in the sweeps (one lane a column, ~190 clocks a level); here
// the sweeps run beside other blocks' level work.  Step of 162 columns x 12 levels 744 -> 666
// us, 2562 x 26 1443 -> 1353, 10242 x 33 4530 -> 4314, 40962 x 55 25.81 -> 25.49 ms; acoustic
// stage at 40962 x 55 1505 -> 1440 us (1391 with S2 on the integer pipes; 215-227 us a first
// substep, 261 a later one).  Bound by the float64 pipe on a large mesh, by the
// chain of its phases on a small one.
// keep: leave rs, ts and the undamped solution in ac_rs, ac_ts, ac_x (the reverse mode).
// last: rho_p and rho_zz too, so that the recovery of u need not wait for that of the cells.
template <int N, bool FIRST>
__global__ void __launch_bounds__(kBlock, 5) k_ac_columns(mpasg_mesh m, mpasg_fields f, FastDiv fl, FastDiv fl1,
                                                          int cols, bool keep, bool last, double dts, double ww_lo,
                                                          double ww_hi, double resm) {
  extern __shared__ fx::Weight s_w[];  // first: its alignment is the wider one
  const uint32_t L = (uint32_t)m.nVertLevels, pitch = (uint32_t)cols | 1u, nlp = L * pitch;
  double* sx = (double*)(s_w + cols * N);  // (L + 1) x pitch, the others L x pitch
  double* sa = sx + nlp + pitch;
  double* sal = sa + nlp;
  double* sg = sal + nlp;
  double* srs = sg + nlp;
  double* sts = srs + nlp;
  double* sR = FIRST ? srs : sts + nlp;  // R = rs, P = ts in the first substep
  double* sP = FIRST ? sts : sR + nlp;
  const uint32_t c0 = blockIdx.x * (uint32_t)cols, ncol = min((uint32_t)cols, (uint32_t)m.nCells - c0);
  const uint32_t nl = ncol * L, nw = nl + ncol;
  const size_t o0 = (size_t)c0 * L, ow0 = o0 + c0;
  for (uint32_t t = threadIdx.x; t < ncol * N; t += kBlock) {
    const uint32_t cl = t / N, j = t - cl * N, c = c0 + cl;
    const size_t g = (size_t)c * m.maxEdges;
    const int n = m.nEdgesOnCell[c];
    s_w[t] = ((int)j < n && n <= N) ? fx::weight(m.cell_edge_geo[g + j], m.edgesOnCell[g + j])
                                    : fx::Weight{0, 0, n > N ? fx::kBadWeight : 0u, n > 0 ? m.edgesOnCell[g] : 0};
  }
  for (uint32_t i = threadIdx.x; i < nl; i += kBlock) {
    const uint32_t col = fl.div(i), q = (i - col * L) * pitch + col;
    sa[q] = f.a_tri[o0 + i];
    sal[q] = f.alpha_tri[o0 + i];
    sg[q] = f.gamma_tri[o0 + i];
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nl; i += kBlock) {
    const uint32_t col = fl.div(i), k = i - col * L, q = k * pitch + col;
    const AcLevel lv = ac_level<N, FIRST>(m, f, s_w + col * N, c0 + col, k, dts, resm);
    srs[q] = lv.rs;
    sts[q] = lv.ts;
    if (!FIRST) {
      sR[q] = lv.R;
      sP[q] = lv.P;
    }
    if (keep) {
      f.ac_rs[o0 + i] = lv.rs;
      f.ac_ts[o0 + i] = lv.ts;
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nw; i += kBlock) {
    const uint32_t col = fl1.div(i), k = i - col * (L + 1), q = k * pitch + col;
    const double rwp = FIRST ? 0.0 : f.rw_p[ow0 + i];
    sx[q] = (k == 0 || k == L) ? rwp  // boundary values pass through the solve unchanged
                               : ac_rhs<FIRST>(m, f, o0 + col * L + k, ow0 + i, rwp, sR[q], sP[q], sR[q - pitch],
                                               sP[q - pitch], dts);
  }
  __syncthreads();
  if (threadIdx.x < ncol) {
    const uint32_t t = threadIdx.x;
    thomas_column(sx + t, sa + t, sal + t, sg + t, L, pitch);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nw; i += kBlock) {
    const uint32_t col = fl1.div(i), k = i - col * (L + 1), q = k * pitch + col;
    const double x = sx[q];
    if (keep) f.ac_x[ow0 + i] = x;
    const double xr = ac_damped(m, f, o0 + col * L, ow0 + col * (L + 1), k, L, x, dts);
    sx[q] = xr;
    if (k == 0 || k == L) {
      if (FIRST) f.wwAvg[ow0 + i] = 0.0;
    } else {
      f.wwAvg[ow0 + i] = fma(ww_hi, xr, FIRST ? 0.0 : fma(ww_lo, f.rw_p[ow0 + i], f.wwAvg[ow0 + i]));
    }
    f.rw_p[ow0 + i] = xr;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nl; i += kBlock) {
    const uint32_t col = fl.div(i), k = i - col * L, q = k * pitch + col;
    f.rtheta_pp_old[o0 + i] = FIRST ? 0.0 : f.rtheta_pp[o0 + i];
    const double rho = ac_level_out(m, f, o0 + i, ow0 + col * (L + 1) + k, k, srs[q], sts[q], sx[q], sx[q + pitch]);
    if (last) recover_rho(m, f, o0 + i, rho);
  }
}

size_t ac_columns_smem_bytes(int L, int cols, int N, bool first) {
  return ((size_t)(first ? 6 : 8) * L + 1) * (cols | 1) * sizeof(double) + (size_t)cols * N * sizeof(fx::Weight);
}

// The mixed form's substep columns in one launch, as k_ac_columns; the float32 increments
// and inputs of a level wait in shared memory as one 16-byte entry.
__global__ void __launch_bounds__(kBlock, 5) k_ac_columns_mixed(mpasg_mesh m, mpasg_fields f, FastDiv fl, FastDiv fl1,
                                                                int cols, bool keep, bool last, int small_step,
                                                                double dts, float epssm, float resm) {
  extern __shared__ AcLevelF s_lv[];  // L x pitch
  const bool first = small_step == 1;
  const float dtsf = (float)dts;
  const uint32_t L = (uint32_t)m.nVertLevels, pitch = (uint32_t)cols | 1u, nlp = L * pitch;
  double* sx = (double*)(s_lv + nlp);  // (L + 1) x pitch, the others L x pitch
  double* sm = sx + nlp + pitch;
  double* sal = sm + nlp;
  double* sg = sal + nlp;
  double* srs = sg + nlp;
  double* sts = srs + nlp;
  const uint32_t c0 = blockIdx.x * (uint32_t)cols, ncol = min((uint32_t)cols, (uint32_t)m.nCells - c0);
  const uint32_t nl = ncol * L, nw = nl + ncol;
  const size_t o0 = (size_t)c0 * L, ow0 = o0 + c0;
  for (uint32_t i = threadIdx.x; i < nl; i += kBlock) {
    const uint32_t col = fl.div(i), k = i - col * L, q = k * pitch + col;
    sm[q] = f.tri_m[o0 + i];
    sal[q] = f.alpha_tri[o0 + i];
    sg[q] = f.gamma_tri[o0 + i];
    double rs, ts;
    s_lv[q] = ac_level_mixed(m, f, c0 + col, k, first, dtsf, resm, &rs, &ts);
    srs[q] = rs;
    sts[q] = ts;
    if (keep) {
      f.ac_rs[o0 + i] = rs;
      f.ac_ts[o0 + i] = ts;
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nw; i += kBlock) {
    const uint32_t col = fl1.div(i), k = i - col * (L + 1), q = k * pitch + col;
    const double rwp = first ? 0.0 : f.rw_p[ow0 + i];
    sx[q] = (k == 0 || k == L) ? rwp  // boundary values pass through the solve unchanged
                               : rwp + f64(ac_rhs_mixed(m, f, o0 + col * L, ow0 + col * (L + 1), k, s_lv[q],
                                                        s_lv[q - pitch], dtsf, resm));
  }
  __syncthreads();
  if (threadIdx.x < ncol) {
    const uint32_t t = threadIdx.x;
    thomas_column<true>(sx + t, sm + t, sal + t, sg + t, L, pitch);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nw; i += kBlock) {
    const uint32_t col = fl1.div(i), k = i - col * (L + 1), q = k * pitch + col;
    const double x = sx[q];
    if (keep) f.ac_x[ow0 + i] = x;
    const double xr = ac_damped_mixed(m, f, o0 + col * L, ow0 + col * (L + 1), k, L, x, dts);
    sx[q] = xr;
    if (k == 0 || k == L) {
      if (first) f.wwAvg[ow0 + i] = 0.0;
    } else {
      const double ww = (first ? 0.0 : f.wwAvg[ow0 + i]) +
                        f64(0.5f * (1.0f - epssm) * (first ? 0.0f : cv<float>(f.rw_p[ow0 + i])));
      f.wwAvg[ow0 + i] = ww + f64(0.5f * (1.0f + epssm) * cv<float>(xr));
    }
    f.rw_p[ow0 + i] = xr;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nl; i += kBlock) {
    const uint32_t col = fl.div(i), k = i - col * L, q = k * pitch + col;
    f.rtheta_pp_old[o0 + i] = first ? 0.0 : f.rtheta_pp[o0 + i];
    const double rho =
        ac_level_out_mixed(m, f, o0 + i, ow0 + col * (L + 1) + k, k, srs[q], sts[q], sx[q], sx[q + pitch]);
    if (last) recover_rho(m, f, o0 + i, rho);
  }
}

size_t ac_columns_mixed_smem_bytes(int L, int cols) {
  return (size_t)(cols | 1) * (L * sizeof(AcLevelF) + (size_t)(6 * L + 1) * sizeof(double));
}

__global__ void k_recover_rho(mpasg_mesh m, mpasg_fields f, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) recover_rho(m, f, i, f.rho_pp[i]);
}

// ---------------------------------------------------------------- divergence damping
template <typename T>
__global__ void k_divergence_damping(mpasg_mesh m, mpasg_fields f, FastDiv fl, double coef) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nEdges * L) return;
  uint32_t e = fl.div(i), k = i - e * L;
  int c1 = m.cellsOnEdge[2 * e], c2 = m.cellsOnEdge[2 * e + 1];
  f.ru_p[i] = damped_ru_p<T>(f, i, (size_t)c1 * L + k, (size_t)c2 * L + k, coef);
}

// ---------------------------------------------------------------- small-step perturbation
// dynamics/smlstep_pert.py:197-373
template <typename T>
__global__ void k_smlstep_pert(mpasg_mesh m, mpasg_fields f, FastDiv fl1) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nCells * (L + 1)) return;
  uint32_t c = fl1.div(i), k = i - c * (L + 1);
  if (k == 0 || k == (uint32_t)L) {
    f.tend_rw[i] = f.tend_w[i];
    return;
  }
  const int me = m.maxEdges;
  const T fzm = cv<T>(m.fzm[k]), fzp = cv<T>(m.fzp[k]);
  T acc = cv<T>(f.tend_w[i]);
  const int n = m.flatTerrain ? 0 : m.nEdgesOnCell[c];  // zero-slope terms add exact zeros
  if constexpr (sizeof(T) == sizeof(double)) {
    for (int j = 0; j < n; ++j) {
      const size_t i = (size_t)m.edgesOnCell[c * me + j] * L + k, zi = ((size_t)c * me + j) * (L + 1) + k;
      const double ut_k = f.tend_u[i];
      acc = fma(-flip_by(fma(fzm, ut_k, fzp * f.tend_u[i - 1]), m.edgesOnCell_sign[c * me + j]),
                m.zb_cell[zi] + flip_below(m.zb3_cell[zi], ut_k), acc);
    }
  } else {
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      T ut_k = cv<T>(f.tend_u[(size_t)e * L + k]);
      T u_i = fzm * ut_k + fzp * cv<T>(f.tend_u[(size_t)e * L + k - 1]);
      T flux = cv<T>(m.edgesOnCell_sign[c * me + j]) * u_i;
      size_t zi = ((size_t)c * me + j) * (L + 1) + k;
      T coef = cv<T>(m.zb_cell[zi]) + (ut_k >= T(0) ? T(1) : T(-1)) * cv<T>(m.zb3_cell[zi]);
      acc = acc - coef * flux;
    }
  }
  size_t o = (size_t)c * L;
  if constexpr (sizeof(T) == sizeof(double))  // (as k_tend_w_theta forms it over flat terrain)
    f.tend_rw[i] = fma(fzm, m.zz[o + k], fzp * m.zz[o + k - 1]) * acc;
  else
    f.tend_rw[i] = f64((fzm * cv<T>(m.zz[o + k]) + fzp * cv<T>(m.zz[o + k - 1])) * acc);
}

// ---------------------------------------------------------------- large-step recovery
// dynamics/recover_large_step.py:414-466 (density / theta / Exner), :485-513 (edges),
// :329-411 (w from omega with zb/zb3 slot fluxes)
// Binomial coefficients C(a, n) = a (a-1) ... (a-n+1) / n!, n = 0..11 (compile time).
struct BinomTable {
  double c[12];
};
__host__ __device__ constexpr BinomTable binom_table(double a) {
  BinomTable b{};
  double t = 1.0;
  b.c[0] = 1.0;
  for (int n = 1; n < 12; ++n) {
    t = t * (a - (n - 1)) / n;
    b.c[n] = t;
  }
  return b;
}

// (1 + x)^(R/cv) - 1 for |x| < 0.02 by its binomial series, 11 terms in float64 Horner
// form (truncation below 1e-19 relative): no cancellation against 1, unlike pow - 1.
MPASG_D double pow1p_rcv_m1(double x) {
  constexpr BinomTable t = binom_table(kRgas / (kCp - kRgas));
  double p = t.c[11];
#pragma unroll
  for (int n = 10; n >= 1; --n) p = fma(p, x, t.c[n]);
  return p * x;
}

// a mean flux and the sum of the substeps' (RecoverTail)
MPASG_D double tail_flux(const RecoverTail& t, double* sum, double v) {
  if (t.sum == RecoverTail::kNone) return v;
  const double all = t.sum == RecoverTail::kNext ? *sum + v : v;
  *sum = all;
  return t.scale != 0.0 ? t.scale * all : v;
}

// Float64 in both forms; T selects the division (exact / Newton reciprocal) and, at
// rk 3, the Exner function: pow in the float64 form; in the mixed form the identity
// exner = exner_base (1 + x)^(R/cv), x = rtheta_p / rtheta_base, with the increment
// exner - exner_base = exner_base pow1p_rcv_m1(x) (pow when |x| >= 0.02), so the
// pressure perturbation needs no difference of nearly equal Exner values.
// FLAT (flat terrain, no slope terms): w itself is finished here as well, omega-derived
// part over the interface density, with the level below's density from the neighbouring
// thread (shared memory) -- the same expressions k_recover_w evaluates, one launch fewer.
template <typename T, bool FLAT = false>
__global__ void __launch_bounds__(kBlock) k_recover_cells(mpasg_mesh m, mpasg_fields f, FastDiv fl1, int rk_step,
                                                          double inv_ns, double rk_dt, bool rho_done, RecoverTail tail) {
  __shared__ double s_rho[FLAT ? kBlock : 1];
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < (uint32_t)m.nCells * (L + 1);
  if (!FLAT && !active) return;
  uint32_t c = 0, k = 0;
  if (active) {
    c = fl1.div(i);
    k = i - c * (L + 1);
  }
  const size_t o = (size_t)c * L + k;
  if (FLAT) {
    double rho = 0.0;
    if (active && k < (uint32_t)L) rho = rho_done ? f.rho_zz[o] : f.rho_p_save[o] + f.rho_pp[o] + m.rho_base[o];
    s_rho[threadIdx.x] = rho;
    __syncthreads();
    if (!active) return;
  }
  if (k < (uint32_t)L) {
    const double rho_zz = rho_done ? f.rho_zz[o] : recover_rho(m, f, o, f.rho_pp[o]);
    double rtheta_p;
    if (rk_step == 3)
      rtheta_p = f.rtheta_p_save[o] + f.rtheta_pp[o] - rk_dt * rho_zz * f.rt_diabatic_tend[o];
    else
      rtheta_p = f.rtheta_p_save[o] + f.rtheta_pp[o];
    double rtb = f.rtheta_base[o];
    f.rtheta_p[o] = rtheta_p;
    const double theta =
        sizeof(T) == sizeof(double) ? fx::quotient(rtheta_p + rtb, rho_zz) : (rtheta_p + rtb) * rcp_nr1(rho_zz);
    f.theta_m[o] = theta;
    if (tail.saves) {
      f.rtheta_p_save[o] = rtheta_p;
      f.theta_m_save[o] = theta;
      f.rr_save[o] = f.rho_p_save[o] = f.rho_p[o];
    }
    if (rk_step == 3) {
      const double rcv = kRgas / (kCp - kRgas);
      double zz = m.zz[o];
      if (sizeof(T) == sizeof(double)) {
        const double ex = mpasg_pow::pow_exner_fx(zz * (kRgas / kP0) * (rtheta_p + rtb), rcv);
        f.exner[o] = ex;
        f.pressure_p[o] = zz * kRgas * __dadd_rn(__dmul_rn(ex, rtheta_p), __dmul_rn(rtb, ex - f.exner_base[o]));
      } else {
        const double exb = f.exner_base[o];
        const double x = fdiv<T>(rtheta_p, rtb);
        double ex, dex;  // exner and exner - exner_base
        if (fabs(x) < 0.02) {
          dex = exb * pow1p_rcv_m1(x);
          ex = exb + dex;
        } else {
          ex = mpasg_pow::pow_exner(zz * (kRgas / kP0) * (rtheta_p + rtb), rcv);
          dex = ex - exb;
        }
        f.exner[o] = ex;
        f.pressure_p[o] = zz * kRgas * (ex * rtheta_p + rtb * dex);
      }
    }
  }
  if (k >= 1 && k < (uint32_t)L) {
    size_t ow = (size_t)c * (L + 1) + k;
    double rws = f.rw_save[ow];
    f.wwAvg[ow] = tail_flux(tail, f.wwAvg_split + ow, rws + f.wwAvg[ow] * inv_ns);
    double rw = rws + f.rw_p[ow];
    f.rw[ow] = rw;
    if (tail.saves) f.rw_save[ow] = rw;
    if (sizeof(T) != sizeof(double)) f.rw_f32[ow] = d2f_bits(rw);
    size_t oc = (size_t)c * L;
    const double den = m.fzm[k] * m.zz[oc + k] + m.fzp[k] * m.zz[oc + k - 1];
    const double wo = fx::is_one(den) ? rw : fdiv<T>(rw, den);
    if (!FLAT) {
      f.w[ow] = wo;
    } else {
      const double rho_k = s_rho[threadIdx.x];
      const double rho_km1 = threadIdx.x >= 1 ? s_rho[threadIdx.x - 1]
                             : rho_done       ? f.rho_zz[oc + k - 1]
                                              : f.rho_p_save[oc + k - 1] + f.rho_pp[oc + k - 1] + m.rho_base[oc + k - 1];
      const double wk = fdiv<T>(wo, m.fzm[k] * rho_k + m.fzp[k] * rho_km1);
      f.w[ow] = wk;
      if (sizeof(T) != sizeof(double)) f.w_f32[ow] = d2f_bits(wk);
    }
  } else {  // bottom and top interfaces
    const size_t ow = (size_t)c * (L + 1) + k;
    if (tail.sum != RecoverTail::kNone) f.wwAvg[ow] = tail_flux(tail, f.wwAvg_split + ow, f.wwAvg[ow]);
    if (FLAT) {  // no slope flux, w = 0
      f.w[ow] = 0.0;
      if (sizeof(T) != sizeof(double)) f.w_f32[ow] = 0.0f;
    }
  }
}

// FINISH: with the last acoustic substep's divergence damping before it and the diagnostics'
// edge fields (k_diag_edges_a) after it: one pass over the edges instead of three.  Bound by the
// float64 pipe (73-75 % of the time at 10242 x 41): 13 operations an edge level, 18 with the saves
// and flux sums of a substep's end, 168 and 233 us at 40962 x 55.
template <typename T, bool FINISH, bool FROM_ZERO>
__global__ void k_recover_edges(mpasg_mesh m, mpasg_fields f, FastDiv fl, double inv_ns, double damp_coef,
                                RecoverTail tail) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nEdges * L) return;
  uint32_t e = fl.div(i), k = i - e * L;
  constexpr bool kDouble = sizeof(T) == sizeof(double);
  const size_t i1 = (size_t)m.cellsOnEdge[2 * e] * L + k, i2 = (size_t)m.cellsOnEdge[2 * e + 1] * L + k;
  double rus = f.ru_save[i];
  f.ruAvg[i] = tail_flux(tail, f.ruAvg_split + i, rus + f.ruAvg[i] * inv_ns);
  double rup;
  if (FINISH) {
    rup = damped_ru_p<T, FROM_ZERO>(f, i, i1, i2, damp_coef);
    f.ru_p[i] = rup;
  } else {
    rup = f.ru_p[i];
  }
  double ru = rus + rup;
  f.ru[i] = ru;
  if (tail.saves) f.ru_save[i] = ru;
  const double rho_1 = f.rho_zz[i1], rho_2 = f.rho_zz[i2];
  const double rho2 = rho_1 + rho_2;
  // 2 ru / rho2 (the factor two is exact wherever it is applied)
  const double h = kDouble ? fx::half(rho2) : 0.0;
  const double u = kDouble ? fx::quotient(ru, h) : 2.0 * ru * rcp_nr1(rho2);
  f.u[i] = u;
  if (!kDouble) f.u_f32[i] = d2f_bits(u);
  if (FINISH) {
    f.h_edge[i] = kDouble ? h : f64(T(0.5) * (cv<T>(rho_1) + cv<T>(rho_2)));
    const T u_t = cv<T>(u);
    const T dcdv = kDouble ? cv<T>(m.edge_dcdv[e]) : G(dcEdge)[e] * G(dvEdge)[e];
    fpw<T>(f.ke_edge, f.ke_edge_f32)[i] = dcdv * (u_t * u_t);
  }
}

template <typename T>
__global__ void k_recover_w(mpasg_mesh m, mpasg_fields f, FastDiv fl1) {
  const int L = m.nVertLevels;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)m.nCells * (L + 1)) return;
  uint32_t c = fl1.div(i), k = i - c * (L + 1);
  constexpr bool kMixed = sizeof(T) != sizeof(double);  // also refresh the float32 copy of w
  if (k == (uint32_t)L) {
    f.w[i] = 0.0;
    if (kMixed) f.w_f32[i] = 0.0f;
    return;
  }
  const int me = m.maxEdges;
  const int n = m.flatTerrain ? 0 : m.nEdgesOnCell[c];  // zero-slope terms add exact zeros
  const size_t oc = (size_t)c * L;
  if (k == 0) {
    double surf = 0.0;
    for (int j = 0; j < n; ++j) {
      int e = m.edgesOnCell[c * me + j];
      const double* ru = f.ru + (size_t)e * L;
      double fs = m.cf1 * ru[0] + m.cf2 * ru[1] + m.cf3 * ru[2];
      size_t zi = ((size_t)c * me + j) * (L + 1);
      double cs = m.zb_cell[zi] + sgn(fs) * m.zb3_cell[zi];
      double sc = m.edgesOnCell_sign[c * me + j] * cs * fs;
      surf = (j == 0) ? sc : surf + sc;
    }
    const double w0 = fdiv<T>(surf, m.cf1 * f.rho_zz[oc] + m.cf2 * f.rho_zz[oc + 1] + m.cf3 * f.rho_zz[oc + 2]);
    f.w[i] = w0;
    if (kMixed) f.w_f32[i] = d2f_bits(w0);
    return;
  }
  double fzm = m.fzm[k], fzp = m.fzp[k];
  double acc = f.w[i];  // omega-derived part from k_recover_cells
  for (int j = 0; j < n; ++j) {
    int e = m.edgesOnCell[c * me + j];
    size_t zi = ((size_t)c * me + j) * (L + 1) + k;
    if (kMixed) {
      double fi = fzm * f.ru[(size_t)e * L + k] + fzp * f.ru[(size_t)e * L + k - 1];
      double ci = m.zb_cell[zi] + sgn(fi) * m.zb3_cell[zi];
      acc = acc + m.edgesOnCell_sign[c * me + j] * ci * fi;
    } else {
      const size_t i = (size_t)e * L + k;
      const double fi = fma(fzm, f.ru[i], fzp * f.ru[i - 1]);
      acc = fma(flip_by(fi, m.edgesOnCell_sign[c * me + j]), m.zb_cell[zi] + flip_by(m.zb3_cell[zi], fi), acc);
    }
  }
  const double wk = fdiv<T>(acc, fzm * f.rho_zz[oc + k] + fzp * f.rho_zz[oc + k - 1]);
  f.w[i] = wk;
  if (kMixed) f.w_f32[i] = d2f_bits(wk);
}

// part 0: cells, 1: edges, 2: w over terrain, 3: rho alone
template <typename T>
int launch_recover(const mpasg_mesh* m, mpasg_fields* f, int rk_step, double inv_ns, double rk_dt, cudaStream_t s,
                   bool finish, double damp_coef, bool one_substep, int part, const RecoverTail& tail) {
  const int L = m->nVertLevels;
  const int nw = nblocks((long long)m->nCells * (L + 1)), ne = nblocks((long long)m->nEdges * L);
  const FastDiv fl(L), fl1(L + 1);
  if (part == 0) {
    if (m->flatTerrain) k_recover_cells<T, true><<<nw, kBlock, 0, s>>>(*m, *f, fl1, rk_step, inv_ns, rk_dt, finish, tail);
    else k_recover_cells<T><<<nw, kBlock, 0, s>>>(*m, *f, fl1, rk_step, inv_ns, rk_dt, finish, tail);
  } else if (part == 1) {
    if (finish && one_substep) k_recover_edges<T, true, true><<<ne, kBlock, 0, s>>>(*m, *f, fl, inv_ns, damp_coef, tail);
    else if (finish) k_recover_edges<T, true, false><<<ne, kBlock, 0, s>>>(*m, *f, fl, inv_ns, damp_coef, tail);
    else k_recover_edges<T, false, false><<<ne, kBlock, 0, s>>>(*m, *f, fl, inv_ns, 0.0, tail);
  } else if (part == 3) {
    k_recover_rho<<<nblocks((long long)m->nCells * L), kBlock, 0, s>>>(*m, *f, (uint32_t)m->nCells * L);
  } else if (!m->flatTerrain) {  // slope fluxes need the new ru of k_recover_edges
    k_recover_w<T><<<nw, kBlock, 0, s>>>(*m, *f, fl1);
  }
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

}  // namespace

// The columns of a substep in one launch; *done is false where their arrays do not fit in
// shared memory.
static int launch_ac_columns(const mpasg_mesh* m, const mpasg_fields* f, bool mixed, int small_step, double dts,
                             double epssm, double resm, bool keep, bool last, cudaStream_t s, bool* done) {
  const int L = m->nVertLevels, N = m->maxEdges <= 6 ? 6 : 10;
  const bool first = small_step == 1;
  const int cols = columns_per_block(m->nCells, L + 1, 600, 18, 2), nb = nblocks(m->nCells, cols);
  const size_t smem = mixed ? ac_columns_mixed_smem_bytes(L, cols) : ac_columns_smem_bytes(L, cols, N, first);
  // (the mixed form takes up to 193 levels, 32 columns of its solve's four arrays)
  *done = smem <= kMaxSmem && !(mixed && thomas_smem_bytes(L) > kMaxSmem);
  if (!*done) return MPASG_OK;
  const auto run = [&](auto kernel, auto... args) -> int {
    if (!allow_smem(kernel, smem)) return MPASG_E_CUDA;
    kernel<<<nb, kBlock, smem, s>>>(*m, *f, FastDiv(L), FastDiv(L + 1), cols, keep, last, args...);
    MPASG_LAUNCH_CHECK();
    return MPASG_OK;
  };
  if (mixed) return run(k_ac_columns_mixed, small_step, dts, (float)epssm, (float)resm);
  const double ww_lo = 0.5 * (1.0 - epssm), ww_hi = 0.5 * (1.0 + epssm);
  if (N == 6 && first) return run(k_ac_columns<6, true>, dts, ww_lo, ww_hi, resm);
  if (N == 6) return run(k_ac_columns<6, false>, dts, ww_lo, ww_hi, resm);
  if (first) return run(k_ac_columns<10, true>, dts, ww_lo, ww_hi, resm);
  return run(k_ac_columns<10, false>, dts, ww_lo, ww_hi, resm);
}

static double damping_coefficient(const mpasg_config* c, double dts) {
  return 2.0 * c->smdiv * c->len_disp / dts;
}

// ================================================================= C ABI
extern "C" int mpasg_moist_coefficients(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f,
                                        void* stream) {
  if (!m || !c || !f) return MPASG_E_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const int L = m->nVertLevels;
  k_moist_cells<<<nblocks(m->nCells), kBlock, 0, s>>>(m->nCells, L, c->num_scalars, c->moist_start,
                                                      c->moist_end, f->scalars, f->qtot, f->cqw);
  MPASG_LAUNCH_CHECK();
  k_moist_edges<<<nblocks((long long)m->nEdges * L), kBlock, 0, s>>>(
      m->nEdges, L, FastDiv(L), c->moist_start, c->moist_end, m->cellsOnEdge, f->qtot, f->cqu_e);
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

extern "C" int mpasg_vert_imp_coefs(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f,
                                    double dts, void* stream) {
  if (!m || !c || !f) return MPASG_E_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const int L = m->nVertLevels;
  const VimpScalars vs = vimp_scalars(dts, c->epssm);
  const FastDiv fl(L);
  const int cols = columns_per_block(m->nCells, L, 400, 31, 6);
  // all five arrays in shared memory as long as an SM still holds five blocks of them
  const bool shared = vimp_columns_smem_bytes(L, cols, true) <= 44 * 1024;
  const size_t smem = vimp_columns_smem_bytes(L, cols, shared);
  const bool mixed = c->precision == MPASG_PRECISION_MIXED;
  if (smem <= kMaxSmem) {
    const auto run = [&](auto kernel) -> int {
      if (!allow_smem(kernel, smem)) return MPASG_E_CUDA;
      kernel<<<nblocks(m->nCells, cols), kBlock, smem, s>>>(*m, *f, fl, cols, vs);
      MPASG_LAUNCH_CHECK();
      return MPASG_OK;
    };
    if (mixed) return shared ? run(k_vimp_columns<float, true>) : run(k_vimp_columns<float, false>);
    return shared ? run(k_vimp_columns<double, true>) : run(k_vimp_columns<double, false>);
  }
  const int nb = nblocks((long long)m->nCells * L), nf = nblocks(m->nCells, 64);
  if (mixed) k_vimp_coefs<float><<<nb, kBlock, 0, s>>>(*m, *f, fl, vs);
  else k_vimp_coefs<double><<<nb, kBlock, 0, s>>>(*m, *f, fl, vs);
  MPASG_LAUNCH_CHECK();
  if (mixed) k_vimp_factor<float><<<nf, 64, 0, s>>>(*m, *f);
  else k_vimp_factor<double><<<nf, 64, 0, s>>>(*m, *f);
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

extern "C" int mpasg_acoustic_step(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f,
                                   int small_step, double dts, void* stream) {
  return mpasgi_acoustic_step(m, c, f, small_step, dts, (cudaStream_t)stream, false);
}

int mpasgi_theta_edge(const mpasg_mesh* m, mpasg_fields* f, bool mixed, cudaStream_t s) {
  const int L = m->nVertLevels;
  if (mixed)
    k_theta_edge<true><<<nblocks((long long)m->nEdges * L), kBlock, 0, s>>>(*m, *f, FastDiv(L));
  else
    k_theta_edge<false><<<nblocks((long long)m->nEdges * L), kBlock, 0, s>>>(*m, *f, FastDiv(L));
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

int mpasgi_acoustic_step(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f, int small_step, double dts,
                         cudaStream_t s, bool copies_current, const AcousticFusion& fuse) {
  if (!m || !c || !f || small_step < 1) return MPASG_E_ARG;
  if (!copies_current) {
    // the edge theta the right-hand side reads
    const int rc = mpasgi_theta_edge(m, f, c->precision == MPASG_PRECISION_MIXED, s);
    if (rc != MPASG_OK) return rc;
  }
  if (c->precision == MPASG_PRECISION_MIXED && !copies_current) {
    const int rc = mpasgi_theta_dev(m, f, s);  // the float32 theta deviations read below
    if (rc != MPASG_OK) return rc;
    const long long n = (long long)m->nCells * m->nVertLevels;
    k_tri_m<<<nblocks(n), kBlock, 0, s>>>(n, f->a_tri, f->alpha_tri, f->tri_m);  // forward-sweep factor
    MPASG_LAUNCH_CHECK();
  }
  return mpasgi_acoustic_parts(m, c, f, small_step, dts, s, -1, fuse);
}

// The acoustic substep in two parts (part -1: both): part 0 updates ru_p / ruAvg on the
// edges and builds the columns' right-hand sides (ac_x holds the tridiagonal right-hand
// side after it); part 1 solves and finishes the columns.
int mpasgi_acoustic_parts(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f, int small_step, double dts,
                          cudaStream_t s, int part, const AcousticFusion& fuse) {
  const int L = m->nVertLevels;
  const double rcv = kRgas / (kCp - kRgas);
  const double c2 = kCp * rcv;
  const double resm = (1.0 - c->epssm) / (1.0 + c->epssm);
  const long long ncw = (long long)m->nCells * (L + 1);
  const bool mixed = c->precision == MPASG_PRECISION_MIXED;
  if (part != 1) {
    if (!(small_step == 1 && fuse.edges_done)) {
      const int ne = nblocks((long long)m->nEdges * L);
      const double coef = damping_coefficient(c, dts);
      const FastDiv fl(L);
      if (mixed && fuse.damp_before && small_step == 2)
        k_acoustic_edges<float, true, true><<<ne, kBlock, 0, s>>>(*m, *f, fl, small_step, dts, c2, coef);
      else if (fuse.damp_before && small_step == 2)
        k_acoustic_edges<double, true, true><<<ne, kBlock, 0, s>>>(*m, *f, fl, small_step, dts, 0.5 * c2, coef);
      else if (mixed && fuse.damp_before)
        k_acoustic_edges<float, true><<<ne, kBlock, 0, s>>>(*m, *f, fl, small_step, dts, c2, coef);
      else if (mixed)
        k_acoustic_edges<float, false><<<ne, kBlock, 0, s>>>(*m, *f, fl, small_step, dts, c2, coef);
      else if (fuse.damp_before)
        k_acoustic_edges<double, true><<<ne, kBlock, 0, s>>>(*m, *f, fl, small_step, dts, 0.5 * c2, coef);
      else
        k_acoustic_edges<double, false><<<ne, kBlock, 0, s>>>(*m, *f, fl, small_step, dts, 0.5 * c2, coef);
      MPASG_LAUNCH_CHECK();
    }
    if (part == -1) {
      bool done = false;
      const int rc = launch_ac_columns(m, f, mixed, small_step, dts, c->epssm, resm, !fuse.scratch, fuse.last, s, &done);
      if (rc != MPASG_OK || done) return rc;
    }
    if (mixed) return MPASG_E_ARG;  // its columns in one launch only
    const int rc = launch_ac_prep(m, f, small_step, dts, c->epssm, resm, s);
    if (rc != MPASG_OK || part == 0) return rc;
  }
  const size_t smem = thomas_smem_bytes(L);
  if (smem <= kMaxSmem) {
    if (!allow_smem(k_ac_thomas_staged, smem)) return MPASG_E_CUDA;
    k_ac_thomas_staged<<<nblocks(m->nCells, kThomasCols), kThomasThreads, smem, s>>>(*m, *f, FastDiv(L), FastDiv(L + 1));
  } else {
    k_ac_thomas<<<nblocks(m->nCells, 64), 64, 0, s>>>(*m, *f);
  }
  MPASG_LAUNCH_CHECK();
  k_ac_post<<<nblocks(ncw), kBlock, 0, s>>>(*m, *f, FastDiv(L + 1), dts, 0.5 * (1.0 + c->epssm));
  MPASG_LAUNCH_CHECK();
  if (fuse.last) {
    k_recover_rho<<<nblocks((long long)m->nCells * L), kBlock, 0, s>>>(*m, *f, (uint32_t)m->nCells * L);
    MPASG_LAUNCH_CHECK();
  }
  return MPASG_OK;
}

extern "C" int mpasg_divergence_damping(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f,
                                        double dts, void* stream) {
  return mpasgi_divergence_damping(m, c, f, dts, (cudaStream_t)stream, false);
}

int mpasgi_divergence_damping(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f, double dts,
                              cudaStream_t stream, bool copies_current) {
  if (!m || !c || !f) return MPASG_E_ARG;
  const int L = m->nVertLevels;
  if (!copies_current) {
    // the reciprocal edge sums read below
    const int rc = mpasgi_theta_edge(m, f, c->precision == MPASG_PRECISION_MIXED, stream);
    if (rc != MPASG_OK) return rc;
  }
  const double coef = damping_coefficient(c, dts);
  if (c->precision == MPASG_PRECISION_MIXED)
    k_divergence_damping<float><<<nblocks((long long)m->nEdges * L), kBlock, 0, (cudaStream_t)stream>>>(
        *m, *f, FastDiv(L), coef);
  else
    k_divergence_damping<double><<<nblocks((long long)m->nEdges * L), kBlock, 0, (cudaStream_t)stream>>>(
        *m, *f, FastDiv(L), coef);
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

extern "C" int mpasg_smlstep_pert(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f,
                                  void* stream) {
  if (!m || !c || !f) return MPASG_E_ARG;
  const int L = m->nVertLevels;
  if (c->precision == MPASG_PRECISION_MIXED)
    k_smlstep_pert<float><<<nblocks((long long)m->nCells * (L + 1)), kBlock, 0, (cudaStream_t)stream>>>(
        *m, *f, FastDiv(L + 1));
  else
    k_smlstep_pert<double><<<nblocks((long long)m->nCells * (L + 1)), kBlock, 0, (cudaStream_t)stream>>>(
        *m, *f, FastDiv(L + 1));
  MPASG_LAUNCH_CHECK();
  return MPASG_OK;
}

namespace {
int recover(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f, int rk_step, int ns, double rk_dt,
            cudaStream_t s, bool finish, double damp_coef, int part, const RecoverTail& tail = RecoverTail()) {
  if (!m || !c || !f || ns < 1) return MPASG_E_ARG;
  const double inv_ns = 1.0 / (double)ns;
  if (c->precision == MPASG_PRECISION_MIXED)
    return launch_recover<float>(m, f, rk_step, inv_ns, rk_dt, s, finish, damp_coef, ns == 1, part, tail);
  return launch_recover<double>(m, f, rk_step, inv_ns, rk_dt, s, finish, damp_coef, ns == 1, part, tail);
}
}  // namespace

extern "C" int mpasg_recover_large_step(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f,
                                        int rk_step, int ns, double rk_dt, void* stream) {
  int rc = MPASG_OK;
  for (int part = 0; part < 3 && rc == MPASG_OK; ++part)
    rc = recover(m, c, f, rk_step, ns, rk_dt, (cudaStream_t)stream, false, 0.0, part);
  return rc;
}

int mpasgi_recover_finish(const mpasg_mesh* m, const mpasg_config* c, mpasg_fields* f, int rk_step, int ns,
                          double rk_dt, double dts, cudaStream_t s, int part, const RecoverTail& tail) {
  return recover(m, c, f, rk_step, ns, rk_dt, s, true, c ? damping_coefficient(c, dts) : 0.0, part, tail);
}
