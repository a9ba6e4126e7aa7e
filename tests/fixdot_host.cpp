// Host build of the fixed-point sums (mpas_dycore_pytorch_gb300/csrc/fixdot.cuh) for
// tests/test_fixdot.py: the same source the kernels use.  A refused sum returns NaN.
#include "../mpas_dycore_pytorch_gb300/csrc/fixdot.cuh"

template <int N>
static void dots(const double* x, const double* w, double* out, long n) {
  for (long i = 0; i < n; ++i) {
    fx::Weight t[N];
    double v[N];
    for (int j = 0; j < N; ++j) {
      t[j] = fx::weight(w[i * N + j], j);
      v[j] = x[i * N + j];
    }
    if (!fx::dot<N>(v, t, out + i)) out[i] = __builtin_nan("");
  }
}

extern "C" void fx_dot10(const double* x, const double* w, double* out, long n) { dots<10>(x, w, out, n); }
extern "C" void fx_dot14(const double* x, const double* w, double* out, long n) { dots<14>(x, w, out, n); }
extern "C" void fx_sum6(const double* x, const double* s, double* out, long n) {
  for (long i = 0; i < n; ++i) {
    double v[6];
    uint32_t g[6];
    for (int j = 0; j < 6; ++j) {
      v[j] = x[i * 6 + j];
      g[j] = s[i * 6 + j] < 0.0 ? 0x80000000u : 0u;
    }
    if (!fx::sum<6>(v, g, out + i)) out[i] = __builtin_nan("");
  }
}

// x -> positive(x), clamp01(x), order key, and the positive / negative parts of rows of six
extern "C" void fx_select(const double* x, double* pos, double* clamp, long long* key, double* back, long n) {
  for (long i = 0; i < n; ++i) {
    pos[i] = fx::positive(x[i]);
    clamp[i] = fx::clamp01(x[i]);
    key[i] = fx::order_key(x[i]);
    back[i] = fx::from_order_key(key[i]);
  }
}
extern "C" void fx_parts6(const double* x, double* pos, double* neg, int* ok, long n) {
  for (long i = 0; i < n; ++i) {
    double v[6];
    uint32_t g[6];
    for (int j = 0; j < 6; ++j) {
      v[j] = x[i * 6 + j];
      g[j] = j & 1 ? 0x80000000u : 0u;
    }
    ok[i] = fx::sum_parts<6>(v, g, pos + i, neg + i);
  }
}
