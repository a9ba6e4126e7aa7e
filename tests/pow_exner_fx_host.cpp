// Host build of pow_exner_fx (mpas_dycore_pytorch_gb300/csrc/pow_exner_fx.cuh) for
// tests/test_pow_exner_fx.py: the same source the kernels use.
#include "../mpas_dycore_pytorch_gb300/csrc/pow_exner_fx.cuh"

extern "C" void pow_fx_many(const double* x, const double* y, double* out, long n) {
  for (long i = 0; i < n; ++i) out[i] = mpasg_pow::pow_exner_fx(x[i], y[i]);
}
extern "C" void pow_dd_many(const double* x, const double* y, double* out, long n) {
  for (long i = 0; i < n; ++i) out[i] = mpasg_pow::pow_exner(x[i], y[i]);
}
