// Host build of the float64 quotient and reciprocal (mpas_dycore_pytorch_gb300/csrc/
// fastdiv64.cuh) for tests/test_fastdiv64.py; `ulps` moves the float32 seed, as the device's
// approximate reciprocal may.
#include "../mpas_dycore_pytorch_gb300/csrc/fastdiv64.cuh"

extern "C" void quotients(const double* a, const double* b, double* out, long n, int ulps) {
  for (long i = 0; i < n; ++i) {
    if (ulps == 0 || !fx::plain_divisor(b[i]) || !fx::plain_dividend(a[i])) {
      out[i] = fx::quotient(a[i], b[i]);
      continue;
    }
    const float s = fx::float_of_bits(fx::bits_of_float(fx::seed_of(b[i])) + (uint32_t)ulps);
    out[i] = fx::quotient_from(a[i], b[i], fx::rcp44(b[i], s));
  }
}
extern "C" void reciprocals(const double* b, double* out, long n) {
  for (long i = 0; i < n; ++i) out[i] = fx::rcp(b[i]);
}
