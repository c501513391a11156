// Host build of the FP32 quotient estimate and its comparison with a bound,
// for tests/test_quotient_estimate.py.
#include "../dwarf-p-ice3_gb300/csrc/ice3gb_device.cuh"

extern "C" void quot_above_host(long n, const double *num, const double *den, const double *bound, int *out)
{
  for (long i = 0; i < n; ++i) out[i] = quot_above(num[i], den[i], bound[i]);
}
