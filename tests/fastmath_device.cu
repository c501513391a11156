// Device build of the functions of fastmath.cuh (same source as the kernels),
// exported for tests/test_gpu_device_functions.py.  Pointers are device memory.
#include "../dwarf-p-ice3_gb300/csrc/fastmath.cuh"

namespace {

__global__ void eval_kernel(int fn, const double *a, const double *b, double *q, double *q2, long n)
{
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i];
  q2[i] = 0.0;
  switch (fn) {
    case 0: q[i] = fm::fexp(x); break;
    case 1: q[i] = fm::fexp10(x); break;
    case 2: q[i] = fm::flog(x); break;
    case 3: q[i] = fm::frcp(x); break;
    case 4: q[i] = fm::fatan(x); break;
    case 5: q[i] = fm::frsqrt(x); break;
    case 6: q[i] = fm::fdiv_rn(x, b[i]); break;
    case 7: fm::fdiv_rn2(x, 2.5 * x, b[i], q[i], q2[i]); break;
    case 8: q[i] = fm::fsqrt_rn(x); break;
    case 9: { const fm::Pair p = fm::flog2(x, b[i]); q[i] = p.a; q2[i] = p.b; break; }
    default: { const fm::Pair p = fm::fexp2(x, b[i]); q[i] = p.a; q2[i] = p.b; break; }
  }
}

// The seed of the reciprocal for every significand truncated to FP32: its
// distance from 2^23-significand i's rounded reciprocal, in units of the last
// place below 1 (2^-24).
__global__ void seed_kernel(int *distance)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (1 << 23)) return;
  const float x = __int_as_float(0x3f800000 | i);
  distance[i] = __float_as_int(fm::rcp_seed_(x)) - __float_as_int(__frcp_rn(x));
}

}  // namespace

extern "C" int fm_eval_device(int fn, const double *a, const double *b, double *q, double *q2, long n)
{
  eval_kernel<<<(unsigned)((n + 255) / 256), 256>>>(fn, a, b, q, q2, n);
  return cudaDeviceSynchronize();
}

extern "C" int fm_seed_device(int *distance)
{
  seed_kernel<<<(1 << 23) / 256, 256>>>(distance);
  return cudaDeviceSynchronize();
}
