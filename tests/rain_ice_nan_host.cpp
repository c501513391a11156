// Host build of compute_pdf's soft-pass form and its full form, for
// tests/test_rain_ice_nan.py: the ice high-content indicator of each; and the
// test of a temperature crossing.
#include "../dwarf-p-ice3_gb300/csrc/rain_ice_point.cuh"

extern "C" void ice_high_host(const Ice3gbConstants *c, long n, const double *t, const double *rit, double *soft,
                              double *full)
{
  ice3pt::Derived d;
  ice3pt::make_derived(*c, d);
  for (long p = 0; p < n; ++p)
    for (int s = 0; s < 2; ++s) {
      double hl[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0}, criauti = 0.0;
      ice3pt::compute_pdf(*c, d, 5e-4, 1e-4, rit[p], 1.0, t[p], 0.0, 5e-4, 5e-4, hl, hi, criauti, s == 0);
      (s == 0 ? soft : full)[p] = hi[0];
    }
}

extern "C" void crosses_host(long n, const double *a, const double *b, const double *z, int *out)
{
  for (long p = 0; p < n; ++p) out[p] = ice3pt::crosses(a[p], b[p], z[p]);
}
