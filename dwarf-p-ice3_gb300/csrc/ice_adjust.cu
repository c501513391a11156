// ice_adjust.cu — saturation adjustment with CB02 subgrid condensation.
//
// Restates src/ice3/jax/stencils/ice_adjust.py:26-398 (IceAdjustJAX) for one
// grid point per lane.  Pure map over the nij*nk points: 19 3-D fields read
// (+ sigqsat per column), 16 written, 280 algorithmic bytes per point.
#include <cmath>

#include "ice3gb_device.cuh"
#include "ice3gb_kernels.h"
#include "ice_adjust_point.cuh"

namespace {
using namespace ice3ia;

// One point per thread.  ADV: the state adjusted is adv_dt times the sources
// (th = dt*ths, r = dt*rs, the state after the microphysics in the chained
// physics step) instead of th/rv/.../rg, which are then not read; rrs/rss/rgs
// are read instead.  Output pointers may be NULL in the internal chained use
// (store skipped).
// Bound: the FP64 pipe.  At 1024x1024x90 a launch takes 15.9 ms (1.7 TB/s of
// HBM); 16.8 ms before the ice fraction was decided on the high words, the
// products of sbar shared and sigma formed only where there is a condensate,
// 19.3 ms with the arc tangent in FP64 as well.  One point per thread: two
// with 128-bit accesses took 22.45 ms when this form took 19.26, and with the
// registers capped for two / three / four blocks either stayed within
// 19.2-19.5 ms.
template <bool ADV, bool SRC>
__global__ void __launch_bounds__(256) ice_adjust_kernel(const __grid_constant__ Cst c,
                                                            const __grid_constant__ IaKernelFields kf,
                                                            long n, int nij, double dt, double inv_dt, const __grid_constant__ IaDerived d)
{
  const Ice3gbIceAdjustFields &f = kf.f;
  for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < n; p += (long)gridDim.x * blockDim.x) {
    IaIn x;
    x.sigqsat = f.sigqsat_3d ? ld1(f.sigqsat, p) : ld1(f.sigqsat, column_of(p, nij));
    x.pabs = ld1(f.pabs, p); x.sigs = ld1(f.sigs, p); x.exn = ld1(f.exn, p);
    x.exn_ref = ld1(f.exn_ref, p); x.rho = ld1(f.rho_dry_ref, p);
    x.cf_mf = ld1(f.cf_mf, p); x.rc_mf = ld1(f.rc_mf, p); x.ri_mf = ld1(f.ri_mf, p);
    x.rvs = f.rvs[p]; x.rcs = f.rcs[p]; x.ris = f.ris[p]; x.ths = f.ths[p];
    if (ADV) {
      const double a = kf.adv_dt;
      x.th = a * x.ths; x.rv = a * x.rvs; x.rc = a * x.rcs; x.ri = a * x.ris;
      x.rr = a * ld1(kf.rrs, p); x.rs = a * ld1(kf.rss, p); x.rg = a * ld1(kf.rgs, p);
    } else {
      x.th = ld1(f.th, p); x.rv = ld1(f.rv, p); x.rc = ld1(f.rc, p); x.ri = ld1(f.ri, p);
      x.rr = ld1(f.rr, p); x.rs = ld1(f.rs, p); x.rg = ld1(f.rg, p);
    }
    IaOut o;
    double s0 = 0.0;
    ia_point(c, d, dt, inv_dt, x, o, SRC ? &s0 : nullptr);
    if (SRC) f.srcs[p] = s0;
#define ST1(field) if (f.field) f.field[p] = o.field;
    ST1(t) ST1(rv_out) ST1(rc_out) ST1(ri_out) ST1(cldfr) ST1(hlc_hrc) ST1(hlc_hcf) ST1(hli_hri) ST1(hli_hcf)
    ST1(cph) ST1(lv) ST1(ls) ST1(rvs) ST1(rcs) ST1(ris) ST1(ths)
#undef ST1
  }
}

// OCND2 (separate liquid and ice clouds): one point per thread; the level
// above (below at the top) gives the layer thickness of ICECLOUD.
template <bool SRC>
__global__ void __launch_bounds__(256) ice_adjust_ocnd2_kernel(const __grid_constant__ Cst c,
                                                               const __grid_constant__ IaKernelFields kf, long n,
                                                               int nij, int nk, double dt, double inv_dt, const __grid_constant__ IaDerived d)
{
  const Ice3gbIceAdjustFields &f = kf.f;
  for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < n; p += (long)gridDim.x * blockDim.x) {
    IaIn x;
    x.sigqsat = f.sigqsat_3d ? ld1(f.sigqsat, p) : ld1(f.sigqsat, column_of(p, nij));
    x.pabs = ld1(f.pabs, p); x.sigs = ld1(f.sigs, p); x.exn = ld1(f.exn, p);
    x.exn_ref = ld1(f.exn_ref, p); x.rho = ld1(f.rho_dry_ref, p);
    x.cf_mf = ld1(f.cf_mf, p); x.rc_mf = ld1(f.rc_mf, p); x.ri_mf = ld1(f.ri_mf, p);
    x.rvs = f.rvs[p]; x.rcs = f.rcs[p]; x.ris = f.ris[p]; x.ths = f.ths[p];
    x.th = ld1(f.th, p); x.rv = ld1(f.rv, p); x.rc = ld1(f.rc, p); x.ri = ld1(f.ri, p);
    x.rr = ld1(f.rr, p); x.rs = ld1(f.rs, p); x.rg = ld1(f.rg, p);
    const long k = p / nij, col = p - k * nij;
    const long kp = k + 1 < nk ? k + 1 : nk - 1;
    Ocnd2In oi;
    oi.estw = kf.tiwmx;
    oi.esti = kf.tiwmx + kTiwmxN;
    oi.z = ld1(f.zz, p);
    oi.dz = ld1(f.zz, kp * nij + col) - ld1(f.zz, (kp - 1) * nij + col);
    oi.ice_cld_wgt = ld1(f.ice_cld_wgt, col);
    oi.bottom = k == 0;
    IaOut o;
    Ocnd2Out oo;
    double s0 = 0.0;
    ia_point<true>(c, d, dt, inv_dt, x, o, SRC ? &s0 : nullptr, &oi, &oo);
    if (SRC) f.srcs[p] = s0;
#define ST1(field) if (f.field) f.field[p] = o.field;
    ST1(t) ST1(rv_out) ST1(rc_out) ST1(ri_out) ST1(cldfr) ST1(hlc_hrc) ST1(hlc_hcf) ST1(hli_hri) ST1(hli_hcf)
    ST1(cph) ST1(lv) ST1(ls) ST1(rvs) ST1(rcs) ST1(ris) ST1(ths)
#undef ST1
    if (f.icldfr) f.icldfr[p] = oo.icldfr;
    if (f.wcldfr) f.wcldfr[p] = oo.wcldfr;
    if (f.ssio) f.ssio[p] = oo.ssio;
    if (f.ssiu) f.ssiu[p] = oo.ssiu;
    if (f.ifr) f.ifr[p] = 10.0;   // PIFR, condensation.F90:259
  }
}

}  // namespace

static_assert(kTiwmxTableN == kTiwmxN && kTiwmxTables == TW_N, "TIWMX table size");

void tiwmx_tables(const Cst &c, double *tab)
{
  // mode_tiwmx_fun.F90 ESATW / ESATI / AA2 / BB3 / AM3 / REDIN as INI_TIWMX
  // fills its tables (the water values above 273.15 K for ESTABI, AM3TAB = 0 there)
  for (int j = kTiwmxStart; j <= kTiwmxStop; ++j) {
    const double t = (double)j / 100.0;
    const long i = j - kTiwmxStart;
    const double w = std::exp(c.ALPW - c.BETAW / t - c.GAMW * std::log(t));
    const double ei = t >= c.TT ? w : std::exp(c.ALPI - c.BETAI / t - c.GAMI * std::log(t));  // ESATI
    tab[TW_ESW * kTiwmxN + i] = w;
    tab[TW_ESI * kTiwmxN + i] = t > 273.15 ? w : std::exp(c.ALPI - c.BETAI / t - c.GAMI * std::log(t));
    const double l = c.LSTT + (c.CPV - c.CI) * (t - c.TT);
    tab[TW_A2 * kTiwmxN + i] = l * l / (2.38e-2 + 0.0071e-2 * (t - c.TT)) / (t * t * c.RV);
    tab[TW_BB3 * kTiwmxN + i] = c.RV / (0.211e-4 * std::pow(t / c.TT, 1.94) * c.P00) * t / ei;
    tab[TW_AM3 * kTiwmxN + i] = t > 273.15 ? 0.0 : 1000. * std::exp(12.96 * (w / ei - 1.) - 0.639);
    const double z = std::fmax(0., std::fmin(1., (c.TT - t) / 20.));
    tab[TW_REDIN * kTiwmxN + i] = 1. - (1. - z) / std::pow(z * z * z + (1. - z) * (1. - z) * (1. - z), .333);
  }
}

cudaError_t launch_ice_adjust(const Cst &c, const IaKernelFields &kf, int nij, int nk, double dt, int num_sms,
                              cudaStream_t s)
{
  const long n = (long)nij * nk;
  const int threads = 256;
  const long cap = (long)num_sms * 64;
  const bool adv = kf.adv_dt != 0.0;
  const bool src = kf.f.srcs != nullptr;
  const double inv_dt = 1.0 / dt;
  const IaDerived d = ia_derived(c);
  if (c.OCND2 != 0.0) {   // (the host rejects OCND2 with adv_dt)
    long blocks = (n + threads - 1) / threads;
    if (blocks > cap) blocks = cap;
    if (src) ice_adjust_ocnd2_kernel<true><<<(unsigned)blocks, threads, 0, s>>>(c, kf, n, nij, nk, dt, inv_dt, d);
    else ice_adjust_ocnd2_kernel<false><<<(unsigned)blocks, threads, 0, s>>>(c, kf, n, nij, nk, dt, inv_dt, d);
  } else {
    long blocks = (n + threads - 1) / threads;
    if (blocks > cap) blocks = cap;
    if (src) {
      if (adv) ice_adjust_kernel<true, true><<<(unsigned)blocks, threads, 0, s>>>(c, kf, n, nij, dt, inv_dt, d);
      else ice_adjust_kernel<false, true><<<(unsigned)blocks, threads, 0, s>>>(c, kf, n, nij, dt, inv_dt, d);
    } else {
      if (adv) ice_adjust_kernel<true, false><<<(unsigned)blocks, threads, 0, s>>>(c, kf, n, nij, dt, inv_dt, d);
      else ice_adjust_kernel<false, false><<<(unsigned)blocks, threads, 0, s>>>(c, kf, n, nij, dt, inv_dt, d);
    }
  }
  return cudaGetLastError();
}
