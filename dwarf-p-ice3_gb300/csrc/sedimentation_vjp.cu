// sedimentation_vjp.cu — adjoint (vector-Jacobian product) of the
// statistical sedimentation sweep.
//
// The forward sweep (sedimentation.cu) first recomputes the fluxes F_k of the
// five species into a scratch array (nothing is kept from the forward call);
// the reverse sweep then walks the columns bottom-up with the cotangent of
// the flux entering each level in a register (sed_vjp_level).  As in the
// forward kernel a block holds 32 columns and a warp per species; per SED_CH
// levels the warps form what the species share, one level each, and at the end
// add up the species' parts of the gradients in the species' order (deterministic),
// one level each.
//
// Bound: the FP64 pipe (61 instructions per warp, species and level; 71 % busy)
// and the integer exp / log / division.  A thread per column with its five species
// one after the other, forward and reverse in one kernel, took 8.03 ms for
// 65,536 x 90; the two kernels take 1.74 + 4.06 ms.
#include "ice3gb_device.cuh"
#include "ice3gb_kernels.h"
#include "sedimentation_point.cuh"

namespace {
using namespace ice3sed;

constexpr int SED_CH = 5;

__global__ void __launch_bounds__(32 * 5) sedimentation_vjp_kernel(const __grid_constant__ Cst c,
                                                                   const __grid_constant__ SedVjpArgs a)
{
  __shared__ double lev[SED_CH][RV_N][32];
  __shared__ double part[SED_CH][5][3][32];            // the species' parts: gradients of rho, dz, cotangent of wlbda
  __shared__ double to[SED_CH][2][32];                 // SedCloud's factors
  __shared__ unsigned falls[SED_CH];                   // and its lanes
  const int lane = threadIdx.x & 31, s = threadIdx.x >> 5;
  const long nij = a.nij, col = blockIdx.x * 32L + lane;
  const bool valid = col < nij, fortran = a.fortran;
  const double dt = a.dt, inv_dt = 1.0 / dt;
  const bool moves = !(s == 0 && fortran && c.LSEDIC == 0.0);
  const double *const src = a.src[s], *const g_src = a.g.src[s], *const g_fpr = a.g.fpr[s];
  const double *const flux = a.flux + (long)s * a.nij * a.nk;
  double *const gx_src = a.gx.src[s];
  CloudPar cp = {0.0, 0.0, 0.0};
  if (s == 0 && moves) {
    const bool has_st = a.sea != nullptr && a.town != nullptr;
    const double sea = (a.sea && valid) ? a.sea[col] : 0.0, town = (a.town && valid) ? a.town[col] : 0.0;
    cp = cloud_params(c, fortran, has_st, sea, town);
  }
  const double rtmin = sed_rtmin(c, s);
  // cotangent of F_k (flux leaving level k downward), starting at the surface
  double bF = (a.g.inpr[s] && moves && valid) ? a.g.inpr[s][col] / c.RHOLW : 0.0;
  for (int k0 = 0; k0 < a.nk; k0 += SED_CH) {
    if (k0 + s < a.nk) {
      const long p = (long)(k0 + s) * nij + col;
      sed_vjp_shared(dt, valid ? ld1(a.rhodref, p) : 1.0, valid ? ld1(a.dzz, p) : 1.0, LaneLev{lev[s], lane});
    }
    __syncthreads();
    const int nlev = a.nk - k0 < SED_CH ? a.nk - k0 : SED_CH;
#pragma unroll 1
    for (int j = 0; j < nlev; ++j) {
      const int k = k0 + j;
      const long p = (long)k * nij + col;
      double c_rho = 0.0, c_dz = 0.0, b_wlbda = 0.0;
      SedCloud cloud = {false, 0.0, 0.0};
      if (valid) {
        const double gS = g_src ? ld1(g_src, p) : 0.0;
        if (!moves) {                                  // source passed through unchanged
          if (gx_src) gx_src[p] = gS;
        } else {
          const double pabs = s == 0 ? ld1(a.pabs, p) : 1.0, tht = s == 0 ? ld1(a.tht, p) : 1.0;
          if (g_fpr) bF += ld1(g_fpr, p);
          const double fa = (k + 1 < a.nk) ? flux[p + nij] : 0.0;
          double b_src;
          bF = sed_vjp_level(c, s, fortran, cp, dt, inv_dt, LaneLev{lev[j], lane}, ld1(src, p), rtmin, fa, flux[p], gS, bF,
                             pabs, tht, b_src, c_rho, c_dz, b_wlbda, cloud);
          if (gx_src) gx_src[p] = b_src;
        }
      }
      part[j][s][0][lane] = c_rho;
      part[j][s][1][lane] = c_dz;
      part[j][s][2][lane] = b_wlbda;
      if (s == 0) {
        to[j][0][lane] = cloud.to_pabs;
        to[j][1][lane] = cloud.to_tht;
        const unsigned m = __ballot_sync(0xffffffffu, cloud.falls);
        if (lane == 0) falls[j] = m;
      }
    }
    __syncthreads();
    if (s < nlev && valid) {
      const long p = (long)(k0 + s) * nij + col;
      double r = part[s][0][0][lane], d = part[s][0][1][lane], w = part[s][0][2][lane];
#pragma unroll
      for (int q = 1; q < 5; ++q) {
        r += part[s][q][0][lane];
        d += part[s][q][1][lane];
        w += part[s][q][2][lane];
      }
      const bool cloud = (falls[s] >> lane) & 1u;
      if (a.gx.pabs) a.gx.pabs[p] = sed_cloud_gradient(cloud, to[s][0][lane], w);
      if (a.gx.tht) a.gx.tht[p] = sed_cloud_gradient(cloud, to[s][1][lane], w);
      if (a.gx.rhodref) a.gx.rhodref[p] = r;
      if (a.gx.dzz) a.gx.dzz[p] = d;
    }
  }
}

}  // namespace

cudaError_t launch_sedimentation_vjp(const Ice3gbConstants &c, const SedVjpArgs &a, cudaStream_t s)
{
  SedArgs f = {};
  f.rhodref = a.rhodref; f.dzz = a.dzz; f.pabs = a.pabs; f.tht = a.tht; f.sea = a.sea; f.town = a.town;
  for (int i = 0; i < 5; ++i) {
    f.src[i] = const_cast<double *>(a.src[i]);         // read only (FLUX_ONLY)
    f.fpr[i] = a.flux + (long)i * a.nij * a.nk;
  }
  f.nij = a.nij; f.nk = a.nk; f.dt = a.dt; f.fortran = a.fortran;
  cudaError_t e = launch_sedimentation_fluxes(c, f, s);
  if (e != cudaSuccess) return e;
  sedimentation_vjp_kernel<<<(unsigned)(((long)a.nij + 31) / 32), 32 * 5, 0, s>>>(c, a);
  return cudaGetLastError();
}
