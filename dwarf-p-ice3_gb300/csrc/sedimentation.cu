// sedimentation.cu — statistical sedimentation, one column and species per
// thread.
//
// Restates ICE4_SEDIMENTATION_STAT (PHYEX-IAL_CY50T1/micro/
// mode_ice4_sedimentation_stat.F90:143-229) and the reference JAX
// sedimentation_stat (src/ice3/jax/stencils/sedimentation.py:58-352), the two
// differing in the cloud mean-radius factor and the flux-divergence scaling
// (selected by `fortran`).  The species of a column do not act on each other,
// so a block holds 32 columns and one warp per species (cloud, rain, ice,
// snow, graupel, and hail where there is any): a thread walks k from the top
// level to the surface with its species' incoming flux F_{k+1} in a register;
// consecutive lanes own consecutive columns, so every level access is
// coalesced.  What the species share at a level (rho, log rho, rho dz / dt,
// dt / (rho dz), dz / dt) is formed once per column: the warps take one level
// each of the next SED_CH and leave it in shared memory (two buffers, one
// barrier per SED_CH levels).
//
// Bound: per warp and level the FP64 pipe (18 instructions per species, 23 in
// the JAX form; 61 % busy at 256x256x90), the barrier between warps of unequal
// work, and the issue of the integer exp / log / reciprocal; a column's chain of nk
// levels where the columns are few.  One thread per column with its five
// species one after the other (their fall speeds dealt out over the warp with
// shuffles) took 2.88 ms for 65,535 x 87 and 1.64 ms for a single block of 32
// columns x 90; five warps per 32 columns took 2.01 and 0.40 ms, and with the
// two fall speeds of a level formed as a pair 1.89 and 0.30 ms.
#include "ice3gb_device.cuh"
#include "ice3gb_kernels.h"
#include "sedimentation_point.cuh"

namespace {
using namespace ice3sed;

// Levels a block forms the shared quantities of at a time, one per species
// warp (a hail warp forms none).
constexpr int SED_CH = 5;

// FLUX_ONLY: the fluxes alone (the adjoint's recomputed forward sweep); the
// sources and the surface precipitation are not written.
template <bool FLUX_ONLY>
__global__ void __launch_bounds__(32 * 6) sedimentation_kernel(const __grid_constant__ Cst c,
                                                               const __grid_constant__ SedArgs a)
{
  __shared__ double lev[2][SED_CH][LV_N][32];
  const int lane = threadIdx.x & 31, s = threadIdx.x >> 5;       // the warp's species
  const long nij = a.nij, col = blockIdx.x * 32L + lane;
  const bool valid = col < nij, hail = s == 5;
  const double dt = a.dt, inv_dt = 1.0 / dt;
  // PHYEX skips the cloud species when LSEDIC is off: its warp only takes
  // its share of the levels
  const bool moves = !(s == 0 && a.fortran && c.LSEDIC == 0.0);
  double *const src = hail ? a.hsrc : a.src[s];
  double *const fpr = hail ? a.hfpr : a.fpr[s];
  double *const inpr = hail ? a.hinpr : a.inpr[s];
  CloudPar cp = {0.0, 0.0, 0.0};
  if (s == 0 && moves) {
    const bool has_st = a.sea != nullptr && a.town != nullptr;
    const double sea = (a.sea && valid) ? a.sea[col] : 0.0, town = (a.town && valid) ? a.town[col] : 0.0;
    cp = cloud_params(c, a.fortran, has_st, sea, town);
  }
  const SpeciesPar par = species_par(c, s);
  double fabove = 0.0;
  // one level ahead: the species' source and, per chunk, the warp's shared level
  double next_src = valid && moves ? src[(long)(a.nk - 1) * nij + col] : 0.0;
  double next_rho = 1.0, next_dz = 1.0;
  auto fetch_level = [&](int k) {
    if (s < SED_CH && k >= 0 && valid) {
      next_rho = ld1(a.rhodref, (long)k * nij + col);
      next_dz = ld1(a.dzz, (long)k * nij + col);
    }
  };
  fetch_level(a.nk - 1 - s);
  int buf = 0;
  for (int top = a.nk - 1; top >= 0; top -= SED_CH, buf ^= 1) {
    if (s < SED_CH && top - s >= 0) {
      sed_shared(a.fortran, dt, inv_dt, next_rho, next_dz, LaneLev{lev[buf][s], lane});
    }
    __syncthreads();
    fetch_level(top - SED_CH - s);
    if (!moves) continue;                                        // uniform over the warp; the barrier is above
    const int nlev = top + 1 < SED_CH ? top + 1 : SED_CH;
#pragma unroll 1
    for (int j = 0; j < nlev; ++j) {
      const long p = (long)(top - j) * nij + col;
      const double sr = next_src;
      if (valid && top - j > 0) next_src = src[p - nij];
      const LaneLev l = {lev[buf][j], lane};
      const double rt = sr * dt, qp = fabove * l[LV_TSO];
      const bool c1 = valid && gtp(rt, par.rtmin), c2 = valid && gtp(qp, par.rtmin);
      // no lane moves the species here (the adjoint's fluxes: at a level whose
      // rho dz is a positive normal number, elsewhere they may be NaN)
      if (__all_sync(0xffffffffu, sed_idle(c1, c2, rt, fabove) && (!FLUX_ONLY || fm::frsqrt_ok(l[LV_RHODZ_IDT])))) {
        if (valid && fpr) fpr[p] = 0.0;
        fabove = 0.0;
        continue;
      }
      const double flux = sed_species_flux(c, s, par, cp, l, rt, qp, c1, c2, fabove, a.pabs, a.tht, p);
      if (valid) {
        if (!FLUX_ONLY) src[p] = sed_species_source(a.fortran, l[LV_IDIV], sr, fabove, flux);
        if (fpr) fpr[p] = flux;
      }
      fabove = flux;
    }
  }
  if (!valid) return;
  if (!moves && fpr)
    for (int k = 0; k < a.nk; ++k) fpr[(long)k * nij + col] = 0.0;
  if (!FLUX_ONLY && inpr) inpr[col] = moves ? fabove / c.RHOLW : 0.0;
}

// SEDIM = SPLI: one column per thread (sed_split_column).
__global__ void __launch_bounds__(128) sedimentation_split_kernel(const __grid_constant__ Cst c,
                                                                  const __grid_constant__ SplitArgs a)
{
  const long col = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (col >= a.sed.nij) return;
  const bool has_st = a.sed.sea != nullptr && a.sed.town != nullptr;
  const double sea = has_st ? a.sed.sea[col] : 0.0, town = has_st ? a.sed.town[col] : 0.0;
  const CloudPar cp = cloud_params(c, true, has_st, sea, town);
  const long n = (long)a.sed.nij * a.sed.nk;
  SplitColumnIO io;
  io.rhodref = a.sed.rhodref; io.dzz = a.sed.dzz; io.pabs = a.sed.pabs; io.tht = a.sed.tht; io.exn = a.exn;
  io.rvt = a.rvt; io.rvs = a.rvs; io.ths = a.ths;
  for (int s = 0; s < 5; ++s) {
    io.rt[s] = a.rt[s];
    io.src[s] = a.sed.src[s];
    io.fpr[s] = a.sed.fpr[s];
    io.inpr[s] = a.sed.inpr[s];
  }
  io.nsp = a.rht ? 6 : 5;
  io.rt[5] = a.rht;
  io.src[5] = a.sed.hsrc;
  io.fpr[5] = a.sed.hfpr;
  io.inpr[5] = a.sed.hinpr;
  io.rtmp = a.scratch;
  io.ext = a.scratch + n;
  io.nij = a.sed.nij;
  io.nk = a.sed.nk;
  if (!sed_split_column(c, cp, a.sed.dt, io, col, a.max_iter)) atomicOr(a.status, ICE3GB_DEV_SED_CAP);
}

// Fog deposition on the lowest level (rain_ice.F90:876-895).
__global__ void fog_deposition_kernel(const __grid_constant__ Cst c, FogArgs a)
{
  const long col = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (col >= a.nij) return;
  if (a.enabled) {
    const double rct = a.rct[col];
    const double indep = c.VDEPOSC * rct * a.rhodref[col] / c.RHOLW;
    a.rcs[col] -= c.VDEPOSC * rct / a.dzz[col];
    a.inprc[col] += indep;
    if (a.indep) a.indep[col] = indep;
  } else if (a.indep) {
    a.indep[col] = 0.0;
  }
}

}  // namespace

cudaError_t launch_sedimentation(const Cst &c, const SedArgs &a, cudaStream_t s)
{
  const int warps = a.hsrc ? 6 : 5;
  sedimentation_kernel<false><<<(unsigned)(((long)a.nij + 31) / 32), 32 * warps, 0, s>>>(c, a);
  return cudaGetLastError();
}

cudaError_t launch_sedimentation_fluxes(const Cst &c, const SedArgs &a, cudaStream_t s)
{
  sedimentation_kernel<true><<<(unsigned)(((long)a.nij + 31) / 32), 32 * 5, 0, s>>>(c, a);
  return cudaGetLastError();
}

cudaError_t launch_sedimentation_split(const Cst &c, const SplitArgs &a, cudaStream_t s)
{
  const long n = a.sed.nij;
  const int threads = 128;
  sedimentation_split_kernel<<<(unsigned)((n + threads - 1) / threads), threads, 0, s>>>(c, a);
  return cudaGetLastError();
}

cudaError_t launch_fog_deposition(const Cst &c, const FogArgs &a, cudaStream_t s)
{
  const int threads = 256;
  fog_deposition_kernel<<<(unsigned)((a.nij + threads - 1) / threads), threads, 0, s>>>(c, a);
  return cudaGetLastError();
}
