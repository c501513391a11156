// sedimentation_point.cuh — one species at one level of the statistical
// sedimentation (ICE4_SEDIMENTATION_STAT, mode_ice4_sedimentation_stat.F90 and
// src/ice3/jax/stencils/sedimentation.py) and of its adjoint: the code of the
// kernels (sedimentation.cu, sedimentation_vjp.cu), which bring the columns,
// the levels' shared quantities and the fluxes.  The sed_column_* functions
// are sweeps of one column over the same levels for the host builds of the
// tests.  Then the time-split form, whole columns.
#pragma once

#include "ice3gb_device.cuh"

namespace ice3sed {

struct CloudPar {
  double log_lbc_conc, ray_inv, fsedc;
};

ICE3_HD CloudPar cloud_params(const Cst &c, bool fortran, bool has_st, double sea, double town)
{
  double lbc, fsedc, conc, ray;
  if (fortran) {
    const double gac_gc = c.GAC / c.GC, gac2_gc2 = c.GAC2 / c.GC2;
    if (has_st) {
      ray = fmax(1.0, 0.5 * ((1.0 - sea) * gac_gc + sea * gac2_gc2));
      lbc = fmax(fmin(c.LBC_1, c.LBC_2), sea * c.LBC_2 + (1.0 - sea) * c.LBC_1);
      fsedc = fmax(fmin(c.FSEDC_1, c.FSEDC_2), sea * c.FSEDC_2 + (1.0 - sea) * c.FSEDC_1);
      conc = (1.0 - town) * (sea * c.CONC_SEA + (1.0 - sea) * c.CONC_LAND) + town * c.CONC_URBAN;
    } else {
      ray = fmax(1.0, 0.5 * gac_gc);
      lbc = c.LBC_1;
      fsedc = c.FSEDC_1;
      conc = c.CONC_LAND;
    }
  } else {
    ray = 1.0;
    lbc = (1.0 - sea) * c.LBC_1 + sea * c.LBC_2;
    fsedc = (1.0 - sea) * c.FSEDC_1 + sea * c.FSEDC_2;
    conc = (1.0 - town) * ((1.0 - sea) * c.CONC_LAND + sea * c.CONC_SEA) + town * c.CONC_URBAN;
  }
  CloudPar p;
  p.log_lbc_conc = fm::flog(lbc * conc);
  p.ray_inv = 1.0 / ray;
  p.fsedc = fsedc;
  return p;
}

// The power-law fall speed F r^a rho^b = F exp(a log r + b log rho) of rain,
// snow, graupel and hail (a = EXSED - 1, b = EXSED - CEXVT - 1), the sum of
// products fused as fma(a, log r, b log rho) wherever it is formed.
ICE3_HD double power_speed(double f, double a, double b, double lr, double lrho)
{
  return f * fm::fexp(fm::fma_(a, lr, b * lrho));
}

// Fall speed for content r (> threshold checked by the caller); lrho = log(rho).
ICE3_HD double fall_speed(const Cst &c, int s, double r, double lrho, double wlbda, const CloudPar &cp)
{
  const double lr = fm::flog(r);
  switch (s) {
    case 0: {  // cloud droplets: sedimentation.py:206-209, F90:264-267
      const double lwlbdc = c.LBEXC * (cp.log_lbc_conc - lrho - lr);
      const double cc = c.CC * (1.0 + 1.26 * wlbda * fm::fexp(lwlbdc) * cp.ray_inv);
      return fm::fexp(-c.CEXVT * lrho - c.DC * lwlbdc) * cc * cp.fsedc;
    }
    case 1:  // rain
      return power_speed(c.FSEDR, c.EXSEDR - 1.0, c.EXSEDR - c.CEXVT - 1.0, lr, lrho);
    case 2: {  // pristine ice: sedimentation.py:46-55, F90:307-311
      const double dmax_ = dmax(0.05e6, -0.15319e6 - 0.021454e6 * (lrho + lr));
      return c.FSEDI * fm::fexp(-c.CEXVT * lrho + c.EXCSEDI * fm::flog(dmax_));
    }
    case 3:  // snow
      return power_speed(c.FSEDS, c.EXSEDS - 1.0, c.EXSEDS - c.CEXVT - 1.0, lr, lrho);
    case 5:  // hail (NRR = 7): OTHER_SPECIES with XFSEDH / XEXSEDH, F90:186-187
      return power_speed(c.FSEDH, c.EXSEDH - 1.0, c.EXSEDH - c.CEXVT - 1.0, lr, lrho);
    default:  // graupel
      return power_speed(c.FSEDG, c.EXSEDG - 1.0, c.EXSEDG - c.CEXVT - 1.0, lr, lrho);
  }
}


// Fall speed as fall_speed() (same operations, same value) with its partial
// derivatives with respect to log r, log rho and wlbda.
ICE3_HD double fall_speed_d(const Cst &c, int s, double r, double lrho, double wlbda, const CloudPar &cp, double &d_lr,
                            double &d_lrho, double &d_wl)
{
  const double lr = fm::flog(r);
  d_wl = 0.0;
  switch (s) {
    case 0: {
      const double lwlbdc = c.LBEXC * (cp.log_lbc_conc - lrho - lr);
      const double e2 = fm::fexp(lwlbdc);
      const double cc = c.CC * (1.0 + 1.26 * wlbda * e2 * cp.ray_inv);
      const double e1 = fm::fexp(-c.CEXVT * lrho - c.DC * lwlbdc);
      const double v = e1 * cc * cp.fsedc;
      // dv/dlwlbdc = e1 fsedc CC (-DC (1 + 1.26 wlbda e2 ray_inv) + 1.26 wlbda e2 ray_inv)
      const double d_lw = e1 * cp.fsedc * c.CC * (-c.DC * (1.0 + 1.26 * wlbda * e2 * cp.ray_inv) +
                                                  1.26 * wlbda * e2 * cp.ray_inv);
      d_lr = -c.LBEXC * d_lw;
      d_lrho = -c.CEXVT * v - c.LBEXC * d_lw;
      d_wl = e1 * cp.fsedc * c.CC * 1.26 * e2 * cp.ray_inv;
      return v;
    }
    case 2: {
      bool first;
      const double arg = -0.15319e6 - 0.021454e6 * (lrho + lr);
      first = gtd(0.05e6, arg);
      const double dmax_ = first ? 0.05e6 : arg;
      const double v = c.FSEDI * fm::fexp(-c.CEXVT * lrho + c.EXCSEDI * fm::flog(dmax_));
      const double dld = first ? 0.0 : fm::fdiv(-0.021454e6, dmax_);
      d_lr = v * c.EXCSEDI * dld;
      d_lrho = v * (-c.CEXVT + c.EXCSEDI * dld);
      return v;
    }
    default: {
      double fsed, ex;
      if (s == 1) { fsed = c.FSEDR; ex = c.EXSEDR; }
      else if (s == 3) { fsed = c.FSEDS; ex = c.EXSEDS; }
      else { fsed = c.FSEDG; ex = c.EXSEDG; }
      const double v = power_speed(fsed, ex - 1.0, ex - c.CEXVT - 1.0, lr, lrho);
      d_lr = (ex - 1.0) * v;
      d_lrho = (ex - c.CEXVT - 1.0) * v;
      return v;
    }
  }
}

ICE3_HD double sed_rtmin(const Cst &c, int s)
{
  return (s == 0) ? c.C_RTMIN : (s == 1) ? c.R_RTMIN : (s == 2) ? dmax(c.I_RTMIN, 1.0e-7) : (s == 3) ? c.S_RTMIN
                                                                                     : (s == 4) ? c.G_RTMIN
                                                                                                : c.H_RTMIN;
}

ICE3_HD double sed_load(const double *p, long i)
{
#if defined(__CUDA_ARCH__)
  return __ldg(p + i);
#else
  return p[i];
#endif
}

// What a species needs of the constants: its threshold and the power law
// F exp(a log r + b log rho) (rain, snow, graupel, hail), the sum fused as in
// power_speed.
struct SpeciesPar {
  double rtmin, f, a, b;
};
ICE3_HD SpeciesPar species_par(const Cst &c, int s)
{
  const double ex = s == 1 ? c.EXSEDR : s == 3 ? c.EXSEDS : s == 4 ? c.EXSEDG : c.EXSEDH;
  return {sed_rtmin(c, s), s == 1 ? c.FSEDR : s == 3 ? c.FSEDS : s == 4 ? c.FSEDG : c.FSEDH, ex - 1.0,
          ex - c.CEXVT - 1.0};
}

// What the species share at a level; LV_IDIV is dt / (rho dz) / dt (Fortran
// scaling) or rho dz dt (the divisor of the JAX form).  Lev: anything indexed by
// these (the kernel's columns lie 32 apart and are read where they are used;
// held in registers across the fall speeds they made the kernel spill).
enum { LV_RHO = 0, LV_LRHO, LV_RHODZ_IDT, LV_TSO, LV_IDIV, LV_DZ_IDT, LV_N };
#if defined(__CUDACC__)
struct LaneLev {                                       // a lane's column in shared memory
  double (*l)[32];
  int lane;
  __device__ __forceinline__ double &operator[](int q) const { return l[q][lane]; }
};
#endif
template <class Lev>
ICE3_HD void sed_shared(bool fortran, double dt, double inv_dt, double rho, double dz, Lev &&l)
{
  const double rhodz = rho * dz, tso = fm::fdiv(dt, rhodz);
  l[LV_RHO] = rho;
  l[LV_LRHO] = fm::flog(rho);
  l[LV_RHODZ_IDT] = rhodz * inv_dt;
  l[LV_TSO] = tso;
  l[LV_IDIV] = fortran ? tso * inv_dt : rhodz * dt;
  l[LV_DZ_IDT] = dz * inv_dt;
}

// The species does not move at the level: content rt at or below its threshold
// (c1) and not negative, nothing falling in (c2): a zero flux, the source kept.
ICE3_HD bool sed_idle(bool c1, bool c2, double rt, double fabove) { return !c1 && !c2 && !negd(rt) && zerod_(fabove); }

// The flux leaving the level: content rt, incoming flux fabove as the content
// qp = fabove dt / (rho dz), c1 / c2 whether each is above the threshold.  The
// two fall speeds are formed as pairs; one that is not wanted carries 1/2
// through.
template <class Lev>
ICE3_HD double sed_species_flux(const Cst &c, int s, const SpeciesPar &par, const CloudPar &cp, const Lev &l,
                                double rt, double qp, bool c1, bool c2, double fabove, const double *pabs,
                                const double *tht, long p)
{
  const double lrho = l[LV_LRHO];
  const fm::Pair lr = fm::flog2(c1 ? rt : 0.5, c2 ? qp : 0.5);
  fm::Pair w;
  if (s == 0) {          // as fall_speed's cloud droplets
    double wlbda = 0.0;
    if (c1 || c2) wlbda = 6.6e-8 * fm::fdiv(101325.0, sed_load(pabs, p)) * (sed_load(tht, p) * (1.0 / 293.15));
    const double lc = cp.log_lbc_conc - lrho, lx = -c.CEXVT * lrho;
    const fm::Pair lw = {c.LBEXC * (lc - lr.a), c.LBEXC * (lc - lr.b)};
    const fm::Pair e2 = fm::fexp2(lw.a, lw.b), e1 = fm::fexp2(lx - c.DC * lw.a, lx - c.DC * lw.b);
    const double k = 1.26 * wlbda * cp.ray_inv;
    w = {e1.a * (c.CC * (1.0 + k * e2.a)) * cp.fsedc, e1.b * (c.CC * (1.0 + k * e2.b)) * cp.fsedc};
  } else if (s == 2) {   // as fall_speed's pristine ice
    const fm::Pair ld = fm::flog2(dmax(0.05e6, -0.15319e6 - 0.021454e6 * (lrho + lr.a)),
                                  dmax(0.05e6, -0.15319e6 - 0.021454e6 * (lrho + lr.b)));
    const double lx = -c.CEXVT * lrho;
    const fm::Pair e = fm::fexp2(lx + c.EXCSEDI * ld.a, lx + c.EXCSEDI * ld.b);
    w = {c.FSEDI * e.a, c.FSEDI * e.b};
  } else {
    const double blr = par.b * lrho;
    const fm::Pair e = fm::fexp2(fm::fma_(par.a, lr.a, blr), fm::fma_(par.a, lr.b, blr));
    w = {par.f * e.a, par.f * e.b};
  }
  const double w1 = c1 ? w.a : 0.0, w2 = c2 ? w.b : 0.0;
  double flux = dmin(l[LV_RHODZ_IDT] * rt, w1 * l[LV_RHO] * rt);
  if (!zerod_(w2)) flux += pmax0(1.0 - l[LV_DZ_IDT] * fm::frcp(w2)) * fabove;
  return flux;
}

// The source after the level's fluxes.
ICE3_HD double sed_species_source(bool fortran, double idiv, double src, double fabove, double flux)
{
  return fortran ? src + idiv * (fabove - flux) : src + fm::fdiv(fabove - flux, idiv);
}

// Fields of one sedimentation sweep; element (k, col) at k * nij + col.
struct SedColumnIO {
  const double *rhodref, *dzz, *pabs, *tht;
  const double *src_in[5];   // sources read (rcs, rrs, ris, rss, rgs)
  double *src_out[5];        // updated sources (may alias src_in), or NULL
  double *fpr[5];            // fluxes F_k, or NULL
  double *inpr[5];           // [nij] surface precipitation, or NULL
  long nij;
  int nk;
};

// Top-down sweep of one column and species (mode_ice4_sedimentation_stat.F90:
// 143-229, sedimentation.py:58-352) with the flux from the level above carried
// along.  src_out, fpr and inpr may be NULL.
ICE3_HD void sed_species_column(const Cst &c, int s, bool fortran, const CloudPar &cp, double dt, const SedColumnIO &io,
                                const double *src_in, double *src_out, double *fpr, double *inpr, long col)
{
  const double inv_dt = 1.0 / dt;
  const SpeciesPar par = species_par(c, s);
  double fabove = 0.0;
  for (int k = io.nk - 1; k >= 0; --k) {
    const long p = (long)k * io.nij + col;
    double l[LV_N];
    sed_shared(fortran, dt, inv_dt, sed_load(io.rhodref, p), sed_load(io.dzz, p), l);
    const double sr = src_in[p], rt = sr * dt, qp = fabove * l[LV_TSO];
    const bool c1 = gtp(rt, par.rtmin), c2 = gtp(qp, par.rtmin), idle = sed_idle(c1, c2, rt, fabove);
    const double flux = idle ? 0.0 : sed_species_flux(c, s, par, cp, l, rt, qp, c1, c2, fabove, io.pabs, io.tht, p);
    if (src_out) src_out[p] = idle ? sr : sed_species_source(fortran, l[LV_IDIV], sr, fabove, flux);
    if (fpr) fpr[p] = flux;
    fabove = flux;
  }
  if (inpr) inpr[col] = fabove / c.RHOLW;
}

// The five species of a column; skip_c: PHYEX's LSEDIC = .FALSE. (cloud not
// sedimented, its outputs left to the caller).
ICE3_HD void sed_column_forward(const Cst &c, bool fortran, bool skip_c, const CloudPar &cp, double dt,
                                const SedColumnIO &io, long col)
{
  for (int s = skip_c ? 1 : 0; s < 5; ++s)
    sed_species_column(c, s, fortran, cp, dt, io, io.src_in[s], io.src_out[s], io.fpr[s], io.inpr[s], col);
}

// Hail in the statistical sweep (NRR = 7; species 7 of
// mode_ice4_sedimentation_stat.F90:186-222, Fortran semantics) for one
// column: the hail content is rhs * dt (mode_ice4_sedimentation.F90:179).
ICE3_HD void sed_hail_column(const Cst &c, double dt, const double *rhodref, const double *dzz, double *rhs,
                             double *fpr, double *inpr, long nij, int nk, long col)
{
  SedColumnIO io = {};
  io.rhodref = rhodref; io.dzz = dzz;
  io.nij = nij;
  io.nk = nk;
  sed_species_column(c, 5, true, CloudPar{}, dt, io, rhs, rhs, fpr, inpr, col);
}

// Cotangents of the sweep's outputs (NULL = zero) and the wanted gradients
// of its inputs (NULL = not wanted), same layouts as SedColumnIO.
struct SedCotangents {
  const double *src[5];      // updated sources
  const double *inpr[5];     // [nij]
  const double *fpr[5];      // fluxes
};
struct SedGradients {
  double *src[5];            // input sources
  double *rhodref, *dzz, *pabs, *tht;
};

// What the species share at a level of the reverse sweep, indexed as in
// sed_shared: RV_TSOR is RV_TSO / (rho dz), RV_IRHO 1 / rho.
enum { RV_RHO = 0, RV_DZ, RV_RHODZ, RV_TSO, RV_LRHO, RV_TSOR, RV_IRHO, RV_N };
template <class Lev>
ICE3_HD void sed_vjp_shared(double dt, double rho, double dz, Lev &&l)
{
  const double rhodz = rho * dz, tso = fm::fdiv(dt, rhodz);
  l[RV_RHO] = rho;
  l[RV_DZ] = dz;
  l[RV_RHODZ] = rhodz;
  l[RV_TSO] = tso;
  l[RV_LRHO] = fm::flog(rho);
  l[RV_TSOR] = fm::fdiv(tso, rhodz);
  l[RV_IRHO] = fm::frcp(rho);
}
// A species' view of them (tso = dt / (rho dz); wlbda: cloud only) and the
// cotangents that it adds to.
struct SedLevel {
  double rho, dz, rhodz, tso, lrho, wlbda;
};
struct SedLevelCot {
  double rho, dz, rhodz, tso, lrho, wlbda;
};

// One species at one level of the reverse sweep: the source and the fluxes
// entering (fa) and leaving (fk) the level, the cotangents gS of the updated
// source and bF of fk.  Returns the cotangent of fa; b_src receives that of
// the source and b the level's.  Derivatives of the branch the forward took at
// the kinks (the min of the two flux bounds, the max(0, .) of the transfer
// factor, the thresholds rt, qp > XRTMIN).
ICE3_HD double sed_vjp_species(const Cst &c, int s, bool fortran, const CloudPar &cp, double dt, double inv_dt,
                               const SedLevel &l, double src, double rtmin, double fa, double fk, double gS, double bF,
                               double &b_src, SedLevelCot &b)
{
  const double rt = src * dt, qp = fa * l.tso;
  const bool c1 = gtp(rt, rtmin), c2 = gtp(qp, rtmin);
  double d1_lr = 0.0, d1_lrho = 0.0, d1_wl = 0.0, d2_lr = 0.0, d2_lrho = 0.0, d2_wl = 0.0;
  const double w1 = c1 ? fall_speed_d(c, s, rt, l.lrho, l.wlbda, cp, d1_lr, d1_lrho, d1_wl) : 0.0;
  const double w2 = c2 ? fall_speed_d(c, s, qp, l.lrho, l.wlbda, cp, d2_lr, d2_lrho, d2_wl) : 0.0;
  const double a1 = l.rhodz * rt * inv_dt, a2 = w1 * l.rho * rt;
  const bool sel1 = !gtd(a1, a2);
  double Bv = 0.0, u = 0.0, idw = 0.0;               // idw = 1 / (dt w2)
  const bool nz2 = !zerod_(w2);
  if (nz2) {
    idw = fm::frcp(dt * w2);
    u = 1.0 - l.dz * idw;
    Bv = pmax0(u);
  }
  // source update
  double b_fa, bFt;
  if (fortran) {
    const double coef = l.tso * inv_dt;
    b_fa = coef * gS;
    bFt = bF - coef * gS;
    b.tso += (fa - fk) * inv_dt * gS;
  } else {
    const double iden = fm::frcp(l.rhodz * dt);
    b_fa = gS * iden;
    bFt = bF - gS * iden;
    b.rhodz += -(fa - fk) * dt * (iden * iden) * gS;
  }
  // F_k = min(a1, a2) + Bv F_{k+1}
  b_fa += Bv * bFt;
  double b_rt = 0.0;
  if (sel1) {
    b_rt = l.rhodz * inv_dt * bFt;
    b.rhodz += rt * inv_dt * bFt;
  } else {
    const double b_w1 = l.rho * rt * bFt;
    b.rho += w1 * rt * bFt;
    b_rt = w1 * l.rho * bFt;
    if (c1) {
      b_rt += fm::fdiv(d1_lr, rt) * b_w1;
      b.lrho += d1_lrho * b_w1;
      b.wlbda += d1_wl * b_w1;
    }
  }
  if (nz2 && pos(u)) {
    const double b_B = fa * bFt, g2 = idw * b_B;
    const double b_w2 = fm::fdiv(l.dz * g2, w2);      // dz / (dt w2^2) b_B
    b.dz -= g2;
    if (c2) {
      const double b_qp = fm::fdiv(d2_lr, qp) * b_w2;
      b.lrho += d2_lrho * b_w2;
      b.wlbda += d2_wl * b_w2;
      b_fa += l.tso * b_qp;
      b.tso += fa * b_qp;
    }
  }
  b_src = gS + dt * b_rt;
  return b_fa;
}

// Where a cloud speed is formed at a level, the factors that take the cotangent
// of wlbda (proportional to theta / pressure) to the pressure and to theta.
struct SedCloud {
  bool falls;
  double to_pabs, to_tht;
};
// The gradient from the sum of the species' cotangents of wlbda (that of a
// species other than cloud is 0, or NaN where it has no finite value): formed
// wherever cloud falls, also where the sum is 0, so that a NaN input gives a NaN
// gradient; 0 at a level without falling cloud.
ICE3_HD double sed_cloud_gradient(bool falls, double factor, double b_wlbda) { return falls ? factor * b_wlbda : 0.0; }

// sed_vjp_species with the level's gradients: c_rho and c_dz receive the
// species' parts of those of rho and dz (all its cotangents taken back to the
// two), b_wlbda its cotangent of wlbda, and cloud the factors (s = 0 only, for
// which pabs and tht are read).
template <class Lev>
ICE3_HD double sed_vjp_level(const Cst &c, int s, bool fortran, const CloudPar &cp, double dt, double inv_dt,
                             const Lev &lv, double src, double rtmin, double fa, double fk, double gS, double bF,
                             double pabs, double tht, double &b_src, double &c_rho, double &c_dz, double &b_wlbda,
                             SedCloud &cloud)
{
  SedLevel l = {lv[RV_RHO], lv[RV_DZ], lv[RV_RHODZ], lv[RV_TSO], lv[RV_LRHO], 0.0};
  if (s == 0) l.wlbda = 6.6e-8 * fm::fdiv(101325.0, pabs) * (tht * (1.0 / 293.15));
  SedLevelCot b = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const double b_fa = sed_vjp_species(c, s, fortran, cp, dt, inv_dt, l, src, rtmin, fa, fk, gS, bF, b_src, b);
  b.rhodz -= lv[RV_TSOR] * b.tso;
  c_rho = b.rho + l.dz * b.rhodz + b.lrho * lv[RV_IRHO];
  c_dz = b.dz + l.rho * b.rhodz;
  b_wlbda = b.wlbda;
  if (s == 0) {
    cloud.falls = gtp(src * dt, rtmin) || gtp(fa * l.tso, rtmin);
    cloud.to_pabs = cloud.falls ? -fm::fdiv(l.wlbda, pabs) : 0.0;
    cloud.to_tht = cloud.falls ? fm::fdiv(l.wlbda, tht) : 0.0;
  }
  return b_fa;
}

// Reverse sweep of one column (hand-written adjoint of sed_column_forward):
// bottom-up, carrying the cotangent of the flux entering each level from
// above.  `flux` holds the forward fluxes F_k of the column (io.fpr layout),
// recomputed by sed_column_forward just before.
ICE3_HD void sed_column_vjp(const Cst &c, bool fortran, bool skip_c, const CloudPar &cp, double dt,
                            const SedColumnIO &io, double *const flux[5], const SedCotangents &g,
                            const SedGradients &gx, long col)
{
  const double inv_dt = 1.0 / dt;
  // cotangent of F_k (flux leaving level k downward), starting at the surface
  double bF[5];
  for (int s = 0; s < 5; ++s) bF[s] = (g.inpr[s] && !(s == 0 && skip_c)) ? g.inpr[s][col] / c.RHOLW : 0.0;
  for (int k = 0; k < io.nk; ++k) {
    const long p = (long)k * io.nij + col;
    double l[RV_N];
    sed_vjp_shared(dt, sed_load(io.rhodref, p), sed_load(io.dzz, p), l);
    double r = 0.0, d = 0.0, w = 0.0;
    SedCloud cloud = {false, 0.0, 0.0};
    for (int s = 0; s < 5; ++s) {
      const double gS = g.src[s] ? g.src[s][p] : 0.0;
      if (s == 0 && skip_c) {                       // sources passed through unchanged
        if (gx.src[s]) gx.src[s][p] = gS;
        continue;
      }
      if (g.fpr[s]) bF[s] += g.fpr[s][p];
      const double fa = (k + 1 < io.nk) ? flux[s][p + io.nij] : 0.0;
      double b_src, c_rho, c_dz, b_wlbda;
      bF[s] = sed_vjp_level(c, s, fortran, cp, dt, inv_dt, l, io.src_in[s][p], sed_rtmin(c, s), fa, flux[s][p], gS,
                            bF[s], sed_load(io.pabs, p), sed_load(io.tht, p), b_src, c_rho, c_dz, b_wlbda, cloud);
      if (gx.src[s]) gx.src[s][p] = b_src;
      r += c_rho;
      d += c_dz;
      w += b_wlbda;
    }
    if (gx.rhodref) gx.rhodref[p] = r;
    if (gx.dzz) gx.dzz[p] = d;
    if (gx.pabs) gx.pabs[p] = sed_cloud_gradient(cloud.falls, cloud.to_pabs, w);
    if (gx.tht) gx.tht[p] = sed_cloud_gradient(cloud.falls, cloud.to_tht, w);
  }
}

// ---- time-split sedimentation (SEDIM = SPLI) ------------------------------
// mode_ice4_sedimentation_split.F90 (INTERNAL_SEDIM_SPLI, without the
// electric charges and the Beard velocity correction) and the negativity
// correction that ICE4_SEDIMENTATION applies after it
// (mode_ice4_sedimentation.F90:196-229).  Per species, in CFL-limited
// sub-steps until the time step is used up: the flux of each level from the
// temporary mixing ratio (initialised with the value at t), the column's
// sub-step = min(remaining time, SPLIT_MAXCFL rho r dz / flux), then the
// temporary mixing ratio moves by the flux divergence plus its external
// tendency (source - r_t / dt) over the sub-step and the source by the flux
// divergence.
struct SplitColumnIO {
  const double *rhodref, *dzz, *pabs, *tht, *exn;
  const double *rt[6];       // mixing ratios at t: rc rr ri rs rg (rh)
  const double *rvt;
  double *src[6];            // in-out sources rcs rrs ris rss rgs (rhs)
  double *rvs, *ths;         // in-out (negativity correction)
  double *fpr[6];            // accumulated fluxes, or NULL
  double *inpr[6];           // [nij]
  double *rtmp, *ext;        // [nk][nij] scratch: temporary mixing ratio, external tendency
  long nij;
  int nk;
  int nsp;                   // 5, or 6 with hail (NRR = 7, species 7 of :340-347)
};

// Flux rho r v(r) of species s at content r (0 below the species' threshold;
// ice: max(XRTMIN, 1e-7)), INTERNAL_SEDIM_SPLI :500-700.
ICE3_HD double split_flux(const Cst &c, int s, double r, double rho, double lrho, double p, double th,
                          const CloudPar &cp)
{
  if (!gtp(r, sed_rtmin(c, s))) return 0.0;
  double wlbda = 0.0;
  if (s == 0) {
    // ZZT = theta (p / P00)^(RD/CPD): the temperature (:520)
    const double t = th * fm::fexp((c.RD / c.CPD) * fm::flog(fm::fdiv(p, c.P00)));
    wlbda = 6.6e-8 * fm::fdiv(101325.0, p) * (t * (1.0 / 293.15));
  }
  return fall_speed(c, s, r, lrho, wlbda, cp) * rho * r;
}

// ICE4_CORRECT_NEGATIVITIES on the sources (mode_ice4_correct_negativities.F90)
// with the latent-heat factors lv / ls.
ICE3_HD void correct_negativities(const Cst &c, double lv, double ls, double &ths, double &rvs, double &rcs,
                                  double &rrs, double &ris, double &rss, double &rgs, double *rhs = nullptr)
{
  double w;
  w = rcs - pmax0(rcs); rvs += w; ths -= w * lv; rcs -= w;
  w = rrs - pmax0(rrs); rvs += w; ths -= w * lv; rrs -= w;
  w = ris - pmax0(ris); rvs += w; ths -= w * ls; ris -= w;
  w = rss - pmax0(rss); rvs += w; ths -= w * ls; rss -= w;
  w = rgs - pmax0(rgs); rvs += w; ths -= w * ls; rgs -= w;
  if (rhs) { w = *rhs - pmax0(*rhs); rvs += w; ths -= w * ls; *rhs -= w; }   // :115-120
  w = dmin(1., fm::fdiv(pmax0(c.V_RTMIN - rvs), dmax(rcs + ris, 1.e-20)));
  ths -= w * (rcs * lv + ris * ls);
  rvs += w * (rcs + ris);
  rcs = (1. - w) * rcs;
  ris = (1. - w) * ris;
  w = dmin(pmax0(rrs), pmax0(c.V_RTMIN - rvs)); rvs += w; rrs -= w; ths -= w * lv;
  w = dmin(pmax0(rss), pmax0(c.V_RTMIN - rvs)); rvs += w; rss -= w; ths -= w * ls;
  w = dmin(pmax0(rgs), pmax0(c.V_RTMIN - rvs)); rvs += w; rgs -= w; ths -= w * ls;
  if (rhs) { w = dmin(pmax0(*rhs), pmax0(c.V_RTMIN - rvs)); rvs += w; *rhs -= w; ths -= w * ls; }   // :165-171
}

// One column; returns false if a species needed more than max_iter sub-steps
// (the sub-stepping then stops for that species).
ICE3_HD bool sed_split_column(const Cst &c, const CloudPar &cp, double dt, const SplitColumnIO &io, long col,
                              int max_iter)
{
  const double inv_dt = 1.0 / dt;
  bool ok = true;
  for (int s = 0; s < io.nsp; ++s) {
    if (s == 0 && c.LSEDIC == 0.0) {          // GSEDIC = .FALSE.: cloud not sedimented
      if (io.inpr[0]) io.inpr[0][col] = 0.0;
      if (io.fpr[0])
        for (int k = 0; k < io.nk; ++k) io.fpr[0][(long)k * io.nij + col] = 0.0;
      continue;
    }
    const double rtmin = s == 0 ? c.C_RTMIN : s == 1 ? c.R_RTMIN : s == 2 ? c.I_RTMIN : s == 3 ? c.S_RTMIN
                                                                                  : s == 4 ? c.G_RTMIN : c.H_RTMIN;
    for (int k = 0; k < io.nk; ++k) {
      const long p = (long)k * io.nij + col;
      const double r = sed_load(io.rt[s], p);
      io.rtmp[p] = r;
      io.ext[p] = io.src[s][p] - r * inv_dt;    // ZPR.S (:180-190)
      if (io.fpr[s]) io.fpr[s][p] = 0.0;
    }
    double remaint = dt, inpr = 0.0;
    int it = 0;
    while (gtp(remaint, 0.0)) {
      if (++it > max_iter) { ok = false; break; }
      // the column's sub-step (:780-805)
      double mt = remaint;
      for (int k = 0; k < io.nk; ++k) {
        const long p = (long)k * io.nij + col;
        const double r = io.rtmp[p];
        if (!gtp(r, rtmin)) continue;
        const double rho = sed_load(io.rhodref, p);
        const double w = split_flux(c, s, r, rho, fm::flog(rho), sed_load(io.pabs, p), sed_load(io.tht, p), cp);
        if (gtp(w, 1.e-20)) mt = dmin(mt, fm::fdiv(c.SPLIT_MAXCFL * rho * r * sed_load(io.dzz, p), w));
      }
      remaint -= mt;
      // update, top-down with the flux of the level above (:806-830)
      const double frac = mt * inv_dt;
      double wa = 0.0;
      for (int k = io.nk - 1; k >= 0; --k) {
        const long p = (long)k * io.nij + col;
        const double r = io.rtmp[p];
        const double rho = sed_load(io.rhodref, p);
        const double w = gtp(r, sed_rtmin(c, s))
                             ? split_flux(c, s, r, rho, fm::flog(rho), sed_load(io.pabs, p), sed_load(io.tht, p), cp)
                             : 0.0;
        const double change = mt * fm::fdiv(1.0, rho * sed_load(io.dzz, p)) * (wa - w);
        io.rtmp[p] = r + change + io.ext[p] * mt;
        io.src[s][p] += change * inv_dt;
        if (io.fpr[s]) io.fpr[s][p] += w * frac;
        if (k == 0) inpr += w / c.RHOLW * frac;
        wa = w;
      }
    }
    if (io.inpr[s]) io.inpr[s][col] = inpr;
  }
  // ICE4_CORRECT_NEGATIVITIES with L/cph of the time-t state (rain_ice.F90:334-345)
  for (int k = 0; k < io.nk; ++k) {
    const long p = (long)k * io.nij + col;
    const double rv = sed_load(io.rvt, p), rc = sed_load(io.rt[0], p), rr = sed_load(io.rt[1], p);
    const double ri = sed_load(io.rt[2], p), rs = sed_load(io.rt[3], p), rg = sed_load(io.rt[4], p);
    const bool hail = io.nsp == 6;
    const double zice = hail ? ri + rs + rg + sed_load(io.rt[5], p) : ri + rs + rg;
    const double zdev = c.CPD + c.CPV * rv + c.CL * (rc + rr) + c.CI * zice;
    const double t = sed_load(io.tht, p) * sed_load(io.exn, p);
    const double ls = (c.LSTT + (c.CPV - c.CI) * (t - c.TT)) / zdev;
    const double lv = (c.LVTT + (c.CPV - c.CL) * (t - c.TT)) / zdev;
    double ths = io.ths[p], rvs = io.rvs[p], rcs = io.src[0][p], rrs = io.src[1][p], ris = io.src[2][p];
    double rss = io.src[3][p], rgs = io.src[4][p];
    double rhs = hail ? io.src[5][p] : 0.0;
    correct_negativities(c, lv, ls, ths, rvs, rcs, rrs, ris, rss, rgs, hail ? &rhs : nullptr);
    io.ths[p] = ths; io.rvs[p] = rvs; io.src[0][p] = rcs; io.src[1][p] = rrs; io.src[2][p] = ris;
    io.src[3][p] = rss; io.src[4][p] = rgs;
    if (hail) io.src[5][p] = rhs;
  }
  return ok;
}

}  // namespace ice3sed
