// The mixture of sub-mixtures as the assembly takes it (interior and boundary points), the time
// step and the secondary variables: mix_point of gales_magma.cuh rearranged for few FP64
// operations (see magma_props), the same to rounding, and rho and cv alone for the state at the
// previous time level.  The property calls and the gas fractions keep gales_magma.cuh's
// operations, which follow the reference's one by one.
// Also built for the host by the CPU tests.
#pragma once

#include "gales_magma.cuh"

namespace magma_mix {
namespace fast {

// ir = 1/rho, ic2 = 1/(rho c)^2 (the sound speed enters the mixture as that only).
struct Props {
  double rho, ir, cv, cp, kappa, D, mu, ic2, alpha, beta;
};

// The solubilities of H2O and CO2 at (p, T): linear interpolation on the equispaced pressure
// table (mixtures.hpp:342-356) or bilinear in (T, p) (380-412, tables [n_T][n_p]); both tables
// share the interval and the weights.
GALES_MAGMA_HD void lookup(const DevMagma& g, double T, double p, double& h2o, double& co2, unsigned& st) {
  const double* pt = g.p_tab;
  if (g.n_T == 0) {
    const double dp = pt[1] - pt[0];
    const double f = floor((p - pt[0]) / dp);
    long long i = (long long)f;
    if (!(f >= 0.0) || i + 1 >= g.n_p) {
      st |= GALES_MAGMA_LOOKUP_RANGE;
      i = i < 0 ? 0 : (i > g.n_p - 2 ? g.n_p - 2 : i);
      if (!(f == f)) i = 0;
    }
    const double t = (p - pt[i]) / dp;
    h2o = g.h2o_tab[i] + (g.h2o_tab[i + 1] - g.h2o_tab[i]) * t;
    co2 = g.co2_tab[i] + (g.co2_tab[i + 1] - g.co2_tab[i]) * t;
    return;
  }
  const double* Tt = g.T_tab;
  const double dp = fabs(pt[1] - pt[0]);
  const double dT = fabs(Tt[1] - Tt[0]);
  const double fp = floor(fabs(p - pt[0]) / dp), fT = floor(fabs(T - Tt[0]) / dT);
  long long pc = (long long)fp, Tr = (long long)fT;
  if (!(fp >= 0.0) || !(fT >= 0.0) || pc + 1 >= g.n_p || Tr + 1 >= g.n_T) {
    st |= GALES_MAGMA_LOOKUP_RANGE;
    pc = pc < 0 ? 0 : (pc > g.n_p - 2 ? g.n_p - 2 : pc);
    Tr = Tr < 0 ? 0 : (Tr > g.n_T - 2 ? g.n_T - 2 : Tr);
    if (!(fp == fp)) pc = 0;
    if (!(fT == fT)) Tr = 0;
  }
  const long long at = Tr * (long long)g.n_p + pc, up = at + g.n_p;
  const double r = 1.0 / (dT * dp);
  const double t2 = Tt[Tr + 1] - T, t1 = T - Tt[Tr], p2 = pt[pc + 1] - p, p1 = p - pt[pc];
  const double w0 = t2 * p2, w1 = t2 * p1, w2 = t1 * p2, w3 = t1 * p1;
  h2o = (w0 * g.h2o_tab[at] + w1 * g.h2o_tab[at + 1] + w2 * g.h2o_tab[up] + w3 * g.h2o_tab[up + 1]) * r;
  co2 = (w0 * g.co2_tab[at] + w1 * g.co2_tab[at + 1] + w2 * g.co2_tab[up] + w3 * g.co2_tab[up + 1]) * r;
}

// computeViscosity (GiordanoEtAlViscosityModel.hpp:88-116); WANT false: its checks alone.
template <bool WANT>
GALES_MAGMA_HD double giordano_mu(const DevMagma& g, double T, double wf_h2o_l, double wf_co2_l, unsigned& st) {
  const double b5 = -84.1, b6 = 141.5, c5 = -99.5;
  if (1.0 - wf_co2_l == 0.0) {
    st |= GALES_MAGMA_VISCOSITY;
    return 0.0;
  }
  // mole fraction of H2O in the melt without its CO2
  const double wm = wf_h2o_l * g.visc_M;
  const double x = wm / (wm + 18.015 * ((1 - wf_co2_l) - wf_h2o_l));
  const double x_no = 1 - x;
  const double pct = 100.0 * x;
  const double* P = g.visc_P;
  const double lg = log(1 + pct);
  const double Cv = P[4] * x_no + c5 * lg + P[5] * x_no * x_no + P[6] * x_no * pct;
  if (T - Cv == 0.0) {
    st |= GALES_MAGMA_VISCOSITY;
    return 0.0;
  }
  if (!WANT) return 0.0;
  const double Bv = P[1] * x_no + P[2] * x_no * x_no + P[3] * x_no * pct + (b5 + b6) * pct + b6 * lg;
#ifdef __CUDA_ARCH__
  return exp10(P[0] + Bv / (T - Cv));
#else
  return pow(10., P[0] + Bv / (T - Cv));
#endif
}

// x where the reference's square root of y has a value.
GALES_MAGMA_HD double where_real(double y, double x) { return y >= 0.0 ? x : NAN; }

// magma_mixture::properties (mixtures.hpp:163-176, submix_of_comp 187-250) of the melt
// (Lange-Carmichael volume), dissolved H2O and CO2 (one molar volume polynomial V(p, T),
// chemicals.hpp:155-160) and the two gases.  FULL false: rho (and 1/rho), cv and the status bits alone.
//
// Bound: FP64 operations, of which a division or square root is about ten and a library power
// over a hundred.  The constituents enter through 1/rho_c, alpha_c/rho_c, beta_c/rho_c and
// 1/(rho_c c_c)^2 = beta_c/rho_c (gases: over gamma), which are polynomials over p here; with
// every constituent's rho, alpha, beta and c formed and divided by again, std::pow for squares and
// the viscosity of both states, a point's two states of two magmas took some 8,000 operations
// (point stage of 25,600 triangles 1.14 ms); now 0.27 ms.  Against 80-bit arithmetic every
// property is as accurate as in the reference's order or more so (rho 1.5e-16 for 1.9e-16, beta
// 3.2e-16 for 3.3e-16; the viscosity's 7.4e-15 come from its exponent).
template <bool FULL>
GALES_MAGMA_HD void magma_props(const DevMagma& g, double p, double T, double sr, Props& o, double& vf_gas,
                                unsigned& st) {
  double wl1, wl2;
  lookup(g, T, p, wl1, wl2, st);
  const double wl0 = 1.0 - wl1 - wl2;
  double wf[5];
  wf[0] = g.wf_comp[0];
  const double wl_ph = wf[0] / wl0;
  wf[1] = wl1 * wl_ph;
  wf[2] = wl2 * wl_ph;
  wf[3] = g.wf_comp[1] - wf[1];
  wf[4] = g.wf_comp[2] - wf[2];
  // melt volume; the dissolved volatiles' molar volume V, dV/dT and -dV/dp
  const double mv = g.melt_V + g.melt_dVdT * (T - 1673.0) + g.melt_dVdp * (p - 1.e5);
  const double a[10] = {9.144e-06, 3.685e-09, 1.168e-11, -1.990e-15, 1.220e-16,
                        -1.945e-17, -1.580e-21, 4.680e-24, 1.144e-26, -3.960e-33};
  const double V = a[0] + a[1] * T + a[2] * T * T + a[3] * T * T * T + p * (a[4] + a[5] * T + a[6] * T * T) +
                   p * p * (a[7] + a[8] * T) + a[9] * p * p * p;
  const double VT = a[1] + 2 * a[2] * T + 3 * a[3] * T * T + p * (a[5] + 2 * a[6] * T) + p * p * a[8];
  const double Vp = -((a[4] + a[5] * T + a[6] * T * T) + 2 * p * (a[7] + a[8] * T) + 3 * a[9] * p * p);
  const double ip = 1.0 / p, Tp = T * ip;
  const double ir3 = g.gas_R[0] * Tp, ir4 = g.gas_R[1] * Tp;
  // wf_c over the molar masses
  const double m0 = g.melt_m0, m12 = wf[1] * g.vol_iM[0] + wf[2] * g.vol_iM[1];
  const double ir = fma(m0, mv, fma(m12, V, fma(wf[3], ir3, wf[4] * ir4)));
  double rho = 1. / ir;
  rho = (1.0 - g.crystal_vf) * rho + g.crystal_vf * g.crystal_rho;
  // cv = cp - T alpha^2/(rho beta)
  const double qV = T * (VT * VT / Vp);
  o.rho = rho;
  o.ir = g.crystal_vf == 0.0 ? ir : 1.0 / rho;
  o.cv = wf[0] * (g.melt_cp - T * g.melt_q) + wf[1] * (g.vol_cp[0] - qV * g.vol_iM[0]) +
         wf[2] * (g.vol_cp[1] - qV * g.vol_iM[1]) + wf[3] * g.gas_cv[0] + wf[4] * g.gas_cv[1];
  if (!FULL) {
    giordano_mu<false>(g, T, wl1, wl2, st);
    return;
  }
  const double Rg = wf[3] * g.gas_R[0] + wf[4] * g.gas_R[1];
  const double bl = where_real(-g.melt_dVdp, m0 * -g.melt_dVdp) + where_real(Vp, m12 * Vp);
  o.alpha = rho * fma(m0, g.melt_dVdT, fma(m12, VT, Rg * ip));
  o.beta = rho * fma(m0, -g.melt_dVdp, fma(m12, Vp, Rg * (Tp * ip)));
  o.ic2 = bl + (T > 0.0 ? (wf[3] * g.gas_R[0] * g.gas_ig[0] + wf[4] * g.gas_R[1] * g.gas_ig[1]) * (Tp * ip) : NAN);
  o.cp = wf[0] * g.melt_cp + wf[1] * g.vol_cp[0] + wf[2] * g.vol_cp[1] + wf[3] * g.gas_cp[0] + wf[4] * g.gas_cp[1];
  o.kappa = wf[0] * g.melt_kappa + wf[1] * g.vol_kappa[0] + wf[2] * g.vol_kappa[1] + wf[3] * g.gas_kappa[0] +
            wf[4] * g.gas_kappa[1];
  o.D = (wf[0] + wf[1] + wf[2] + wf[3] + wf[4]) * 1.e-10;
  vf_gas = wf[3] * rho * ir3 + wf[4] * rho * ir4;
  double mu = giordano_mu<true>(g, T, wl1, wl2, st);
  if (g.gas_on_mu == GALES_GAS_MU_ISHII_ZUBER) {
    mu = mu / (1.0 - vf_gas);
  } else if (g.gas_on_mu == GALES_GAS_MU_PAL_2003 && !(sr < 2.220446049250313e-16)) {
    const double Ca = g.bubble_r * mu * sr / 0.36;
    const double a2 = 2.4 * (Ca * Ca);
    const double TT = pow(1.0 - a2, -0.8) * pow(1.0 - vf_gas / 0.9999, -0.9999);
    const double TT2 = TT * TT, TT5 = TT2 * TT2 * TT;
    double x = 1.e-5, F;
    int it = 0;
    do {
      const double x2 = x * x, x4 = x2 * x2, y = 1.0 - a2 * x2, y2 = y * y, y4 = y2 * y2;
      F = x4 * x / y4 - TT5;
      const double Fp = 5 * x4 / y4 + 8 * a2 * (x4 * x2) / (y4 * y);
      x -= F / Fp;
    } while (F < 1.e-9 && ++it < 200);
    if (it >= 200) st |= GALES_MAGMA_PAL_ITER;
    mu = mu * x;
  }
  if (g.crystal_on_mu == GALES_CRYSTAL_MU_EINSTEIN_ROSCOE) {
    mu = mu * g.crystal_er;
  } else if (g.crystal_on_mu == GALES_CRYSTAL_MU_CARICCHI) {
    const double s = sr < 2.220446049250313e-16 ? 1.e-6 : sr;
    const double ls = log10(s);
    const double phi_max = 0.066499 * tanh(0.913424 * ls + 3.850623) + 0.591806;
    const double delta = -6.301095 * tanh(0.818496 * ls + 2.86) + 7.462405;
    const double alpha_c = -0.000378 * tanh(1.148101 * ls + 3.92) + 0.999572;
    const double gamma = 3.987815 * tanh(0.8908 * ls + 3.24) + 5.099645;
    const double phi = g.crystal_vf;
    const double num = 1.0 + pow(phi / phi_max, delta);
    const double xx = sqrt(3.142) * phi / (2 * alpha_c * phi_max) * (1.0 + pow(phi / phi_max, gamma));
    const double den = pow(1.0 - alpha_c * erf(xx), 2.5 * phi_max);
    mu = mu * (num / den);
  }
  o.mu = mu;
}

// A sub-mixture of any kind at (p, T) (see sub_props of gales_magma.cuh).
template <bool FULL>
GALES_MAGMA_HD void sub_props(const DevMagma& g, double p, double T, double sr, Props& o, double& vf_gas,
                              unsigned& st) {
  if (g.kind == GALES_SUBMIX_MAGMA) {
    magma_props<FULL>(g, p, T, sr, o, vf_gas, st);
    return;
  }
  vf_gas = 0.0;
  o.D = 1.e-10;
  double c;
  if (g.ch_kind == GALES_CH_CUSTOM) {
    o.rho = g.ch_rho;
    o.mu = g.ch_mu;
    o.cp = g.ch_cp;
    o.kappa = g.ch_kappa;
    o.alpha = g.ch_alpha;
    o.beta = g.ch_beta;
    c = (o.beta == 0.0) ? 1.e20 : 1.0 / sqrt(o.rho * o.beta);
    o.cv = (o.beta == 0.0) ? o.cp : o.cp - T * o.alpha * o.alpha / (o.rho * o.beta);
  } else {
    o.rho = p / (g.ch_R * T);
    o.beta = 1.0 / p;
    o.alpha = 1.0 / T;
    c = sqrt(g.ch_gamma * g.ch_R * T);
    o.cv = g.ch_cv;
    o.cp = g.ch_cp;
    o.mu = g.ch_mu;
    o.kappa = g.ch_kappa;
  }
  o.ir = 1.0 / o.rho;
  o.ic2 = 1.0 / ((o.rho * o.rho) * (c * c));
}

// One point of the mixture of sub-mixtures (fluid_properties.hpp:171-200):
// f = rho, mu, cp, cv, kappa, sound speed, alpha, beta; comp[c] = rho_c, cv_c T, chemical
// diffusivity, gas volume fraction.  Returns the status bits.
GALES_MAGMA_HD unsigned mix_point(const DevMagma* mg, int nc, double p, double T, const double* Y, double sr,
                                  double* f, double (*comp)[4]) {
  unsigned st = 0;
  double irho = 0, mu = 0, cp = 0, cv = 0, kappa = 0, ss = 0, alpha = 0, beta = 0;
  for (int c = 0; c < nc; ++c) {
    Props m;
    double vfg;
    sub_props<true>(mg[c], p, T, sr, m, vfg, st);
    const double y = Y[c], yr = y * m.ir;
    irho = fma(y, m.ir, irho);
    mu += y * m.mu;
    cp += y * m.cp;
    cv = fma(y, m.cv, cv);
    kappa += y * m.kappa;
    ss += y * m.ic2;
    alpha = fma(yr, m.alpha, alpha);
    beta = fma(yr, m.beta, beta);
    comp[c][0] = m.rho;
    comp[c][1] = m.cv * T;
    comp[c][2] = m.D;
    comp[c][3] = vfg;
  }
  const double rho = 1.0 / irho;
  f[0] = rho;
  f[1] = mu;
  f[2] = cp;
  f[3] = cv;
  f[4] = kappa;
  f[5] = irho / sqrt(ss);
  f[6] = alpha * rho;
  f[7] = beta * rho;
  return st;
}

// rho and cv of mix_point at shear rate 0, with its status bits (the state at the previous time
// level, of which the assembly reads nothing else): its operations, so that equal states have
// equal rho and cv.
GALES_MAGMA_HD unsigned mix_rho_cv(const DevMagma* mg, int nc, double p, double T, const double* Y, double& rho,
                                   double& cv) {
  unsigned st = 0;
  double irho = 0, x = 0;
  for (int c = 0; c < nc; ++c) {
    Props m;
    double vfg;
    sub_props<false>(mg[c], p, T, 0.0, m, vfg, st);
    irho = fma(Y[c], m.ir, irho);
    x = fma(Y[c], m.cv, x);
  }
  rho = 1.0 / irho;
  cv = x;
  return st;
}

}  // namespace fast
}  // namespace magma_mix
