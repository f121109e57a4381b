// Exact vector-Jacobian product of the assembled rhs, point level.
//
// The interior element residual of fluid_2d.hpp:251-305 at one quadrature point is
//   r_b += JxW [ N_b phi0 + sum_d dN_b/dx_d phi_d ]            with
//   phi0  = (U - U_P)/dt - S - S0 tau Res
//   phi_d = F_dif,d - F_adv,d + nu DUDY dI/dx_d + A_d tau Res
// (the least-squares weight FPT_b = (sum_d dN_b/dx_d A_d - N_b S0) tau split by node
// factor).  point_forward evaluates (phi0, phi_d) from the interpolated state Iq, its
// gradient dI and the previous level Pq in FP64 with every coefficient a function of
// the state and of the material parameters theta_c = (density parameter, mu_c, cp_c);
// point_reverse propagates cotangents (phi0_bar, phi_d_bar) back to Iq, dI and theta
// by hand-written reverse mode through tau (with compute_h and the DUDY inverse),
// the dc viscosity, the mixture EOS and U_P.  Nothing is stored between calls: the
// caller recomputes the point from the state.  The dc scaling u_ref_inv is itself a
// function of theta (fluid_2d.hpp:123-135, the mixture at p_ref, T_ref, Y_ref); its
// cotangent is returned in urib for the caller to fold into theta.
//
// Parameterisation (the derivative's meaning):
//   custom chemical (chemicals.hpp:19-49): theta = (rho_c, mu_c, cp_c); alpha, beta,
//     kappa fixed; cv_c = cp_c - T alpha^2/(rho_c beta) (beta != 0), else cp_c.
//   ideal gas (chemicals.hpp:198-271): theta = (M_c, mu_c, cp_c) with R_c = R_u/M_c,
//     cv_c = cp_c - R_c, gamma_c = cp_c/cv_c; kappa fixed.
// Everything here is __host__ __device__ so the same code can be checked on the CPU.
#pragma once

#include <cmath>

#include "gales_physics.cuh"

namespace gales {
namespace vjp {

#define GV_HD __host__ __device__ __forceinline__

constexpr double kRu = 8.314462;  // chemicals.hpp:229

template <int DIM, int NC>
struct Ctx {
  static constexpr int ND = Layout<DIM, NC>::ND;
  const DevChem* ch;
  double dt, inv_dt, dc_sharp, dc_scale;
  double gravity[3];
  const double* u_ref_inv;
  int tau, dc_2006, steady;
};

// Per point geometry used by tau and dc.
template <int DIM, int NEN>
struct PGeo {
  double G[DIM][DIM], trG;
  double ds[DIM][NEN];
};

template <int DIM>
GV_HD double dot(const double* a, const double* b) {
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < DIM; ++i) s += a[i] * b[i];
  return s;
}

// ---------------------------------------------------------------------------
// Mixture EOS (fluid_properties.hpp:199-227) with its tape, in reciprocals: ir_c = 1/rho_c
// (a gas has R T/p), A_c = alpha_c/rho_c and B_c = beta_c/rho_c, so that a state takes 1/p,
// 1/rho and 1/sqrt(c2) and no division per component; the component constants of a point's two
// states are formed once (CompK).
struct CompK {
  double ir, cvs, ig;   // custom: 1/rho, alpha^2/(rho beta); gas: 1/gamma = (cp - R)/cp
};

template <int NC>
struct Mix {
  double Y[NC];
  double ir[NC], cvc[NC], c2t[NC];   // 1/rho_c, cv_c, Y-free sound-speed term 1/(rho_c^2 s_c^2)
  double A[NC], B[NC];
  double ip, irho, rho, mu, cp, cv, kappa, c2, isc, c, alpha, beta;
};

GV_HD void comp_const(const DevChem& q, CompK& k) {
  if (q.kind == GALES_CH_CUSTOM) {
    k.ir = 1.0 / q.rho;
    k.cvs = q.beta == 0.0 ? 0.0 : q.alpha * q.alpha / (q.rho * q.beta);
    k.ig = 0.0;
  } else {
    k.ir = k.cvs = 0.0;
    k.ig = (q.cp - q.R) / q.cp;
  }
}

template <int NC>
GV_HD void mix_forward(const DevChem* ch, const CompK* kc, double p, double T, const double* Y, Mix<NC>& m) {
  double irho = 0.0, mu = 0.0, cp = 0.0, cv = 0.0, kappa = 0.0, c2 = 0.0, al = 0.0, be = 0.0;
  bool gas = false;   // a material without a gas never divides by p
#pragma unroll
  for (int c = 0; c < NC; ++c) gas |= ch[c].kind != GALES_CH_CUSTOM;
  m.ip = gas ? 1.0 / p : 0.0;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const DevChem& q = ch[c];
    m.Y[c] = Y[c];
    if (q.kind == GALES_CH_CUSTOM) {
      m.ir[c] = kc[c].ir;
      m.cvc[c] = q.cp - T * kc[c].cvs;
      m.A[c] = q.alpha * kc[c].ir;
      m.B[c] = q.beta * kc[c].ir;
      m.c2t[c] = q.beta == 0.0 ? 1.e-40 * kc[c].ir * kc[c].ir : m.B[c];   // s^2 = 1/(rho beta)
    } else {
      m.A[c] = q.R * m.ip;
      m.ir[c] = m.A[c] * T;
      m.B[c] = m.ir[c] * m.ip;
      m.cvc[c] = q.cp - q.R;
      m.c2t[c] = m.B[c] * kc[c].ig;
    }
    irho += Y[c] * m.ir[c];
    mu += Y[c] * q.mu;
    cp += Y[c] * q.cp;
    cv += Y[c] * m.cvc[c];
    kappa += Y[c] * q.kappa;
    c2 += Y[c] * m.c2t[c];
    al += Y[c] * m.A[c];
    be += Y[c] * m.B[c];
  }
  m.irho = irho;
  m.rho = 1.0 / irho;
  m.mu = mu; m.cp = cp; m.cv = cv; m.kappa = kappa; m.c2 = c2;
  m.isc = 1.0 / sqrt(c2);
  m.c = irho * m.isc;
  m.alpha = m.rho * al;
  m.beta = m.rho * be;
}

// Cotangents of the mixture outputs.
struct MixBar {
  double rho, mu, cp, cv, kappa, c, alpha, beta;
};

// irb, cvcb: the components' 1/rho_c and cv_c cotangents from the coefficient layer.
template <int NC>
GV_HD void mix_reverse(const DevChem* ch, const CompK* kc, double T, const Mix<NC>& m, const MixBar& o,
                       const double* irb_in, const double* cvcb, double& pb, double& Tb, double* Yb, double* th) {
  // outputs: rho = 1/irho, c = irho/sqrt(c2), alpha = rho sum Y A, beta = rho sum Y B
  const double rhob = o.rho + (o.alpha * m.alpha + o.beta * m.beta) * m.irho;
  const double alb = o.alpha * m.rho, beb = o.beta * m.rho;
  const double irhob = o.c * m.isc - rhob * m.rho * m.rho;
  const double c2b = o.c * (-0.5 * m.irho * m.isc * m.isc * m.isc);
  double ipb = 0.0;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const DevChem& q = ch[c];
    const double Yc = m.Y[c];
    const double irb = irb_in[c] + irhob * Yc, cvb = cvcb[c] + o.cv * Yc;
    const double c2tb = c2b * Yc, Ab = alb * Yc, Bb = beb * Yc;
    Yb[c] += irhob * m.ir[c] + o.mu * q.mu + o.cp * q.cp + o.cv * m.cvc[c] + o.kappa * q.kappa + c2b * m.c2t[c] +
             alb * m.A[c] + beb * m.B[c];
    th[3 * c + 1] += o.mu * Yc;
    th[3 * c + 2] += o.cp * Yc + cvb;
    if (q.kind == GALES_CH_CUSTOM) {
      const double ir = kc[c].ir;
      const double it = irb + Ab * q.alpha + Bb * q.beta + c2tb * (q.beta == 0.0 ? 2.e-40 * ir : q.beta);
      th[3 * c] += cvb * T * kc[c].cvs * ir - it * ir * ir;   // cv = cp - T alpha^2/(rho beta)
      Tb -= cvb * kc[c].cvs;
    } else {
      // A = R/p, ir = A T, B = ir/p, c2t = B (cp - R)/cp
      const double Bt = Bb + c2tb * kc[c].ig;
      const double it = irb + Bt * m.ip, At = Ab + it * T;
      ipb += Bt * m.ir[c] + At * q.R;
      Tb += it * m.A[c];
      const double x = c2tb * m.B[c] / q.cp;     // (cp - R)/cp: -1/cp in R, R/cp^2 in cp
      const double Rb = At * m.ip - x - cvb;
      th[3 * c + 2] += x * (1.0 - kc[c].ig);
      th[3 * c] += Rb * (-q.R * q.R / kRu);      // theta_0 = M, R = R_u/M
    }
  }
  pb -= ipb * m.ip * m.ip;
}

// The previous level: rho and cv alone (what U_P needs), and their parameter cotangents.
template <int NC>
struct MixP {
  double Y[NC], ir[NC], ip, rho, cv;
};

template <int NC>
GV_HD void mixp_forward(const DevChem* ch, const CompK* kc, double p, double T, const double* Y, MixP<NC>& m) {
  double irho = 0.0, cv = 0.0;
  bool gas = false;
#pragma unroll
  for (int c = 0; c < NC; ++c) gas |= ch[c].kind != GALES_CH_CUSTOM;
  m.ip = gas ? 1.0 / p : 0.0;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const DevChem& q = ch[c];
    const bool custom = q.kind == GALES_CH_CUSTOM;
    m.Y[c] = Y[c];
    m.ir[c] = custom ? kc[c].ir : q.R * m.ip * T;
    irho += Y[c] * m.ir[c];
    cv += Y[c] * (custom ? q.cp - T * kc[c].cvs : q.cp - q.R);
  }
  m.rho = 1.0 / irho;
  m.cv = cv;
}

template <int NC>
GV_HD void mixp_reverse(const DevChem* ch, const CompK* kc, double T, const MixP<NC>& m, double rhob, double cvb_mix,
                        double* th) {
  const double irhob = -rhob * m.rho * m.rho;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const DevChem& q = ch[c];
    const double irb = irhob * m.Y[c], cvb = cvb_mix * m.Y[c];
    th[3 * c + 2] += cvb;
    if (q.kind == GALES_CH_CUSTOM) {
      const double ir = kc[c].ir;
      th[3 * c] += cvb * T * kc[c].cvs * ir - irb * ir * ir;
    } else {
      th[3 * c] += (irb * T * m.ip - cvb) * (-q.R * q.R / kRu);
    }
  }
}

// ---------------------------------------------------------------------------
// Coefficient scalars (fluid_2d.hpp:393-404, 531-533) and the structure vectors of
// DUDY = w r0^T + rho M: w = (1, v, E, Y), r0 its first row, mE the energy row of M,
// u' = U + p e_E.
template <int DIM, int NC>
struct Cf {
  using L = Layout<DIM, NC>;
  static constexpr int ND = L::ND;
  double p, v[DIM], T, Y[NC];
  double rho, E, drho_dp, drho_dT, de_dp, de_dT, mu, lam, kappa, cv, cp;
  double drho_dY[L::NYA], dE_dY[L::NYA], H[L::NYA], rhoD[L::NYA], rhoDH[L::NYA];
  double w[ND], r0[ND], mE[ND];
};

template <int DIM, int NC>
struct CfBar {
  using L = Layout<DIM, NC>;
  static constexpr int ND = L::ND;
  double p, v[DIM], T, Y[NC];
  double rho, E, drho_dp, drho_dT, de_dp, de_dT, mu, lam, kappa;
  double drho_dY[L::NYA], dE_dY[L::NYA], rhoD[L::NYA], rhoDH[L::NYA];
  double w[ND], r0[ND], mE[ND];
};

template <int DIM, int NC>
GV_HD void coef_forward(const Mix<NC>& m, const DevChem* ch, double p, const double* v, double T, Cf<DIM, NC>& c) {
  using L = Layout<DIM, NC>;
  c.p = p; c.T = T;
#pragma unroll
  for (int k = 0; k < DIM; ++k) c.v[k] = v[k];
#pragma unroll
  for (int i = 0; i < NC; ++i) c.Y[i] = m.Y[i];
  const double rho = m.rho;
  c.rho = rho; c.cv = m.cv; c.cp = m.cp;
  c.E = m.cv * T + 0.5 * dot<DIM>(v, v);
  c.drho_dp = rho * m.beta;
  c.drho_dT = -rho * m.alpha;
  c.de_dp = (m.beta * p - m.alpha * T) * m.irho;
  c.de_dT = m.cp - p * m.alpha * m.irho;
  c.mu = m.mu;
  c.lam = (-2.0 / 3.0) * m.mu;
  c.kappa = m.kappa;
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) {
    c.drho_dY[i] = -rho * rho * (m.ir[i] - m.ir[NC - 1]);
    c.dE_dY[i] = m.cvc[i] * T - m.cvc[NC - 1] * T;
    c.H[i] = m.cvc[i] * T + p * m.ir[i];
    c.rhoD[i] = rho * ch[i].D;
    c.rhoDH[i] = c.rhoD[i] * c.H[i];
  }
  c.w[0] = 1.0; c.r0[0] = c.drho_dp; c.mE[0] = c.de_dp;
#pragma unroll
  for (int k = 0; k < DIM; ++k) { c.w[1 + k] = v[k]; c.r0[1 + k] = 0.0; c.mE[1 + k] = v[k]; }
  c.w[L::iT] = c.E; c.r0[L::iT] = c.drho_dT; c.mE[L::iT] = c.de_dT;
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) {
    c.w[L::iY + i] = m.Y[i]; c.r0[L::iY + i] = c.drho_dY[i]; c.mE[L::iY + i] = c.dE_dY[i];
  }
}

template <int DIM, int NC>
GV_HD void cfbar_zero(CfBar<DIM, NC>& b) {
  double* x = reinterpret_cast<double*>(&b);
  for (unsigned i = 0; i < sizeof(CfBar<DIM, NC>) / sizeof(double); ++i) x[i] = 0.0;
}

// Fold the structure-vector cotangents (w, r0, mE) into the scalar ones.
template <int DIM, int NC>
GV_HD void cfbar_fold(CfBar<DIM, NC>& b) {
  using L = Layout<DIM, NC>;
  b.drho_dp += b.r0[0]; b.de_dp += b.mE[0];
#pragma unroll
  for (int k = 0; k < DIM; ++k) b.v[k] += b.w[1 + k] + b.mE[1 + k];
  b.E += b.w[L::iT]; b.drho_dT += b.r0[L::iT]; b.de_dT += b.mE[L::iT];
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) {
    b.Y[i] += b.w[L::iY + i]; b.drho_dY[i] += b.r0[L::iY + i]; b.dE_dY[i] += b.mE[L::iY + i];
  }
}

// Coefficient layer reverse: scalar cotangents -> mixture cotangents, per-component
// 1/rho_c / cv_c cotangents, and direct state cotangents (p, v, T).
template <int DIM, int NC>
GV_HD void coef_reverse(const Mix<NC>& m, const DevChem* ch, const Cf<DIM, NC>& c, const CfBar<DIM, NC>& b,
                        MixBar& o, double* irb, double* cvcb, double& pb, double* vb, double& Tb, double* Yb) {
  const double rho = m.rho, irho = m.irho, p = c.p, T = c.T;
  o = MixBar{0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < NC; ++i) { irb[i] = 0.0; cvcb[i] = 0.0; }
  // E = cv T + |v|^2/2
  o.cv += b.E * T; Tb += b.E * m.cv;
#pragma unroll
  for (int k = 0; k < DIM; ++k) vb[k] += b.E * c.v[k] + b.v[k];
  pb += b.p; Tb += b.T;
#pragma unroll
  for (int i = 0; i < NC; ++i) Yb[i] += b.Y[i];
  o.rho += b.rho;
  // drho_dp = rho beta, drho_dT = -rho alpha
  o.rho += b.drho_dp * m.beta - b.drho_dT * m.alpha;
  o.beta += b.drho_dp * rho;
  o.alpha -= b.drho_dT * rho;
  // de_dp = (beta p - alpha T)/rho, de_dT = cp - p alpha/rho
  const double g = b.de_dp * irho, f = b.de_dT * irho;
  o.beta += g * p;
  o.alpha -= g * T + f * p;
  pb += g * m.beta - f * m.alpha;
  Tb -= g * m.alpha;
  o.rho += (f * p * m.alpha) * irho - g * c.de_dp;
  o.cp += b.de_dT;
  o.mu += b.mu - (2.0 / 3.0) * b.lam;
  o.kappa += b.kappa;
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) {
    const int n = NC - 1;
    // drho_dY = -rho^2 (1/rho_i - 1/rho_n)
    o.rho += b.drho_dY[i] * (-2.0 * rho * (m.ir[i] - m.ir[n]));
    irb[i] -= b.drho_dY[i] * (rho * rho);
    irb[n] += b.drho_dY[i] * (rho * rho);
    // dE_dY = (cv_i - cv_n) T
    cvcb[i] += b.dE_dY[i] * T;
    cvcb[n] -= b.dE_dY[i] * T;
    Tb += b.dE_dY[i] * (m.cvc[i] - m.cvc[n]);
    // rhoD = rho D, rhoDH = rho D H with H = cv_i T + p/rho_i
    o.rho += b.rhoD[i] * ch[i].D + b.rhoDH[i] * ch[i].D * c.H[i];
    const double Hb = b.rhoDH[i] * c.rhoD[i];
    cvcb[i] += Hb * T;
    Tb += Hb * m.cvc[i];
    pb += Hb * m.ir[i];
    irb[i] += Hb * p;
  }
}

// ---------------------------------------------------------------------------
// Products with DUDY and the adjoint of the bilinear form x^T DUDY y (weight s):
//   x^T DUDY y = (x.w)(r0.y) + rho (sum_{r in v,Y} x_r y_r + x_E mE.y)
//   x^T A_d y  = v_d x^T DUDY y + (x.u') y_{v_d} + (x_{v_d} + v_d x_E) y_p
template <int DIM, int NC>
GV_HD void Dy(const Cf<DIM, NC>& c, const double* y, double* out) {  // DUDY y
  using L = Layout<DIM, NC>;
  constexpr int ND = L::ND;
  double ry = 0.0, my = 0.0;
#pragma unroll
  for (int j = 0; j < ND; ++j) {
    if (j < 1 || j >= L::iT) ry += c.r0[j] * y[j];
    my += c.mE[j] * y[j];
  }
#pragma unroll
  for (int r = 0; r < ND; ++r) {
    const double m = r == L::iT ? my : y[r];
    out[r] = r == 0 ? ry : c.w[r] * ry + c.rho * m;
  }
}

template <int DIM, int NC>
GV_HD double xw_of(const Cf<DIM, NC>& c, const double* x) {  // x.w
  double xw = x[0];
#pragma unroll
  for (int j = 1; j < Layout<DIM, NC>::ND; ++j) xw += x[j] * c.w[j];
  return xw;
}

template <int DIM, int NC>
GV_HD void DTx(const Cf<DIM, NC>& c, const double* x, double* out) {  // DUDY^T x
  using L = Layout<DIM, NC>;
  constexpr int ND = L::ND;
  const double xw = xw_of<DIM, NC>(c, x), re = c.rho * x[L::iT];
#pragma unroll
  for (int j = 0; j < ND; ++j) {
    double o = re * c.mE[j];
    if (j >= 1 && j != L::iT) o += c.rho * x[j];
    if (j < 1 || j >= L::iT) o += c.r0[j] * xw;
    out[j] = o;
  }
}

template <int DIM, int NC>
GV_HD void xDy_rev(const Cf<DIM, NC>& c, const double* x, const double* y, double s, CfBar<DIM, NC>& b) {
  using L = Layout<DIM, NC>;
  constexpr int ND = L::ND;
  double ry = 0.0, my = 0.0, d = 0.0;
#pragma unroll
  for (int j = 0; j < ND; ++j) {
    if (j < 1 || j >= L::iT) ry += c.r0[j] * y[j];
    my += c.mE[j] * y[j];
    if (j >= 1 && j != L::iT) d += x[j] * y[j];
  }
  const double sw = s * xw_of<DIM, NC>(c, x), sr = s * ry, sm = s * c.rho * x[L::iT];
#pragma unroll
  for (int j = 0; j < ND; ++j) {
    if (j > 0) b.w[j] += sr * x[j];
    if (j < 1 || j >= L::iT) b.r0[j] += sw * y[j];
    b.mE[j] += sm * y[j];
  }
  b.rho += s * (d + x[L::iT] * my);
}

// ---------------------------------------------------------------------------
// compute_h (quad.hpp:356-383, 701-739) with its tape and adjoint.
template <int DIM>
struct HTape {
  double nv, s0[DIM], acc[DIM], ip, s1[DIM], n1, s1n[DIM], s2[3], n2, s2n[3], alpha[3], Q;
  bool norm1, norm2;
};

// The steps that decide compute_h's branches are never fused into multiply-adds, whatever the
// translation unit's setting (on the host the unit is compiled without contraction).
#ifdef __CUDA_ARCH__
GV_HD double hmul(double a, double b) { return __dmul_rn(a, b); }
GV_HD double hadd(double a, double b) { return __dadd_rn(a, b); }
GV_HD double hsub(double a, double b) { return __dsub_rn(a, b); }
#else
GV_HD double hmul(double a, double b) { return a * b; }
GV_HD double hadd(double a, double b) { return a + b; }
GV_HD double hsub(double a, double b) { return a - b; }
#endif

template <int DIM>
GV_HD double hdot(const double* a, const double* b) {
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < DIM; ++i) s = hadd(s, hmul(a[i], b[i]));
  return s;
}

template <int DIM>
GV_HD double quadform(const double (&G)[DIM][DIM], const double* s) {
  double r = 0.0;
#pragma unroll
  for (int i = 0; i < DIM; ++i) {
    double t = 0.0;
#pragma unroll
    for (int j = 0; j < DIM; ++j) t += G[i][j] * s[j];
    r += s[i] * t;
  }
  return r;
}

template <int DIM>
GV_HD void quadform_rev(const double (&G)[DIM][DIM], const double* s, double ab, double* sb) {
#pragma unroll
  for (int i = 0; i < DIM; ++i) {
    double t = 0.0;
#pragma unroll
    for (int j = 0; j < DIM; ++j) t += (G[i][j] + G[j][i]) * s[j];
    sb[i] += ab * t;
  }
}

template <int DIM>
GV_HD double compute_h_fwd(const double (&G)[DIM][DIM], const double* v, const double (&dv)[DIM][DIM],
                           HTape<DIM>& t) {
  t.nv = sqrt(hdot<DIM>(v, v));
#pragma unroll
  for (int i = 0; i < DIM; ++i) t.s0[i] = v[i] / t.nv;
  t.alpha[0] = quadform<DIM>(G, t.s0);
#pragma unroll
  for (int i = 0; i < DIM; ++i) t.acc[i] = hdot<DIM>(dv[i], v);
  t.ip = hdot<DIM>(t.acc, t.s0);
#pragma unroll
  for (int i = 0; i < DIM; ++i) t.s1[i] = hsub(t.acc[i], hmul(t.ip, t.s0[i]));
  t.n1 = sqrt(hdot<DIM>(t.s1, t.s1));
  t.norm1 = t.n1 > kEps;
  const double in1 = t.norm1 ? 1.0 / t.n1 : 1.0;
#pragma unroll
  for (int i = 0; i < DIM; ++i) t.s1n[i] = t.s1[i] * in1;
  t.alpha[1] = quadform<DIM>(G, t.s1n);
  t.alpha[2] = 0.0;
  t.norm2 = false;
  if constexpr (DIM == 3) {
    t.s2[0] = hsub(hmul(t.s0[1], t.s1n[2]), hmul(t.s0[2], t.s1n[1]));
    t.s2[1] = hsub(hmul(t.s1n[0], t.s0[2]), hmul(t.s1n[2], t.s0[0]));
    t.s2[2] = hsub(hmul(t.s0[0], t.s1n[1]), hmul(t.s0[1], t.s1n[0]));
    t.n2 = sqrt(hdot<3>(t.s2, t.s2));
    t.norm2 = t.n2 > kEps;
    const double in2 = t.norm2 ? 1.0 / t.n2 : 1.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) t.s2n[i] = t.s2[i] * in2;
    t.alpha[2] = quadform<DIM>(G, t.s2n);
  }
  double Q = 0.0;
#pragma unroll
  for (int i = 0; i < DIM; ++i)
    if (t.alpha[i] != 0.0) Q += 1.0 / t.alpha[i];
  t.Q = Q;
  return 2.0 * sqrt(fabs(Q));
}

template <int DIM>
GV_HD void normalise_rev(const double* sn, double n, bool norm, const double* snb, double* sb) {
  if (!norm) {
#pragma unroll
    for (int i = 0; i < DIM; ++i) sb[i] += snb[i];
    return;
  }
  const double pr = dot<DIM>(snb, sn), in = 1.0 / n;
#pragma unroll
  for (int i = 0; i < DIM; ++i) sb[i] += (snb[i] - pr * sn[i]) * in;
}

template <int DIM>
GV_HD void compute_h_rev(const double (&G)[DIM][DIM], const double* v, const double (&dv)[DIM][DIM],
                         const HTape<DIM>& t, double hb, double* vb, double (&dvb)[DIM][DIM]) {
  if (t.Q == 0.0) return;
  const double Qb = hb * (t.Q > 0.0 ? 1.0 : -1.0) / sqrt(fabs(t.Q));
  double s0b[DIM], s1nb[DIM], s1b[DIM], accb[DIM];
#pragma unroll
  for (int i = 0; i < DIM; ++i) { s0b[i] = 0.0; s1nb[i] = 0.0; s1b[i] = 0.0; accb[i] = 0.0; }
  if constexpr (DIM == 3) {
    if (t.alpha[2] != 0.0) {
      double s2nb[3] = {0, 0, 0}, s2b[3] = {0, 0, 0};
      quadform_rev<DIM>(G, t.s2n, -Qb / (t.alpha[2] * t.alpha[2]), s2nb);
      normalise_rev<3>(t.s2n, t.n2, t.norm2, s2nb, s2b);
      // s2 = s0 x s1n: s0b += s1n x s2b, s1nb += s2b x s0
      s0b[0] += t.s1n[1] * s2b[2] - t.s1n[2] * s2b[1];
      s0b[1] += t.s1n[2] * s2b[0] - t.s1n[0] * s2b[2];
      s0b[2] += t.s1n[0] * s2b[1] - t.s1n[1] * s2b[0];
      s1nb[0] += s2b[1] * t.s0[2] - s2b[2] * t.s0[1];
      s1nb[1] += s2b[2] * t.s0[0] - s2b[0] * t.s0[2];
      s1nb[2] += s2b[0] * t.s0[1] - s2b[1] * t.s0[0];
    }
  }
  if (t.alpha[1] != 0.0) quadform_rev<DIM>(G, t.s1n, -Qb / (t.alpha[1] * t.alpha[1]), s1nb);
  normalise_rev<DIM>(t.s1n, t.n1, t.norm1, s1nb, s1b);
  // s1 = acc - ip s0
  double ipb = 0.0;
#pragma unroll
  for (int i = 0; i < DIM; ++i) {
    accb[i] += s1b[i];
    ipb -= s1b[i] * t.s0[i];
    s0b[i] -= t.ip * s1b[i];
  }
  // ip = acc . s0
#pragma unroll
  for (int i = 0; i < DIM; ++i) {
    accb[i] += ipb * t.s0[i];
    s0b[i] += ipb * t.acc[i];
  }
  // acc = dv v
#pragma unroll
  for (int i = 0; i < DIM; ++i)
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      dvb[i][j] += accb[i] * v[j];
      vb[j] += accb[i] * dv[i][j];
    }
  if (t.alpha[0] != 0.0) quadform_rev<DIM>(G, t.s0, -Qb / (t.alpha[0] * t.alpha[0]), s0b);
  // s0 = v/|v|
  normalise_rev<DIM>(t.s0, t.nv, true, s0b, vb);
}

// ---------------------------------------------------------------------------
// X = DUDY^{-1} in closed form (see tau_closed): dense rows p and T (x0, xT), the velocity and
// mass-fraction rows are (e_j - w_j e_p)/rho.
template <int DIM, int NC>
struct Inv {
  double x0[Layout<DIM, NC>::ND], xT[Layout<DIM, NC>::ND], irho;
};

template <int DIM, int NC>
GV_HD void dudy_inverse(const Cf<DIM, NC>& c, double irho, Inv<DIM, NC>& X) {
  using L = Layout<DIM, NC>;
  const double idet = 1.0 / (c.drho_dp * c.de_dT - c.drho_dT * c.de_dp), q = irho * idet;
  double sY = 0.0, sE = -c.E;
#pragma unroll
  for (int j = 0; j < DIM; ++j) sE += c.v[j] * c.v[j];
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) {
    sY += c.drho_dY[i] * c.Y[i];
    sE += c.dE_dY[i] * c.Y[i];
  }
  const double R1 = 1.0 + irho * sY, R2 = irho * sE;
  X.irho = irho;
  X.x0[0] = (R1 * c.de_dT - c.drho_dT * R2) * idet;
  X.xT[0] = (c.drho_dp * R2 - c.de_dp * R1) * idet;
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    X.x0[1 + j] = c.drho_dT * q * c.v[j];
    X.xT[1 + j] = -c.drho_dp * q * c.v[j];
  }
  X.x0[L::iT] = -c.drho_dT * q;
  X.xT[L::iT] = c.drho_dp * q;
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) {
    X.x0[L::iY + i] = (c.drho_dT * c.dE_dY[i] - c.drho_dY[i] * c.de_dT) * q;
    X.xT[L::iY + i] = (c.de_dp * c.drho_dY[i] - c.drho_dp * c.dE_dY[i]) * q;
  }
}

template <int DIM, int NC>
GV_HD void inv_mul(const Cf<DIM, NC>& c, const Inv<DIM, NC>& X, const double* y, double* out) {  // X y
  using L = Layout<DIM, NC>;
  double a = 0.0, b = 0.0;
#pragma unroll
  for (int j = 0; j < L::ND; ++j) {
    a += X.x0[j] * y[j];
    b += X.xT[j] * y[j];
  }
#pragma unroll
  for (int j = 1; j < L::ND; ++j) out[j] = X.irho * (y[j] - c.w[j] * y[0]);
  out[0] = a;
  out[L::iT] = b;
}

template <int DIM, int NC>
GV_HD void inv_tmul(const Cf<DIM, NC>& c, const Inv<DIM, NC>& X, const double* y, double* out) {  // X^T y
  using L = Layout<DIM, NC>;
  double s = 0.0;
#pragma unroll
  for (int j = 0; j < L::ND; ++j) {
    double o = X.x0[j] * y[0] + X.xT[j] * y[L::iT];
    if (j >= 1 && j != L::iT) {
      o += X.irho * y[j];
      s += c.w[j] * y[j];
    }
    out[j] = o;
  }
  out[0] -= X.irho * s;
}

// ---------------------------------------------------------------------------
// The point residual (phi0, phi_d) and its reverse.
template <int DIM, int NEN, int NC>
struct PTape {
  using L = Layout<DIM, NC>;
  static constexpr int ND = L::ND;
  CompK kc[NC];
  Mix<NC> m;
  MixP<NC> mP;
  Cf<DIM, NC> c;
  double vP[DIM], TP, EP;
  double U[ND], UP[ND], S[ND];
  double dd[ND], Res[ND];
  // tau
  bool tau_on, lowm;
  HTape<DIM> ht;
  Inv<DIM, NC> X;
  double vn, h, use, hv, td[ND], tpre00, tpre11, Bm, t00;
  double wv[ND], xy0;          // tau Res; row p of DUDY^{-1} diag(td) Res
  int use_branch;            // 0: dt/2, 1: h/(2(v+c)) + h/(2v)
  int td_branch[ND];         // 0: use, 1: the capped term
  // dc
  bool dc_on;
  double dU[DIM][ND], grho[DIM], gn, Jv[DIM], sJ, hdc, AdI[ND], Z[ND], Zn, Un, use1, nu0, nu;
  double sg[NEN];
};

template <int DIM, int NEN, int NC>
GV_HD void point_forward(const Ctx<DIM, NC>& x, const PGeo<DIM, NEN>& q, const double* Iq,
                         const double (&dI)[DIM][Layout<DIM, NC>::ND], const double* Pq,
                         PTape<DIM, NEN, NC>& t, double* phi0, double (&phi)[DIM][Layout<DIM, NC>::ND]) {
  using L = Layout<DIM, NC>;
  constexpr int ND = L::ND;
  const double dt = x.dt;
  // primitive state at I and at P (fluid_2d.hpp:112-121)
  double p = Iq[0], T = Iq[L::iT], v[DIM], Y[NC], YP[NC];
  double sY = 0.0, sYP = 0.0;
#pragma unroll
  for (int k = 0; k < DIM; ++k) { v[k] = Iq[1 + k]; t.vP[k] = Pq[1 + k]; }
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) {
    Y[i] = Iq[L::iY + i]; sY += Y[i];
    YP[i] = Pq[L::iY + i]; sYP += YP[i];
  }
  Y[NC - 1] = 1.0 - sY;
  YP[NC - 1] = 1.0 - sYP;
  t.TP = Pq[L::iT];
#pragma unroll
  for (int i = 0; i < NC; ++i) comp_const(x.ch[i], t.kc[i]);
  mixp_forward<NC>(x.ch, t.kc, Pq[0], t.TP, YP, t.mP);
  mix_forward<NC>(x.ch, t.kc, p, T, Y, t.m);
  coef_forward<DIM, NC>(t.m, x.ch, p, v, T, t.c);
  const Cf<DIM, NC>& c = t.c;
  // U, U_P, S and the mass term (fluid_2d.hpp:372-385, 597-599)
  t.EP = t.mP.cv * t.TP + 0.5 * dot<DIM>(t.vP, t.vP);
#pragma unroll
  for (int j = 0; j < ND; ++j) {
    t.U[j] = t.m.rho * c.w[j];
    double wP = (j == 0) ? 1.0 : (j < L::iT ? t.vP[j - 1] : (j == L::iT ? t.EP : YP[j - L::iY]));
    t.UP[j] = t.mP.rho * wP;
    t.S[j] = 0.0;
  }
  double gv = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    t.S[1 + d] = t.m.rho * x.gravity[d];
    gv += x.gravity[d] * v[d];
  }
  t.S[L::iT] = t.m.rho * gv;
  // least-squares residual Res = DUDY (I - P)/dt + sum_d A_d dI_d - S  (fluid_2d.hpp:282)
#pragma unroll
  for (int j = 0; j < ND; ++j) t.dd[j] = (Iq[j] - Pq[j]) * x.inv_dt;
  Dy<DIM, NC>(c, t.dd, t.Res);
#pragma unroll
  for (int d = 0; d < DIM; ++d) Dy<DIM, NC>(c, dI[d], t.dU[d]);
  double div = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) div += dI[d][1 + d];
  // sum_d A_d dI_d, A_d = v_d DUDY + u' e_vd^T + (e_vd + v_d e_E) e_p^T
#pragma unroll
  for (int j = 0; j < ND; ++j) {
    double a = (t.U[j] + (j == L::iT ? p : 0.0)) * div;
#pragma unroll
    for (int d = 0; d < DIM; ++d) a += v[d] * t.dU[d][j];
    t.AdI[j] = a;
  }
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    t.AdI[1 + d] += dI[d][0];
    t.AdI[L::iT] += v[d] * dI[d][0];
  }
#pragma unroll
  for (int j = 0; j < ND; ++j) t.Res[j] += t.AdI[j] - t.S[j];
  // tau (fluid_2d.hpp:877-960), 2019 or none
#pragma unroll
  for (int r = 0; r < ND; ++r) t.wv[r] = 0.0;
  t.vn = sqrt(hdot<DIM>(v, v));
  t.tau_on = t.vn >= kEps && x.tau == GALES_TAU_NON_DIAG_COMP_2019;
  t.lowm = false;
  if (t.tau_on) {
    double dv[DIM][DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
      for (int d = 0; d < DIM; ++d) dv[a][d] = dI[d][1 + a];
    t.h = compute_h_fwd<DIM>(q.G, v, dv, t.ht);
    const double cs = t.m.c, h = t.h, vn = t.vn;
    t.hv = (0.5 * h) * (2.0 * vn + cs) / (vn * (vn + cs));   // h/(2(|v| + c)) + h/(2|v|)
    t.use_branch = (x.steady || t.hv <= dt * 0.5) ? 1 : 0;
    t.use = t.use_branch ? t.hv : dt * 0.5;
    const double use = t.use, rho = t.m.rho;
    const double hh = h * h * (1.0 / 12.0);
    double cap[ND];
    cap[0] = use;
    const double capv = hh * rho / t.m.mu;
#pragma unroll
    for (int d = 0; d < DIM; ++d) cap[1 + d] = capv;
    cap[L::iT] = hh * rho * t.m.cv / t.m.kappa;
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) cap[L::iY + i] = hh / x.ch[i].D;
    t.td_branch[0] = 0;
    t.td[0] = use;
#pragma unroll
    for (int j = 1; j < ND; ++j) {
      t.td_branch[j] = cap[j] < use ? 1 : 0;
      t.td[j] = t.td_branch[j] ? cap[j] : use;
    }
    dudy_inverse<DIM, NC>(c, t.m.irho, t.X);
    double y[ND];
#pragma unroll
    for (int j = 0; j < ND; ++j) y[j] = t.td[j] * t.Res[j];
    inv_mul<DIM, NC>(c, t.X, y, t.wv);
    t.xy0 = t.wv[0];
    if (vn < 0.1 * cs) {
      // row p: tau00 = 1/(1/a + 1/B), zero elsewhere
      t.lowm = true;
      t.tpre00 = t.X.x0[0] * t.td[0];
      t.tpre11 = t.m.irho * t.td[1];
      t.Bm = rho * t.tpre11 * q.trG;
      t.t00 = t.tpre00 * t.Bm / (t.tpre00 + t.Bm);
      t.wv[0] = t.t00 * t.Res[0];
    }
  }
  // dc viscosity (fluid_2d.hpp:1027-1065)
  t.nu = 0.0;
  t.dc_on = false;
  if (x.dc_2006) {
    double s = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) { t.grho[d] = t.dU[d][0]; s += t.grho[d] * t.grho[d]; }
    t.gn = sqrt(s);
    if (!(t.gn < kEps)) {
      const double ign = 1.0 / t.gn;
#pragma unroll
      for (int d = 0; d < DIM; ++d) t.Jv[d] = t.grho[d] * ign;
      double hs = 0.0;
#pragma unroll
      for (int i = 0; i < NEN; ++i) {
        double tt = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) tt += t.Jv[d] * q.ds[d][i];
        t.sg[i] = tt >= 0.0 ? 1.0 : -1.0;
        hs += fabs(tt);
      }
      t.sJ = hs;
      if (hs > kEps) {
        t.dc_on = true;
        t.hdc = 1.0 / hs;
        double Zn = 0.0, Un = 0.0;
#pragma unroll
        for (int j = 0; j < ND; ++j) {
          t.Z[j] = x.u_ref_inv[j] * (t.AdI[j] - t.S[j]);
          const double u = x.u_ref_inv[j] * t.U[j];
          Zn += t.Z[j] * t.Z[j];
          Un += u * u;
        }
        t.Zn = sqrt(Zn);
        t.Un = sqrt(Un);
        const double a = x.dc_sharp, hd = t.hdc;
        double use1 = 0.0;
        if (a != 2.0)
#pragma unroll
          for (int d = 0; d < DIM; ++d)
#pragma unroll
            for (int j = 0; j < ND; ++j) {
              const double u = x.u_ref_inv[j] * t.dU[d][j];
              use1 += u * u;
            }
        t.use1 = use1;
        double nu = 0.0;
        if (a == 1.0) nu = t.Zn * hd * (1.0 / sqrt(use1));
        else if (a == 2.0) nu = t.Zn * hd * hd / t.Un;
        else if (a == 1.5) nu = t.Zn * hd * ((1.0 / sqrt(use1)) + hd / t.Un) / 2.0;
        t.nu0 = nu;
        t.nu = x.dc_scale * nu;
      }
    }
  }
  // phi0 = rv - S0 tau Res,  phi_d = F_dif,d - F_adv,d + nu dU_d + A_d tau Res
  const double* wv = t.wv;
  double Dw[ND];
  Dy<DIM, NC>(c, wv, Dw);
#pragma unroll
  for (int j = 0; j < ND; ++j) phi0[j] = (t.U[j] - t.UP[j]) * x.inv_dt - t.S[j];
  {
    double s0w = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) s0w += x.gravity[d] * wv[1 + d];
    phi0[L::iT] -= t.m.rho * s0w;
  }
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    // viscous stress row d
    double tsd[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) tsd[j] = c.mu * (dI[d][1 + j] + dI[j][1 + d]) + (j == d ? c.lam * div : 0.0);
    double fd[ND];
    fd[0] = 0.0;
#pragma unroll
    for (int j = 0; j < DIM; ++j) fd[1 + j] = tsd[j];
    double en = c.kappa * dI[d][L::iT];
#pragma unroll
    for (int j = 0; j < DIM; ++j) en += v[j] * tsd[j];
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) {
      en += c.rhoDH[i] * dI[d][L::iY + i];
      fd[L::iY + i] = c.rhoD[i] * dI[d][L::iY + i];
    }
    fd[L::iT] = en;
    // A_d tau Res - F_adv,d = v_d (DUDY tau Res) + u' (wv_vd - v_d) + (wv_p - p) e_vd + v_d wv_p e_E
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      const double up = t.U[j] + (j == L::iT ? p : 0.0);
      phi[d][j] = fd[j] + t.nu * t.dU[d][j] + v[d] * Dw[j] + up * (wv[1 + d] - v[d]);
    }
    phi[d][1 + d] += wv[0] - p;
    phi[d][L::iT] += v[d] * wv[0];
  }
}

// Reverse of point_forward.  Outputs are accumulated (+=).
template <int DIM, int NEN, int NC>
GV_HD void point_reverse(const Ctx<DIM, NC>& x, const PGeo<DIM, NEN>& q, const double* Iq,
                         const double (&dI)[DIM][Layout<DIM, NC>::ND], const double* Pq,
                         const PTape<DIM, NEN, NC>& t, const double* phi0b,
                         const double (&phib)[DIM][Layout<DIM, NC>::ND], double* Ib,
                         double (&dIb)[DIM][Layout<DIM, NC>::ND], double* th, double* urib = nullptr) {
  using L = Layout<DIM, NC>;
  constexpr int ND = L::ND;
  const Cf<DIM, NC>& c = t.c;
  const double dt = x.dt, rho = t.m.rho;
  CfBar<DIM, NC> b;
  cfbar_zero<DIM, NC>(b);
  double Ub[ND], Sb[ND], Resb[ND], wvb[ND], nub = 0.0;
#pragma unroll
  for (int j = 0; j < ND; ++j) { Ub[j] = 0.0; Sb[j] = 0.0; Resb[j] = 0.0; wvb[j] = 0.0; }
  double dUb[DIM][ND];
#pragma unroll
  for (int d = 0; d < DIM; ++d)
#pragma unroll
    for (int j = 0; j < ND; ++j) dUb[d][j] = 0.0;
  const double* wv = t.wv;
  double Dw[ND];
  Dy<DIM, NC>(c, wv, Dw);
  // ---- phi_d
  double div = 0.0;
#pragma unroll
  for (int k = 0; k < DIM; ++k) div += dI[k][1 + k];
  double divb = 0.0, xs[ND], wu[ND];
#pragma unroll
  for (int j = 0; j < ND; ++j) xs[j] = wu[j] = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const double* pb = phib[d];
    // A_d wv - F_adv,d = v_d DUDY wv + u' (wv_vd - v_d) + (wv_p - p) e_vd + v_d wv_p e_E
    const double vd = c.v[d], tt = wv[1 + d] - vd;
    const double pw = xw_of<DIM, NC>(c, pb), pu = rho * pw + c.p * pb[L::iT];
    double pDw = 0.0, du = 0.0;
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      pDw += pb[j] * Dw[j];
      xs[j] += vd * pb[j];
      wu[j] += tt * pb[j];
      du += pb[j] * t.dU[d][j];
      dUb[d][j] = t.nu * pb[j];
    }
    nub += du;
    wvb[1 + d] += pu;
    wvb[0] += pb[1 + d] + vd * pb[L::iT];
    b.v[d] += pDw + pb[L::iT] * wv[0] - pu;
    b.rho += tt * pw;
    b.p += tt * pb[L::iT] - pb[1 + d];
    // F_dif,d: momentum rows tau_dj, energy row v.tau_d + kappa dT + sum rhoDH dY, species rhoD dY
    double tsd[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) tsd[j] = c.mu * (dI[d][1 + j] + dI[j][1 + d]) + (j == d ? c.lam * div : 0.0);
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const double Phi = pb[1 + j] + pb[L::iT] * c.v[j];
      b.v[j] += pb[L::iT] * tsd[j];
      // tsd_j = mu (dI[d][1+j] + dI[j][1+d]) + [j==d] lam div
      b.mu += Phi * (dI[d][1 + j] + dI[j][1 + d]);
      dIb[d][1 + j] += Phi * c.mu;
      dIb[j][1 + d] += Phi * c.mu;
      if (j == d) {
        b.lam += Phi * div;
        divb += Phi * c.lam;
      }
    }
    b.kappa += pb[L::iT] * dI[d][L::iT];
    dIb[d][L::iT] += pb[L::iT] * c.kappa;
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) {
      b.rhoDH[i] += pb[L::iT] * dI[d][L::iY + i];
      b.rhoD[i] += pb[L::iY + i] * dI[d][L::iY + i];
      dIb[d][L::iY + i] += pb[L::iT] * c.rhoDH[i] + pb[L::iY + i] * c.rhoD[i];
    }
  }
#pragma unroll
  for (int k = 0; k < DIM; ++k) dIb[k][1 + k] += divb;
  {
    double at[ND];
    DTx<DIM, NC>(c, xs, at);
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      wvb[j] += at[j];
      if (j > 0) b.w[j] += rho * wu[j];
    }
    xDy_rev<DIM, NC>(c, xs, wv, 1.0, b);
  }
  // ---- phi0 = (U - U_P)/dt - S - S0 wv
  double UPb[ND];
#pragma unroll
  for (int j = 0; j < ND; ++j) {
    Ub[j] += phi0b[j] * x.inv_dt;
    UPb[j] = -phi0b[j] * x.inv_dt;
    Sb[j] -= phi0b[j];
  }
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    b.rho -= phi0b[L::iT] * x.gravity[d] * wv[1 + d];
    wvb[1 + d] -= phi0b[L::iT] * rho * x.gravity[d];
  }
  // ---- dc viscosity: nu = dc_scale nu0(Zn, Un, hdc, use1)
  double AdIb[ND];
#pragma unroll
  for (int j = 0; j < ND; ++j) AdIb[j] = 0.0;
  if (t.dc_on && nub != 0.0) {
    const double a = x.dc_sharp, hd = t.hdc;
    const double nu0b = nub * x.dc_scale;
    double Znb = 0.0, Unb = 0.0, hdb = 0.0, use1b = 0.0;
    if (a == 1.0) {
      const double is = 1.0 / sqrt(t.use1);
      Znb = nu0b * hd * is;
      hdb = nu0b * t.Zn * is;
      use1b = nu0b * t.Zn * hd * (-0.5 * is / t.use1);
    } else if (a == 2.0) {
      Znb = nu0b * hd * hd / t.Un;
      hdb = nu0b * 2.0 * t.Zn * hd / t.Un;
      Unb = -nu0b * t.Zn * hd * hd / (t.Un * t.Un);
    } else if (a == 1.5) {
      const double is = 1.0 / sqrt(t.use1);
      const double inner = is + hd / t.Un;
      Znb = nu0b * hd * inner / 2.0;
      hdb = nu0b * t.Zn * (inner + hd / t.Un) / 2.0;
      Unb = -nu0b * t.Zn * hd * hd / (2.0 * t.Un * t.Un);
      use1b = nu0b * t.Zn * hd / 2.0 * (-0.5 * is / t.use1);
    }
    // Zn = |Z|, Z = u_ref_inv (AdI - S)
    if (t.Zn > 0.0) {
      const double zf = Znb / t.Zn;
#pragma unroll
      for (int j = 0; j < ND; ++j) {
        const double zj = zf * t.Z[j], g = zj * x.u_ref_inv[j];
        AdIb[j] += g;
        Sb[j] -= g;
        if (urib) urib[j] += zj * (t.AdI[j] - t.S[j]);
      }
    }
    // Un = |u_ref_inv U|
    if (t.Un > 0.0) {
      const double uf = Unb / t.Un;
#pragma unroll
      for (int j = 0; j < ND; ++j) {
        const double uj = uf * x.u_ref_inv[j] * t.U[j];
        Ub[j] += uj * x.u_ref_inv[j];
        if (urib) urib[j] += uj * t.U[j];
      }
    }
    // use1 = sum_d |u_ref_inv dU_d|^2
    if (use1b != 0.0)
#pragma unroll
    for (int d = 0; d < DIM; ++d)
#pragma unroll
      for (int j = 0; j < ND; ++j) {
        dUb[d][j] += use1b * 2.0 * x.u_ref_inv[j] * x.u_ref_inv[j] * t.dU[d][j];
        if (urib) urib[j] += use1b * 2.0 * x.u_ref_inv[j] * t.dU[d][j] * t.dU[d][j];
      }
    // hdc = 1/sJ, sJ = sum_i |J . dN_i|, J = grho/|grho|, grho_d = dU_d[0]
    const double sJb = -hdb / (t.sJ * t.sJ);
    double Jb[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      double sum = 0.0;
#pragma unroll
      for (int i = 0; i < NEN; ++i) sum += t.sg[i] * q.ds[d][i];
      Jb[d] = sJb * sum;
    }
    const double pr = dot<DIM>(Jb, t.Jv), ign = 1.0 / t.gn;
#pragma unroll
    for (int d = 0; d < DIM; ++d) dUb[d][0] += (Jb[d] - pr * t.Jv[d]) * ign;
  }
  // ---- tau: the loss term wv . wvb with wv = tau Res, tau = DUDY^{-1} diag(td) but for row p
  // at low Mach numbers
  double vb_h[DIM], dvb[DIM][DIM];
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    vb_h[a] = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) dvb[a][d] = 0.0;
  }
  double cvb_tau = 0.0, csb_tau = 0.0;
  if (t.tau_on) {
    // With X = DUDY^{-1}, y = diag(td) Res and pX = X^T wvb, the loss pX . (DUDY dX y) has the
    // cotangents diag(td) pX of Res, diag(Res) pX of td and -pX (X y)^T of DUDY
    double wl[ND], pX[ND], tdb[ND], qX[ND];
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      wl[j] = (j == 0 && t.lowm) ? 0.0 : wvb[j];
      qX[j] = j == 0 ? t.xy0 : wv[j];
    }
    inv_tmul<DIM, NC>(c, t.X, wl, pX);
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      tdb[j] = t.Res[j] * pX[j];
      Resb[j] += t.td[j] * pX[j];
    }
    xDy_rev<DIM, NC>(c, pX, qX, -1.0, b);
    if (t.lowm) {
      // tau00 = 1/(1/a + 1/B), a = X00 td_0, B = rho (td_1/rho) trG
      Resb[0] += t.t00 * wvb[0];
      const double tb = wvb[0] * t.Res[0], fa = t.t00 / t.tpre00, fB = t.t00 / t.Bm;
      const double ab = tb * fa * fa, Bb = tb * fB * fB;
      tdb[0] += ab * t.X.x0[0];
      tdb[1] += Bb * q.trG;
      const double al = ab * t.td[0];
      double px[ND], qx[ND];
#pragma unroll
      for (int j = 0; j < ND; ++j) {
        px[j] = al * t.X.x0[j];
        qx[j] = j == 0 ? t.X.x0[0] : (j == L::iT ? t.X.xT[0] : -c.w[j] * t.m.irho);
      }
      xDy_rev<DIM, NC>(c, px, qx, -1.0, b);
    }
    // td_0 = use, td_j = min(use, cap_j)
    const double h = t.h, vn = t.vn, cs = t.m.c;
    double useb = tdb[0], hb = 0.0, hs = 0.0, gv_ = 0.0, gT = 0.0;
#pragma unroll
    for (int j = 1; j < ND; ++j) {
      if (!t.td_branch[j]) {
        useb += tdb[j];
        continue;
      }
      // td_j is its cap: h^2 rho/(12 mu), h^2 rho cv/(12 kappa), h^2/(12 D)
      const double g = tdb[j] * t.td[j];
      hs += g;
      if (j < L::iT) {
        gv_ += g;
      } else if (j == L::iT) {
        gT += g;
      }
    }
    if (hs != 0.0) hb += 2.0 * hs / h;
    if (gv_ != 0.0) b.mu -= gv_ / t.m.mu;
    if (gT != 0.0) {
      cvb_tau += gT / t.m.cv;
      b.kappa -= gT / t.m.kappa;
    }
    b.rho += (gv_ + gT) * t.m.irho;
    double vnb = 0.0;
    if (t.use_branch) {
      // use = h/(2(vn + c)) + h/(2 vn)
      const double i1 = 0.5 / (vn + cs), i2 = 0.5 / vn;
      hb += useb * (i1 + i2);
      csb_tau -= useb * h * 2.0 * i1 * i1;
      vnb -= useb * h * 2.0 * (i1 * i1 + i2 * i2);
    }
    double dv[DIM][DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
      for (int d = 0; d < DIM; ++d) dv[a][d] = dI[d][1 + a];
    compute_h_rev<DIM>(q.G, c.v, dv, t.ht, hb, vb_h, dvb);
    vnb /= vn;
#pragma unroll
    for (int k = 0; k < DIM; ++k) vb_h[k] += vnb * c.v[k];
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
      for (int d = 0; d < DIM; ++d) dIb[d][1 + a] += dvb[a][d];
  }
  // ---- Res = DUDY dd + AdI - S
#pragma unroll
  for (int j = 0; j < ND; ++j) {
    AdIb[j] += Resb[j];
    Sb[j] -= Resb[j];
  }
  xDy_rev<DIM, NC>(c, Resb, t.dd, 1.0, b);
  {
    double ddb[ND];
    DTx<DIM, NC>(c, Resb, ddb);
#pragma unroll
    for (int j = 0; j < ND; ++j) Ib[j] += ddb[j] * x.inv_dt;
  }
  // sum_d A_d dI_d and dU_d = DUDY dI_d: the cotangent of DUDY dI_d is dUb_d + v_d AdIb
  const double aw = xw_of<DIM, NC>(c, AdIb), au = rho * aw + c.p * AdIb[L::iT];
  b.rho += div * aw;
  b.p += div * AdIb[L::iT];
#pragma unroll
  for (int j = 1; j < ND; ++j) b.w[j] += div * rho * AdIb[j];
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    double xd[ND], at[ND], s = AdIb[L::iT] * dI[d][0];
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      xd[j] = dUb[d][j] + c.v[d] * AdIb[j];
      s += AdIb[j] * t.dU[d][j];
    }
    b.v[d] += s;
    xDy_rev<DIM, NC>(c, xd, dI[d], 1.0, b);
    DTx<DIM, NC>(c, xd, at);
#pragma unroll
    for (int j = 0; j < ND; ++j) dIb[d][j] += at[j];
    dIb[d][1 + d] += au;
    dIb[d][0] += AdIb[1 + d] + c.v[d] * AdIb[L::iT];
  }
  // S = (0, rho g, rho g.v, 0)
  {
    double gv = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      gv += x.gravity[d] * c.v[d];
      b.rho += Sb[1 + d] * x.gravity[d];
      b.v[d] += Sb[L::iT] * rho * x.gravity[d];
    }
    b.rho += Sb[L::iT] * gv;
  }
  // U = rho w
#pragma unroll
  for (int j = 0; j < ND; ++j) {
    b.rho += Ub[j] * c.w[j];
    b.w[j] += Ub[j] * rho;
  }
  cfbar_fold<DIM, NC>(b);
  // ---- coefficients -> mixture -> state and parameters
  MixBar o;
  double irb[NC], cvcb[NC], pb = 0.0, Tb = 0.0, vb[DIM], Yb[NC];
#pragma unroll
  for (int k = 0; k < DIM; ++k) vb[k] = vb_h[k];
#pragma unroll
  for (int i = 0; i < NC; ++i) Yb[i] = 0.0;
  coef_reverse<DIM, NC>(t.m, x.ch, c, b, o, irb, cvcb, pb, vb, Tb, Yb);
  o.cv += cvb_tau;
  o.c += csb_tau;
  mix_reverse<NC>(x.ch, t.kc, c.T, t.m, o, irb, cvcb, pb, Tb, Yb, th);
  // U_P = rho_P (1, v_P, E_P, Y_P): parameters only
  {
    double rPb = 0.0;
#pragma unroll
    for (int j = 0; j < ND; ++j)
      rPb += UPb[j] * (j == 0 ? 1.0 : (j < L::iT ? t.vP[j - 1] : (j == L::iT ? t.EP : t.mP.Y[j - L::iY])));
    mixp_reverse<NC>(x.ch, t.kc, t.TP, t.mP, rPb, UPb[L::iT] * t.mP.rho * t.TP, th);
  }
  // state cotangents: p, v, T, Y_i (Y_nc = 1 - sum Y_i)
  Ib[0] += pb;
#pragma unroll
  for (int k = 0; k < DIM; ++k) Ib[1 + k] += vb[k];
  Ib[L::iT] += Tb;
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) Ib[L::iY + i] += Yb[i] - Yb[NC - 1];
}

// ---------------------------------------------------------------------------
// Boundary point (execute_b, fluid_2d.hpp:341-349, 610-817): rb = sum_k (F_adv,k -
// F_dif,k) JNxW_k with the side's Neumann and mass-flux overrides, and its reverse.
template <int DIM, int NC>
struct BTape {
  using L = Layout<DIM, NC>;
  CompK kc[NC];
  Mix<NC> m;
  Cf<DIM, NC> c;
  double ts[DIM][DIM], qf[DIM], Jf[DIM][L::NYA], div;
  bool tsf[DIM][DIM], qff[DIM], Jff[DIM][L::NYA];   // entry set by an override
};

template <int DIM, int NC>
GV_HD void bpoint_forward(const Ctx<DIM, NC>& x, const gales_side_bc& bc, const double* Iq,
                          const double (&dI)[DIM][Layout<DIM, NC>::ND], const double* JN, BTape<DIM, NC>& t,
                          double* rb) {
  using L = Layout<DIM, NC>;
  constexpr int ND = L::ND;
  double p = Iq[0], T = Iq[L::iT], v[DIM], Y[NC], sY = 0.0;
#pragma unroll
  for (int k = 0; k < DIM; ++k) v[k] = Iq[1 + k];
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) { Y[i] = Iq[L::iY + i]; sY += Y[i]; }
  Y[NC - 1] = 1.0 - sY;
#pragma unroll
  for (int i = 0; i < NC; ++i) comp_const(x.ch[i], t.kc[i]);
  mix_forward<NC>(x.ch, t.kc, p, T, Y, t.m);
  coef_forward<DIM, NC>(t.m, x.ch, p, v, T, t.c);
  const Cf<DIM, NC>& c = t.c;
  const double rho = t.m.rho;
  double div = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) div += dI[d][1 + d];
  t.div = div;
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int b = 0; b < DIM; ++b) {
      const int lo = a < b ? a : b, hi = a < b ? b : a;
      t.tsf[a][b] = (bc.tau_mask >> (lo * 3 + hi)) & 1u;
      if (t.tsf[a][b]) t.ts[a][b] = bc.tau[lo * 3 + hi];
      else if (a == b) t.ts[a][b] = c.lam * div + 2.0 * c.mu * dI[a][1 + a];
      else t.ts[a][b] = c.mu * (dI[hi][1 + lo] + dI[lo][1 + hi]);
    }
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    t.qff[d] = (bc.q_mask >> d) & 1u;
    t.qf[d] = t.qff[d] ? bc.q[d] : -c.kappa * dI[d][L::iT];
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) {
      t.Jff[d][i] = (bc.J_mask >> (d * 8 + i)) & 1u;
      t.Jf[d][i] = t.Jff[d][i] ? bc.J[d][i] : rho * x.ch[i].D * dI[d][L::iY + i];
    }
  }
#pragma unroll
  for (int j = 0; j < ND; ++j) rb[j] = 0.0;
#pragma unroll
  for (int k = 0; k < DIM; ++k) {
    double fa[ND], fd[ND];
    if ((bc.mass_flux_mask >> k) & 1u) {
      const double mf = bc.mass_flux[k];
      fa[0] = mf;
#pragma unroll
      for (int j = 0; j < DIM; ++j) fa[1 + j] = mf * v[j] + (j == k ? p : 0.0);
      fa[L::iT] = mf * c.E + p * v[k];
#pragma unroll
      for (int i = 0; i < NC - 1; ++i) fa[L::iY + i] = mf * Y[i];
    } else {
      fa[0] = rho * v[k];
#pragma unroll
      for (int j = 0; j < DIM; ++j) fa[1 + j] = rho * v[k] * v[j] + (j == k ? p : 0.0);
      fa[L::iT] = v[k] * (rho * c.E + p);
#pragma unroll
      for (int i = 0; i < NC - 1; ++i) fa[L::iY + i] = rho * v[k] * Y[i];
    }
    fd[0] = 0.0;
    double en = -t.qf[k];
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      fd[1 + j] = t.ts[k][j];
      en += t.ts[k][j] * v[j];
    }
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) {
      en -= c.H[i] * t.Jf[k][i];
      fd[L::iY + i] = t.Jf[k][i];
    }
    fd[L::iT] = en;
#pragma unroll
    for (int j = 0; j < ND; ++j) rb[j] += (fa[j] - fd[j]) * JN[k];
  }
}

template <int DIM, int NC>
GV_HD void bpoint_reverse(const Ctx<DIM, NC>& x, const gales_side_bc& bc, const double* Iq,
                          const double (&dI)[DIM][Layout<DIM, NC>::ND], const double* JN, const BTape<DIM, NC>& t,
                          const double* rbb, double* Ib, double (&dIb)[DIM][Layout<DIM, NC>::ND], double* th) {
  using L = Layout<DIM, NC>;
  constexpr int ND = L::ND;
  const Cf<DIM, NC>& c = t.c;
  const double rho = t.m.rho;
  CfBar<DIM, NC> b;
  cfbar_zero<DIM, NC>(b);
  double tsb[DIM][DIM], Hb[L::NYA];
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int e = 0; e < DIM; ++e) tsb[a][e] = 0.0;
#pragma unroll
  for (int i = 0; i < L::NYA; ++i) Hb[i] = 0.0;
#pragma unroll
  for (int k = 0; k < DIM; ++k) {
    double fab[ND], fdb[ND];
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      fab[j] = rbb[j] * JN[k];
      fdb[j] = -rbb[j] * JN[k];
    }
    const double vk = c.v[k];
    if ((bc.mass_flux_mask >> k) & 1u) {
      const double mf = bc.mass_flux[k];
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        b.v[j] += fab[1 + j] * mf;
        if (j == k) b.p += fab[1 + j];
      }
      b.E += fab[L::iT] * mf;
      b.p += fab[L::iT] * vk;
      b.v[k] += fab[L::iT] * c.p;
#pragma unroll
      for (int i = 0; i < NC - 1; ++i) b.Y[i] += fab[L::iY + i] * mf;
    } else {
      b.rho += fab[0] * vk;
      b.v[k] += fab[0] * rho;
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        b.rho += fab[1 + j] * vk * c.v[j];
        b.v[k] += fab[1 + j] * rho * c.v[j];
        b.v[j] += fab[1 + j] * rho * vk;
        if (j == k) b.p += fab[1 + j];
      }
      b.v[k] += fab[L::iT] * (rho * c.E + c.p);
      b.rho += fab[L::iT] * vk * c.E;
      b.E += fab[L::iT] * vk * rho;
      b.p += fab[L::iT] * vk;
#pragma unroll
      for (int i = 0; i < NC - 1; ++i) {
        b.rho += fab[L::iY + i] * vk * c.Y[i];
        b.v[k] += fab[L::iY + i] * rho * c.Y[i];
        b.Y[i] += fab[L::iY + i] * rho * vk;
      }
    }
    // fd: (0, ts[k][:], ts[k].v - qf_k - sum_i H_i Jf_ki, Jf_k:)
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      tsb[k][j] += fdb[1 + j] + fdb[L::iT] * c.v[j];
      b.v[j] += fdb[L::iT] * t.ts[k][j];
    }
    const double qfb = -fdb[L::iT];
    if (!t.qff[k]) {
      b.kappa -= qfb * dI[k][L::iT];
      dIb[k][L::iT] -= qfb * c.kappa;
    }
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) {
      Hb[i] -= fdb[L::iT] * t.Jf[k][i];
      const double Jb = -fdb[L::iT] * c.H[i] + fdb[L::iY + i];
      if (!t.Jff[k][i]) {
        b.rho += Jb * x.ch[i].D * dI[k][L::iY + i];
        dIb[k][L::iY + i] += Jb * rho * x.ch[i].D;
      }
    }
  }
  // stresses (symmetric overrides are constants)
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int e = 0; e < DIM; ++e) {
      if (t.tsf[a][e]) continue;
      const double g = tsb[a][e];
      if (a == e) {
        b.lam += g * t.div;
#pragma unroll
        for (int d = 0; d < DIM; ++d) dIb[d][1 + d] += g * c.lam;
        b.mu += g * 2.0 * dI[a][1 + a];
        dIb[a][1 + a] += g * 2.0 * c.mu;
      } else {
        const int lo = a < e ? a : e, hi = a < e ? e : a;
        b.mu += g * (dI[hi][1 + lo] + dI[lo][1 + hi]);
        dIb[hi][1 + lo] += g * c.mu;
        dIb[lo][1 + hi] += g * c.mu;
      }
    }
  cfbar_fold<DIM, NC>(b);
  MixBar o;
  double irb[NC], cvcb[NC], pb = 0.0, Tb = 0.0, vb[DIM], Yb[NC];
#pragma unroll
  for (int k = 0; k < DIM; ++k) vb[k] = 0.0;
#pragma unroll
  for (int i = 0; i < NC; ++i) Yb[i] = 0.0;
  coef_reverse<DIM, NC>(t.m, x.ch, c, b, o, irb, cvcb, pb, vb, Tb, Yb);
  // H_i = cv_i T + p/rho_i
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) {
    cvcb[i] += Hb[i] * c.T;
    Tb += Hb[i] * t.m.cvc[i];
    pb += Hb[i] * t.m.ir[i];
    irb[i] += Hb[i] * c.p;
  }
  mix_reverse<NC>(x.ch, t.kc, c.T, t.m, o, irb, cvcb, pb, Tb, Yb, th);
  Ib[0] += pb;
#pragma unroll
  for (int k = 0; k < DIM; ++k) Ib[1 + k] += vb[k];
  Ib[L::iT] += Tb;
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) Ib[L::iY + i] += Yb[i] - Yb[NC - 1];
}

#undef GV_HD

}  // namespace vjp
}  // namespace gales
