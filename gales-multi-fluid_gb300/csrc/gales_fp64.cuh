// FP64 form of the interior pass.
//
// On this GPU an FP64 instruction of a warp holds the SM's FP64 pipe for 16 cycles (2 lanes
// per clock), so everything here is arranged for few FP64 operations; loads, integer work and
// DRAM traffic are nearly free beside them.  Two kernels per chunk of elements:
//   point64_kernel  - one thread per (element, quadrature point): interpolation, mixture,
//                     tau and dc viscosity (as the mixed form's point stage, without its
//                     rounding to binary32), the whole residual of the point and the vectors
//                     from which the element block is built.
//   rows64_kernel   - simplices: one thread per (element, dof row r), see below.
//   tensor64_kernel - quadrilaterals and hexahedra, see below.
//   residual64_kernel - the rhs alone.
//   dirichlet64_kernel - the diagonal of blocked rows, which needs the block's whole trace.
//
// Structure (fluid_2d.hpp:407-575).  With w = (1, v, E, Y), r0 the first row of DUDY, mE the
// energy row of M (M = 0 but for the velocity and mass-fraction diagonal and mE),
//   DUDY = w r0^T + rho M,  A_k = v_k DUDY + u' e_vk^T + (e_vk + v_k e_E) e_p^T,
//   u' = rho w + p e_E,     S0 = e_E (rho g)^T on the velocity columns,
// and every tau variant has dense rows p and E only: tau[v_d] = a_d e_p + m_d e_vd,
// tau[Y_i] = b_i e_p + n_i e_Yi.  So with z = r0^T tau, y = mE^T tau, f_d = a_d + m_d v_d,
// h_i = b_i + n_i Y_i, and for a test function with gradient g_b (s_b = g_b.v, e_b = g_b.f)
//   (FPT_b DUDY)[r] = s_b ((w_r z + rho (M tau)[r]) DUDY) + u'_r (e_b r0 + rho (m g_b) on V)
//                     + kappa_br tau0 DUDY - N_b [r = E] rho (e_g r0 + rho (m g) on V),
// where (M tau)[v_j] DUDY = f_j r0 + rho m_j e_vj, (M tau)[Y_i] DUDY = h_i r0 + rho n_i e_Yi
// and kappa_b is g_b on the velocity rows and s_b on E.  zeta = z DUDY, Z = tau0 DUDY and, for
// the energy row, Theta = E zeta + rho y DUDY + Z (and the same for the few entries of FPT_b
// itself that are needed) come from the point stage; a row of FPT_b DUDY is then two or three
// vector multiply-adds for each test function, and its least-squares products with A_a are
// s_a (FPT_b DUDY)[r] plus a velocity and a pressure column.
#pragma once

#include "gales_kernels.cuh"

namespace gales {

// Place of the product of directions k <= l in a record.
__host__ __device__ constexpr int gg_at(int dim, int k, int l) { return k * dim - k * (k - 1) / 2 + (l - k); }

// Words of a point's record and of an element's, in doubles.  Words named J.., r0, DE, zeta,
// Z, Theta and their scalars and entries (ZU .. THE, ZV .. THV) carry the point's weight JxW.  A block holds EB elements, word
// major with the element innermost: word f of point q of element l at [(q RW + f) EB + l], so
// a warp whose lanes are elements reads 256 contiguous bytes a word (quadrilaterals and
// hexahedra, whose matrix stage has a CTA per element, keep a sector of 4 together).
template <int DIM, int NEN, int NC>
struct Rec64 {
  using L = Layout<DIM, NC>;
  static constexpr int ND = L::ND, NQ = NEN, N = NEN * ND;
  static constexpr bool SIMPLEX = NEN == DIM + 1;
  static constexpr int EB = SIMPLEX ? 32 : 4;
  static constexpr int NGG = SIMPLEX ? 0 : DIM * (DIM + 1) / 2;   // products of two directions
  static constexpr int NG = SIMPLEX ? 0 : DIM * DIM;              // the directions themselves
  static constexpr int NR = 1 + NC;    // columns p, T, Y_1.. of r0 and of the energy row of DUDY
  static constexpr int JX = 0, JR = 1, RHO = 2, PR = 3, NU = 4, JMU = 5, JKAP = 6, EG = 7, ZU = 8, T0U = 9, THU = 10;
  static constexpr int ZE = 11, T0E = 12, THE = 13, E = 14;
  static constexpr int V = 15, F = V + DIM, JM = F + DIM, S = JM + DIM, EK = S + DIM;
  static constexpr int ZV = EK + DIM, T0V = ZV + DIM, THV = T0V + DIM;
  static constexpr int Y = THV + DIM, H = Y + L::NYA, JRN = H + L::NYA, JRD = JRN + L::NYA, JRDH = JRD + L::NYA;
  static constexpr int R0 = JRDH + L::NYA, DE = R0 + NR;
  static constexpr int ZETA = DE + NR, ZZ = ZETA + ND, THETA = ZZ + ND;
  static constexpr int GG = THETA + ND, G = GG + NGG;
  static constexpr int RV = G + NG, PHI = RV + ND;
  static constexpr int RW = PHI + DIM * ND;
  // element words: the rows' shares of the trace, then the scatter descriptors as 32-bit
  // integers: node, CSR row length, Dirichlet mask of each node b, then per (b, a) the unit
  // offset u = node_rp(b) nd + slot(b, a) (dof row jb of node b holds node a's columns from
  // nd u + jb rowlen on)
  static constexpr int TR = NQ * RW;
  static constexpr int INTS = TR + ND;
  static constexpr int NI = 3 * NEN + NEN * NEN;
  static constexpr int EW = INTS + (NI + 1) / 2;    // doubles per element
  static constexpr int I_NODE = 0, I_ROWLEN = NEN, I_BLOCKED = 2 * NEN, I_OFF = 3 * NEN;
  static constexpr size_t ELEM_BYTES = (size_t)EW * sizeof(double);
  static __host__ __device__ constexpr int col_r0(int c) {  // index of column c in r0, -1 on velocities
    return c == 0 ? 0 : (c >= L::iT ? c - L::iT + 1 : -1);
  }
};

// The largest |dv[i][j]|, rounded up in its last 32 bits (integer comparisons: free beside FP64).
template <int DIM>
__device__ __forceinline__ double max_entry(const double (&dv)[DIM][DIM]) {
  int m = 0;
#pragma unroll
  for (int i = 0; i < DIM; ++i)
#pragma unroll
    for (int j = 0; j < DIM; ++j) m = max(m, __double2hiint(dv[i][j]) & 0x7fffffff);
  return __hiloint2double(m, -1);
}

// compute_h with fused operations and no divisions but the last, where the direction s1 is
// well conditioned: |s1| > 1e-3 max|dv| |v| keeps its relative error below ~1e-12.  The bound has
// the size of the terms that dv v sums, not of the sum: a shear flow oblique to the axes has
// dv v = 0, and what rounding leaves of it points anywhere.  Elsewhere decided = false and
// the caller takes the reference's operations (compute_h_reference), whose branches hang on
// rounding.  dv carries the reference's roundings; mm = max|dv|^2.
template <int DIM>
__device__ __forceinline__ double compute_h64(const double (&G)[DIM][DIM], const double* v, double vv, double iv,
                                              const double (&dv)[DIM][DIM], double mm, bool& decided) {
  decided = false;
  double s0[DIM], acc[DIM], w1[DIM];
#pragma unroll
  for (int i = 0; i < DIM; ++i) s0[i] = v[i] * iv;
  double ip = 0.0;
#pragma unroll
  for (int i = 0; i < DIM; ++i) {
    double t = dv[i][0] * v[0];
#pragma unroll
    for (int j = 1; j < DIM; ++j) t = fma(dv[i][j], v[j], t);
    acc[i] = t;
    ip = fma(t, s0[i], ip);
  }
  double n1 = 0.0;
#pragma unroll
  for (int i = 0; i < DIM; ++i) {
    w1[i] = fma(-ip, s0[i], acc[i]);
    n1 = fma(w1[i], w1[i], n1);
  }
  constexpr double kMin2 = 1.0e6 * kEps * kEps;  // (1e3 DBL_EPSILON)^2
  if (!(n1 > fmax(1.0e-6 * (vv * mm), kMin2))) return 0.0;
  const double A0 = qform_fma<DIM>(G, s0), A1 = qform_fma<DIM>(G, w1);
  if (A0 == 0.0 || A1 == 0.0) return 0.0;
  // h = 2 sqrt|1/A0 + n1/A1 (+ n2/A2)| = 2 sqrt|num / den|
  double num, den;
  if constexpr (DIM == 3) {
    double w2[3];
    w2[0] = fma(s0[1], w1[2], -s0[2] * w1[1]);
    w2[1] = fma(w1[0], s0[2], -w1[2] * s0[0]);
    w2[2] = fma(s0[0], w1[1], -s0[1] * w1[0]);
    const double n2 = fma(w2[0], w2[0], fma(w2[1], w2[1], w2[2] * w2[2]));
    const double A2 = qform_fma<DIM>(G, w2);
    if (!(n2 > kMin2 * n1) || A2 == 0.0) return 0.0;
    num = fma(A1, A2, A0 * fma(n1, A2, n2 * A1));
    den = A0 * A1 * A2;
  } else {
    num = fma(n1, A0, A1);
    den = A0 * A1;
  }
  decided = true;
  return 2.0 * sqrt(fabs(num / den));
}

// y = DUDY x
template <int DIM, int NC>
__device__ __forceinline__ void dudy_mul(const Coef<DIM, NC>& c, const double* x, double* y) {
  using L = Layout<DIM, NC>;
  double r = fma(c.drho_dp, x[0], c.drho_dT * x[L::iT]), m = fma(c.de_dp, x[0], c.de_dT * x[L::iT]);
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) {
    r = fma(c.drho_dY[i], x[L::iY + i], r);
    m = fma(c.dE_dY[i], x[L::iY + i], m);
  }
#pragma unroll
  for (int d = 0; d < DIM; ++d) m = fma(c.v[d], x[1 + d], m);
  y[0] = r;
#pragma unroll
  for (int d = 0; d < DIM; ++d) y[1 + d] = fma(c.v[d], r, c.rho * x[1 + d]);
  y[L::iT] = fma(c.E, r, c.rho * m);
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) y[L::iY + i] = fma(c.Y[i], r, c.rho * x[L::iY + i]);
}

// y = x^T DUDY; returns x.u'
template <int DIM, int NC>
__device__ __forceinline__ double dudy_left(const Coef<DIM, NC>& c, const double* x, double* y) {
  using L = Layout<DIM, NC>;
  double xw = fma(c.E, x[L::iT], x[0]);
#pragma unroll
  for (int d = 0; d < DIM; ++d) xw = fma(c.v[d], x[1 + d], xw);
#pragma unroll
  for (int i = 0; i < NC - 1; ++i) xw = fma(c.Y[i], x[L::iY + i], xw);
  const double re = c.rho * x[L::iT];
  y[0] = fma(xw, c.drho_dp, re * c.de_dp);
#pragma unroll
  for (int d = 0; d < DIM; ++d) y[1 + d] = fma(re, c.v[d], c.rho * x[1 + d]);
  y[L::iT] = fma(xw, c.drho_dT, re * c.de_dT);
#pragma unroll
  for (int i = 0; i < NC - 1; ++i)
    y[L::iY + i] = fma(xw, c.drho_dY[i], fma(re, c.dE_dY[i], c.rho * x[L::iY + i]));
  return fma(c.rho, xw, c.p * x[L::iT]);
}

// Diagonal parameters td of tau (fluid_2d.hpp:877-1022); true for the variants whose tau is
// DUDY^{-1} diag(td).
template <int DIM, int NEN, int NC, int EOS>
__device__ __forceinline__ bool tau_params(const KParams& k, const ElemGeo<DIM, NEN>& q, const Coef<DIM, NC>& c,
                                           const Props<NC>& pr, const double* v, double v_nrm, double h, double trG,
                                           double* td) {
  using L = Layout<DIM, NC>;
  constexpr int ND = L::ND;
  const double dt = k.dt, cs = c.c, rho = c.rho, mu = c.mu, cv = c.cv, kappa = c.kappa;
  const double hh12 = h * h * (1.0 / 12.0);
  // min(use, x/d), without the division where a positive d leaves no doubt
  auto cap = [](double use, double x, double d) { return (d > 0.0 && x >= use * d) ? use : fmin(use, x / d); };
  if (k.tau == GALES_TAU_NON_DIAG_COMP_2001 || k.tau == GALES_TAU_NON_DIAG_COMP_2019) {
    double use;
    if (k.tau == GALES_TAU_NON_DIAG_COMP_2019) {
      // h/(2(|v| + c)) + h/(2|v|)
      use = (0.5 * h) * fma(2.0, v_nrm, cs) / (v_nrm * (v_nrm + cs));
    } else {
      // the reference's alpha vector is never filled: lambda^2 = 4/dt^2 (unsteady) or 0
      const double lambda_sqr = k.steady ? 0.0 : 4 / (dt * dt);
      use = 1.0 / sqrt(lambda_sqr) + h / (2 * v_nrm);
    }
    if (!k.steady) use = fmin(dt * 0.5, use);
    td[0] = use;
    const double tm = cap(use, hh12 * rho, mu);
#pragma unroll
    for (int d = 0; d < DIM; ++d) td[1 + d] = tm;
    td[L::iT] = cap(use, hh12 * rho * cv, kappa);
#pragma unroll
    for (int i = 0; i < NC - 1; ++i)
      td[L::iY + i] = EOS == kEosMagma ? cap(use, hh12, pr.D_c[i]) : fmin(use, hh12 * k.ch[i].inv_D);
    return true;
  }
#pragma unroll
  for (int i = 0; i < ND; ++i) td[i] = 0.0;
  if (k.tau == GALES_TAU_DIAG_INCOMP_2007) {
    double use = 0.0;
#pragma unroll
    for (int i = 0; i < DIM; ++i)
#pragma unroll
      for (int j = 0; j < DIM; ++j) use = fma(q.G[i][j], q.G[i][j], use);
    const double vGv = qform_fma<DIM>(q.G, v);
    const double nu = mu / rho, de = kappa / (rho * cv);
    double tau_m = vGv + 9.0 * use * (nu * nu), tau_e = vGv + 9.0 * use * (de * de);
    if (!k.steady) {
      tau_m += 4.0 / (dt * dt);
      tau_e += 4.0 / (dt * dt);
    }
    tau_m = 1.0 / sqrt(tau_m);
    tau_e = 1.0 / sqrt(tau_e);
    double gg = 0.0;
#pragma unroll
    for (int i = 0; i < DIM; ++i) gg = fma(q.g[i], q.g[i], gg);
    td[0] = 1.0 / (rho * tau_m * gg);
#pragma unroll
    for (int d = 0; d < DIM; ++d) td[1 + d] = tau_m / rho;
    td[L::iT] = tau_e / (rho * cv);
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) td[L::iY + i] = tau_m;
  } else if (k.tau == GALES_TAU_DIAG_2014) {
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      const double a0 = dudy_entry<DIM, NC, double>(c, i, i);
      const double tt = 4.0 / (dt * dt) * (a0 * a0);
      double ta = 0.0, tk = 0.0;
#pragma unroll
      for (int kk = 0; kk < DIM; ++kk)
#pragma unroll
        for (int ll = 0; ll < DIM; ++ll) {
          const double ak = a_entry<DIM, NC, double>(c, kk, i, i);
          const double al = a_entry<DIM, NC, double>(c, ll, i, i);
          const double kv = k_entry<DIM, NC, double>(c, kk, ll, i, i);
          ta += q.G[kk][ll] * (ak * al);
          tk += q.G[kk][ll] * q.G[kk][ll] * (kv * kv);
        }
      td[i] = 1.0 / (sqrt(tt) + sqrt(ta) + sqrt(tk) + 1.e-8);
    }
    td[0] = 1.0 / (td[0] + rho * td[1] * trG);
  }
  return false;
}

// Directions the element block is built in, the gradients of the reference coordinates: those
// of the barycentric coordinates 1..DIM of a simplex (its nodes' shape gradients), of xi, eta,
// zeta of a quadrilateral or hexahedron (xi = sum_i xi_i N_i with the nodes' xi_i = +-1).
template <int DIM, int NEN>
__device__ __forceinline__ void directions(const ElemGeo<DIM, NEN>& q, double (&g)[DIM][DIM]) {
  if constexpr (NEN == DIM + 1) {
#pragma unroll
    for (int k = 0; k < DIM; ++k)
#pragma unroll
      for (int d = 0; d < DIM; ++d) g[k][d] = q.ds[d][k + 1];
  } else {
#pragma unroll
    for (int k = 0; k < DIM; ++k)
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < NEN; ++i) {
          // element.hpp node order: x+ at 1, 2 (mod 4), y+ at 2, 3 (mod 4), z+ at 4..7
          const bool plus = k == 0 ? ((i & 3) == 1 || (i & 3) == 2) : (k == 1 ? (i & 3) >= 2 : i >= 4);
          s = plus ? s + q.ds[d][i] : s - q.ds[d][i];
        }
        g[k][d] = s;
      }
  }
}

// The point stage of one (element, point): about 1,130 FP64 operations, the FP64 pipe 84% busy
// (7.8 ms for 4.0M points, 0.3 of them the unfused gradients; 29 with the reference's operations
// one by one, among them the LU inverse of DUDY, two mixtures with a division per component and 20
// more divisions).  l is the element's place in its block.
template <int DIM, int NEN, int NC, int EOS, bool WANT_M>
__device__ __forceinline__ void point64(const KParams& k, long long e, int iq, double* __restrict__ blk, int l) {
  using L = Layout<DIM, NC>;
  using R = Rec64<DIM, NEN, NC>;
  constexpr int ND = L::ND, NQ = NEN, iT = L::iT, iY = L::iY, EB = R::EB;
  constexpr int NG = geo_per_element<DIM, NEN>(NQ);
  auto W = [&](int f) -> double& { return blk[(size_t)(iq * R::RW + f) * EB + l]; };
  int nodes[NEN];
#pragma unroll
  for (int a = 0; a < NEN; ++a) nodes[a] = __ldg(k.conn + e * NEN + a);
  {
    // scatter descriptor of node b = iq
    int nb = nodes[0];
#pragma unroll
    for (int a = 1; a < NEN; ++a) nb = (iq == a) ? nodes[a] : nb;
    const int fl = k.node_flag ? __ldg(k.node_flag + nb) : 0;
    const uint32_t blocked = (fl >= 0 && fl < GALES_MAX_FLAGS) ? k.dirichlet_mask[fl] : 0u;
    int32_t* di = reinterpret_cast<int32_t*>(blk + (size_t)R::INTS * EB);
    di[(R::I_NODE + iq) * EB + l] = nb;
    di[(R::I_BLOCKED + iq) * EB + l] = (int32_t)blocked;
    if constexpr (WANT_M) {
      const int64_t rr0 = __ldg(k.node_rp + nb), rr1 = __ldg(k.node_rp + nb + 1);
      di[(R::I_ROWLEN + iq) * EB + l] = (int32_t)((rr1 - rr0) * ND);
      const uint16_t* sl = k.slot + ((long long)e * NEN + iq) * NEN;
#pragma unroll
      for (int a = 0; a < NEN; ++a) di[(R::I_OFF + iq * NEN + a) * EB + l] = (int32_t)(rr0 * ND + __ldg(sl + a));
    }
  }
  const ElemGeo<DIM, NEN>& q = reinterpret_cast<const ElemGeo<DIM, NEN>*>(k.geo)[e * NG + (NG == 1 ? 0 : iq)];
  double sh[NEN];
#pragma unroll
  for (int i = 0; i < NEN; ++i) sh[i] = k.sh_tab[iq][i];
  const double jx = q.J * k.W_in;
  double Ie[NEN][ND], Pq[ND], Iq[ND];
#pragma unroll
  for (int i = 0; i < NEN; ++i)
#pragma unroll
    for (int j = 0; j < ND; ++j) Ie[i][j] = __ldg(k.I + (long long)nodes[i] * ND + j);
#pragma unroll
  for (int j = 0; j < ND; ++j) Pq[j] = Iq[j] = 0.0;
#pragma unroll
  for (int i = 0; i < NEN; ++i) {
    const double* pi = k.P + (long long)nodes[i] * ND;
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      Pq[j] = fma(sh[i], __ldg(pi + j), Pq[j]);
      Iq[j] = fma(sh[i], Ie[i][j], Iq[j]);
    }
  }
  // Gradients, summed with the reference's operations: where a field is uniform over the element
  // what rounding leaves of its gradient decides the directions of h and, through grad rho,
  // whether and along what the discontinuity capturing acts.  (With fused sums the blocks of such
  // elements differed from the reference's in their leading digits.)
  double dI[DIM][ND];
  if constexpr (NEN == DIM + 1 && NQ <= 32 && (32 % NQ) == 0) {
    // a simplex's gradient is the same at its points, whose lanes are consecutive: lane iq
    // forms the columns iq, iq + NQ, ... and the element's lanes exchange them
    constexpr int NSL = (ND + NQ - 1) / NQ;
    const unsigned int lane = threadIdx.x & 31u;
    const unsigned int base = lane & ~(unsigned int)(NQ - 1);
    const unsigned int gmask = NQ == 32 ? 0xffffffffu : (((1u << NQ) - 1u) << base);
    double colv[NSL][DIM];
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) {
      const int jj = iq + NQ * sl;
      const int jc = jj < ND ? jj : ND - 1;
#pragma unroll
      for (int d = 0; d < DIM; ++d) colv[sl][d] = 0.0;
#pragma unroll
      for (int i = 0; i < NEN; ++i) {
        double a = Ie[i][0];
#pragma unroll
        for (int j = 1; j < ND; ++j) a = (jc == j) ? Ie[i][j] : a;
#pragma unroll
        for (int d = 0; d < DIM; ++d) colv[sl][d] = add_rn(colv[sl][d], mul_rn(q.ds[d][i], a));
      }
    }
#pragma unroll
    for (int j = 0; j < ND; ++j)
#pragma unroll
      for (int d = 0; d < DIM; ++d) dI[d][j] = __shfl_sync(gmask, colv[j / NQ][d], (int)(base + j % NQ));
  } else {
#pragma unroll
    for (int d = 0; d < DIM; ++d)
#pragma unroll
      for (int j = 0; j < ND; ++j) {
        double b = mul_rn(q.ds[d][0], Ie[0][j]);
#pragma unroll
        for (int i = 1; i < NEN; ++i) b = add_rn(b, mul_rn(q.ds[d][i], Ie[i][j]));
        dI[d][j] = b;
      }
  }
  double dv[DIM][DIM];
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int d = 0; d < DIM; ++d) dv[a][d] = dI[d][1 + a];
  // mixture at P (shear rate 0) and I, conservative variables
  double p, v[DIM], T, Y[NC], U[ND], UP[ND];
  Props<NC> pr;
  Coef<DIM, NC> c;
  double vv, trG = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) trG += q.G[d][d];
  const double mdv = max_entry<DIM>(dv), mm = mdv * mdv;
  {
    double pP, vP[DIM], TP, YP[NC], rhoP, cvP;
    assign<DIM, NC>(Pq, pP, vP, TP, YP);
    assign<DIM, NC>(Iq, p, v, T, Y);
    if constexpr (EOS == kEosMagma) {
      double oP[2];
      unsigned st = magma_rho_cv(k.mg, NC, pP, TP, YP, oP);
      st |= magma_mixture<NC>(k.mg, p, T, Y, shear_rate<DIM>(dv), pr);
      if (st) flag_error(k, GALES_ERR_MAGMA, e);
      rhoP = oP[0];
      cvP = oP[1];
      pr.irho = 1.0 / pr.rho;
#pragma unroll
      for (int i = 0; i < NC; ++i) pr.irho_c[i] = 1.0 / pr.rho_c[i];
    } else {
      mixture_pair_fast<NC, true>(k.ch, k.has_gas != 0, pP, TP, YP, p, T, Y, rhoP, cvP, pr);
      // a gas has no sound speed below T = 0 (chemicals.hpp:258-264)
      if (k.has_gas && !(T >= 0.0)) pr.c = __longlong_as_double(0x7ff8000000000000ll);
    }
    auto speed2 = [&]() {
      double s = v[0] * v[0];
#pragma unroll
      for (int d = 1; d < DIM; ++d) s = fma(v[d], v[d], s);
      return s;
    };
    vv = speed2();
    // |v| below 1e-6 of its variation over the element: the reference's sums decide whether it
    // is zero and where it points
    if (vv * trG < 1.0e-12 * mm) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        double x = 0.0, y = 0.0;
#pragma unroll
        for (int i = 0; i < NEN; ++i) {
          x = add_rn(x, mul_rn(sh[i], __ldg(k.I + (long long)nodes[i] * ND + 1 + d)));
          y = add_rn(y, mul_rn(sh[i], __ldg(k.P + (long long)nodes[i] * ND + 1 + d)));
        }
        Iq[1 + d] = v[d] = x;
        Pq[1 + d] = vP[d] = y;
      }
      vv = speed2();
    }
    conservative<DIM, NC>(rhoP, cvP, vP, TP, YP, UP);
  }
  make_coef_fast<DIM, NC>(pr, p, v, vv, T, Y, c);
  conservative<DIM, NC>(pr.rho, pr.cv, v, T, Y, U);
  const double iv = rsqrt(vv), v_nrm = vv > 0.0 ? vv * iv : 0.0;
  const double uE = U[iT] + p;   // energy entry of u'
  // tau (fluid_2d.hpp:877-1022): dense rows p and E, the velocity and mass-fraction rows'
  // column p and diagonal
  double t0[ND], tE[ND], ta[DIM], tm[DIM], tb[L::NYA], tn[L::NYA];
#pragma unroll
  for (int j = 0; j < ND; ++j) t0[j] = tE[j] = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) ta[d] = tm[d] = 0.0;
#pragma unroll
  for (int i = 0; i < L::NYA; ++i) tb[i] = tn[i] = 0.0;
  if (v_nrm >= kEps && k.tau != GALES_TAU_NONE) {
    bool decided;
    double h = compute_h64<DIM>(q.G, v, vv, iv, dv, mm, decided);
    if (!decided) h = compute_h_reference<DIM, NEN, ND>(k.I, nodes, sh, q);
    double td[ND];
    const bool nondiag = tau_params<DIM, NEN, NC, EOS>(k, q, c, pr, v, v_nrm, h, trG, td);
    if (nondiag) {
      const double det = tau_det<DIM, NC>(c);
      // DUDY is singular exactly where LU meets a zero pivot column: rho = 0 or det = 0
      if (det == 0.0 || c.rho == 0.0) flag_error(k, GALES_ERR_SINGULAR, e);
      double tau[ND][ND];
      tau_closed<DIM, NC, double>(c, pr.irho, 1.0 / det, td, v_nrm < 0.1 * c.c, c.rho * trG, tau);
#pragma unroll
      for (int j = 0; j < ND; ++j) {
        t0[j] = tau[0][j];
        tE[j] = tau[iT][j];
      }
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        ta[d] = tau[1 + d][0];
        tm[d] = tau[1 + d][1 + d];
      }
#pragma unroll
      for (int i = 0; i < NC - 1; ++i) {
        tb[i] = tau[iY + i][0];
        tn[i] = tau[iY + i][iY + i];
      }
    } else {
      t0[0] = td[0];
      tE[iT] = td[iT];
#pragma unroll
      for (int d = 0; d < DIM; ++d) tm[d] = td[1 + d];
#pragma unroll
      for (int i = 0; i < NC - 1; ++i) tn[i] = td[iY + i];
    }
  }
  // least-squares residual Res = DUDY (I - P)/dt + sum_d A_d dI_d - S (fluid_2d.hpp:280-290)
  double dU[DIM][ND], AdI[ND], x[ND], Sv[ND];
#pragma unroll
  for (int j = 0; j < ND; ++j) Sv[j] = 0.0;
  {
    double gv = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      Sv[1 + d] = c.rho * k.gravity[d];
      gv = fma(k.gravity[d], v[d], gv);
    }
    Sv[iT] = c.rho * gv;
  }
  double div = dI[0][1];
#pragma unroll
  for (int d = 1; d < DIM; ++d) div += dI[d][1 + d];
#pragma unroll
  for (int d = 0; d < DIM; ++d) dudy_mul<DIM, NC>(c, dI[d], dU[d]);
#pragma unroll
  for (int j = 0; j < ND; ++j) {
    double s = (j == iT ? uE : U[j]) * div;
#pragma unroll
    for (int d = 0; d < DIM; ++d) s = fma(v[d], dU[d][j], s);
    AdI[j] = s;
  }
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    AdI[1 + d] += dI[d][0];
    AdI[iT] = fma(v[d], dI[d][0], AdI[iT]);
  }
  {
    double dd[ND], Res[ND];
#pragma unroll
    for (int j = 0; j < ND; ++j) dd[j] = (Iq[j] - Pq[j]) * k.inv_dt;
    dudy_mul<DIM, NC>(c, dd, Res);
#pragma unroll
    for (int j = 0; j < ND; ++j) Res[j] = Res[j] + (AdI[j] - Sv[j]);
    // x = tau Res
    double x0 = t0[0] * Res[0], xE = tE[0] * Res[0];
#pragma unroll
    for (int j = 1; j < ND; ++j) {
      x0 = fma(t0[j], Res[j], x0);
      xE = fma(tE[j], Res[j], xE);
    }
    x[0] = x0;
    x[iT] = xE;
#pragma unroll
    for (int d = 0; d < DIM; ++d) x[1 + d] = fma(ta[d], Res[0], tm[d] * Res[1 + d]);
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) x[iY + i] = fma(tb[i], Res[0], tn[i] * Res[iY + i]);
  }
  // discontinuity capturing (fluid_2d.hpp:1027-1065): with s = |grad rho|^2 and
  // S1 = sum_i |grad rho . dN_i| its length is sqrt(s)/S1
  double nu = 0.0;
  if (k.dc_2006) {
    double s = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) s = fma(dU[d][0], dU[d][0], s);
    if (!(s < kEps * kEps)) {
      double S1 = 0.0;
#pragma unroll
      for (int i = 0; i < NEN; ++i) {
        double t = dU[0][0] * q.ds[0][i];
#pragma unroll
        for (int d = 1; d < DIM; ++d) t = fma(dU[d][0], q.ds[d][i], t);
        S1 += fabs(t);
      }
      if (S1 * S1 > (kEps * kEps) * s) {
        double Z2 = 0.0, U2 = 0.0;
#pragma unroll
        for (int j = 0; j < ND; ++j) {
          const double zj = k.u_ref_inv[j] * (AdI[j] - Sv[j]), uj = k.u_ref_inv[j] * U[j];
          Z2 = fma(zj, zj, Z2);
          U2 = fma(uj, uj, U2);
        }
        const double a = k.dc_sharp;
        if (a == 2.0) {
          nu = sqrt(Z2 / U2) * (s / (S1 * S1));
        } else if (a == 1.0 || a == 1.5) {
          const double hd = sqrt(s) / S1;
          double use1 = 0.0;
#pragma unroll
          for (int d = 0; d < DIM; ++d)
#pragma unroll
            for (int j = 0; j < ND; ++j) {
              const double u = k.u_ref_inv[j] * dU[d][j];
              use1 = fma(u, u, use1);
            }
          const double b = 1.0 / sqrt(use1);
          if (a == 1.0) nu = sqrt(Z2) * hd * b;
          else nu = sqrt(Z2) * hd * (b + hd / sqrt(U2)) / 2.0;
        }
        nu = k.dc_scale * nu;
      }
    }
  }
  // the point's residual: N_b rv + sum_d dN_b/dx_d phi_d, least-squares terms included
  {
    double Dx[ND];
    dudy_mul<DIM, NC>(c, x, Dx);
    double gx = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) gx = fma(k.gravity[d], x[1 + d], gx);
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      double rv = fma(U[j] - UP[j], k.inv_dt, -Sv[j]);
      if (j == iT) rv = fma(-c.rho, gx, rv);
      W(R::RV + j) = jx * rv;
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      double ph[ND];
      // A_d x - F_adv + nu dU: v_d (Dx - u') + u' x_vd, then the columns of e_p and p
#pragma unroll
      for (int j = 0; j < ND; ++j) {
        const double up = j == iT ? uE : U[j];
        ph[j] = fma(up, x[1 + d] - v[d], fma(v[d], Dx[j], nu * dU[d][j]));
      }
      ph[1 + d] += x[0] - p;
      ph[iT] = fma(v[d], x[0], ph[iT]);
      // F_dif
      double en = fma(c.kappa, dI[d][iT], 0.0);
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        double ts = c.mu * (dI[d][1 + j] + dI[j][1 + d]);
        if (j == d) ts = fma(c.lambda, div, ts);
        ph[1 + j] += ts;
        en = fma(v[j], ts, en);
      }
#pragma unroll
      for (int i = 0; i < NC - 1; ++i) {
        ph[iY + i] = fma(c.rhoD[i], dI[d][iY + i], ph[iY + i]);
        en = fma(c.rhoDH[i], dI[d][iY + i], en);
      }
      ph[iT] += en;
#pragma unroll
      for (int j = 0; j < ND; ++j) W(R::PHI + d * ND + j) = jx * ph[j];
    }
  }
  if constexpr (WANT_M) {
    // f, h and the sums of e_k from tau as it is, everything else from JxW tau
    double f[DIM], h[L::NYA], eg = 0.0, g[DIM][DIM];
    directions<DIM, NEN>(q, g);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      f[d] = fma(tm[d], v[d], ta[d]);
      eg = fma(k.gravity[d], f[d], eg);
      ta[d] *= jx;
      tm[d] *= jx;
    }
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) {
      h[i] = fma(tn[i], Y[i], tb[i]);
      tb[i] *= jx;
      tn[i] *= jx;
    }
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      t0[j] *= jx;
      tE[j] *= jx;
    }
    double z[ND], y[ND], zd[ND], yd[ND], Zd[ND];
    double bY = 0.0, bE = 0.0;
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) {
      bY = fma(c.drho_dY[i], tb[i], bY);
      bE = fma(c.dE_dY[i], tb[i], bE);
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) bE = fma(v[d], ta[d], bE);
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      double a = j == 0 ? bY : 0.0, b = j == 0 ? bE : 0.0;
      if (j >= 1 && j < iT) b = v[j < 1 ? 0 : (j - 1) % DIM] * tm[j < 1 ? 0 : (j - 1) % DIM];
      if (j >= iY) {
        a = c.drho_dY[(j - iY) % L::NYA] * tn[(j - iY) % L::NYA];
        b = c.dE_dY[(j - iY) % L::NYA] * tn[(j - iY) % L::NYA];
      }
      z[j] = fma(c.drho_dp, t0[j], fma(c.drho_dT, tE[j], a));
      y[j] = fma(c.de_dp, t0[j], fma(c.de_dT, tE[j], b));
    }
    const double zu = dudy_left<DIM, NC>(c, z, zd), yu = dudy_left<DIM, NC>(c, y, yd);
    const double t0u = dudy_left<DIM, NC>(c, t0, Zd);
    const double jr = jx * c.rho, jE = jx * c.E;
    auto theta = [&](double a, double b, double t) { return fma(c.E, a, fma(c.rho, b, t)); };
    W(R::JX) = jx;
    W(R::JR) = jr;
    W(R::RHO) = c.rho;
    W(R::PR) = p;
    W(R::NU) = nu;
    W(R::JMU) = jx * c.mu;
    W(R::JKAP) = jx * c.kappa;
    W(R::EG) = eg;
    W(R::ZU) = zu;
    W(R::T0U) = t0u;
    W(R::THU) = theta(zu, yu, t0u);
    W(R::ZE) = z[iT];
    W(R::T0E) = t0[iT];
    W(R::THE) = theta(z[iT], y[iT], t0[iT]);
    W(R::E) = c.E;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      W(R::V + d) = v[d];
      W(R::F + d) = f[d];
      W(R::JM + d) = tm[d];
      W(R::ZV + d) = z[1 + d];
      W(R::T0V + d) = t0[1 + d];
      W(R::THV + d) = theta(z[1 + d], y[1 + d], t0[1 + d]);
    }
    if constexpr (!R::SIMPLEX) {
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) W(R::G + a * DIM + d) = g[a][d];
#pragma unroll
        for (int b = a; b < DIM; ++b) {
          double s = g[a][0] * g[b][0];
#pragma unroll
          for (int d = 1; d < DIM; ++d) s = fma(g[a][d], g[b][d], s);
          W(R::GG + gg_at(DIM, a, b)) = s;
        }
      }
    }
#pragma unroll
    for (int kk = 0; kk < DIM; ++kk) {
      double s = g[kk][0] * v[0], ek = g[kk][0] * f[0];
#pragma unroll
      for (int d = 1; d < DIM; ++d) {
        s = fma(g[kk][d], v[d], s);
        ek = fma(g[kk][d], f[d], ek);
      }
      W(R::S + kk) = s;
      W(R::EK + kk) = ek;
    }
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) {
      W(R::Y + i) = Y[i];
      W(R::H + i) = h[i];
      W(R::JRN + i) = c.rho * tn[i];
      W(R::JRD + i) = jx * c.rhoD[i];
      W(R::JRDH + i) = jx * c.rhoDH[i];
      W(R::R0 + 2 + i) = jx * c.drho_dY[i];
      W(R::DE + 2 + i) = fma(jE, c.drho_dY[i], jr * c.dE_dY[i]);
    }
    W(R::R0) = jx * c.drho_dp;
    W(R::R0 + 1) = jx * c.drho_dT;
    W(R::DE) = fma(jE, c.drho_dp, jr * c.de_dp);
    W(R::DE + 1) = fma(jE, c.drho_dT, jr * c.de_dT);
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      W(R::ZETA + j) = zd[j];
      W(R::ZZ + j) = Zd[j];
      W(R::THETA + j) = theta(zd[j], yd[j], Zd[j]);
    }
  }
  if (!finite_bits(jx) || !finite_bits(pr.rho) || !finite_bits(nu)) flag_error(k, GALES_ERR_NONFINITE, e);
}

template <int DIM, int NEN, int NC, int EOS, bool WANT_M>
__global__ void __launch_bounds__(128) point64_kernel(const KParams k, double* __restrict__ out, long long first,
                                                      long long n) {
  using R = Rec64<DIM, NEN, NC>;
  constexpr int NQ = NEN;
  const int t = (int)blockIdx.x * 128 + (int)threadIdx.x;
  const int li = t / NQ, iq = t - li * NQ;
  if (li < n) {
    const long long g = first + li;
    const long long e = k.el_list ? (long long)k.el_list[g] : g;
    const int b = li / R::EB;
    point64<DIM, NEN, NC, EOS, WANT_M>(k, e, iq, out + (size_t)b * R::EW * R::EB, li - b * R::EB);
  }
  if (k.clear_n[0] > 0 || k.clear_n[1] > 0) clear_arrays(k);
}

// rhs of row r of the element at place l: -(sum_q N_b rv + sum_d dN_b/dx_d phi_d); a simplex's
// gradients do not depend on the point.
template <int DIM, int NEN, int NC, typename Sink>
__device__ __forceinline__ void row_residual64(const KParams& k, const double* __restrict__ blk, int l, int r,
                                               const ElemGeo<DIM, NEN>* __restrict__ geo, Sink sink) {
  using R = Rec64<DIM, NEN, NC>;
  constexpr int NQ = NEN, ND = R::ND;
  auto W = [&](int p, int f) -> double { return blk[(size_t)(p * R::RW + f) * R::EB + l]; };
  if constexpr (R::SIMPLEX) {
    double rv[NQ], ph[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) ph[d] = W(0, R::PHI + d * ND + r);
#pragma unroll
    for (int p = 0; p < NQ; ++p) {
      rv[p] = W(p, R::RV + r);
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        if (p > 0) ph[d] += W(p, R::PHI + d * ND + r);
    }
#pragma unroll
    for (int b = 0; b < NEN; ++b) {
      double s = geo->ds[0][b] * ph[0];
#pragma unroll
      for (int d = 1; d < DIM; ++d) s = fma(geo->ds[d][b], ph[d], s);
#pragma unroll
      for (int p = 0; p < NQ; ++p) s = fma(k.sh_tab[p][b], rv[p], s);
      sink(b, -s);
    }
  } else {
    double s[NEN];
#pragma unroll
    for (int b = 0; b < NEN; ++b) s[b] = 0.0;
#pragma unroll 1
    for (int p = 0; p < NQ; ++p) {
      const double rv = W(p, R::RV + r);
      double ph[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) ph[d] = W(p, R::PHI + d * ND + r);
#pragma unroll
      for (int b = 0; b < NEN; ++b) {
        s[b] = fma(k.sh_tab[p][b], rv, s[b]);
#pragma unroll
        for (int d = 0; d < DIM; ++d) s[b] = fma(geo[p].ds[d][b], ph[d], s[b]);
      }
    }
#pragma unroll
    for (int b = 0; b < NEN; ++b) sink(b, -s[b]);
  }
}

// The rhs alone: a thread per (element, dof row), lanes along the elements of a block.
template <int DIM, int NEN, int NC>
__global__ void __launch_bounds__(128) residual64_kernel(const KParams k, const double* __restrict__ in, long long first,
                                                         long long n) {
  using R = Rec64<DIM, NEN, NC>;
  constexpr int ND = R::ND, EB = R::EB, NGE = geo_per_element<DIM, NEN>(NEN);
  const long long t = (long long)blockIdx.x * 128 + threadIdx.x;
  const int l = (int)(t % EB);
  const long long task = t / EB;
  const int r = (int)(task % ND);
  const long long b = task / ND, li = b * EB + l;
  if (li >= n) return;
  const long long e = k.el_list ? (long long)k.el_list[first + li] : first + li;
  const double* blk = in + (size_t)b * R::EW * EB;
  const int32_t* di = reinterpret_cast<const int32_t*>(blk + (size_t)R::INTS * EB);
  row_residual64<DIM, NEN, NC>(k, blk, l, r, reinterpret_cast<const ElemGeo<DIM, NEN>*>(k.geo) + e * NGE, [&](int nb, double v) {
    if (k.local_r) {
      k.local_r[(first + li) * R::N + nb * ND + r] = v;
    } else if (!(((uint32_t)di[(R::I_BLOCKED + nb) * EB + l] >> r) & 1u)) {
      add_to(k.rhs + (long long)di[(R::I_NODE + nb) * EB + l] * ND + r, v, k.scatter_mode);
    }
  });
}

// Row r = ROW of the element blocks of a simplex, a thread per element (see the head of this
// file).  The block is built in the barycentric directions 1..DIM: rows of node b and columns
// of node a for b, a >= 1, the columns of node 0 from sum_a (N_a, dN_a) = (1, 0), the rows of
// node 0 from the same sum over the test functions.  The points of the simplex rules have
// N_a(q) = beta but for N_q(q) = alpha, so sum_q N_a(q) W_q = beta sum_q W_q + (alpha - beta) W_a.
// acc (shared memory, NQ ND words of the lane) holds the rows of node 0: the sum over all test
// functions less the others.  emit(b, a, c, value) receives every entry.
template <int DIM, int NC, int ROW, typename Emit>
__device__ __forceinline__ void simplex_row64(const KParams& k, const double* __restrict__ rec,
                                              const ElemGeo<DIM, DIM + 1>& geo, double* acc, Emit emit) {
  using L = Layout<DIM, NC>;
  using R = Rec64<DIM, DIM + 1, NC>;
  constexpr int ND = L::ND, NQ = DIM + 1, iT = L::iT, iY = L::iY, EB = R::EB;
  constexpr bool rE = ROW == iT, rV = ROW >= 1 && ROW < iT, rY = ROW >= iY;
  constexpr int J = rV ? ROW - 1 : 0, IY = rY ? ROW - iY : 0;
  auto W = [&](int p, int f) -> double { return __ldg(rec + (size_t)(p * R::RW + f) * EB); };
  const double dt = k.dt;
  const double beta = k.sh_tab[0][1], alpha = k.sh_tab[1][1];
  const double bdt = beta * k.inv_dt, adt = (alpha - beta) * k.inv_dt;
  // sums over the points that do not depend on the test function: nu DUDY[r] and the
  // viscous scalars of the row
  double Dn[ND], kmu = 0.0, kap = 0.0, kmv[DIM], krd[L::NYA];
#pragma unroll
  for (int c = 0; c < ND; ++c) Dn[c] = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) kmv[d] = 0.0;
#pragma unroll
  for (int i = 0; i < L::NYA; ++i) krd[i] = 0.0;
  // columns of DUDY[r] that can be nonzero
  auto d_nz = [](int c) { return rE || R::col_r0(c) >= 0 || c == ROW; };

  // one test function: b >= 1, or the sum of all of them (N = 1, gradient 0); the sum's
  // least-squares part is the source's, on the energy row alone
  auto test_function = [&](int b, auto sum) {
    constexpr bool total = decltype(sum)::value, ls = !total || rE;
    double gb[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) gb[d] = total ? 0.0 : geo.ds[d][b];
    const double gJ = rV ? gb[J] : 0.0, dgJ = rV ? dt * gJ : 0.0;
    // Wq: dt JxW (FPT (DUDY/dt - S0) + X_b) of point q, X_b = N_b (DUDY/dt - S0) - WA_b;
    // M[a] etc.: sums over the points of the least-squares products with A_a
    double Wq[NQ][ND], Ws[ND], M[DIM][ND], fuM = 0.0, FV[DIM], FE[DIM];
#pragma unroll
    for (int p = 0; p < NQ; ++p) {
      const double rho = W(p, R::RHO), jx = W(p, R::JX);
      const double Nb = total ? 1.0 : (b == p ? alpha : beta);
      const double s = total ? 0.0 : W(p, R::S + b - 1), eb = total ? 0.0 : W(p, R::EK + b - 1);
      const double wr = rE ? W(p, R::E) : (rV ? W(p, R::V + J) : (rY ? W(p, R::Y + IY) : 1.0));
      const double ur = rE ? fma(rho, wr, W(p, R::PR)) : (ROW == 0 ? rho : rho * wr);  // u'_r
      const double rN = rE ? rho * Nb : 0.0;
      const double sdt = total ? 0.0 : s * dt;
      const double cD = total ? 1.0 : Nb - sdt;        // dt (N_b/dt - s_b)
      double FD[ND], fe = 0.0;
      if constexpr (ls) {
        // coefficients of zeta (Theta), r0 and m in FPT_b and FPT_b DUDY
        const double cz = (rE || ROW == 0) ? s : s * wr;
        double cr;
        if constexpr (rE) cr = total ? -rN * W(p, R::EG) : fma(ur, eb, -rN * W(p, R::EG));
        else if constexpr (rV) cr = rho * fma(wr, eb, s * W(p, R::F + J));
        else if constexpr (rY) cr = rho * fma(wr, eb, s * W(p, R::H + IY));
        else cr = rho * eb;
        const double sr = (rV || rY) ? s * rho : 0.0;
        auto comb = [&](int fz, int f0) {   // cz zeta + gb_J tau0
          double t = cz * W(p, fz);
          if constexpr (rV) t = fma(gJ, W(p, f0), t);
          return t;
        };
        if constexpr (!total) fe = comb(rE ? R::THE : R::ZE, R::T0E);
        const double fu = total ? cr * W(p, R::JR) : fma(cr, W(p, R::JR), comb(rE ? R::THU : R::ZU, R::T0U));
        fuM = p == 0 ? fu : fuM + fu;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          double t = total ? 0.0 : ur * gb[d];
          if constexpr (rE) t = total ? -rN * k.gravity[d] : fma(-rN, k.gravity[d], t);
          if (rV && d == J) t += sr;
          const double fv = total ? t * W(p, R::JM + d) : fma(t, W(p, R::JM + d), comb((rE ? R::THV : R::ZV) + d, R::T0V + d));
          FV[d] = p == 0 ? fv : FV[d] + fv;
          FD[1 + d] = rho * (total ? fv : fma(fe, W(p, R::V + d), fv));
        }
#pragma unroll
        for (int c = 0; c < ND; ++c) {
          if (R::col_r0(c) < 0) continue;
          const double r0c = W(p, R::R0 + R::col_r0(c));
          double t = total ? cr * r0c : fma(cr, r0c, comb((rE ? R::THETA : R::ZETA) + c, R::ZZ + c));
          if (rY && c == ROW) t = fma(sr, W(p, R::JRN + IY), t);
          FD[c] = t;
        }
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
          const double sa = W(p, R::S + a);
          if constexpr (!total) FE[a] = p == 0 ? sa * fe : fma(sa, fe, FE[a]);
#pragma unroll
          for (int c = 0; c < ND; ++c) M[a][c] = p == 0 ? sa * FD[c] : fma(sa, FD[c], M[a][c]);
        }
      }
      const double cDr = total && ROW == 0 ? 0.0 : cD * W(p, R::JR);   // on the diagonal of M
      const double ug = total ? 0.0 : -(dt * jx) * ur, gr = -dt * (rE ? fma(fe, rho, rN * jx) : fe * rho);
#pragma unroll
      for (int c = 0; c < ND; ++c) {
        double t = ls ? FD[c] : 0.0;
        if (R::col_r0(c) >= 0) {
          const int ci = R::col_r0(c) < 0 ? 0 : R::col_r0(c);
          const double cc = (rE || ROW == 0) ? cD : cD * wr;
          const double r0c = W(p, (rE ? R::DE : R::R0) + ci);
          t = ls ? fma(cc, r0c, t) : cc * r0c;
        } else if (ls) {
          const int d = (c < 1 ? 0 : (c - 1) % DIM);
          if constexpr (rE) t = fma(cDr, W(p, R::V + d), t);
          if constexpr (!total) t = fma(ug, gb[d], t);
          t = fma(gr, k.gravity[d], t);
        }
        if (c == 0 && rV && !total) t = fma(-dgJ, jx, t);
        if (c == 0 && rE && !total) t = fma(-sdt, jx, t);
        if ((rV || rY) && c == ROW) t = (ls || R::col_r0(c) >= 0) ? t + cDr : cDr;
        Wq[p][c] = t;
        Ws[c] = p == 0 ? t : Ws[c] + t;
      }
    }
    double o0[ND];   // columns of node 0: the sum over the trial functions less the others
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      o0[c] = Ws[c] * k.inv_dt;
      Ws[c] *= bdt;
    }
#pragma unroll
    for (int a = 1; a < NQ; ++a) {
      double ga[DIM], gg = 0.0;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        ga[d] = geo.ds[d][a];
        if constexpr (!total) gg = d == 0 ? gb[0] * ga[0] : fma(gb[d], ga[d], gg);
      }
      double o[ND];
#pragma unroll
      for (int c = 0; c < ND; ++c) {
        o[c] = fma(adt, Wq[a][c], Ws[c]);
        if constexpr (ls) o[c] += M[a - 1][c];
        if constexpr (!total)
          if (d_nz(c)) o[c] = fma(gg, Dn[c], o[c]);
      }
      if constexpr (ls) {
        if constexpr (!total) o[0] += FE[a - 1];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          o[0] = fma(ga[d], FV[d], o[0]);
          o[1 + d] = fma(ga[d], fuM, o[1 + d]);
        }
      }
      if constexpr (!total) {
        // viscous and diffusive terms (fluid_2d.hpp:531-571; the closed form beside viscous_row32)
        if constexpr (rV) {
          const double p1 = kmu * ga[J], p2 = (-2.0 / 3.0) * kmu * gb[J];
#pragma unroll
          for (int m = 0; m < DIM; ++m) o[1 + m] = fma(gb[m], p1, fma(ga[m], p2, o[1 + m]));
          o[1 + J] = fma(kmu, gg, o[1 + J]);
        }
        if constexpr (rE) {
          double gamv = ga[0] * kmv[0], gbmv = gb[0] * kmv[0];
#pragma unroll
          for (int d = 1; d < DIM; ++d) {
            gamv = fma(ga[d], kmv[d], gamv);
            gbmv = fma(gb[d], kmv[d], gbmv);
          }
          gbmv *= -2.0 / 3.0;
#pragma unroll
          for (int m = 0; m < DIM; ++m)
            o[1 + m] = fma(gb[m], gamv, fma(ga[m], gbmv, fma(kmv[m], gg, o[1 + m])));
          o[iT] = fma(kap, gg, o[iT]);
#pragma unroll
          for (int i = 0; i < NC - 1; ++i) o[iY + i] = fma(krd[i], gg, o[iY + i]);
        }
        if constexpr (rY) o[ROW] = fma(krd[IY], gg, o[ROW]);
      }
#pragma unroll
      for (int c = 0; c < ND; ++c) {
        o0[c] -= o[c];
        if constexpr (total) {
          acc[a * ND + c] = o[c];
        } else {
          acc[a * ND + c] -= o[c];
          emit(b, a, c, o[c]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      if constexpr (total) {
        acc[c] = o0[c];
      } else {
        acc[c] -= o0[c];
        emit(b, 0, c, o0[c]);
      }
    }
  };
  test_function(0, std::true_type());
#pragma unroll
  for (int p = 0; p < NQ; ++p) {
    const double nu = W(p, R::NU), jnr = nu * W(p, R::JR);
    const double wr = rV ? W(p, R::V + J) : (rY ? W(p, R::Y + IY) : 1.0);
    const double nw = (rE || ROW == 0) ? nu : nu * wr;
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      if (R::col_r0(c) >= 0)
        Dn[c] = fma(nw, W(p, (rE ? R::DE : R::R0) + (R::col_r0(c) < 0 ? 0 : R::col_r0(c))), Dn[c]);
      else if constexpr (rE)
        Dn[c] = fma(jnr, W(p, R::V + (c < 1 ? 0 : (c - 1) % DIM)), Dn[c]);
      if ((rV || rY) && c == ROW) Dn[c] += jnr;
    }
    if constexpr (rV) kmu += W(p, R::JMU);
    if constexpr (rE) {
      kap += W(p, R::JKAP);
      const double jm = W(p, R::JMU);
#pragma unroll
      for (int d = 0; d < DIM; ++d) kmv[d] = fma(jm, W(p, R::V + d), kmv[d]);
#pragma unroll
      for (int i = 0; i < NC - 1; ++i) krd[i] += W(p, R::JRDH + i);
    }
    if constexpr (rY) krd[IY] += W(p, R::JRD + IY);
  }
#pragma unroll 1
  for (int b = 1; b < NQ; ++b) test_function(b, std::false_type());
#pragma unroll
  for (int a = 0; a < NQ; ++a)
#pragma unroll
    for (int c = 0; c < ND; ++c) emit(0, a, c, acc[a * ND + c]);
}

// Matrix stage of the simplices.  A warp takes one dof row of the EB = 32 elements of a block,
// a lane per element, so that the row's structure is known at compile time and no lane idles
// (a lane per block row kept 28 of 32 busy and paid for every row type in each).  The rows of
// one node are staged in shared memory and scattered one after the other, consecutive lanes
// on consecutive columns of the CSR row.  Each row is several thousand instructions of its
// own, so neighbouring CTAs take the same row of other blocks, a group of kRows64Group at a
// time: with the rows of one block side by side two thirds of the cycles waited for
// instructions (54 ms for 998,250 tets with 7 dofs, 25 in this order; any group from 152 CTAs
// up does).  Bound: the FP64 pipe, 83% busy with 1,757 instructions per row and 32 elements:
// 23.3 ms for those tets, where a lane per block row that formed FPT_b took 57.  CTAs of
// kRows64Warps warps; of one where the launch has fewer than 16 warps for each SM, which they
// spread evenly (4,096 triangles with 5 dofs: 53 us against 63; 4,374 tets with 7: 151 against
// 163; from 16 warps on no difference).
constexpr int kRows64Warps = 4;
constexpr int kRows64Group = 304;   // CTAs whose blocks are taken row by row (two per SM)

template <int DIM, int NC>
struct Rows64Smem {
  static constexpr int N = (DIM + 1) * Layout<DIM, NC>::ND, NS = N + 1;
  double st[32 * NS], acc[32 * NS];   // a warp's
};

template <int DIM, int NC>
__global__ void __launch_bounds__(32 * kRows64Warps)
    rows64_kernel(const KParams k, double* in, long long first, long long n) {
  constexpr int NEN = DIM + 1;
  using R = Rec64<DIM, NEN, NC>;
  using SM = Rows64Smem<DIM, NC>;
  constexpr int ND = R::ND, N = R::N, EB = R::EB, NS = SM::NS;
  static_assert(EB == 32, "a lane per element of a block");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SM& sm = reinterpret_cast<SM*>(smem_raw)[threadIdx.x >> 5];
  double* st = sm.st;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  double* acc = sm.acc + lane * NS;
  const long long nblk = (n + EB - 1) / EB, ncta = (nblk + warps - 1) / warps;
  // CTA order: groups of kRows64Group CTAs' blocks, all of a group's first rows, then its second
  const long long gi = (long long)blockIdx.x / ((long long)kRows64Group * ND);
  const long long c0 = gi * kRows64Group, nc = ncta - c0 < kRows64Group ? ncta - c0 : kRows64Group;
  const long long u = (long long)blockIdx.x - c0 * ND;
  const int r = (int)(u / nc);
  const long long b0 = (c0 + u % nc) * warps + (threadIdx.x >> 5);
  if (b0 >= nblk) return;
  const int cnt = (int)(n - b0 * EB < EB ? n - b0 * EB : EB);
  const long long li = b0 * EB + (lane < cnt ? lane : cnt - 1);
  const int l = lane < cnt ? lane : cnt - 1;   // idle lanes of a last block repeat its last element
  const long long e = k.el_list ? (long long)k.el_list[first + li] : first + li;
  const double* blk = in + (size_t)b0 * R::EW * EB;
  const int32_t* di = reinterpret_cast<const int32_t*>(blk + (size_t)R::INTS * EB);
  const ElemGeo<DIM, NEN>& geo = reinterpret_cast<const ElemGeo<DIM, NEN>*>(k.geo)[e];
  const bool local = k.local_r != nullptr, vjp = k.vjp_lam != nullptr;
  const int mode = k.scatter_mode;
  double tr = 0.0;
  if (vjp) {
    for (int c = 0; c < N; ++c) st[lane * NS + c] = 0.0;
  } else {
    row_residual64<DIM, NEN, NC>(k, blk, l, r, &geo, [&](int nb, double v) {
      if (lane >= cnt) return;
      if (local) k.local_r[(first + li) * N + nb * ND + r] = v;
      else if (!(((uint32_t)di[(R::I_BLOCKED + nb) * EB + l] >> r) & 1u))
        add_to(k.rhs + (long long)di[(R::I_NODE + nb) * EB + l] * ND + r, v, mode);
    });
  }
  // scatters the staged rows of node b (their lane's element per row of st)
  auto flush = [&](int b) {
    __syncwarp();
    for (int t = lane; t < cnt * N; t += 32) {
      const int el = t / N, cx = t - el * N, a = cx / ND;
      const double val = st[el * NS + cx];
      if (local) {
        k.local_m[(first + b0 * EB + el) * (long long)(N * N) + (b * ND + r) * N + cx] = val;
        continue;
      }
      if (((uint32_t)di[(R::I_BLOCKED + b) * EB + el] >> r) & 1u) continue;
      if (val != 0.0)
        add_to(k.vals + (int64_t)di[(R::I_OFF + b * NEN + a) * EB + el] * ND +
                   (int64_t)r * di[(R::I_ROWLEN + b) * EB + el] + (cx - a * ND),
               val, mode);
    }
    __syncwarp();
  };
  auto run = [&](auto row) {
    constexpr int ROW = decltype(row)::value;
    if (vjp) {
      double lam = 0.0;
      int at = -1;
      simplex_row64<DIM, NC, ROW>(k, blk + l, geo, acc, [&](int b, int a, int c, double v) {
        if (a == b && c == ROW) tr += v;
        if (b != at) {
          at = b;
          const bool off = ((uint32_t)di[(R::I_BLOCKED + b) * EB + l] >> ROW) & 1u;
          lam = off ? 0.0 : __ldg(k.vjp_lam + (long long)di[(R::I_NODE + b) * EB + l] * ND + ROW);
        }
        st[lane * NS + a * ND + c] = fma(lam, v, st[lane * NS + a * ND + c]);
      });
    } else {
      simplex_row64<DIM, NC, ROW>(k, blk + l, geo, acc, [&](int b, int a, int c, double v) {
        if (a == b && c == ROW) tr += v;
        st[lane * NS + a * ND + c] = v;
        // a test function's last entry: node 0's last column
        const bool done = b == 0 ? (a == NEN - 1 && c == ND - 1) : (a == 0 && c == ND - 1);
        if (done && (!local || k.local_m)) flush(b);
      });
    }
  };
  switch (r) {
    case 0: run(std::integral_constant<int, 0>()); break;
    case 1: run(std::integral_constant<int, 1>()); break;
    case 2: run(std::integral_constant<int, 2>()); break;
    case 3: run(std::integral_constant<int, 3>()); break;
    case 4: if constexpr (ND > 4) run(std::integral_constant<int, 4 < ND ? 4 : 0>()); break;
    case 5: if constexpr (ND > 5) run(std::integral_constant<int, 5 < ND ? 5 : 0>()); break;
    case 6: if constexpr (ND > 6) run(std::integral_constant<int, 6 < ND ? 6 : 0>()); break;
    default: if constexpr (ND > 7) run(std::integral_constant<int, 7 < ND ? 7 : 0>()); break;
  }
  static_assert(ND >= 4 && ND <= 8, "rows dispatched above");
  if (lane < cnt && !local)
    in[((size_t)b0 * R::EW + R::TR + r) * EB + l] = tr;
  if (vjp) {
    __syncwarp();
    for (int t = lane; t < cnt * N; t += 32) {
      const int el = t / N, cx = t - el * N, a = cx / ND;
      const double val = st[el * NS + cx];
      if (val != 0.0) atomicAdd(k.vjp_g + (long long)di[(R::I_NODE + a) * EB + el] * ND + (cx - a * ND), val);
    }
  }
}

// Matrix stage of quadrilaterals and hexahedra, a CTA per element.  In the reference
// directions the block is
//   block(b, a) = sum_q sum_ij phi_b^i(q) H_ij(q) phi_a^j(q),  phi^0 = N, phi^k = dN/dxi_k,
// with nd x nd matrices H_ij of the point that do not know the nodes:
//   H_00 = JxW (DUDY/dt - S0) + source's least squares     H_k0 = JxW (FPT_k (DUDY/dt - S0) - A_k)
//   H_0l = -JxW S0 tau A_l (energy row alone)               H_kl = JxW (FPT_k A_l + K'_kl),
// FPT_k = A_k tau for the test function with gradient e_k (see the head of this file).  A
// thread per (point, dof row) forms the H_ij in shared memory (about 540 FP64 operations with
// 8 dofs), then a thread per (row, column) contracts one direction after the other with the
// one-dimensional shape functions (sum factorisation): 1,600 operations for its 64 entries of
// the hexahedron against 3,072 for a direct contraction.  With FPT_b and the block rows formed
// per test function and point it was 481,000 operations per hexahedron; now 131,000.  Bound:
// the FP64 pipe.
template <int DIM, int NC>
struct Tensor64 {
  static constexpr int NEN = 1 << DIM;
  using R = Rec64<DIM, NEN, NC>;
  static constexpr int ND = R::ND, NQ = NEN, NF = DIM + 1;
  static constexpr int RS = ND | 1;             // row stride of a matrix (conflict-free stores by row)
  static constexpr int HS = ND * RS;            // words of one matrix
  static constexpr int T1 = NQ * ND, T2 = ND * ND;
  static constexpr int THREADS = ((T1 > T2 ? T1 : T2) + 31) / 32 * 32;
  struct Smem {
    double H[NF * NF][NQ][HS];
    int32_t off[NEN][NEN], rowlen[NEN], node[NEN];
    uint32_t blocked[NEN];
  };
  // node and point of the corner with the given signs (element.hpp order)
  static __device__ __forceinline__ int corner(int x, int y, int z) { return (z << 2) | (y ? 3 - x : x); }
};

// H_ij of point q, row r.
template <int DIM, int NC>
__device__ __forceinline__ void tensor_point64(const KParams& k, const double* __restrict__ blk, int l, int q, int r,
                                               double (*H)[Tensor64<DIM, NC>::NQ][Tensor64<DIM, NC>::HS]) {
  using T = Tensor64<DIM, NC>;
  using R = typename T::R;
  using L = Layout<DIM, NC>;
  constexpr int ND = T::ND, iT = L::iT, iY = L::iY, NF = T::NF;
  const bool rE = r == iT, rV = r >= 1 && r < iT, rY = r >= iY;
  auto W = [&](int f) -> double { return blk[(size_t)(q * R::RW + f) * R::EB + l]; };
  auto out = [&](int i, int j, int c) -> double& { return H[i * NF + j][q][r * T::RS + c]; };
  const double rho = W(R::RHO), jx = W(R::JX), jr = W(R::JR), nu = W(R::NU), jmu = W(R::JMU);
  const double wr = r == 0 ? 1.0 : W(rV ? R::V + r - 1 : (rE ? R::E : R::Y + r - iY));
  const double wz = rE ? 1.0 : wr;
  const double ur = fma(rho, wr, rE ? W(R::PR) : 0.0);
  const double rhf = rV ? rho * W(R::F + r - 1) : (rY ? rho * W(R::H + r - iY) : 0.0);
  const int fz = rE ? R::THETA : R::ZETA;
  double v[DIM], g[DIM][DIM], s[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    v[d] = W(R::V + d);
    s[d] = W(R::S + d);
#pragma unroll
    for (int a = 0; a < DIM; ++a) g[a][d] = W(R::G + a * DIM + d);
  }
  // FPT_k DUDY = s_k Q + gZ_k Z + u'_r e_k r0 (p, T, Y columns), rho (FPT_k + FPT_k[E] v) (velocities);
  // Qv, Qe, Qu: the part of FPT_k's velocity and energy entries and of FPT_k.u' that goes with s_k
  double Q[L::iT + NC], Qv[DIM], DR[ND], KD[ND];
  const double Qe = wz * W(rE ? R::THE : R::ZE);
  const double Qu = fma(rhf, jr, wz * W(rE ? R::THU : R::ZU));
  const double t0e = W(R::T0E), t0u = W(R::T0U);
  double t0v[DIM], jm[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    t0v[d] = W(R::T0V + d);
    jm[d] = W(R::JM + d);
    Qv[d] = fma(rV && d == r - 1 ? rho : 0.0, jm[d], wz * W((rE ? R::THV : R::ZV) + d));
  }
  double r0[R::NR], Z[R::NR];
#pragma unroll
  for (int c = 0; c < ND; ++c) {
    const int ci = R::col_r0(c);
    if (ci >= 0) {
      r0[ci < 0 ? 0 : ci] = W(R::R0 + (ci < 0 ? 0 : ci));
      Z[ci < 0 ? 0 : ci] = W(R::ZZ + c);
      double x = fma(rhf, r0[ci < 0 ? 0 : ci], wz * W(fz + c));
      if (c >= iY) x = fma(rY && c == r ? rho : 0.0, W(R::JRN + (c - iY) % L::NYA), x);
      Q[c] = x;
      DR[c] = rE ? W(R::DE + (ci < 0 ? 0 : ci)) : wr * r0[ci < 0 ? 0 : ci];
    } else {
      Q[c] = 0.0;
      DR[c] = rE ? jr * v[(c - 1) % DIM] : 0.0;
    }
    if (c >= 1 && c != iT) DR[c] += c == r ? jr : 0.0;
    // what multiplies grad.grad: the diffusive entries of K and nu DUDY
    double kd = 0.0;
    if (c >= 1 && c < iT) kd = rE ? jmu * v[(c < 1 ? 0 : c - 1) % DIM] : (c == r ? jmu : 0.0);
    if (c == iT) kd = rE ? W(R::JKAP) : 0.0;
    if (c >= iY) kd = rE ? W(R::JRDH + (c - iY) % L::NYA) : (c == r ? W(R::JRD + (c - iY) % L::NYA) : 0.0);
    KD[c] = fma(nu, DR[c], kd);
  }
  // the viscous entries on the velocity columns: jmu a_l g_k + jlam a_k g_l, a = g[., r] or s (energy row)
  double av[DIM];
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    double x = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) x = (rV && d == r - 1) ? g[a][d] : x;
    av[a] = rE ? s[a] : x;
  }
  const double jlam = (-2.0 / 3.0) * jmu;
#pragma unroll
  for (int kk = 0; kk < DIM; ++kk) {
    const double sk = s[kk], gZ = rV ? av[kk] : 0.0, ue = ur * W(R::EK + kk);
    const double fe = fma(gZ, t0e, sk * Qe);
    double fu = fma(ue, jr, fma(gZ, t0u, sk * Qu));
    double fv[DIM], FD[ND];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      fv[d] = fma(ur * g[kk][d], jm[d], fma(gZ, t0v[d], sk * Qv[d]));
      FD[1 + d] = rho * fma(fe, v[d], fv[d]);
    }
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      const int ci = R::col_r0(c);
      if (ci >= 0) FD[c] = fma(ue, r0[ci < 0 ? 0 : ci], fma(gZ, Z[ci < 0 ? 0 : ci], sk * Q[c]));
    }
    // H_k0
    const double ug = jx * ur, fr = fe * rho;
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      double x = fma(k.inv_dt, FD[c], -sk * DR[c]);
      if (c >= 1 && c < iT) {
        x = fma(-ug, g[kk][(c < 1 ? 0 : c - 1) % DIM], x);
        x = fma(-fr, k.gravity[(c < 1 ? 0 : c - 1) % DIM], x);
      }
      if (c == 0) x = fma(-jx, av[kk], x);
      out(1 + kk, 0, c) = x;
    }
    // H_kl
    fu = fma(jlam, av[kk], fu);
#pragma unroll
    for (int ll = 0; ll < DIM; ++ll) {
      const double gg = W(R::GG + (kk <= ll ? gg_at(DIM, kk, ll) : gg_at(DIM, ll, kk)));
      const double p1 = jmu * av[ll];
      double xp = fe * s[ll];
#pragma unroll
      for (int d = 0; d < DIM; ++d) xp = fma(fv[d], g[ll][d], xp);
#pragma unroll
      for (int c = 0; c < ND; ++c) {
        double x = c == 0 ? fma(s[ll], FD[c], xp) : s[ll] * FD[c];
        x = fma(gg, KD[c], x);
        if (c >= 1 && c < iT) {
          x = fma(fu, g[ll][(c < 1 ? 0 : c - 1) % DIM], x);
          x = fma(p1, g[kk][(c < 1 ? 0 : c - 1) % DIM], x);
        }
        out(1 + kk, 1 + ll, c) = x;
      }
    }
  }
  // H_00, and the energy row's H_0l: FPT_0 = -rho t_g
  double F0[ND];
#pragma unroll
  for (int c = 0; c < ND; ++c) F0[c] = 0.0;
  if (rE) {
    const double c0 = -rho * W(R::EG);
    double fv[DIM];
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      const int ci = R::col_r0(c);
      if (ci >= 0) F0[c] = c0 * r0[ci < 0 ? 0 : ci];
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      fv[d] = (-rho * k.gravity[d]) * jm[d];
      F0[1 + d] = rho * fv[d];
    }
#pragma unroll
    for (int ll = 0; ll < DIM; ++ll) {
      double xp = fv[0] * g[ll][0];
#pragma unroll
      for (int d = 1; d < DIM; ++d) xp = fma(fv[d], g[ll][d], xp);
#pragma unroll
      for (int c = 0; c < ND; ++c) {
        double x = c == 0 ? fma(s[ll], F0[c], xp) : s[ll] * F0[c];
        if (c >= 1 && c < iT) x = fma(c0 * jr, g[ll][(c < 1 ? 0 : c - 1) % DIM], x);
        out(0, 1 + ll, c) = x;
      }
    }
  }
#pragma unroll
  for (int c = 0; c < ND; ++c) {
    double x = k.inv_dt * (DR[c] + F0[c]);
    if (c >= 1 && c < iT && rE) x = fma(-jr, k.gravity[(c < 1 ? 0 : c - 1) % DIM], x);
    out(0, 0, c) = x;
  }
}

template <int DIM, int NC>
__global__ void __launch_bounds__(Tensor64<DIM, NC>::THREADS)
    tensor64_kernel(const KParams k, double* in, long long first, long long n) {
  using T = Tensor64<DIM, NC>;
  using R = typename T::R;
  constexpr int NEN = T::NEN, NQ = T::NQ, ND = T::ND, N = R::N, EB = R::EB, iT = Layout<DIM, NC>::iT;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  typename T::Smem& S = *reinterpret_cast<typename T::Smem*>(smem_raw);
  const int tid = threadIdx.x;
  const long long li = blockIdx.x;
  const long long e = k.el_list ? (long long)k.el_list[first + li] : first + li;
  const int l = (int)(li % EB);
  const double* blk = in + (size_t)(li / EB) * R::EW * EB;
  const int32_t* di = reinterpret_cast<const int32_t*>(blk + (size_t)R::INTS * EB);
  for (int t = tid; t < NEN * NEN; t += T::THREADS) S.off[t / NEN][t % NEN] = di[(R::I_OFF + t) * EB + l];
  if (tid < NEN) {
    S.rowlen[tid] = di[(R::I_ROWLEN + tid) * EB + l];
    S.node[tid] = di[(R::I_NODE + tid) * EB + l];
    S.blocked[tid] = (uint32_t)di[(R::I_BLOCKED + tid) * EB + l];
  }
  const bool local = k.local_r != nullptr, vjp = k.vjp_lam != nullptr;
  const int mode = k.scatter_mode;
  if (tid < T::T1) tensor_point64<DIM, NC>(k, blk, l, tid / ND, tid % ND, S.H);
  __syncthreads();
  // rhs: a thread per (node, row)
  if (!vjp && tid < N) {
    const int b = tid / ND, rr = tid - b * ND;
    const ElemGeo<DIM, NEN>* geo = reinterpret_cast<const ElemGeo<DIM, NEN>*>(k.geo) + e * NQ;
    double x = 0.0;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      auto W = [&](int f) -> double { return blk[(size_t)(q * R::RW + f) * EB + l]; };
      x = fma(k.sh_tab[q][b], W(R::RV + rr), x);
#pragma unroll
      for (int d = 0; d < DIM; ++d) x = fma(geo[q].ds[d][b], W(R::PHI + d * ND + rr), x);
    }
    if (local) k.local_r[(first + li) * N + tid] = -x;
    else if (!((S.blocked[b] >> rr) & 1u)) add_to(k.rhs + (long long)S.node[b] * ND + rr, -x, mode);
  }
  if (local && !k.local_m) return;
  const bool active = tid < T::T2;
  const int r = active ? tid / ND : 0, c = active ? tid - r * ND : 0;
  const int at = r * T::RS + c;
  // the H_0l are there on the energy row alone
  const bool src = r == iT;
  const bool any_src = __any_sync(0xffffffffu, src);
  // one-dimensional shape functions at the lower point: near and far node (the upper point's are
  // mirrored); derivatives -1/2, 1/2
  double nA, nB;
  if constexpr (DIM == 2) {
    nA = k.sh_tab[0][0] + k.sh_tab[0][3];
    nB = k.sh_tab[0][1] + k.sh_tab[0][2];
  } else {
    nA = (k.sh_tab[0][0] + k.sh_tab[0][3]) + (k.sh_tab[0][4] + k.sh_tab[0][7]);
    nB = (k.sh_tab[0][1] + k.sh_tab[0][2]) + (k.sh_tab[0][5] + k.sh_tab[0][6]);
  }
  auto n1 = [&](int a, int q) { return a == q ? nA : nB; };
  double tr = 0.0, vacc[NEN];
#pragma unroll
  for (int a = 0; a < NEN; ++a) vacc[a] = 0.0;
  auto sink = [&](int b, int a, double x) {
    if (a == b && r == c) tr += x;
    if (vjp) {
      const bool off = (S.blocked[b] >> r) & 1u;
      const double lam = off ? 0.0 : __ldg(k.vjp_lam + (long long)S.node[b] * ND + r);
#pragma unroll
      for (int q = 0; q < NEN; ++q) vacc[q] = q == a ? fma(lam, x, vacc[q]) : vacc[q];
      return;
    }
    if (!active) return;
    if (local) {
      k.local_m[(first + li) * (long long)(N * N) + (b * ND + r) * N + a * ND + c] = x;
      return;
    }
    if ((S.blocked[b] >> r) & 1u) return;
    if (x != 0.0) add_to(k.vals + (int64_t)S.off[b][a] * ND + (int64_t)r * S.rowlen[b] + c, x, mode);
  };
  // V[qy][qx][i][j], i, j in {0, xi, eta}: the plane's matrices after the contraction over zeta
  // for the pair (bz, az)
  auto plane = [&](int bz, int az) {
    double V[2][2][3][3];
#pragma unroll
    for (int qy = 0; qy < 2; ++qy)
#pragma unroll
      for (int qx = 0; qx < 2; ++qx) {
        if constexpr (DIM == 2) {
          const int q = T::corner(qx, qy, 0);
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) V[qy][qx][i][j] = (i > 0 || j == 0 || src) ? S.H[i * T::NF + j][q][at] : 0.0;
        } else {
          const int q0 = T::corner(qx, qy, 0), q1 = T::corner(qx, qy, 1);
          const double b0 = n1(bz, 0), b1 = n1(bz, 1), a0 = n1(az, 0), a1 = n1(az, 1);
          const double w0 = b0 * a0, w1 = b1 * a1;
          const double db = bz ? 0.5 : -0.5, da = az ? 0.5 : -0.5;
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              if (i == 0 && j > 0) continue;
              V[qy][qx][i][j] = fma(w1, S.H[i * T::NF + j][q1][at], w0 * S.H[i * T::NF + j][q0][at]);
            }
#pragma unroll
          for (int j = 0; j < 3; ++j) {   // zeta derivative of the test function
            const double x = fma(db * a1, S.H[3 * T::NF + j][q1][at], (db * a0) * S.H[3 * T::NF + j][q0][at]);
            if (j == 0) V[qy][qx][0][0] += x;
            else V[qy][qx][0][j] = x;
          }
#pragma unroll
          for (int i = 1; i < 3; ++i)     // of the trial function
            V[qy][qx][i][0] = fma(da * b1, S.H[i * T::NF + 3][q1][at],
                                  fma(da * b0, S.H[i * T::NF + 3][q0][at], V[qy][qx][i][0]));
          V[qy][qx][0][0] = fma(db * da, S.H[15][q0][at] + S.H[15][q1][at], V[qy][qx][0][0]);
          if (any_src) {
            // lanes of other rows read words that no thread writes: selected away
#pragma unroll
            for (int j = 1; j < 3; ++j) {
              const double h0 = src ? S.H[j][q0][at] : 0.0, h1 = src ? S.H[j][q1][at] : 0.0;
              V[qy][qx][0][j] = fma(w1, h1, fma(w0, h0, V[qy][qx][0][j]));
            }
            const double h0 = src ? S.H[3][q0][at] : 0.0, h1 = src ? S.H[3][q1][at] : 0.0;
            V[qy][qx][0][0] = fma(da * b1, h1, fma(da * b0, h0, V[qy][qx][0][0]));
          }
        }
      }
#pragma unroll 1
    for (int yp = 0; yp < 4; ++yp) {
      const int by = yp >> 1, ay = yp & 1;
      const double b0 = n1(by, 0), b1 = n1(by, 1), a0 = n1(ay, 0), a1 = n1(ay, 1);
      const double w0 = b0 * a0, w1 = b1 * a1;
      const double db = by ? 0.5 : -0.5, da = ay ? 0.5 : -0.5, dd = db * da;
      double U[2][4];   // per qx: 00, x0, 0x, xx
#pragma unroll
      for (int qx = 0; qx < 2; ++qx) {
        const double (&A)[3][3] = V[0][qx], (&B)[3][3] = V[1][qx];
        double x = fma(w1, B[0][0], w0 * A[0][0]);
        x = fma(db * a1, B[2][0], fma(db * a0, A[2][0], x));
        x = fma(da * b1, B[0][2], fma(da * b0, A[0][2], x));
        U[qx][0] = fma(dd, A[2][2] + B[2][2], x);
        x = fma(w1, B[1][0], w0 * A[1][0]);
        U[qx][1] = fma(da * b1, B[1][2], fma(da * b0, A[1][2], x));
        x = fma(w1, B[0][1], w0 * A[0][1]);
        U[qx][2] = fma(db * a1, B[2][1], fma(db * a0, A[2][1], x));
        U[qx][3] = fma(w1, B[1][1], w0 * A[1][1]);
      }
      const double xx = 0.25 * (U[0][3] + U[1][3]);
#pragma unroll
      for (int bx = 0; bx < 2; ++bx)
#pragma unroll
        for (int ax = 0; ax < 2; ++ax) {
          const double hb = bx ? 0.5 : -0.5, ha = ax ? 0.5 : -0.5;
          double x = bx == ax ? xx : -xx;
          x = fma(n1(bx, 1) * n1(ax, 1), U[1][0], fma(n1(bx, 0) * n1(ax, 0), U[0][0], x));
          x = fma(hb * n1(ax, 1), U[1][1], fma(hb * n1(ax, 0), U[0][1], x));
          x = fma(ha * n1(bx, 1), U[1][2], fma(ha * n1(bx, 0), U[0][2], x));
          sink(T::corner(bx, by, bz), T::corner(ax, ay, az), x);
        }
    }
  };
  if constexpr (DIM == 2) {
    plane(0, 0);
  } else {
#pragma unroll 1
    for (int zp = 0; zp < 4; ++zp) plane(zp >> 1, zp & 1);
  }
  if (local) return;
  if (active && r == c) in[((size_t)(li / EB) * R::EW + R::TR + r) * EB + l] = tr;
  if (vjp && active) {
#pragma unroll
    for (int a = 0; a < NEN; ++a)
      if (vacc[a] != 0.0) atomicAdd(k.vjp_g + (long long)S.node[a] * ND + c, vacc[a]);
  }
}

// Diagonal of the blocked rows (Dirichlet): avg = (1 + trace)/n of the element block
// (scatter.hpp:62-78), from the rows' shares of the trace in row order.
template <int DIM, int NEN, int NC>
__global__ void __launch_bounds__(128) dirichlet64_kernel(const KParams k, const double* __restrict__ in, long long n) {
  using R = Rec64<DIM, NEN, NC>;
  constexpr int ND = R::ND, EB = R::EB;
  const long long li = (long long)blockIdx.x * 128 + threadIdx.x;
  if (li >= n) return;
  const int l = (int)(li % EB);
  const double* blk = in + (size_t)(li / EB) * R::EW * EB;
  const int32_t* di = reinterpret_cast<const int32_t*>(blk + (size_t)R::INTS * EB);
  uint32_t any = 0u;
#pragma unroll
  for (int b = 0; b < NEN; ++b) any |= (uint32_t)di[(R::I_BLOCKED + b) * EB + l];
  if (any == 0u) return;
  double tr = 0.0;
#pragma unroll
  for (int r = 0; r < ND; ++r) tr += blk[(size_t)(R::TR + r) * EB + l];
  const double avg = (1.0 + tr) * (1.0 / R::N);
  for (int b = 0; b < NEN; ++b) {
    const uint32_t bl = (uint32_t)di[(R::I_BLOCKED + b) * EB + l];
    for (int r = 0; r < ND; ++r) {
      if (!((bl >> r) & 1u)) continue;
      if (k.vjp_lam) {
        const long long dof = (long long)di[(R::I_NODE + b) * EB + l] * ND + r;
        atomicAdd(k.vjp_g + dof, __ldg(k.vjp_lam + dof) * avg);
      } else {
        add_to(k.vals + (int64_t)di[(R::I_OFF + b * NEN + b) * EB + l] * ND + (int64_t)r * di[(R::I_ROWLEN + b) * EB + l] + r,
               avg, k.scatter_mode);
      }
    }
  }
}

}  // namespace gales
