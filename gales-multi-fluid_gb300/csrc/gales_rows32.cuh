// Matrix stage of the mixed form: the FP32 element blocks from the point records of
// gales_kernels.cuh's point stage.
//
// Row (b, r) of the element block (test node b, dof r) is built per quadrature point
// (fluid_2d.hpp:264-331) from
//   JxW [ FPT_b RM_a + N_a X_b ]   with
//   WA_b  = sum_k dN_b/dx_k A_k
//   FPT_b = (WA_b - N_b S0) tau                       least-squares weight
//   RM_a  = N_a DUDY/dt + WA_a - N_a S0               least-squares operator
//   X_b   = N_b (DUDY/dt - S0) - WA_b                 Galerkin mass, source, advection
// plus the viscous/diffusive and dc terms sum_kl dN_b/dx_k K'_kl dN_a/dx_l with
// K'_kl = K_kl + nu d_kl DUDY.
// None of the nd x nd matrices is formed.  DUDY = w r0^T + rho M (w = (1, v, E, Y),
// r0 its first row, M zero but for the velocity and mass-fraction diagonal and the
// energy row mE), A_k = v_k DUDY + u' e_{v_k}^T + (e_{v_k} + v_k e_E) e_p^T with
// u' = U + p e_E, and S0 = e_E sigma^T with sigma = rho g on the velocity columns
// (fluid_2d.hpp:407-575).  With s_b = dN_b/dx . v these give, for row r,
//   FPT_b[r]   = s_b (w_r z + rho Mtau[r]) + u'_r t_b + kappa_br tau[0] - N_b [r=E] rho t_g
//   (FPT_b RM_a)[r] = alpha_a (FPT_b DUDY)[r] + (FPT_b[r].u') gamma_a
//                     + (FPT_b[r].kappa_a) e_p - N_a FPT_b[r][E] sigma
//   X_b[r]     = beta_b DUDY[r] - u'_r gamma_b - kappa_br e_p - N_b [r=E] sigma
// where z = r0^T tau, Mtau = M tau, t_b = sum_k dN_b/dx_k tau[v_k], t_g = sum_k g_k
// tau[v_k], gamma_a = dN_a/dx on the velocity columns, kappa_a = dN_a/dx on the
// velocity rows + s_a e_E, alpha_a = N_a/dt + s_a, beta_b = N_b/dt - s_b.  K'_kl is
// applied in closed form from a few point scalars (mu, lambda, mu v, lambda v, kappa,
// rho D_i, rho D_i H_i) and nu DUDY: per point for non-affine elements, once from
// JxW-weighted sums for simplices (their shape gradients do not depend on the point).
//
// Mapping.  A warp takes row (b, r) of the 32 elements of a block of records, a lane per
// element; the NEN warps of a CTA take the test nodes b of one dof row r.  So r is known at
// compile time: the terms that a row does not have (r0 on velocity columns, M, kappa, t_g, the
// structural zeros of tau and K') are never issued, every lane works, and a record word is one
// conflict-free load.  The words that a row needs of a point lie together in the record; two
// bulk copies bring them into one of two buffers in shared memory while the CTA works on the
// other point.  CTAs of one row r of kRows32Group blocks run side by side: with all rows of a
// block side by side the code of eight rows would not stay in the instruction cache.
// Bound: instruction issue (2.6 of 4 per cycle, 57% of them FP32 arithmetic before its
// multiply-adds over the columns were paired, see fma2; ncu on 64,000 hexahedra with 6 dofs).
// Whole pass of 1.0M tets with 7 dofs: 6.11 ms, 6.21 without the pairs; of half a million
// hexahedra with 8: 14.4 and 15.1.  The rows alone, without the pairs: 2.61 and 8.70 ms; a lane
// per (element, row), with r and b known at run time only and t_b formed in shared memory by an
// extra pass, took 3.73 and 13.6; this mapping with the words loaded where they are used,
// without the bulk copies, 3.26 and 10.9.  Five CTAs of 4 warps a multiprocessor, two of 8: 2.58
// and 2.78 ms with six and four CTAs of tets, 12.3 with three of hexahedra.
#pragma once

#include "gales_kernels.cuh"

namespace gales {

// Structural zeros of tau[1 + d]: column p and the diagonal.
template <int DIM>
__device__ __forceinline__ float tb_entry(const float* gb, const float* t_p, const float* t_d, int j) {
  if (j == 0) {
    float x = __fmul_rn(gb[0], t_p[0]);
#pragma unroll
    for (int d = 1; d < DIM; ++d) x = fmaf(gb[d], t_p[d], x);
    return x;
  }
  return __fmul_rn(gb[(j - 1) % DIM], t_d[(j - 1) % DIM]);
}

// Bulk copies of point records into shared memory with transaction barriers
// (cp.async.bulk and mbarrier, sm_90+).  Every wait is bounded.
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// orders earlier accesses to shared memory before later bulk copies into it
__device__ __forceinline__ void bulk_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void bulk_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0u;
}
// Bounded wait on phase `parity` of a transaction barrier: false after kMbarTries
// polls (each poll may suspend the thread for a while), far beyond any bulk copy.
constexpr long long kMbarTries = 1ll << 24;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (long long i = 0; i < kMbarTries; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

constexpr unsigned kRows32Group = 608;   // blocks whose rows are taken dof by dof

// Point scalars entering K'_kl (JxW-weighted, summed over the points of a simplex).
template <int DIM, int NC, typename S>
struct KSums {
  using L = Layout<DIM, NC>;
  S mu, lambda, kappa, muv[DIM], lamv[DIM], rhoD[L::NYA], rhoDH[L::NYA];
};

// Two binary32 operations in one instruction (fma.rn.f32x2 and its kin): each half rounds like
// the single operation, and the pair takes one issue slot.
__device__ __forceinline__ void fma2(float& x0, float& x1, float s, float y0, float y1) {   // x += s y
  asm("{ .reg .b64 a, b, c;\n mov.b64 a, {%2, %2};\n mov.b64 b, {%3, %4};\n mov.b64 c, {%0, %1};\n"
      " fma.rn.f32x2 c, a, b, c;\n mov.b64 {%0, %1}, c; }"
      : "+f"(x0), "+f"(x1)
      : "f"(s), "f"(y0), "f"(y1));
}
__device__ __forceinline__ void mul2(float& x0, float& x1, float s, float y0, float y1) {   // x = s y
  asm("{ .reg .b64 a, b;\n mov.b64 a, {%2, %2};\n mov.b64 b, {%3, %4};\n mul.rn.f32x2 a, a, b;\n mov.b64 {%0, %1}, a; }"
      : "=f"(x0), "=f"(x1)
      : "f"(s), "f"(y0), "f"(y1));
}
__device__ __forceinline__ void add2(float& x0, float& x1, float y0, float y1) {   // x += y
  asm("{ .reg .b64 a, b;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %3};\n add.rn.f32x2 a, a, b;\n mov.b64 {%0, %1}, a; }"
      : "+f"(x0), "+f"(x1)
      : "f"(y0), "f"(y1));
}
// x[j] += s y[j] over the columns that sel names, in the pairs (v1 v2), (v3 p), (T Y1), ... of 3D
// or (v1 v2), (p T), (Y1 Y2), ... of 2D.
template <int DIM, int ND, typename Sel>
__device__ __forceinline__ void row_axpy(float (&x)[ND], float s, const float (&y)[ND], Sel sel) {
  auto col = [](int i) { return i <= DIM ? (i + 1) % (DIM + 1) : i; };
#pragma unroll
  for (int i = 0; i < ND; i += 2) {
    const int j0 = col(i), j1 = i + 1 < ND ? col(i + 1) : j0;
    if (j1 != j0 && sel(j0) && sel(j1)) {
      fma2(x[j0], x[j1], s, y[j0], y[j1]);
    } else {
      if (sel(j0)) x[j0] = fmaf(s, y[j0], x[j0]);
      if (j1 != j0 && sel(j1)) x[j1] = fmaf(s, y[j1], x[j1]);
    }
  }
}

// Adds sum_kl gb_k K_kl(ROW, :) ga_l to a row of one (b, a) block (the closed form of
// the contraction; fluid_2d.hpp:531-571):
//   velocity row v_j: mu gb_m ga_j + lambda gb_j ga_m + mu (gb.ga) d_mj  on column v_m
//   energy row      : mu v_m (gb.ga) + gb_m (ga.mu v) + ga_m (gb.lambda v) on v_m,
//                     kappa (gb.ga) on T, rho D_i H_i (gb.ga) on Y_i
//   mass-fraction row Y_i: rho D_i (gb.ga) on Y_i.
template <int DIM, int NC, int ROW>
__device__ __forceinline__ void viscous_row32(float (&acc)[Layout<DIM, NC>::ND], const KSums<DIM, NC, float>& ks,
                                              const float* gb, const float* ga) {
  using L = Layout<DIM, NC>;
  constexpr bool cE = ROW == L::iT, cV = ROW >= 1 && ROW < L::iT, cY = ROW >= L::iY;
  constexpr int J = cV ? ROW - 1 : 0, IY = cY ? ROW - L::iY : 0;
  if constexpr (ROW == 0) return;
  float gg = __fmul_rn(gb[0], ga[0]);
#pragma unroll
  for (int d = 1; d < DIM; ++d) gg = fmaf(gb[d], ga[d], gg);
  if constexpr (cV || cE) {
    float p1, p2;
    if constexpr (cV) {
      p1 = __fmul_rn(ks.mu, ga[J]);
      p2 = __fmul_rn(ks.lambda, gb[J]);
    } else {
      p1 = __fmul_rn(ga[0], ks.muv[0]);
      p2 = __fmul_rn(gb[0], ks.lamv[0]);
#pragma unroll
      for (int d = 1; d < DIM; ++d) {
        p1 = fmaf(ga[d], ks.muv[d], p1);
        p2 = fmaf(gb[d], ks.lamv[d], p2);
      }
    }
    float x[DIM];
    mul2(x[0], x[1], p2, ga[0], ga[1]);
    fma2(x[0], x[1], p1, gb[0], gb[1]);
    if constexpr (cE) fma2(x[0], x[1], gg, ks.muv[0], ks.muv[1]);
    if constexpr (DIM == 3) {
      x[2 % DIM] = fmaf(gb[2 % DIM], p1, __fmul_rn(ga[2 % DIM], p2));
      if constexpr (cE) x[2 % DIM] = fmaf(ks.muv[2 % DIM], gg, x[2 % DIM]);
    }
    if constexpr (cV) x[J] = __fadd_rn(x[J], __fmul_rn(ks.mu, gg));
    add2(acc[1], acc[2], x[0], x[1]);
    if constexpr (DIM == 3) acc[3] = __fadd_rn(acc[3], x[2 % DIM]);
  }
  if constexpr (cE) {
    constexpr int ND = L::ND;
    float y[ND];
    y[L::iT] = ks.kappa;
#pragma unroll
    for (int i = 0; i < NC - 1; ++i) y[L::iY + i] = ks.rhoDH[i];
    row_axpy<DIM, ND>(acc, gg, y, [](int j) { return j >= L::iT; });
  }
  if constexpr (cY) acc[ROW] = fmaf(ks.rhoD[IY], gg, acc[ROW]);
}

// The words of a point record that a row reads: LEN words from FIRST on, then row[r].
template <int DIM, int NEN, int NC, bool WANT_M>
struct RowWords {
  using S = float;
  using L = Layout<DIM, NC>;
  using QPT = QP<DIM, NEN, NC, S>;
  static constexpr int FIRST = WANT_M ? GALES_W(mu) : GALES_W(rho);
  static constexpr int MAX = GALES_W(row) - FIRST + QPT::RP;
  __host__ __device__ static constexpr int len(int r) {
    return (r == L::iT ? GALES_W(row) : r >= 1 && r < L::iT ? GALES_W(y) : GALES_W(tau0)) - FIRST;
  }
};

// The two bulk copies of one point's words (a buffer of RowWords::MAX lines of 32 floats).
template <int DIM, int NEN, int NC, bool WANT_M>
__device__ __forceinline__ void load_point32(float* dst, const float* rec, int r, uint64_t* bar) {
  using S = float;
  using QPT = QP<DIM, NEN, NC, S>;
  using W = RowWords<DIM, NEN, NC, WANT_M>;
  const uint32_t len = (uint32_t)W::len(r) * 128u, rp = (uint32_t)QPT::RP * 128u;
  bulk_expect(bar, len + rp);
  bulk_copy(dst, rec + W::FIRST * 32, len, bar);
  bulk_copy(dst + W::len(r) * 32, rec + (GALES_W(row) + r * QPT::RP) * 32, rp, bar);
}

// One element's row (b, ROW): acc[a][c] (WANT_M) and the residual row.  blk: word 0 of point 0
// of the CTA's block of elements; buf: two buffers of a point's words, bar: their transaction
// barriers.  False if a copy did not arrive (see mbar_wait).
template <int DIM, int NEN, int NC, int ROW, bool WANT_M>
__device__ __forceinline__ bool row32(const KParams& k, const float* __restrict__ blk, int b, float* buf, uint64_t* bar,
                                      float (&acc)[NEN][Layout<DIM, NC>::ND], float& racc) {
  using L = Layout<DIM, NC>;
  using S = float;
  using QPT = QP<DIM, NEN, NC, S>;
  using RB = RecBlock<DIM, NEN, NC>;
  using W = RowWords<DIM, NEN, NC, WANT_M>;
  constexpr int ND = L::ND, NQ = NEN, iT = L::iT, iY = L::iY;
  constexpr bool AFF = NEN == DIM + 1;
  constexpr bool cE = ROW == iT, cV = ROW >= 1 && ROW < iT, cY = ROW >= iY, cP = ROW == 0;
  constexpr int J = cV ? ROW - 1 : 0, IY = cY ? ROW - iY : 0;
  auto isV = [](int j) { return j >= 1 && j < iT; };
  // DUDY[r] can be nonzero at column j
  auto dnz = [&](int j) { return cE || !isV(j) || j == ROW; };
  const int lane = threadIdx.x & 31;
  const float idt = k.inv_dt_f;
#pragma unroll
  for (int a = 0; a < NEN; ++a)
#pragma unroll
    for (int j = 0; j < ND; ++j) acc[a][j] = 0.f;
  racc = 0.f;
  float Dnu[ND];
  KSums<DIM, NC, float> ksum;
  if constexpr (AFF) {
#pragma unroll
    for (int j = 0; j < ND; ++j) Dnu[j] = 0.f;
    ksum.mu = ksum.lambda = ksum.kappa = 0.f;
#pragma unroll
    for (int d = 0; d < DIM; ++d) ksum.muv[d] = ksum.lamv[d] = 0.f;
#pragma unroll
    for (int y = 0; y < L::NYA; ++y) ksum.rhoD[y] = ksum.rhoDH[y] = 0.f;
  }
  // shape gradients of a simplex: the same at every point
  float gaf[AFF ? NEN : 1][DIM], gb[DIM];
  if constexpr (AFF) {
#pragma unroll
    for (int a = 0; a < NEN; ++a)
#pragma unroll
      for (int d = 0; d < DIM; ++d) gaf[a][d] = __ldg(blk + (GALES_W(dse) + d * NEN + a) * RB::EB + lane);
#pragma unroll
    for (int d = 0; d < DIM; ++d) gb[d] = __ldg(blk + (GALES_W(dse) + d * NEN + b) * RB::EB + lane);
  }
#pragma unroll 1
  for (int q = 0; q < NQ; ++q) {
    float* pt = buf + (q & 1) * (W::MAX * 32);
    const bool ok = mbar_wait(&bar[q & 1], (uint32_t)(q >> 1) & 1u);
    auto c = [&](int f) -> float { return pt[(f - W::FIRST) * 32 + lane]; };
    auto row = [&](int f) -> float { return pt[(W::len(ROW) + f) * 32 + lane]; };
    const float rho = c(GALES_W(rho)), p = c(GALES_W(p)), jx = c(GALES_W(JxW));
    float vq[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      if constexpr (!AFF) gb[d] = c(GALES_W(ds) + d * NEN + b);
      vq[d] = c(GALES_W(v) + d);
    }
    // w[j]
    auto w = [&](int j) -> float { return j == 0 ? 1.f : isV(j) ? vq[(j - 1) % DIM] : c(j == iT ? GALES_W(E) : GALES_W(Y) + (j - iY)); };
    const float Nb = k.sh_tab_f[q][b];
    float sb = __fmul_rn(gb[0], vq[0]);
#pragma unroll
    for (int d = 1; d < DIM; ++d) sb = fmaf(gb[d], vq[d], sb);
    const float wr = w(ROW);
    const float ur = cE ? fmaf(rho, wr, p) : (cP ? rho : __fmul_rn(rho, wr));
    const float kap = cE ? sb : (cV ? gb[J] : 0.f);
    // row r of FPT_b
    const float cz = cP ? sb : __fmul_rn(sb, wr), cm = __fmul_rn(sb, rho), cg = -__fmul_rn(Nb, rho);
    float t_p[DIM], t_d[DIM], F[ND];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      t_p[d] = c(GALES_W(tvp) + d);
      t_d[d] = c(GALES_W(tvd) + d);
    }
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      float x = __fmul_rn(cz, c(GALES_W(z) + j));
      if (cE) x = fmaf(cm, c(GALES_W(y) + j), x);
      if ((cV || cY) && (j == 0 || j == ROW))
        x = fmaf(cm, cV ? (j == 0 ? t_p[J] : t_d[J]) : row(DIM + 1 + (j == 0 ? 0 : 1)), x);
      if (j < iT) x = fmaf(ur, tb_entry<DIM>(gb, t_p, t_d, j), x);
      if (cV || cE) x = fmaf(kap, c(GALES_W(tau0) + j), x);
      if (cE && j < iT) x = fmaf(cg, c(GALES_W(tg) + j), x);
      F[j] = x;
    }
    // residual row: N_b rv + sum_k dN_b/dx_k rf_k + FPT_b Res (fluid_2d.hpp:253-262, 280-290)
    {
      float x = __fmul_rn(Nb, row(0));
#pragma unroll
      for (int d = 0; d < DIM; ++d) x = fmaf(gb[d], row(1 + d), x);
#pragma unroll
      for (int j = 0; j < ND; ++j) x = fmaf(F[j], c(GALES_W(res) + j), x);
      racc = fmaf(jx, x, racc);
    }
    if constexpr (WANT_M) {
      // FPT_b DUDY, DUDY row r, and the a-independent velocity-column terms
      float fw = F[0];
#pragma unroll
      for (int j = 1; j < ND; ++j) fw = fmaf(F[j], w(j), fw);
      const float fu = fmaf(rho, fw, __fmul_rn(p, F[iT]));
      const float rF = __fmul_rn(rho, F[iT]);
      float FD[ND], Dr[ND];
#pragma unroll
      for (int j = 0; j < ND; ++j) {
        float mEj;
        if (j == 0) mEj = c(GALES_W(de_dp));
        else if (j < iT) mEj = vq[(j - 1) % DIM];
        else if (j == iT) mEj = c(GALES_W(de_dT));
        else mEj = c(GALES_W(dE_dY) + (j - iY));
        float x = (j >= 1 && j != iT) ? fmaf(rF, mEj, __fmul_rn(rho, F[j])) : __fmul_rn(rF, mEj);
        float dd = cE ? __fmul_rn(rho, mEj) : ((cV || cY) && j == ROW ? rho : 0.f);
        if (!isV(j)) {
          const float r0j = j == 0 ? c(GALES_W(drho_dp)) : (j == iT ? c(GALES_W(drho_dT)) : c(GALES_W(drho_dY) + (j - iY)));
          x = fmaf(fw, r0j, x);
          if (cE || (cY && j == ROW)) dd = fmaf(wr, r0j, dd);
          else dd = cP ? r0j : __fmul_rn(wr, r0j);
        }
        FD[j] = x;
        Dr[j] = dd;
      }
      float hv[ND];   // velocity columns
      const float fe = cE ? __fmul_rn(rho, __fadd_rn(F[iT], Nb)) : rF;
#pragma unroll
      for (int d = 0; d < DIM; ++d) hv[1 + d] = -fmaf(ur, gb[d], __fmul_rn(fe, k.gravity_f[d]));
      const float beta = fmaf(Nb, idt, -sb);
      KSums<DIM, NC, float> ks;
      float nu_j = 0.f;
      if constexpr (!AFF) {
        ks.mu = __fmul_rn(jx, c(GALES_W(mu)));
        ks.lambda = __fmul_rn(jx, c(GALES_W(lambda)));
        ks.kappa = __fmul_rn(jx, c(GALES_W(kappa)));
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          ks.muv[d] = __fmul_rn(ks.mu, vq[d]);
          ks.lamv[d] = __fmul_rn(ks.lambda, vq[d]);
        }
#pragma unroll
        for (int y = 0; y < L::NYA; ++y) {
          ks.rhoD[y] = __fmul_rn(jx, c(GALES_W(rhoD) + y));
          ks.rhoDH[y] = __fmul_rn(jx, c(GALES_W(rhoDH) + y));
        }
        nu_j = __fmul_rn(jx, c(GALES_W(nu)));
      }
      const float A3 = __fmul_rn(jx, fu);
#pragma unroll
      for (int a = 0; a < NEN; ++a) {
        float ga[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) ga[d] = AFF ? gaf[AFF ? a : 0][d] : c(GALES_W(ds) + d * NEN + a);
        const float Na = k.sh_tab_f[q][a];
        float sa = __fmul_rn(ga[0], vq[0]);
#pragma unroll
        for (int d = 1; d < DIM; ++d) sa = fmaf(ga[d], vq[d], sa);
        float fk = __fmul_rn(sa, F[iT]);
#pragma unroll
        for (int d = 0; d < DIM; ++d) fk = fmaf(ga[d], F[1 + d], fk);
        const float A1 = __fmul_rn(jx, fmaf(Na, idt, sa)), A4 = __fmul_rn(jx, Na), A2 = __fmul_rn(A4, beta);
        const float f0 = (cV || cE) ? fmaf(-Na, kap, fk) : fk;
        acc[a][0] = fmaf(jx, f0, acc[a][0]);
        float gv[ND];
#pragma unroll
        for (int d = 0; d < DIM; ++d) gv[1 + d] = ga[d];
        row_axpy<DIM, ND>(acc[a], A4, hv, isV);
        row_axpy<DIM, ND>(acc[a], A3, gv, isV);
        row_axpy<DIM, ND>(acc[a], A2, Dr, dnz);
        row_axpy<DIM, ND>(acc[a], A1, FD, [](int) { return true; });
        if constexpr (!AFF) {
          viscous_row32<DIM, NC, ROW>(acc[a], ks, gb, ga);
          float gg = __fmul_rn(gb[0], ga[0]);
#pragma unroll
          for (int d = 1; d < DIM; ++d) gg = fmaf(gb[d], ga[d], gg);
          const float gn = __fmul_rn(gg, nu_j);
          row_axpy<DIM, ND>(acc[a], gn, Dr, dnz);
        }
      }
      if constexpr (AFF) {
        const float jn = __fmul_rn(jx, c(GALES_W(nu)));
        row_axpy<DIM, ND>(Dnu, jn, Dr, dnz);
        if constexpr (cV || cE) {
          const float mu = c(GALES_W(mu)), lam = c(GALES_W(lambda));
          ksum.mu = fmaf(jx, mu, ksum.mu);
          ksum.lambda = fmaf(jx, lam, ksum.lambda);
          if constexpr (cE) {
            ksum.kappa = fmaf(jx, c(GALES_W(kappa)), ksum.kappa);
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
              ksum.muv[d] = fmaf(__fmul_rn(jx, mu), vq[d], ksum.muv[d]);
              ksum.lamv[d] = fmaf(__fmul_rn(jx, lam), vq[d], ksum.lamv[d]);
            }
#pragma unroll
            for (int y = 0; y < NC - 1; ++y) ksum.rhoDH[y] = fmaf(jx, c(GALES_W(rhoDH) + y), ksum.rhoDH[y]);
          }
        }
        if constexpr (cY) ksum.rhoD[IY] = fmaf(jx, c(GALES_W(rhoD) + IY), ksum.rhoD[IY]);
      }
    }
    // the buffer is free for point q + 2
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0 && q + 1 < NQ) mbar_wait(&bar[(q + 1) & 1], (uint32_t)((q + 1) >> 1) & 1u);
      return false;
    }
    if (threadIdx.x == 0 && q + 2 < NQ) {
      bulk_fence();
      load_point32<DIM, NEN, NC, WANT_M>(pt, blk + (size_t)(q + 2) * RB::RW * RB::EB, ROW, &bar[q & 1]);
    }
  }
  if constexpr (WANT_M && AFF) {
    // viscous/diffusive and dc terms of a simplex, from the point sums
#pragma unroll
    for (int a = 0; a < NEN; ++a) {
      viscous_row32<DIM, NC, ROW>(acc[a], ksum, gb, gaf[AFF ? a : 0]);
      float gg = __fmul_rn(gb[0], gaf[AFF ? a : 0][0]);
#pragma unroll
      for (int d = 1; d < DIM; ++d) gg = fmaf(gb[d], gaf[AFF ? a : 0][d], gg);
      row_axpy<DIM, ND>(acc[a], gg, Dnu, dnz);
    }
  }
  return true;
}

// A warp stages its row HN trial nodes at a time for the scatter: their entries and, per
// element, where each node's run of nd entries goes (negative: a blocked row, written by
// dirichlet32_kernel).
template <int DIM, int NEN, int NC>
struct Rows32 {
  using RB = RecBlock<DIM, NEN, NC>;
  static constexpr int ND = Layout<DIM, NC>::ND, N = NEN * ND;
  static constexpr int HN = NEN < 4 ? NEN : 4, HC = HN * ND, NS = HC | 1;
  static_assert(NEN % HN == 0 && HC <= 32, "a lane per staged column");
  static constexpr int THREADS = 32 * NEN;
  struct Stage {
    int64_t at[NEN][32 * HN];
    float st[NEN][32 * NS];
  };
  template <bool WANT_M>
  struct Smem {
    union {
      float pt[2][RowWords<DIM, NEN, NC, WANT_M>::MAX * 32];   // point records
      typename std::conditional<WANT_M, Stage, float>::type s;
    };
    uint64_t bar[2];
  };
};

template <int DIM, int NEN, int NC, bool WANT_M>
__global__ void __launch_bounds__(32 * NEN, NEN == 8 ? 2 : 5) rows32_kernel(const KParams k, unsigned char* in, long long first, long long n) {
  using T = Rows32<DIM, NEN, NC>;
  using RB = RecBlock<DIM, NEN, NC>;
  using S = float;
  using QPT = QP<DIM, NEN, NC, S>;
  constexpr int ND = T::ND, N = T::N, EB = RB::EB, NS = T::NS, HN = T::HN, HC = T::HC;
  __shared__ __align__(128) typename T::template Smem<WANT_M> sm;
  const int lane = threadIdx.x & 31, b = threadIdx.x >> 5;
  const long long nblk = (n + EB - 1) / EB;
  // CTA order: groups of kRows32Group blocks, all of a group's first rows, then its second
  const unsigned c0 = blockIdx.x / (kRows32Group * ND) * kRows32Group;
  const unsigned nc = (unsigned)nblk - c0 < kRows32Group ? (unsigned)nblk - c0 : kRows32Group;
  const unsigned u = blockIdx.x - c0 * ND;
  const int r = (int)(u / nc);
  const long long b0 = c0 + u % nc;
  const int cnt = (int)(n - b0 * EB < EB ? n - b0 * EB : EB);
  // Idle lanes of a last block take the scatter words of its last element; their record words
  // are whatever the buffer holds there, and nothing that they form is stored (below cnt alone).
  const int l = lane < cnt ? lane : cnt - 1;
  unsigned char* blk = in + (size_t)b0 * RB::BYTES;
  const float* rec = reinterpret_cast<const float*>(blk);
  if (threadIdx.x == 0) {
    mbar_init(&sm.bar[0], 1);
    mbar_init(&sm.bar[1], 1);
    mbar_fence_init();
    load_point32<DIM, NEN, NC, WANT_M>(sm.pt[0], rec, r, &sm.bar[0]);
    load_point32<DIM, NEN, NC, WANT_M>(sm.pt[1], rec + RB::RW * EB, r, &sm.bar[1]);
  }
  __syncthreads();
  // scatter descriptor words of node b (carried by point b)
  const float* desc = reinterpret_cast<const float*>(blk) + (size_t)b * RB::RW * EB;
  const int32_t node = word_int(desc[GALES_W(d_node) * EB + l]);
  const bool blocked = ((uint32_t)word_int(desc[GALES_W(d_blocked) * EB + l]) >> r) & 1u;
  const bool local = k.local_r != nullptr;
  float acc[NEN][ND], racc;
  bool ok;
  auto run = [&](auto row) { ok = row32<DIM, NEN, NC, decltype(row)::value, WANT_M>(k, rec, b, sm.pt[0], sm.bar, acc, racc); };
  static_assert(ND >= 4 && ND <= 8, "rows dispatched below");
  float diag = 0.f;
  auto put = [&](auto row) {
    run(row);
    if constexpr (WANT_M) {
#pragma unroll
      for (int a = 0; a < NEN; ++a) diag = a == b ? acc[a][decltype(row)::value] : diag;
    }
  };
  switch (r) {
    case 0: put(std::integral_constant<int, 0>()); break;
    case 1: put(std::integral_constant<int, 1>()); break;
    case 2: put(std::integral_constant<int, 2>()); break;
    case 3: put(std::integral_constant<int, 3>()); break;
    case 4: if constexpr (ND > 4) put(std::integral_constant<int, 4 < ND ? 4 : 0>()); break;
    case 5: if constexpr (ND > 5) put(std::integral_constant<int, 5 < ND ? 5 : 0>()); break;
    case 6: if constexpr (ND > 6) put(std::integral_constant<int, 6 < ND ? 6 : 0>()); break;
    default: if constexpr (ND > 7) put(std::integral_constant<int, 7 < ND ? 7 : 0>()); break;
  }
  const long long g0 = first + b0 * EB;
  if (!ok) {
    if (threadIdx.x == 0) flag_error(k, GALES_ERR_TIMEOUT, g0);
    return;
  }
  if (lane < cnt) {
    if (local) k.local_r[(g0 + lane) * N + b * ND + r] = widen(-racc);
    else if (!blocked) add_to(k.rhs + (long long)node * ND + r, widen(-racc), k.scatter_mode);
  }
  if constexpr (WANT_M) {
    if (local && !k.local_m) return;
    // this row's share of the trace (Dirichlet, see dirichlet32_kernel)
    if (lane < cnt && !local)
      reinterpret_cast<double*>(blk + RB::TR_OFF)[(size_t)(r * NEN + b) * EB + lane] = widen(diag);
    const int64_t rowoff = (int64_t)r * word_int(desc[GALES_W(d_rowlen) * EB + l]);
    float* st = sm.s.st[b];
    int64_t* at = sm.s.at[b];
    const int ca = lane < HC ? lane / ND : 0, cj = lane - ca * ND;
#pragma unroll
    for (int h = 0; h < NEN / HN; ++h) {
      __syncwarp();
#pragma unroll
      for (int i = 0; i < HN; ++i) {
#pragma unroll
        for (int j = 0; j < ND; ++j) st[lane * NS + i * ND + j] = acc[h * HN + i][j];
        at[lane * HN + i] = blocked || lane >= cnt
                                ? -1
                                : (int64_t)word_int(desc[(GALES_W(d_off) + h * HN + i) * EB + l]) * ND + rowoff;
      }
      __syncwarp();
      if (lane >= HC) continue;
      if (local) {
        double* out = k.local_m + g0 * (long long)(N * N) + (b * ND + r) * N + h * HC + lane;
        for (int el = 0; el < cnt; ++el, out += N * N) *out = widen(st[el * NS + lane]);
        continue;
      }
      // one element's row per step, consecutive lanes on consecutive columns
      double* vals = k.vals + cj;
      if (k.scatter_mode != 0) {
        // elements of one colour share no row: their adds are independent, eight in flight
#pragma unroll 1
        for (int e0 = 0; e0 < 32; e0 += 8) {
          double v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int64_t to = at[(e0 + i) * HN + ca];
            v[i] = to >= 0 ? vals[to] : 0.0;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int64_t to = at[(e0 + i) * HN + ca];
            const float x = st[(e0 + i) * NS + lane];
            if (to >= 0 && x != 0.f) vals[to] = v[i] + widen(x);
          }
        }
        continue;
      }
#pragma unroll 1
      for (int e0 = 0; e0 < 32; e0 += 4) {
        double d[4];
        bool normal = true;
#pragma unroll
        for (int i = 0; i < 4; ++i) {   // widen() without its rare branch
          const unsigned w = __float_as_uint(st[(e0 + i) * NS + lane]), m = w & 0x7fffffffu;
          normal &= m == 0u || m - 0x00800000u < 0x7f000000u;
          d[i] = __hiloint2double(m == 0u ? 0 : (int)(((m >> 3) + 0x38000000u) | (w & 0x80000000u)), (int)(w << 29));
        }
        if (!normal) {
#pragma unroll
          for (int i = 0; i < 4; ++i) d[i] = widen(st[(e0 + i) * NS + lane]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int64_t to = at[(e0 + i) * HN + ca];
          if (to >= 0 && __double2hiint(d[i]) != 0) atomicAdd(vals + to, d[i]);
        }
      }
    }
  }
}

// Diagonal of the blocked rows (Dirichlet): avg = (1 + trace)/n of the element block
// (scatter.hpp:62-78), from the rows' shares of the trace.  A CTA takes a block of elements, a
// lane each; its NEN warps sum a part of the shares and then write one node's rows.  Bound:
// latency, of three trips to L2: the masks, the shares with the descriptors, the entries of a
// coloured scatter.  A thread per element with a loop over its nodes and dofs made such a trip
// for each of them: 10 us a launch, and a coloured assembly has one for each colour (2.10 ms for
// 82,800 tets of one component with 32 colours; 1.68 now).
template <int DIM, int NEN, int NC>
__global__ void __launch_bounds__(32 * NEN) dirichlet32_kernel(const KParams k, const unsigned char* __restrict__ in, long long n) {
  using RB = RecBlock<DIM, NEN, NC>;
  using S = float;
  using QPT = QP<DIM, NEN, NC, S>;
  constexpr int ND = Layout<DIM, NC>::ND, N = NEN * ND, EB = RB::EB;
  __shared__ double part[NEN][EB];
  const int b = threadIdx.x >> 5, l = threadIdx.x & 31;
  const unsigned char* blk = in + (size_t)blockIdx.x * RB::BYTES;
  const float* desc = reinterpret_cast<const float*>(blk) + (size_t)b * RB::RW * EB + l;
  const bool on = (long long)blockIdx.x * EB + l < n;
  const uint32_t bl = on ? (uint32_t)word_int(desc[GALES_W(d_blocked) * EB]) : 0u;
  if (!__syncthreads_or(bl != 0u)) return;
  const double* tr = reinterpret_cast<const double*>(blk + RB::TR_OFF) + l;
  double s = 0.0;
  if (on)
#pragma unroll
    for (int i = 0; i < ND; ++i) s += tr[(size_t)(b * ND + i) * EB];
  part[b][l] = s;
  __syncthreads();
  if (bl == 0u) return;
  s = 1.0;
#pragma unroll
  for (int a = 0; a < NEN; ++a) s += part[a][l];
  const double avg = s * (1.0 / N);
  double* row = k.vals + (int64_t)word_int(desc[(GALES_W(d_off) + b) * EB]) * ND;
  const int64_t step = word_int(desc[GALES_W(d_rowlen) * EB]) + 1;
  double v[ND];
#pragma unroll
  for (int r = 0; r < ND; ++r) v[r] = k.scatter_mode != 0 && ((bl >> r) & 1u) ? row[r * step] : 0.0;
#pragma unroll
  for (int r = 0; r < ND; ++r) {
    if (!((bl >> r) & 1u)) continue;
    if (k.scatter_mode != 0) row[r * step] = v[r] + avg;
    else atomicAdd(row + r * step, avg);
  }
}

}  // namespace gales
