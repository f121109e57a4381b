// Linear solve of the assembled system on the GPU: flexible GMRES with a right
// ILU(k) preconditioner, the solver the reference runs after every assembly
// (belos_linear_solver::execute, src/fem/ls/belos_linear_solver_factory.hpp:103-218,
// with Ifpack "ILU" and Belos "Flexible GMRES" as sim/fluid_mc/P0/setup.txt:10-16
// selects).  It reads the CSR values the assembly leaves in device memory, so a
// Newton step needs no host copy of the matrix.
//
// Layout.  The assembled matrix has dense nd x nd blocks per pair of connected nodes
// (its scalar rows i*nd+k of node row i hold deg*nd consecutive values, node by
// node).  Scalar ILU(k) on such a pattern is block ILU(k) on the node graph: the
// scalar level of fill of an entry equals the level of its node block (paths through
// the entry's own node add a level-0 step), so the factor is stored as node blocks,
// F[pos][r][c] row-major, with the node rows' blocks sorted by column and the diagonal
// block's position kept.  The factor entries are computed with the same operations in
// the same order as row-oriented scalar elimination, so they equal it bit for bit.
//
// Parallelism.  A node row of the factor and of the forward substitution depends on
// the rows of its lower blocks, a row of the backward substitution on those of its
// upper blocks: rows are ordered by level (longest dependency chain) on the host.  The
// factorisation (a CTA per node row) and each substitution (a warp per node row) are one
// persistent launch each, which takes rows in level order and waits for single rows (see
// ilu_factor_rows_kernel, ilu_sweep_kernel; ilu_sweep_cluster_kernel where the vector fits in
// shared memory).  The preconditioner application is
// captured once into a CUDA graph whose kernels take the Krylov vector's index from
// device memory.  The Arnoldi step (two classical
// Gram-Schmidt passes) uses blocked dot products with fixed partial-sum order, so
// repeated solves are bit-identical.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/gales_asm.h"

namespace {

constexpr int kWarpsPerBlock = 8;   // node rows per CTA in the level kernels
constexpr int kSweepWarps = 10;     // warps per CTA of the sweeps, one CTA per SM
constexpr int kDotThreads = 256;

template <typename T>
struct Dev {
  T* p = nullptr;
  size_t n = 0;
  cudaError_t alloc(size_t count) {
    if (count <= n && p) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
    if (count == 0) return cudaSuccess;
    cudaError_t e = cudaMalloc(&p, count * sizeof(T));
    if (e == cudaSuccess) n = count;
    return e;
  }
  template <typename U>
  cudaError_t upload(const std::vector<U>& v) {
    cudaError_t e = alloc(v.size());
    if (e != cudaSuccess || v.empty()) return e;
    return cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
};

// ---------------------------------------------------------------------------
// Host: ILU(k) symbolic factorisation of the node graph and the level sets.
// ---------------------------------------------------------------------------

// Ifpack_IlukGraph's level-of-fill rule on node rows: row I starts with its graph
// columns at level 0; for its columns K < I in ascending order, every upper column J of
// row K gets level lev(I,K) + lev(K,J) + 1, kept when <= fill.  A linked list keeps the
// row's columns sorted while fill is inserted.
void iluk_symbolic(int64_t n, const int64_t* rp, const int32_t* col, int fill, std::vector<int64_t>& f_rp,
                   std::vector<int32_t>& f_col, std::vector<int64_t>& f_diag) {
  f_rp.assign(n + 1, 0);
  f_col.clear();
  f_diag.assign(n, -1);
  std::vector<int> f_lev;
  std::vector<int32_t> next(n + 1, -1);  // linked list; index n is the head
  std::vector<int> lev(n, INT32_MAX);
  std::vector<int32_t> touched;
  for (int64_t i = 0; i < n; ++i) {
    touched.clear();
    // graph columns (sorted) plus the diagonal
    int32_t prev = (int32_t)n;
    bool diag_in = false;
    auto push_sorted = [&](int32_t c) {
      next[prev] = c;
      next[c] = -1;
      prev = c;
    };
    next[n] = -1;
    for (int64_t p = rp[i]; p < rp[i + 1]; ++p) {
      const int32_t c = col[p];
      if (!diag_in && c > i) {
        push_sorted((int32_t)i);
        lev[i] = 0;
        touched.push_back((int32_t)i);
        diag_in = true;
      }
      if (c == i) diag_in = true;
      push_sorted(c);
      lev[c] = 0;
      touched.push_back(c);
    }
    if (!diag_in) {
      push_sorted((int32_t)i);
      lev[i] = 0;
      touched.push_back((int32_t)i);
    }
    // eliminate with the rows of the lower columns, in ascending order
    for (int32_t k = next[n]; k >= 0 && k < i; k = next[k]) {
      const int lik = lev[k];
      int32_t at = k;  // insertion cursor: columns after k are > k
      for (int64_t q = f_diag[k] + 1; q < f_rp[k + 1]; ++q) {
        const int l = lik + f_lev[q] + 1;
        if (l > fill) continue;
        const int32_t j = f_col[q];
        if (lev[j] != INT32_MAX) {
          if (l < lev[j]) lev[j] = l;
          continue;
        }
        while (next[at] >= 0 && next[at] < j) at = next[at];
        next[j] = next[at];
        next[at] = j;
        lev[j] = l;
        touched.push_back(j);
      }
    }
    for (int32_t c = next[n]; c >= 0; c = next[c]) {
      if (c == i) f_diag[i] = (int64_t)f_col.size();
      f_col.push_back(c);
      f_lev.push_back(lev[c]);
    }
    f_rp[i + 1] = (int64_t)f_col.size();
    for (int32_t c : touched) lev[c] = INT32_MAX;
  }
}

// Level sets: forward level = 1 + max over lower columns, backward = 1 + max over upper
// columns.  Rows of one level are stored contiguously (ascending) in rows[off[l]..off[l+1]).
void level_sets(int64_t n, const std::vector<int64_t>& f_rp, const std::vector<int32_t>& f_col,
                const std::vector<int64_t>& f_diag, bool forward, std::vector<int32_t>& level,
                std::vector<int64_t>& off, std::vector<int32_t>& rows) {
  level.assign(n, 0);
  int nlev = 0;
  if (forward) {
    for (int64_t i = 0; i < n; ++i) {
      int l = 0;
      for (int64_t p = f_rp[i]; p < f_diag[i]; ++p) l = std::max(l, level[f_col[p]] + 1);
      level[i] = l;
      nlev = std::max(nlev, l + 1);
    }
  } else {
    for (int64_t i = n - 1; i >= 0; --i) {
      int l = 0;
      for (int64_t p = f_diag[i] + 1; p < f_rp[i + 1]; ++p) l = std::max(l, level[f_col[p]] + 1);
      level[i] = l;
      nlev = std::max(nlev, l + 1);
    }
  }
  off.assign(nlev + 1, 0);
  for (int64_t i = 0; i < n; ++i) off[level[i] + 1]++;
  for (int l = 0; l < nlev; ++l) off[l + 1] += off[l];
  rows.assign(n, 0);
  std::vector<int64_t> fillp(off.begin(), off.end() - 1);
  for (int64_t i = 0; i < n; ++i) rows[fillp[level[i]]++] = (int32_t)i;
}

// ---------------------------------------------------------------------------
// Device kernels.
// ---------------------------------------------------------------------------

__device__ __forceinline__ int64_t find_col(const int32_t* __restrict__ c, int64_t lo, int64_t hi, int32_t j) {
  while (lo < hi) {
    const int64_t m = (lo + hi) >> 1;
    const int32_t v = c[m];
    if (v == j) return m;
    if (v < j) lo = m + 1;
    else hi = m;
  }
  return -1;
}

// Scatter the assembled values into the factor blocks (fill blocks stay zero): warp per
// node row, lanes over the row's nd x deg*nd values.
template <int ND, typename T>
__global__ void matrix_to_factor_kernel(const double* __restrict__ vals, const int64_t* __restrict__ node_rp,
                                        const int64_t* __restrict__ a2f, int64_t n_nodes, T* __restrict__ F) {
  const int64_t i = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (i >= n_nodes) return;
  const int lane = threadIdx.x & 31;
  const int64_t t0 = node_rp[i], deg = node_rp[i + 1] - t0;
  const int64_t base = t0 * ND * ND, len = deg * ND;
  for (int k = 0; k < ND; ++k) {
    for (int64_t e = lane; e < len; e += 32) {
      const int64_t t = t0 + e / ND;
      const int kk = (int)(e % ND);
      F[a2f[t] * (ND * ND) + k * ND + kk] = (T)vals[base + k * len + e];
    }
  }
}

// One level of the numeric factorisation: warp per node row I.  For its lower blocks K
// in ascending order: L_IK = A_IK U_KK^-1 (row-wise substitution, lane r < ND owns row
// r), then A_IJ -= L_IK U_KJ for the upper blocks J of row K present in row I (lanes
// over (J, r)).  Then the row-wise Doolittle step of the diagonal block, applied across
// the whole block row.  Every entry sees the subtractions of the scalar ikj order.
template <int ND, typename T>
__global__ void ilu_factor_level_kernel(T* __restrict__ F, const int64_t* __restrict__ f_rp,
                                        const int32_t* __restrict__ f_col, const int64_t* __restrict__ f_diag,
                                        const int32_t* __restrict__ rows, int64_t count,
                                        unsigned int* __restrict__ status) {
  constexpr int BB = ND * ND;
  const int64_t w = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (w >= count) return;
  const int lane = threadIdx.x & 31;
  const int32_t I = rows[w];
  const int64_t p0 = f_rp[I], p1 = f_rp[I + 1], pd = f_diag[I];
  for (int64_t p = p0; p < pd; ++p) {
    const int32_t K = f_col[p];
    const int64_t dK = f_diag[K], pK1 = f_rp[K + 1];
    T* B = F + p * BB;
    const T* UK = F + dK * BB;
    if (lane < ND) {
      T row[ND];
#pragma unroll
      for (int c = 0; c < ND; ++c) row[c] = B[lane * ND + c];
#pragma unroll
      for (int c = 0; c < ND; ++c) {
        T s = row[c];
#pragma unroll
        for (int c2 = 0; c2 < c; ++c2) s -= row[c2] * UK[c2 * ND + c];
        row[c] = s / UK[c * ND + c];
      }
#pragma unroll
      for (int c = 0; c < ND; ++c) B[lane * ND + c] = row[c];
    }
    __syncwarp();
    const int64_t items = (pK1 - dK - 1) * ND;
    for (int64_t it = lane; it < items; it += 32) {
      const int64_t q = dK + 1 + it / ND;
      const int r = (int)(it % ND);
      const int64_t pos = find_col(f_col, p + 1, p1, f_col[q]);
      if (pos < 0) continue;
      T l[ND];
#pragma unroll
      for (int m = 0; m < ND; ++m) l[m] = B[r * ND + m];
      const T* U = F + q * BB;
      T* tgt = F + pos * BB + r * ND;
#pragma unroll
      for (int c = 0; c < ND; ++c) {
        T s = tgt[c];
#pragma unroll
        for (int m = 0; m < ND; ++m) s -= l[m] * U[m * ND + c];
        tgt[c] = s;
      }
    }
    __syncwarp();
  }
  // Diagonal block and the upper blocks: rows r in order, pivots c2 < r in order.
  T* D = F + pd * BB;
  const int64_t ncols = (p1 - pd) * ND;  // columns of the block row from the diagonal block on
  for (int r = 1; r < ND; ++r) {
    for (int c2 = 0; c2 < r; ++c2) {
      const T l = D[r * ND + c2] / D[c2 * ND + c2];
      __syncwarp();
      if (lane == 0) D[r * ND + c2] = l;
      for (int64_t e = lane; e < ncols; e += 32) {
        const int64_t b = e / ND;
        const int c = (int)(e % ND);
        if (b == 0 && c <= c2) continue;
        T* Rb = F + (pd + b) * BB;
        Rb[r * ND + c] -= l * Rb[c2 * ND + c];
      }
      __syncwarp();
    }
  }
  if (lane < ND && D[lane * ND + lane] == T(0)) atomicOr(status, (unsigned)GALES_ERR_SINGULAR);
}

// Waits of the persistent kernels below.  A CTA or warp claims rows from a ticket counter
// in level order (rows[] lists them level by level) and only ever waits on rows of earlier
// levels, whose tickets were claimed before its own by CTAs or warps that are running, so
// these kernels always progress; every wait is still bounded (kSpinMax polls), after which
// GALES_ERR_TIMEOUT is set in a status word and the CTA or warp waits no more: it goes through
// its rows with what there is.  d_status[0] is the factorisation's word, which the call that runs
// it reads; d_status[1] the substitutions', which gales_solver_apply leaves to
// gales_solver_sync or the next factorisation or solve.
constexpr long long kSpinMax = 1ll << 22;

__device__ __forceinline__ int ld_acquire(const int* f) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* f, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(f), "r"(v) : "memory");
}
__device__ __forceinline__ bool wait_flag(const int* f) {
  for (long long i = 0; i < kSpinMax; ++i) {
    if (ld_acquire(f) != 0) return true;
    __nanosleep(32);
  }
  return false;
}

template <typename T>
__device__ __forceinline__ void cp_async_word(T* dst, const T* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(T) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// Shared memory of one factorisation CTA: the block row I, two buffers with a row K's
// diagonal and upper blocks, the row's columns and, per buffer, the upper blocks of row K
// that row I has (their index in row K and their position in row I).
template <int ND, typename T>
struct FactorSmem {
  static constexpr int BB = ND * ND;
  static size_t bytes(int max_row, int max_u) {
    return ((size_t)max_row + 2 * (1 + (size_t)max_u)) * BB * sizeof(T) +
           ((size_t)max_row + 4 * (size_t)max_u) * sizeof(int32_t);
  }
};

// The numeric factorisation in one persistent launch, a CTA per node row I.  For its lower
// blocks K in ascending order: L_IK = A_IK U_KK^-1 (row-wise substitution, lane r < ND of
// warp 0 owns row r), then A_IJ -= L_IK U_KJ for the upper blocks J of row K present in row
// I (a thread per entry), then the Doolittle step of the diagonal block applied across the
// whole block row, pivot by pivot.  Every entry sees the subtractions of the scalar ikj
// order, unfused.
// Bound: the FP64 pipe (2 lanes per SM and clock) by the ~49 ND multiply-subtract pairs of
// each (K, J), and the chain of rows.  A row waits for row K only when it reaches K, so the
// long part of its work runs while its last neighbours are still in progress, and the next
// K's blocks are copied to shared memory (cp.async) during the current update when that row
// is done already.  One warp per row and one launch per level (all of a row's inputs final
// before it starts) took 725 ms on the 157k-node tet system; a level has ~210 rows, too few
// warps for the FP64 pipes of 152 SMs.
constexpr int kFactorThreads = 128;

template <int ND, typename T>
__global__ void __launch_bounds__(kFactorThreads)
    ilu_factor_rows_kernel(T* __restrict__ F, const int64_t* __restrict__ f_rp, const int32_t* __restrict__ f_col,
                           const int64_t* __restrict__ f_diag, const int32_t* __restrict__ rows, int64_t n,
                           unsigned int* ticket, int* ready, unsigned int* __restrict__ status, int max_row,
                           int max_u) {
  constexpr int BB = ND * ND;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T* R = reinterpret_cast<T*>(sm_raw);                      // [max_row][BB] the block row
  T* UB = R + (size_t)max_row * BB;                         // [2][1 + max_u][BB] row K from its diagonal on
  int32_t* RC = (int32_t*)(UB + 2 * (size_t)(1 + max_u) * BB);  // [max_row] the row's columns
  int32_t* MQ = RC + max_row;                               // [2][max_u] matching blocks: index in row K
  int32_t* MP = MQ + 2 * max_u;                             // [2][max_u] and position in row I
  __shared__ int nm[2], s_row, s_next;
  __shared__ T ls[ND];
  const int tid = threadIdx.x;
  bool late = false;   // thread 0: a wait ran out
  for (;;) {
    if (tid == 0) {
      const unsigned int t = atomicAdd(ticket, 1u);
      s_row = (int64_t)t < n ? rows[t] : -1;
      nm[0] = nm[1] = 0;
    }
    __syncthreads();
    const int32_t I = s_row;
    if (I < 0) break;
    const int64_t p0 = f_rp[I];
    const int nb = (int)(f_rp[I + 1] - p0), bd = (int)(f_diag[I] - p0);
    for (int e = tid; e < nb * BB; e += kFactorThreads) R[e] = F[p0 * BB + e];
    for (int e = tid; e < nb; e += kFactorThreads) RC[e] = f_col[p0 + e];
    __syncthreads();
    // starts the copy of lower block b's row K into buffer b & 1 and lists its matches
    auto load = [&](int b) {
      const int64_t dK = f_diag[RC[b]];
      const int nu = (int)(f_rp[RC[b] + 1] - dK - 1), buf = b & 1;
      T* U = UB + (size_t)buf * (1 + max_u) * BB;
      for (int e = tid; e < (nu + 1) * BB; e += kFactorThreads) cp_async_word(U + e, F + dK * BB + e);
      for (int q = tid; q < nu; q += kFactorThreads) {
        const int pos = (int)find_col(RC, b + 1, nb, f_col[dK + 1 + q]);
        if (pos < 0) continue;
        const int at = atomicAdd(&nm[buf], 1);
        MQ[buf * max_u + at] = q;
        MP[buf * max_u + at] = pos;
      }
    };
    bool have = false;
    for (int b = 0; b < bd; ++b) {
      const int buf = b & 1;
      if (!have) {
        if (tid == 0 && !late && !wait_flag(ready + RC[b])) {
          late = true;
          atomicOr(status, (unsigned)GALES_ERR_TIMEOUT);
        }
        __syncthreads();
        load(b);
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      const T* UK = UB + (size_t)buf * (1 + max_u) * BB;
      T* B = R + (size_t)b * BB;
      if (tid < ND) {
        T row[ND];
#pragma unroll
        for (int c = 0; c < ND; ++c) row[c] = B[tid * ND + c];
#pragma unroll
        for (int c = 0; c < ND; ++c) {
          T s = row[c];
#pragma unroll
          for (int c2 = 0; c2 < c; ++c2) s -= row[c2] * UK[c2 * ND + c];
          row[c] = s / UK[c * ND + c];
        }
#pragma unroll
        for (int c = 0; c < ND; ++c) B[tid * ND + c] = row[c];
      } else if (tid == 32) {
        s_next = b + 1 < bd ? ld_acquire(ready + RC[b + 1]) : 0;
        nm[buf ^ 1] = 0;
      }
      __syncthreads();
      have = s_next != 0;
      if (have) load(b + 1);
      const int items = nm[buf] * BB;
      for (int t = tid; t < items; t += kFactorThreads) {
        const int i = t / BB, rc = t - i * BB, r = rc / ND, c = rc - r * ND;
        const T* U = UK + (size_t)(1 + MQ[buf * max_u + i]) * BB + c;
        T* tgt = R + (size_t)MP[buf * max_u + i] * BB + rc;
        T s = *tgt;
#pragma unroll
        for (int m = 0; m < ND; ++m) s -= B[r * ND + m] * U[m * ND];
        *tgt = s;
      }
      __syncthreads();
    }
    // Doolittle step of the diagonal block across the upper blocks: pivots c2 in order, all
    // rows below a pivot at once
    T* D = R + (size_t)bd * BB;
    const int ncols = (nb - bd) * ND;
    for (int c2 = 0; c2 < ND - 1; ++c2) {
      const int nr = ND - 1 - c2;
      if (tid < nr) {
        const int r = c2 + 1 + tid;
        const T l = D[r * ND + c2] / D[c2 * ND + c2];
        D[r * ND + c2] = l;
        ls[r] = l;
      }
      __syncthreads();
      for (int t = tid; t < nr * ncols; t += kFactorThreads) {
        const int rr = t / ncols, e = t - rr * ncols, r = c2 + 1 + rr;
        const int bb = e / ND, c = e - bb * ND;
        if (bb == 0 && c <= c2) continue;
        T* Rb = D + (size_t)bb * BB;
        Rb[r * ND + c] -= ls[r] * Rb[c2 * ND + c];
      }
      __syncthreads();
    }
    for (int e = tid; e < nb * BB; e += kFactorThreads) F[p0 * BB + e] = R[e];
    if (tid < ND && D[tid * ND + tid] == T(0)) atomicOr(status, (unsigned)GALES_ERR_SINGULAR);
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      st_release(ready + I, 1);
    }
  }
}

// Triangular substitutions, one persistent launch per triangle, a warp per node row:
//   lower  y_I = L_II^-1 (v_I - sum_K L_IK y_K), L_II unit lower
//   upper  x_I = U_II^-1 (y_I - sum_J U_IJ x_J)
// A sweep is a chain of levels (204 on a 27k-node system of tets, ~130 rows each), so its
// time is the latency of one level, not the bytes of the factor.  The words of the result
// are their own ready flags: the result vector is filled with a bit pattern that no row
// stores (kUnset, a NaN), lanes poll the words that they need with relaxed loads, which
// leave L1 alone, and a finished row is stored without a fence.  A level is then one
// store-to-load trip through L2 plus the row's own arithmetic; separate flags (release
// store, acquire load, then the load of the values) cost three such trips, and an acquire
// also empties the L1 that the factor had been prefetched into: 9.4 us a level with an FP32
// factor, 15 us with FP64 (M^-1 3.86 and 6.14 ms there; now 0.41 and 0.75 ms, 1.0 and 1.8 us
// a level).  Before it polls, a row loads its factor blocks into registers: lanes form G = 32 /
// ND groups of ND, lane (g, r) holds row r of the blocks g, g + G, ... (KB at a time).
// Blocks are taken in the order in which their rows finish (ascending for the lower sweep,
// descending for the upper one), all first polls in flight together.  With the diagonal
// blocks' rows scaled in advance (scale_diag_kernel) the chain has one multiply-add per
// unknown.  Ten warps per SM keep the next levels' rows loaded (M^-1 on a 157k-node system of
// 372 levels with 4, 8 and 10 warps: 2.57, 1.72, 1.62 ms); a block's columns spread over the groups instead of a
// block per group, with fewer products after the last arrival, was no faster (1.67).
template <int ND>
constexpr int kSweepBlocks = 56 / ND < 8 ? 56 / ND : 8;   // blocks per lane held in registers

template <typename T>
struct SweepWord;
template <>
struct SweepWord<double> {
  using Bits = unsigned long long;
  static constexpr Bits kUnset = ~0ull, kNan = 0x7ff8000000000000ull;
  static __device__ __forceinline__ Bits load(const double* p) {
    Bits v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
  }
  static __device__ __forceinline__ void store(double* p, double x) {
    Bits v = (Bits)__double_as_longlong(x);
    if (v == kUnset) v = kNan;
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
  }
  static __device__ __forceinline__ double value(Bits v) { return __longlong_as_double((long long)v); }
};
template <>
struct SweepWord<float> {
  using Bits = unsigned int;
  static constexpr Bits kUnset = ~0u, kNan = 0x7fc00000u;
  static __device__ __forceinline__ Bits load(const float* p) {
    Bits v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
  }
  static __device__ __forceinline__ void store(float* p, float x) {
    Bits v = __float_as_uint(x);
    if (v == kUnset) v = kNan;
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
  }
  static __device__ __forceinline__ float value(Bits v) { return __uint_as_float(v); }
};

__device__ __forceinline__ double sweep_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float sweep_fma(float a, float b, float c) { return fmaf(a, b, c); }

// The upper sweep's diagonal blocks: row r of U_II divided by its pivot, and the pivot's
// reciprocal on the diagonal (thread per block row, once per factorisation; a division and
// ND products per row and sweep otherwise, a third of the sweep's FP64 work).
template <int ND, typename T>
__global__ void scale_diag_kernel(const T* __restrict__ F, const int64_t* __restrict__ f_diag, int64_t n_rows,
                                  T* __restrict__ Us) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_rows) return;
  const int64_t node = i / ND;
  const int r = (int)(i - node * ND);
  const T* D = F + f_diag[node] * (ND * ND) + r * ND;
  T* o = Us + i * ND;
  const T rd = T(1) / D[r];
#pragma unroll
  for (int c = 0; c < ND; ++c) o[c] = c == r ? rd : D[c] * rd;
}

// In (lower: the FP64 right-hand side vbase; upper: the lower sweep's result yin) and out
// (zw, kUnset before the launch; upper: also the FP64 column zoutbase).  The ticket starts
// at ~0u (it is cleared together with zw), so the first claim is row 0 of the order.
template <int ND, typename T, bool LOWER>
__global__ void __launch_bounds__(32 * kSweepWarps)
    ilu_sweep_kernel(const T* __restrict__ F, const int64_t* __restrict__ f_rp, const int32_t* __restrict__ f_col,
                     const int64_t* __restrict__ f_diag, const T* __restrict__ Us, const int32_t* __restrict__ rows,
                     int64_t n, const double* __restrict__ vbase, const T* __restrict__ yin, T* zw, double* zoutbase,
                     const int* __restrict__ jidx, int64_t ld, unsigned int* ticket, unsigned int* status) {
  using W = SweepWord<T>;
  constexpr int BB = ND * ND, G = 32 / ND, KB = kSweepBlocks<ND>;
  const int lane = threadIdx.x & 31;
  const int g = lane / ND, r = lane < G * ND ? lane - g * ND : 0;
  const int64_t off = jidx ? (int64_t)(*jidx) * ld : 0;
  bool late = false;
  for (;;) {
    unsigned int t = 0;
    if (lane == 0) t = atomicAdd(ticket, 1u) + 1u;
    t = __shfl_sync(0xffffffffu, t, 0);
    if ((int64_t)t >= n) break;
    const int32_t I = rows[t];
    const int64_t pd = f_diag[I];
    const int64_t pa = LOWER ? f_rp[I] : pd + 1;
    const int nblk = (int)((LOWER ? pd : f_rp[I + 1]) - pa);
    // row r of the diagonal block and the right-hand side
    T D[ND];
#pragma unroll
    for (int c = 0; c < ND; ++c) D[c] = LOWER ? F[pd * BB + r * ND + c] : Us[((int64_t)I * ND + r) * ND + c];
    const T rhs = LOWER ? (T)vbase[off + (int64_t)I * ND + r] : yin[(int64_t)I * ND + r];
    T sum = g == 0 ? -rhs : T(0), sum2 = T(0);
    for (int k0 = 0; k0 < nblk; k0 += KB * G) {
      int64_t zc[KB];
      T B[KB][ND];
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        const int i = k0 + k * G + g;
        const bool on = g < G && i < nblk;
        const int64_t p = pa + (LOWER ? i : nblk - 1 - i);
        zc[k] = on ? (int64_t)f_col[p] * ND + r : -1;
#pragma unroll
        for (int c = 0; c < ND; ++c) B[k][c] = on ? F[p * BB + r * ND + c] : T(0);
      }
      typename W::Bits w[KB];
#pragma unroll
      for (int k = 0; k < KB; ++k) w[k] = zc[k] >= 0 ? W::load(zw + zc[k]) : typename W::Bits(0);
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        if (k0 + k * G >= nblk) break;   // the same for every lane
        for (long long spin = 0; !late && __any_sync(0xffffffffu, w[k] == W::kUnset); ++spin) {
          if (w[k] == W::kUnset) w[k] = W::load(zw + zc[k]);
          late = spin >= kSpinMax;
        }
        const T zk = W::value(w[k]);
#pragma unroll
        for (int c = 0; c < ND; ++c) {
          const T x = __shfl_sync(0xffffffffu, zk, (g < G ? g : 0) * ND + c);
          if (c & 1) sum2 = sweep_fma(B[k][c], x, sum2);
          else sum = sweep_fma(B[k][c], x, sum);
        }
      }
    }
    // the groups' sums in a fixed order; s = rhs - sum of the blocks
    sum += sum2;
    T part[G];
#pragma unroll
    for (int q = 0; q < G; ++q) part[q] = __shfl_sync(0xffffffffu, sum, q * ND + r);
#pragma unroll
    for (int h = 1; h < G; h *= 2)
#pragma unroll
      for (int q = 0; q + h < G; q += 2 * h) part[q] += part[q + h];
    T s = -part[0];
    if constexpr (LOWER) {
#pragma unroll
      for (int c = 0; c < ND - 1; ++c) {
        const T x = __shfl_sync(0xffffffffu, s, c);
        if (lane > c) s = sweep_fma(-D[c], x, s);
      }
    } else {
      T rd = D[0];
#pragma unroll
      for (int c = 1; c < ND; ++c) rd = r == c ? D[c] : rd;
      s *= rd;
#pragma unroll
      for (int c = ND - 1; c > 0; --c) {
        const T x = __shfl_sync(0xffffffffu, s, c);
        if (lane < c) s = sweep_fma(-D[c], x, s);
      }
    }
    if (lane < ND) {
      W::store(zw + (int64_t)I * ND + lane, s);
      if constexpr (!LOWER) zoutbase[off + (int64_t)I * ND + lane] = (double)s;
    }
  }
  if (late && lane == 0) atomicOr(status, (unsigned)GALES_ERR_TIMEOUT);
}

// Small systems: each sweep by one thread-block cluster, whose CTAs hold the whole result vector
// in shared memory (n ND words <= kClusterSmem).  A finished row is stored into every CTA's copy
// and polled locally, so a level pays a trip to a neighbour's shared memory in place of one
// through L2.  With an FP64 factor the off-diagonal blocks are multiplied by the inverse of their
// row's diagonal block in advance (scale_rows_kernel), which leaves no solve, ND dependent FP64
// operations, after the last arrival:
//   lower  y_I = L_II^-1 v_I - sum_K (L_II^-1 L_IK) y_K, upper alike with U_II.
// An FP32 factor keeps its blocks: rounding them once more would double the sweeps' error.
// Rows go to the cluster's warps in turn, in level order; all warps are resident, so every wait
// ends (and is bounded, see kSpinMax).  Bound: the FP64 latency of the products and sums after a
// row's last arrival.  M^-1 of a 2,145-node channel (161 levels, 5 dofs): 0.23 ms with an FP64
// factor and 0.13 with FP32, against 0.41 and 0.24 through L2.  4 or 12 warps per CTA: 0.23,
// 0.24; a block's columns spread over the lanes, each polling its own word: 0.22 and 0.15.
// A cluster has 16 of the 152 SMs, so it suits systems whose time is their levels' latency:
// kClusterBusy bounds the register loads of blocks that a warp makes per level (a load is 1.6 us
// FP32, 3 FP64, a level through L2 0.85 and 1.8), kClusterBytes the factor's bytes per level (16
// SMs with a few rows in flight each read 0.2 TB/s).  M^-1 in us, cluster and L2 (loads, KB per
// level).  Better in the cluster: 350, 572 (quads, 4 dofs, FP32; 0.22, 12), 537, 685 (hexes, 8
// dofs, FP64; 0.20, 224), 456, 513 (the same, longer; 0.25, 283), 561, 645 (hexes, ILU(2), FP32; 0.26,
// 167), 266, 302 (triangles, ILU(0), FP32; 0.43, 12).  Through L2: 450, 392 (hexes, FP32; 0.34, 187),
// 1,102, 904 (the same, ILU(3); 0.27, 203), 259, 244 (tets, 5 dofs, FP32; 0.52, 82), 177, 152
// (tets, 7 dofs, ILU(0), FP64; 0.61, 207), 225, 124 (tets, ILU(0), FP32; 1.22, 109).  An FP64 system
// that fits was never above 283 KB a level: that line is its L2 time per level at the same rate.
constexpr int kClusterWarps = 8, kClusterMax = 16;
constexpr size_t kClusterSmem = 200 * 1024;
constexpr double kClusterBusy = 0.48;
template <typename T>
constexpr double kClusterBytes = sizeof(T) == 8 ? 380e3 : 180e3;
template <typename T>
constexpr bool kClusterScaled = sizeof(T) == 8;

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <typename T>
__device__ __forceinline__ typename SweepWord<T>::Bits cluster_poll(uint32_t at) {
  typename SweepWord<T>::Bits v;
  if constexpr (sizeof(T) == 8) asm volatile("ld.relaxed.cluster.shared::cta.b64 %0, [%1];" : "=l"(v) : "r"(at) : "memory");
  else asm volatile("ld.relaxed.cluster.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
  return v;
}
// stores x into CTA rank's copy of the word at shared address at
template <typename T>
__device__ __forceinline__ void cluster_store(uint32_t at, uint32_t rank, T x) {
  using W = SweepWord<T>;
  uint32_t to;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(at), "r"(rank));
  if constexpr (sizeof(T) == 8) {
    typename W::Bits v = (typename W::Bits)__double_as_longlong(x);
    if (v == W::kUnset) v = W::kNan;
    asm volatile("st.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(to), "l"(v) : "memory");
  } else {
    typename W::Bits v = __float_as_uint(x);
    if (v == W::kUnset) v = W::kNan;
    asm volatile("st.relaxed.cluster.shared::cluster.b32 [%0], %1;" ::"r"(to), "r"(v) : "memory");
  }
}

// S = the off-diagonal factor blocks times the inverse of their row's diagonal block (warp per
// node row, a lane per block column; the diagonal of U scaled as in Us).
template <int ND, typename T>
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
    scale_rows_kernel(const T* __restrict__ F, const int64_t* __restrict__ f_rp, const int64_t* __restrict__ f_diag,
                      const T* __restrict__ Us, int64_t n, T* __restrict__ S) {
  constexpr int BB = ND * ND;
  const int64_t I = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (I >= n) return;
  const int lane = threadIdx.x & 31;
  const int64_t p0 = f_rp[I], p1 = f_rp[I + 1], pd = f_diag[I];
  for (int64_t it = lane; it < (p1 - p0) * ND; it += 32) {
    const int64_t p = p0 + it / ND;
    const int c = (int)(it % ND);
    if (p == pd) continue;
    T x[ND];
#pragma unroll
    for (int r = 0; r < ND; ++r) x[r] = F[p * BB + r * ND + c];
    if (p < pd) {
      const T* D = F + pd * BB;
#pragma unroll
      for (int q = 0; q < ND - 1; ++q)
#pragma unroll
        for (int r = q + 1; r < ND; ++r) x[r] = sweep_fma(-D[r * ND + q], x[q], x[r]);
    } else {
      const T* D = Us + I * BB;
#pragma unroll
      for (int r = 0; r < ND; ++r) x[r] *= D[r * ND + r];
#pragma unroll
      for (int q = ND - 1; q > 0; --q)
#pragma unroll
        for (int r = 0; r < q; ++r) x[r] = sweep_fma(-D[r * ND + q], x[q], x[r]);
    }
#pragma unroll
    for (int r = 0; r < ND; ++r) S[p * BB + r * ND + c] = x[r];
  }
}

// In (lower: the FP64 right-hand side vbase; upper: the lower sweep's result y) and out (lower:
// y; upper: the FP64 column zoutbase).  D: the factor (lower) or the scaled diagonal blocks.
template <int ND, typename T, bool LOWER>
__global__ void __launch_bounds__(32 * kClusterWarps)
    ilu_sweep_cluster_kernel(const T* __restrict__ S, const int64_t* __restrict__ f_rp,
                             const int32_t* __restrict__ f_col, const int64_t* __restrict__ f_diag,
                             const T* __restrict__ Dg, const int32_t* __restrict__ rows, int64_t n,
                             const double* __restrict__ vbase, T* __restrict__ y, double* __restrict__ zoutbase,
                             const int* __restrict__ jidx, int64_t ld, unsigned int* status) {
  using W = SweepWord<T>;
  constexpr int BB = ND * ND, G = 32 / ND, KB = kSweepBlocks<ND>;
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  T* z = reinterpret_cast<T*>(sweep_smem);
  const uint32_t z0 = (uint32_t)__cvta_generic_to_shared(z);
  const int lane = threadIdx.x & 31;
  const int g = lane / ND, r = lane < G * ND ? lane - g * ND : 0;
  const uint32_t nc = gridDim.x;   // one cluster
  const int64_t off = jidx ? (int64_t)(*jidx) * ld : 0;
  for (int64_t i = threadIdx.x; i < n * ND; i += blockDim.x)
    reinterpret_cast<typename W::Bits*>(z)[i] = W::kUnset;
  cluster_sync();
  bool late = false;
  for (int64_t t = cluster_rank() + (int64_t)nc * (threadIdx.x >> 5); t < n; t += (int64_t)nc * kClusterWarps) {
    const int32_t I = rows[t];
    const int64_t pd = f_diag[I];
    const int64_t pa = LOWER ? f_rp[I] : pd + 1;
    const int nblk = (int)((LOWER ? pd : f_rp[I + 1]) - pa);
    T D[ND];
#pragma unroll
    for (int c = 0; c < ND; ++c) D[c] = Dg[(LOWER ? pd : (int64_t)I) * BB + r * ND + c];
    // x times the inverse of the diagonal block
    auto solve = [&](T x) {
      if constexpr (LOWER) {
#pragma unroll
        for (int c = 0; c < ND - 1; ++c) {
          const T xc = __shfl_sync(0xffffffffu, x, c);
          if (r > c) x = sweep_fma(-D[c], xc, x);
        }
      } else {
        T rd = D[0];
#pragma unroll
        for (int c = 1; c < ND; ++c) rd = r == c ? D[c] : rd;
        x *= rd;
#pragma unroll
        for (int c = ND - 1; c > 0; --c) {
          const T xc = __shfl_sync(0xffffffffu, x, c);
          if (r < c) x = sweep_fma(-D[c], xc, x);
        }
      }
      return x;
    };
    T rhs = LOWER ? (T)vbase[off + (int64_t)I * ND + r] : y[(int64_t)I * ND + r];
    if constexpr (kClusterScaled<T>) rhs = solve(rhs);
    T sum = g == 0 ? -rhs : T(0), sum2 = T(0);
    for (int k0 = 0; k0 < nblk; k0 += KB * G) {
      int zc[KB];
      T B[KB][ND];
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        const int i = k0 + k * G + g;
        const bool on = g < G && i < nblk;
        const int64_t p = pa + (LOWER ? i : nblk - 1 - i);
        zc[k] = on ? f_col[p] * ND + r : -1;
#pragma unroll
        for (int c = 0; c < ND; ++c) B[k][c] = on ? S[p * BB + r * ND + c] : T(0);
      }
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        if (k0 + k * G >= nblk) break;   // the same for every lane
        typename W::Bits w = zc[k] >= 0 ? W::kUnset : typename W::Bits(0);
        for (long long spin = 0; !late; ++spin) {
          if (w == W::kUnset) w = cluster_poll<T>(z0 + (uint32_t)zc[k] * (uint32_t)sizeof(T));
          if (!__any_sync(0xffffffffu, w == W::kUnset)) break;
          if (spin >= kSpinMax) late = true;
        }
        const T zk = W::value(w);
#pragma unroll
        for (int c = 0; c < ND; ++c) {
          const T x = __shfl_sync(0xffffffffu, zk, (g < G ? g : 0) * ND + c);
          if (c & 1) sum2 = sweep_fma(B[k][c], x, sum2);
          else sum = sweep_fma(B[k][c], x, sum);
        }
      }
    }
    sum += sum2;
    T part[G];
#pragma unroll
    for (int q = 0; q < G; ++q) part[q] = __shfl_sync(0xffffffffu, sum, q * ND + r);
#pragma unroll
    for (int h = 1; h < G; h *= 2)
#pragma unroll
      for (int q = 0; q + h < G; q += 2 * h) part[q] += part[q + h];
    T s = -part[0];
    if constexpr (!kClusterScaled<T>) s = solve(s);
    // lane (g, r) stores word r into the copies of the CTAs g, g + G, ...
    if (g < G)
      for (uint32_t c = (uint32_t)g; c < nc; c += G)
        cluster_store<T>(z0 + (uint32_t)(I * ND + r) * (uint32_t)sizeof(T), c, s);
    if (lane < ND) {
      if constexpr (LOWER) y[(int64_t)I * ND + lane] = s;
      else zoutbase[off + (int64_t)I * ND + lane] = (double)s;
    }
  }
  if (late && lane == 0) atomicOr(status, (unsigned)GALES_ERR_TIMEOUT);
  cluster_sync();   // a CTA's copy is written until every row is done
}

// y = A x (or y = b - A x) on the assembly's CSR values: warp per node row.  Lanes form
// G = 32 / ND groups of ND, lane (g, r) takes scalar row r over the node row's blocks g,
// g + G, ...: ND multiply-adds a block and G - 1 adds at the end.  Bound: the FP64 pipe
// (0.18 ms for the 115M entries of a 157k-node tet system at 2 lanes per SM and clock, DRAM
// 0.14 ms); a warp per scalar row spent more FP64 issue slots on its shuffle sums than on
// products: 1.28 ms there, now 0.32.
template <int ND>
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
    spmv_kernel(const double* __restrict__ vals, const int64_t* __restrict__ node_rp,
                const int32_t* __restrict__ node_col, int64_t n_nodes, const double* __restrict__ x,
                const double* __restrict__ b, double* __restrict__ y) {
  constexpr int G = 32 / ND;
  const int64_t i = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (i >= n_nodes) return;
  const int lane = threadIdx.x & 31;
  const int g = lane / ND, r = lane < G * ND ? lane - g * ND : 0;
  const int64_t t0 = node_rp[i];
  const int deg = (int)(node_rp[i + 1] - t0);
  const double* a = vals + t0 * (ND * ND) + (int64_t)r * deg * ND;
  double s = 0.0;
  if (g < G)
#pragma unroll 2
    for (int k = g; k < deg; k += G) {
      const double* xc = x + (int64_t)node_col[t0 + k] * ND;
#pragma unroll
      for (int c = 0; c < ND; ++c) s = fma(__ldcs(a + k * ND + c), xc[c], s);
    }
  double tot = s;
#pragma unroll
  for (int q = 1; q < G; ++q) tot += __shfl_sync(0xffffffffu, s, q * ND + r);
  if (lane < ND) {
    const int64_t row = i * ND + lane;
    y[row] = b ? b[row] - tot : tot;
  }
}

// One pass of the Arnoldi step, mode kDots: h = V^T w; kSubDots: w -= V h, then h2 = V^T w
// and h += h2; kSubNorm: w -= V h2, then hn[0] = ||w||.  nv columns of V, stride ld.  A CTA takes
// tiles of kTile rows: a thread subtracts its rows, then the warps share the columns of the
// dot products (lane partials in shared memory, kCols columns at a time, carried over the
// tiles).  The last CTA to finish adds the CTAs' partial sums in a fixed order, so repeated
// solves are bit-identical.  Bound: DRAM (V once per pass; a tile's columns come from L2 the
// second time) and, with fused multiply-adds, as much FP64: 44 us per pass over 25 columns of
// 1.1M rows.  Separate launches for the dots, their final sums (one CTA adding 304 partials
// serially, 24 us each) and the updates took 0.47 ms a step on 189k rows, mostly launches; now
// 0.16 ms.  Tiles of 256 rows and four CTAs per SM, against 512 and two, keep enough loads in
// flight and a tile's columns in L2: 164 against 339 us for kSubDots at 1.1M rows, 33 columns.
constexpr int kDots = 0, kSubDots = 1, kSubNorm = 2;
constexpr int kTile = 256, kCols = 96;
constexpr int kHs = 512;   // coefficients held in shared memory; those of more columns are read from L2

template <int MODE>
__global__ void __launch_bounds__(kDotThreads, 4)
    arnoldi_kernel(const double* __restrict__ V, int64_t ld, int nv, double* __restrict__ w, int64_t n,
                   double* __restrict__ h, double* __restrict__ h2, double* __restrict__ hn,
                   double* __restrict__ part, unsigned int* __restrict__ count) {
  __shared__ double ws[kTile];
  __shared__ double acc[MODE == kSubNorm ? 1 : kCols][32];
  __shared__ double red[kDotThreads / 32];
  __shared__ double hs[kHs];
  __shared__ bool last;
  constexpr int NW = kDotThreads / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double* __restrict__ hsub = MODE == kSubDots ? h : h2;
  if (MODE != kDots) {
    for (int c = threadIdx.x; c < nv && c < kHs; c += kDotThreads) hs[c] = __ldcg(hsub + c);
    __syncthreads();
  }
  double nrm = 0.0;
  const int nout = MODE == kSubNorm ? 1 : nv;
  for (int cb = 0; cb == 0 || cb < nv; cb += kCols) {
    const int nc = nv - cb < kCols ? nv - cb : kCols;
    if constexpr (MODE != kSubNorm)
      for (int c = wid; c < nc; c += NW) acc[c][lane] = 0.0;
    for (int64_t lo = (int64_t)blockIdx.x * kTile; lo < n; lo += (int64_t)gridDim.x * kTile) {
      const int m = (int)(n - lo < kTile ? n - lo : kTile);
      for (int i = threadIdx.x; i < m; i += kDotThreads) {
        double x = w[lo + i];
        if (MODE != kDots && cb == 0 && nv > 0) {
          const double* __restrict__ v = V + lo + i;
          const int nh = nv < kHs ? nv : kHs;
          double s0 = 0.0, s1 = 0.0;
          int c = 0;
#pragma unroll 4
          for (; c + 1 < nh; c += 2) {
            s0 = fma(v[(int64_t)c * ld], hs[c], s0);
            s1 = fma(v[(int64_t)(c + 1) * ld], hs[c + 1], s1);
          }
          for (; c < nh; ++c) s0 = fma(v[(int64_t)c * ld], hs[c], s0);
          for (; c < nv; ++c) s0 = fma(v[(int64_t)c * ld], __ldcg(hsub + c), s0);
          x -= s0 + s1;
          w[lo + i] = x;
        }
        if constexpr (MODE == kSubNorm) nrm = fma(x, x, nrm);
        else ws[i] = x;
      }
      if constexpr (MODE == kSubNorm) continue;
      __syncthreads();
      for (int c = wid; c < nc; c += NW) {
        const double* __restrict__ v = V + (int64_t)(cb + c) * ld + lo;
        double a = acc[MODE == kSubNorm ? 0 : c][lane];
        for (int i = lane; i < m; i += 32) a = fma(v[i], ws[i], a);
        acc[MODE == kSubNorm ? 0 : c][lane] = a;
      }
      __syncthreads();
    }
    if constexpr (MODE == kSubNorm) break;
    for (int c = wid; c < nc; c += NW) {
      double a = acc[MODE == kSubNorm ? 0 : c][lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if (lane == 0) part[(int64_t)blockIdx.x * nout + cb + c] = a;
    }
  }
  if constexpr (MODE == kSubNorm) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    if (lane == 0) red[wid] = nrm;
    __syncthreads();
    if (threadIdx.x == 0) {
      double a = 0.0;
      for (int q = 0; q < NW; ++q) a += red[q];
      part[blockIdx.x] = a;
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(count, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int c = wid; c < nout; c += NW) {
    double a = 0.0;
    for (unsigned int q = lane; q < gridDim.x; q += 32) a += __ldcg(part + (int64_t)q * nout + c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane != 0) continue;
    if constexpr (MODE == kDots) h[c] = a;
    else if constexpr (MODE == kSubDots) { h2[c] = a; h[c] += a; }
    else hn[0] = sqrt(a);
  }
  if (threadIdx.x == 0) *count = 0;
}

// x += sum_c Z[c] y[c]
__global__ void update_x_kernel(const double* __restrict__ Z, int64_t ld, int nv, const double* __restrict__ y,
                                double* __restrict__ x, int64_t n) {
  extern __shared__ double ys[];
  for (int c = threadIdx.x; c < nv; c += blockDim.x) ys[c] = y[c];
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int c = 0; c < nv; ++c) s = fma(Z[(int64_t)c * ld + i], ys[c], s);
    x[i] += s;
  }
}

// dst = src / *nrm (dst = 0 when the norm is zero)
__global__ void scale_kernel(const double* __restrict__ src, const double* __restrict__ nrm, double* __restrict__ dst,
                             int64_t n) {
  const double d = *nrm;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = d > 0.0 ? src[i] / d : 0.0;
}

__global__ void set_index_kernel(int* __restrict__ p, int v) { *p = v; }

__global__ void copy_kernel(const double* __restrict__ src, double* __restrict__ dst, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

// fluid_updater::corrector then model::dof_trimmer: I += dx, then the dofs with index
// in [first, last) of every node clamped as max(lo, min(v, hi)).
__global__ void correct_kernel(double* __restrict__ I, const double* __restrict__ dx, int64_t n, int nd, int first,
                               int last, double lo, double hi) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double v = I[i] + dx[i];
    const int k = (int)(i % nd);
    if (k >= first && k < last) v = fmax(lo, fmin(v, hi));
    I[i] = v;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Handle and C ABI.
// ---------------------------------------------------------------------------

struct gales_solver {
  int device = 0;
  int nd = 0;
  int sms = 1;
  int64_t n_nodes = 0, n_rows = 0, nnz = 0;
  gales_solver_params prm{};
  std::vector<int64_t> node_rp, f_rp, f_diag, lev_off_f, lev_off_b;
  std::vector<int32_t> node_col, f_col, lev_f, lev_b, rows_f, rows_b;
  Dev<int64_t> d_node_rp, d_f_rp, d_f_diag, d_a2f;
  Dev<int32_t> d_node_col, d_f_col, d_rows_f, d_rows_b;
  Dev<double> d_F, d_V, d_Z, d_w, d_r, d_x, d_part, d_h, d_h2, d_y, d_vals, d_b;
  Dev<float> d_Ff;           // FP32 factor (GALES_PRECOND_ILU_FP32)
  Dev<int> d_j;
  Dev<int> d_ready;          // factorisation: ticket, then a ready flag per node row
  Dev<unsigned char> d_udiag;  // the upper sweep's scaled diagonal blocks (factor's type)
  Dev<unsigned char> d_scaled;  // cluster sweeps in FP64: off-diagonal blocks times their inverse diagonal block
  Dev<unsigned char> d_sweep;  // substitutions: the two result vectors (factor's type), then two tickets
  Dev<unsigned int> d_status, d_count;  // error bits of factorisation and substitutions; CTAs of an Arnoldi pass that are done
  double* h_buf = nullptr;   // pinned: Hessenberg column and the least-squares solution
  int m = 0;                 // Krylov vectors per cycle
  int max_row = 0, max_u = 0;  // longest factor row, longest upper part (blocks)
  int smem_optin = 0;          // opt-in shared memory per CTA
  size_t factor_smem = 0;      // dynamic shared memory of the factorisation kernel (0: level launches)
  int factor_ctas = 1;         // its resident CTAs per SM
  int cluster = 0;             // CTAs of the sweeps' cluster (0: the sweeps through L2)
  int dot_blocks = 1;
  cudaGraphExec_t prec_graph = nullptr;
  cudaStream_t cap = nullptr;
  int64_t launches = 0;
  std::string err;
};

namespace {

int sfail(gales_solver* s, int code, const std::string& msg) {
  if (s) s->err = msg;
  return code;
}

#define SCK(s, call, what)                                                                               \
  do {                                                                                                   \
    cudaError_t e__ = (call);                                                                            \
    if (e__ != cudaSuccess)                                                                              \
      return sfail(s, e__ == cudaErrorMemoryAllocation ? GALES_ERR_NO_MEMORY : GALES_ERR_CUDA,            \
                   std::string(what) + ": " + cudaGetErrorString(e__));                                  \
  } while (0)

bool dev_ptr(const void* p) {
  if (!p) return false;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

inline unsigned grid_for(int64_t warps) { return (unsigned)((warps + kWarpsPerBlock - 1) / kWarpsPerBlock); }

template <typename T>
T* factor_ptr(gales_solver* s);
template <>
double* factor_ptr<double>(gales_solver* s) { return s->d_F.p; }
template <>
float* factor_ptr<float>(gales_solver* s) { return s->d_Ff.p; }

// Launch wrappers for nd = ND and a factor stored in T (double: the reference's FP64
// arithmetic; float: FP32 factor and substitutions).
template <int ND, typename T>
struct Kernels {
  static cudaError_t to_factor(gales_solver* s, const double* vals, cudaStream_t st) {
    matrix_to_factor_kernel<ND, T><<<grid_for(s->n_nodes), 32 * kWarpsPerBlock, 0, st>>>(
        vals, s->d_node_rp.p, s->d_a2f.p, s->n_nodes, factor_ptr<T>(s));
    return cudaGetLastError();
  }
  // A launch of one cluster of `size` CTAs.
  struct ClusterLaunch {
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg;
    ClusterLaunch(unsigned size, size_t smem, cudaStream_t st) {
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = size;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      std::memset(&cfg, 0, sizeof(cfg));
      cfg.gridDim = dim3(size);
      cfg.blockDim = dim3(32 * kClusterWarps);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = st;
      cfg.attrs = at;
      cfg.numAttrs = 1;
    }
  };
  static size_t cluster_smem(const gales_solver* s) { return (size_t)s->n_rows * sizeof(T); }
  // Cluster size of the sweeps: the largest of 16 and 8 that the device takes, 0 where the
  // result vector is too long for a CTA or the work too much for a cluster's SMs (see
  // kClusterBusy, kClusterBytes).
  template <bool LOWER>
  static cudaError_t prepare_cluster(gales_solver* s, int& size) {
    const auto fn = ilu_sweep_cluster_kernel<ND, T, LOWER>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    for (; size > 4; size /= 2) {
      ClusterLaunch l((unsigned)size, cluster_smem(s), nullptr);
      int nb = 0;
      if (cudaOccupancyMaxActiveClusters(&nb, fn, &l.cfg) == cudaSuccess && nb > 0) return cudaSuccess;
      cudaGetLastError();
    }
    size = 0;
    return cudaSuccess;
  }
  static int cluster_size(gales_solver* s) {
    if (cluster_smem(s) > kClusterSmem || cluster_smem(s) > (size_t)s->smem_optin) return 0;
    constexpr int64_t per = 32 / ND * kSweepBlocks<ND>;   // blocks of a row that a warp loads at once
    int64_t loads = 0;
    for (int64_t i = 0; i < s->n_nodes; ++i) {
      const int64_t lower = s->f_diag[i] - s->f_rp[i], upper = s->f_rp[i + 1] - s->f_diag[i] - 1;
      loads += std::max<int64_t>(1, (lower + per - 1) / per) + std::max<int64_t>(1, (upper + per - 1) / per);
    }
    const double levels = (double)(s->lev_off_f.size() - 1 + s->lev_off_b.size() - 1);
    if ((double)loads > kClusterBusy * levels * (kClusterMax * kClusterWarps) ||
        (double)s->f_col.size() * (ND * ND * sizeof(T)) > kClusterBytes<T> * levels)
      return 0;
    int size = kClusterMax;
    if (size && (prepare_cluster<true>(s, size) != cudaSuccess || prepare_cluster<false>(s, size) != cudaSuccess)) {
      cudaGetLastError();
      size = 0;
    }
    return size;
  }
  // The persistent factorisation where a block row and two rows' upper parts fit the shared
  // memory of an SM; rows too long for that take the level launches on global memory.
  static cudaError_t prepare(gales_solver* s) {
    const size_t bytes = FactorSmem<ND, T>::bytes(s->max_row, s->max_u);
    s->factor_smem = 0;
    if (bytes > (size_t)s->smem_optin) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(ilu_factor_rows_kernel<ND, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)bytes);
    int nb = 0;
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, ilu_factor_rows_kernel<ND, T>, kFactorThreads, bytes);
    if (e == cudaSuccess && nb > 0) {
      s->factor_smem = bytes;
      s->factor_ctas = nb;
    }
    return e;
  }
  static cudaError_t factor(gales_solver* s, cudaStream_t st) {
    if (s->factor_smem) {
      cudaError_t e = cudaMemsetAsync(s->d_ready.p, 0, s->d_ready.n * sizeof(int), st);
      if (e != cudaSuccess) return e;
      const unsigned g = (unsigned)std::min<int64_t>(s->n_nodes, (int64_t)s->sms * s->factor_ctas);
      ilu_factor_rows_kernel<ND, T><<<g, kFactorThreads, s->factor_smem, st>>>(
          factor_ptr<T>(s), s->d_f_rp.p, s->d_f_col.p, s->d_f_diag.p, s->d_rows_f.p, s->n_nodes,
          reinterpret_cast<unsigned int*>(s->d_ready.p), s->d_ready.p + 1, s->d_status.p, s->max_row, s->max_u);
      ++s->launches;
      return cudaGetLastError();
    }
    for (size_t l = 0; l + 1 < s->lev_off_f.size(); ++l) {
      const int64_t o = s->lev_off_f[l], c = s->lev_off_f[l + 1] - o;
      ilu_factor_level_kernel<ND, T><<<grid_for(c), 32 * kWarpsPerBlock, 0, st>>>(
          factor_ptr<T>(s), s->d_f_rp.p, s->d_f_col.p, s->d_f_diag.p, s->d_rows_f.p + o, c, s->d_status.p);
      ++s->launches;
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  static cudaError_t scale_diag(gales_solver* s, cudaStream_t st) {
    scale_diag_kernel<ND, T><<<(unsigned)((s->n_rows + 127) / 128), 128, 0, st>>>(
        factor_ptr<T>(s), s->d_f_diag.p, s->n_rows, reinterpret_cast<T*>(s->d_udiag.p));
    ++s->launches;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !s->cluster || !kClusterScaled<T>) return e;
    scale_rows_kernel<ND, T><<<grid_for(s->n_nodes), 32 * kWarpsPerBlock, 0, st>>>(
        factor_ptr<T>(s), s->d_f_rp.p, s->d_f_diag.p, reinterpret_cast<const T*>(s->d_udiag.p), s->n_nodes,
        reinterpret_cast<T*>(s->d_scaled.p));
    ++s->launches;
    return cudaGetLastError();
  }
  // both substitutions (result vectors and tickets set to all ones by the caller)
  static cudaError_t sweeps(gales_solver* s, const double* v, double* z, const int* j, int64_t ld, cudaStream_t st) {
    T* y = reinterpret_cast<T*>(s->d_sweep.p);
    if (s->cluster) {
      const ClusterLaunch l((unsigned)s->cluster, cluster_smem(s), st);
      const T* S = kClusterScaled<T> ? reinterpret_cast<const T*>(s->d_scaled.p) : factor_ptr<T>(s);
      const cudaError_t e = cudaLaunchKernelEx(
          &l.cfg, ilu_sweep_cluster_kernel<ND, T, true>, S, (const int64_t*)s->d_f_rp.p, (const int32_t*)s->d_f_col.p,
          (const int64_t*)s->d_f_diag.p, (const T*)factor_ptr<T>(s), (const int32_t*)s->d_rows_f.p, s->n_nodes, v, y,
          (double*)nullptr, j, ld, s->d_status.p + 1);
      if (e != cudaSuccess) return e;
      return cudaLaunchKernelEx(&l.cfg, ilu_sweep_cluster_kernel<ND, T, false>, S, (const int64_t*)s->d_f_rp.p,
                                (const int32_t*)s->d_f_col.p, (const int64_t*)s->d_f_diag.p,
                                reinterpret_cast<const T*>(s->d_udiag.p), (const int32_t*)s->d_rows_b.p, s->n_nodes,
                                (const double*)nullptr, y, z, j, ld, s->d_status.p + 1);
    }
    T* x = y + s->n_rows;
    unsigned int* tk = reinterpret_cast<unsigned int*>(x + s->n_rows);
    const unsigned g = (unsigned)std::min<int64_t>((s->n_nodes + kSweepWarps - 1) / kSweepWarps, s->sms);
    ilu_sweep_kernel<ND, T, true><<<g, 32 * kSweepWarps, 0, st>>>(
        factor_ptr<T>(s), s->d_f_rp.p, s->d_f_col.p, s->d_f_diag.p, nullptr, s->d_rows_f.p, s->n_nodes, v, nullptr, y,
        nullptr, j, ld, tk, s->d_status.p + 1);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ilu_sweep_kernel<ND, T, false><<<g, 32 * kSweepWarps, 0, st>>>(
        factor_ptr<T>(s), s->d_f_rp.p, s->d_f_col.p, s->d_f_diag.p, reinterpret_cast<const T*>(s->d_udiag.p),
        s->d_rows_b.p, s->n_nodes, nullptr, y, x, z, j, ld, tk + 1, s->d_status.p + 1);
    return cudaGetLastError();
  }
  static cudaError_t spmv(gales_solver* s, const double* vals, const double* x, const double* b, double* y,
                          cudaStream_t st) {
    spmv_kernel<ND><<<grid_for(s->n_nodes), 32 * kWarpsPerBlock, 0, st>>>(vals, s->d_node_rp.p, s->d_node_col.p,
                                                                         s->n_nodes, x, b, y);
    return cudaGetLastError();
  }
};

struct Ops {
  int (*cluster_size)(gales_solver*);
  cudaError_t (*prepare)(gales_solver*);
  cudaError_t (*to_factor)(gales_solver*, const double*, cudaStream_t);
  cudaError_t (*factor)(gales_solver*, cudaStream_t);
  cudaError_t (*scale_diag)(gales_solver*, cudaStream_t);
  cudaError_t (*sweeps)(gales_solver*, const double*, double*, const int*, int64_t, cudaStream_t);
  cudaError_t (*spmv)(gales_solver*, const double*, const double*, const double*, double*, cudaStream_t);
};

template <int ND, typename T>
Ops ops_for() {
  using K = Kernels<ND, T>;
  return {K::cluster_size, K::prepare, K::to_factor, K::factor, K::scale_diag, K::sweeps, K::spmv};
}

// nd = 2 + dim + nb_comp - 1 with one to four components (gales_asm_create)
template <typename T>
bool ops_t(int nd, Ops& o) {
  switch (nd) {
    case 4: o = ops_for<4, T>(); return true;
    case 5: o = ops_for<5, T>(); return true;
    case 6: o = ops_for<6, T>(); return true;
    case 7: o = ops_for<7, T>(); return true;
    case 8: o = ops_for<8, T>(); return true;
    default: return false;
  }
}

bool ops(const gales_solver* s, Ops& o) {
  return s->prm.precond == GALES_PRECOND_ILU_FP32 ? ops_t<float>(s->nd, o) : ops_t<double>(s->nd, o);
}

inline bool has_ilu(const gales_solver* s) {
  return s->prm.precond == GALES_PRECOND_ILU || s->prm.precond == GALES_PRECOND_ILU_FP32;
}

// z = M^-1 v for columns addressed by *j (graph) or plain pointers (j null): the two sweeps
// after setting their result vectors and tickets to all ones (SweepWord::kUnset).
int apply_prec(gales_solver* s, const Ops& o, const double* v, double* z, const int* j, int64_t ld, cudaStream_t st) {
  if (!s->cluster) SCK(s, cudaMemsetAsync(s->d_sweep.p, 0xff, s->d_sweep.n, st), "clear sweep vectors");
  SCK(s, o.sweeps(s, v, z, j, ld, st), "substitutions");
  s->launches += 2;
  return 0;
}

// One Arnoldi pass over w (see arnoldi_kernel); nv = 0 with kSubNorm is hn[0] = ||w||.
template <int MODE>
int arnoldi(gales_solver* s, const double* V, int nv, double* w, double* hn, cudaStream_t st) {
  arnoldi_kernel<MODE><<<s->dot_blocks, kDotThreads, 0, st>>>(V, s->n_rows, nv, w, s->n_rows, s->d_h.p, s->d_h2.p, hn,
                                                             s->d_part.p, s->d_count.p);
  ++s->launches;
  SCK(s, cudaGetLastError(), "Arnoldi step");
  return 0;
}

unsigned stream_grid(int64_t n, int sms) {
  const int64_t b = (n + 255) / 256;
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)sms * 8));
}

// Waits for the stream and reads both status words; the substitutions' word is cleared, so that
// a wait that ran out is reported once.
int read_status(gales_solver* s, cudaStream_t st, unsigned int (&w)[2]) {
  SCK(s, cudaMemcpyAsync(w, s->d_status.p, sizeof(w), cudaMemcpyDeviceToHost, st), "status");
  SCK(s, cudaStreamSynchronize(st), "status");
  if (w[1]) SCK(s, cudaMemsetAsync(s->d_status.p + 1, 0, sizeof(w[1]), st), "clear status");
  return 0;
}

int factorize(gales_solver* s, const Ops& o, const double* vals, cudaStream_t st) {
  if (s->prm.precond == GALES_PRECOND_ILU_FP32)
    SCK(s, cudaMemsetAsync(s->d_Ff.p, 0, s->d_Ff.n * sizeof(float), st), "clear factor");
  else
    SCK(s, cudaMemsetAsync(s->d_F.p, 0, s->d_F.n * sizeof(double), st), "clear factor");
  SCK(s, cudaMemsetAsync(s->d_status.p, 0, sizeof(unsigned int), st), "clear status");
  SCK(s, o.to_factor(s, vals, st), "matrix to factor");
  ++s->launches;
  SCK(s, o.factor(s, st), "factorisation");
  SCK(s, o.scale_diag(s, st), "diagonal blocks");
  unsigned int w[2];
  const int rc = read_status(s, st, w);
  if (rc) return rc;
  if (w[1]) return sfail(s, GALES_ERR_TIMEOUT, "a substitution wait of an earlier apply ran out");
  if (w[0] & GALES_ERR_TIMEOUT) return sfail(s, GALES_ERR_TIMEOUT, "a factorisation wait ran out");
  if (w[0]) return sfail(s, GALES_ERR_SINGULAR, "zero pivot in the incomplete factorisation");
  return 0;
}

int capture_prec_graph(gales_solver* s, const Ops& o) {
  if (s->prec_graph) return 0;
  SCK(s, cudaStreamCreateWithFlags(&s->cap, cudaStreamNonBlocking), "capture stream");
  SCK(s, cudaStreamBeginCapture(s->cap, cudaStreamCaptureModeThreadLocal), "begin capture");
  const int64_t before = s->launches;
  const int rc = apply_prec(s, o, s->d_V.p, s->d_Z.p, s->d_j.p, s->n_rows, s->cap);
  s->launches = before;
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(s->cap, &g);
  if (rc) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  SCK(s, e, "end capture");
  const cudaError_t ei = cudaGraphInstantiate(&s->prec_graph, g, 0);
  cudaGraphDestroy(g);
  SCK(s, ei, "instantiate graph");
  return 0;
}

}  // namespace

extern "C" {

void gales_solver_default(gales_solver_params* p) {
  if (!p) return;
  p->rel_res_tol = 1e-9;
  p->maxsubspace = 200;
  p->maxrestarts = 5;
  p->maxiters = -1;
  p->fill = 1;
  p->precond = GALES_PRECOND_ILU;
}

int gales_iluk_pattern(int64_t n, const int64_t* row_ptr, const int32_t* col, int32_t fill, int64_t* nnz,
                       int64_t* f_row_ptr, int32_t* f_col, int32_t* level_fwd, int32_t* level_bwd,
                       int32_t* n_levels) {
  if (n < 0 || !row_ptr || (n > 0 && !col) || fill < 0 || !nnz) return GALES_ERR_BAD_INPUT;
  std::vector<int64_t> rp, diag, off;
  std::vector<int32_t> fc, lev, rows;
  iluk_symbolic(n, row_ptr, col, fill, rp, fc, diag);
  *nnz = (int64_t)fc.size();
  if (f_row_ptr) std::memcpy(f_row_ptr, rp.data(), sizeof(int64_t) * (n + 1));
  if (f_col) std::memcpy(f_col, fc.data(), sizeof(int32_t) * fc.size());
  level_sets(n, rp, fc, diag, true, lev, off, rows);
  if (level_fwd) std::memcpy(level_fwd, lev.data(), sizeof(int32_t) * n);
  if (n_levels) n_levels[0] = (int32_t)off.size() - 1;
  level_sets(n, rp, fc, diag, false, lev, off, rows);
  if (level_bwd) std::memcpy(level_bwd, lev.data(), sizeof(int32_t) * n);
  if (n_levels) n_levels[1] = (int32_t)off.size() - 1;
  return 0;
}

int gales_solver_create(gales_asm* h, const gales_solver_params* prm, gales_solver** out) {
  if (!h || !out) return GALES_ERR_BAD_INPUT;
  *out = nullptr;
  gales_solver_params p;
  gales_solver_default(&p);
  if (prm) p = *prm;
  if (!(p.rel_res_tol >= 0.0) || p.maxsubspace < 1 || p.maxrestarts < 0 || p.fill < 0 ||
      (p.precond != GALES_PRECOND_ILU && p.precond != GALES_PRECOND_ILU_FP32 && p.precond != GALES_PRECOND_NONE))
    return GALES_ERR_BAD_INPUT;
  int64_t n_nodes = 0, nnz_nodes = 0, n_rows = 0, nnz = 0;
  const int64_t* nrp = nullptr;
  const int32_t* ncol = nullptr;
  int rc = gales_asm_node_graph(h, &n_nodes, &nnz_nodes, &nrp, &ncol);
  if (rc) return rc;
  rc = gales_asm_pattern(h, &n_rows, &nnz, nullptr, nullptr);
  if (rc) return rc;
  if (n_nodes <= 0 || n_rows % n_nodes) return GALES_ERR_BAD_INPUT;
  auto* s = new gales_solver();
  s->prm = p;
  s->nd = (int)(n_rows / n_nodes);
  s->n_nodes = n_nodes;
  s->n_rows = n_rows;
  s->nnz = nnz;
  s->m = p.maxsubspace;
  Ops o;
  if (!ops(s, o)) {
    delete s;
    return GALES_ERR_UNSUPPORTED;
  }
  s->node_rp.assign(nrp, nrp + n_nodes + 1);
  s->node_col.assign(ncol, ncol + nnz_nodes);
  auto bail = [&](int code) {
    gales_solver_destroy(s);
    return code;
  };
  cudaGetDevice(&s->device);
  cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, s->device);
  s->dot_blocks = (int)std::max<int64_t>(1, std::min<int64_t>(4 * s->sms, (n_rows + kTile - 1) / kTile));
  std::vector<int64_t> a2f;
  if (has_ilu(s)) {
    iluk_symbolic(n_nodes, s->node_rp.data(), s->node_col.data(), p.fill, s->f_rp, s->f_col, s->f_diag);
    level_sets(n_nodes, s->f_rp, s->f_col, s->f_diag, true, s->lev_f, s->lev_off_f, s->rows_f);
    level_sets(n_nodes, s->f_rp, s->f_col, s->f_diag, false, s->lev_b, s->lev_off_b, s->rows_b);
    for (int64_t i = 0; i < n_nodes; ++i) {
      s->max_row = std::max(s->max_row, (int)(s->f_rp[i + 1] - s->f_rp[i]));
      s->max_u = std::max(s->max_u, (int)(s->f_rp[i + 1] - s->f_diag[i] - 1));
    }
    a2f.resize(nnz_nodes);
    for (int64_t i = 0; i < n_nodes; ++i) {
      int64_t q = s->f_rp[i];
      for (int64_t t = s->node_rp[i]; t < s->node_rp[i + 1]; ++t) {
        while (s->f_col[q] != s->node_col[t]) ++q;
        a2f[t] = q;
      }
    }
  }
  const size_t bb = (size_t)s->nd * s->nd;
  if (s->d_node_rp.upload(s->node_rp) || s->d_node_col.upload(s->node_col) || s->d_f_rp.upload(s->f_rp) ||
      s->d_f_col.upload(s->f_col) || s->d_f_diag.upload(s->f_diag) || s->d_a2f.upload(a2f) ||
      s->d_rows_f.upload(s->rows_f) || s->d_rows_b.upload(s->rows_b) || (p.precond == GALES_PRECOND_ILU ? s->d_F.alloc(s->f_col.size() * bb)
                                       : s->d_Ff.alloc(s->f_col.size() * bb)) ||
      s->d_V.alloc((size_t)(s->m + 1) * n_rows) || s->d_Z.alloc((size_t)s->m * n_rows) || s->d_w.alloc(n_rows) ||
      s->d_r.alloc(n_rows) || s->d_x.alloc(n_rows) || s->d_part.alloc((size_t)s->dot_blocks * (s->m + 2)) ||
      s->d_h.alloc(s->m + 2) || s->d_h2.alloc(s->m + 2) || s->d_y.alloc(s->m + 2) || s->d_j.alloc(1) ||
      (has_ilu(s) ? s->d_ready.alloc(1 + (size_t)n_nodes) : cudaSuccess) ||
      (has_ilu(s) ? s->d_udiag.alloc((size_t)n_nodes * bb * (p.precond == GALES_PRECOND_ILU ? sizeof(double) : sizeof(float)))
                  : cudaSuccess) ||
      (has_ilu(s) ? s->d_sweep.alloc(2 * (size_t)n_rows * (p.precond == GALES_PRECOND_ILU ? sizeof(double) : sizeof(float)) +
                                     2 * sizeof(unsigned int))
                  : cudaSuccess) || s->d_status.upload(std::vector<unsigned int>(2, 0u)) || s->d_count.upload(std::vector<unsigned int>(1, 0u))) {
    cudaGetLastError();
    return bail(GALES_ERR_NO_MEMORY);
  }
  if (cudaMallocHost(&s->h_buf, sizeof(double) * 2 * (s->m + 2)) != cudaSuccess) {
    cudaGetLastError();
    return bail(GALES_ERR_NO_MEMORY);
  }
  if (has_ilu(s)) {
    cudaDeviceGetAttribute(&s->smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device);
    if (o.prepare(s) != cudaSuccess) {
      cudaGetLastError();
      s->factor_smem = 0;
    }
    s->cluster = o.cluster_size(s);
    if (s->cluster && p.precond == GALES_PRECOND_ILU && s->d_scaled.alloc(s->f_col.size() * bb * sizeof(double))) {
      cudaGetLastError();
      s->cluster = 0;
    }
    rc = capture_prec_graph(s, o);
    if (rc) {
      // plain launches remain available
      cudaGetLastError();
      s->prec_graph = nullptr;
    }
  }
  *out = s;
  return 0;
}

int gales_solver_factorize(gales_solver* s, const double* vals, void* stream) {
  if (!s || !vals) return GALES_ERR_BAD_INPUT;
  if (!has_ilu(s)) return 0;
  SCK(s, cudaSetDevice(s->device), "cudaSetDevice");
  cudaStream_t st = (cudaStream_t)stream;
  const double* dv = vals;
  if (!dev_ptr(vals)) {
    SCK(s, s->d_vals.alloc(s->nnz), "staging values");
    SCK(s, cudaMemcpyAsync(s->d_vals.p, vals, s->nnz * sizeof(double), cudaMemcpyHostToDevice, st), "copy values");
    dv = s->d_vals.p;
  }
  Ops o;
  ops(s, o);
  return factorize(s, o, dv, st);
}

int gales_solver_apply(gales_solver* s, const double* v, double* z, void* stream) {
  if (!s || !v || !z || !dev_ptr(v) || !dev_ptr(z)) return GALES_ERR_BAD_INPUT;
  SCK(s, cudaSetDevice(s->device), "cudaSetDevice");
  cudaStream_t st = (cudaStream_t)stream;
  if (!has_ilu(s)) {
    copy_kernel<<<stream_grid(s->n_rows, s->sms), 256, 0, st>>>(v, z, s->n_rows);
    SCK(s, cudaGetLastError(), "copy");
    return 0;
  }
  Ops o;
  ops(s, o);
  return apply_prec(s, o, v, z, nullptr, 0, st);
}

int gales_solver_sync(gales_solver* s, void* stream) {
  if (!s) return GALES_ERR_BAD_INPUT;
  SCK(s, cudaSetDevice(s->device), "cudaSetDevice");
  unsigned int w[2];
  const int rc = read_status(s, (cudaStream_t)stream, w);
  if (rc) return rc;
  return w[1] ? sfail(s, GALES_ERR_TIMEOUT, "a substitution wait ran out") : 0;
}

int gales_solver_factor(gales_solver* s, int64_t* n_block_rows, int64_t* nnz_blocks, const int64_t** row_ptr,
                        const int32_t** col, double* vals) {
  if (!s) return GALES_ERR_BAD_INPUT;
  if (n_block_rows) *n_block_rows = s->n_nodes;
  if (nnz_blocks) *nnz_blocks = (int64_t)s->f_col.size();
  if (row_ptr) *row_ptr = s->f_rp.data();
  if (col) *col = s->f_col.data();
  if (vals && !s->f_col.empty()) {
    SCK(s, cudaSetDevice(s->device), "cudaSetDevice");
    SCK(s, cudaDeviceSynchronize(), "synchronize");
    const size_t cnt = s->f_col.size() * s->nd * s->nd;
    if (s->prm.precond == GALES_PRECOND_ILU_FP32) {
      std::vector<float> tmp(cnt);
      SCK(s, cudaMemcpy(tmp.data(), s->d_Ff.p, cnt * sizeof(float), cudaMemcpyDeviceToHost), "copy factor");
      for (size_t i = 0; i < cnt; ++i) vals[i] = tmp[i];
    } else {
      SCK(s, cudaMemcpy(vals, s->d_F.p, cnt * sizeof(double), cudaMemcpyDeviceToHost), "copy factor");
    }
  }
  return 0;
}

int gales_solver_levels(gales_solver* s, int32_t* n_levels_fwd, int32_t* n_levels_bwd) {
  if (!s) return GALES_ERR_BAD_INPUT;
  if (n_levels_fwd) *n_levels_fwd = s->lev_off_f.empty() ? 0 : (int32_t)s->lev_off_f.size() - 1;
  if (n_levels_bwd) *n_levels_bwd = s->lev_off_b.empty() ? 0 : (int32_t)s->lev_off_b.size() - 1;
  return 0;
}

int gales_solver_solve(gales_solver* s, const double* vals, const double* rhs, double* x, gales_solver_result* res,
                       void* stream) {
  if (!s || !vals || !rhs || !x) return GALES_ERR_BAD_INPUT;
  const auto t_start = std::chrono::steady_clock::now();
  SCK(s, cudaSetDevice(s->device), "cudaSetDevice");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t n = s->n_rows;
  const int m = s->m;
  const gales_solver_params& p = s->prm;
  const int64_t maxiters = p.maxiters < 0 ? n - 1 : p.maxiters;
  Ops o;
  ops(s, o);
  const double* dA = vals;
  if (!dev_ptr(vals)) {
    SCK(s, s->d_vals.alloc(s->nnz), "staging values");
    SCK(s, cudaMemcpyAsync(s->d_vals.p, vals, s->nnz * sizeof(double), cudaMemcpyHostToDevice, st), "copy values");
    dA = s->d_vals.p;
  }
  const double* db = rhs;
  if (!dev_ptr(rhs)) {
    SCK(s, s->d_b.alloc(n), "staging rhs");
    SCK(s, cudaMemcpyAsync(s->d_b.p, rhs, n * sizeof(double), cudaMemcpyHostToDevice, st), "copy rhs");
    db = s->d_b.p;
  }
  const bool x_dev = dev_ptr(x);
  double* dx = x_dev ? x : s->d_x.p;
  const bool prec = has_ilu(s);
  if (prec) {
    const int rc = factorize(s, o, dA, st);
    if (rc) return rc;
  }
  SCK(s, cudaMemsetAsync(dx, 0, n * sizeof(double), st), "clear x");
  const unsigned sg = stream_grid(n, s->sms);
  double* V = s->d_V.p;
  double* Z = s->d_Z.p;
  double* hb = s->h_buf;
  std::vector<double> H((size_t)(m + 1) * m), cs(m), sn(m), g(m + 1), y(m), h(m + 2);
  // ||b||; r = b (x0 = 0)
  int rc = arnoldi<kSubNorm>(s, nullptr, 0, const_cast<double*>(db), s->d_h.p + m + 1, st);  // db is only read
  if (rc) return rc;
  SCK(s, cudaMemcpyAsync(hb, s->d_h.p + m + 1, sizeof(double), cudaMemcpyDeviceToHost, st), "norm");
  SCK(s, cudaStreamSynchronize(st), "norm");
  const double bnorm = hb[0];
  double beta = bnorm;
  const double* r = db;
  int64_t iters = 0;
  int cycles = 0;
  bool converged = bnorm == 0.0;
  while (!converged && cycles <= p.maxrestarts && iters < maxiters && beta > 0.0) {
    ++cycles;
    // V0 = r / beta (beta on the device in d_h[m+1])
    scale_kernel<<<sg, 256, 0, st>>>(r, s->d_h.p + m + 1, V, n);
    ++s->launches;
    std::fill(g.begin(), g.end(), 0.0);
    g[0] = beta;
    int j = 0;
    bool est_conv = false;
    for (; j < m && iters < maxiters; ++j) {
      double* vj = V + (int64_t)j * n;
      double* zj = Z + (int64_t)j * n;
      if (prec) {
        if (s->prec_graph) {
          set_index_kernel<<<1, 1, 0, st>>>(s->d_j.p, j);
          SCK(s, cudaGraphLaunch(s->prec_graph, st), "preconditioner graph");
          s->launches += 3;
        } else {
          rc = apply_prec(s, o, vj, zj, nullptr, 0, st);
          if (rc) return rc;
        }
      } else {
        copy_kernel<<<sg, 256, 0, st>>>(vj, zj, n);
        ++s->launches;
      }
      SCK(s, o.spmv(s, dA, zj, nullptr, s->d_w.p, st), "spmv");
      ++s->launches;
      // two classical Gram-Schmidt passes: h = V^T w, w -= V h (twice; h summed)
      rc = arnoldi<kDots>(s, V, j + 1, s->d_w.p, nullptr, st);
      if (rc) return rc;
      rc = arnoldi<kSubDots>(s, V, j + 1, s->d_w.p, nullptr, st);
      if (rc) return rc;
      rc = arnoldi<kSubNorm>(s, V, j + 1, s->d_w.p, s->d_h.p + j + 1, st);
      if (rc) return rc;
      scale_kernel<<<sg, 256, 0, st>>>(s->d_w.p, s->d_h.p + j + 1, V + (int64_t)(j + 1) * n, n);
      ++s->launches;
      SCK(s, cudaGetLastError(), "Arnoldi step");
      SCK(s, cudaMemcpyAsync(hb, s->d_h.p, (j + 2) * sizeof(double), cudaMemcpyDeviceToHost, st), "Hessenberg");
      SCK(s, cudaStreamSynchronize(st), "Arnoldi step");
      for (int c = 0; c <= j + 1; ++c) h[c] = hb[c];
      const double hn = h[j + 1];
      for (int c = 0; c < j; ++c) {
        const double t = cs[c] * h[c] + sn[c] * h[c + 1];
        h[c + 1] = -sn[c] * h[c] + cs[c] * h[c + 1];
        h[c] = t;
      }
      const double d = std::hypot(h[j], h[j + 1]);
      cs[j] = d > 0.0 ? h[j] / d : 1.0;
      sn[j] = d > 0.0 ? h[j + 1] / d : 0.0;
      h[j] = d;
      h[j + 1] = 0.0;
      g[j + 1] = -sn[j] * g[j];
      g[j] = cs[j] * g[j];
      for (int c = 0; c <= j; ++c) H[(size_t)c * m + j] = h[c];
      ++iters;
      if (std::fabs(g[j + 1]) <= p.rel_res_tol * bnorm || hn == 0.0) {
        est_conv = true;
        ++j;
        break;
      }
    }
    for (int c = j - 1; c >= 0; --c) {
      double sum = g[c];
      for (int t = c + 1; t < j; ++t) sum -= H[(size_t)c * m + t] * y[t];
      y[c] = sum / H[(size_t)c * m + c];
    }
    for (int c = 0; c < j; ++c) hb[m + 2 + c] = y[c];
    SCK(s, cudaMemcpyAsync(s->d_y.p, hb + m + 2, j * sizeof(double), cudaMemcpyHostToDevice, st), "solution");
    update_x_kernel<<<sg, 256, j * sizeof(double), st>>>(Z, n, j, s->d_y.p, dx, n);
    // r = b - A x, beta = ||r||
    SCK(s, o.spmv(s, dA, dx, db, s->d_r.p, st), "residual");
    s->launches += 2;
    rc = arnoldi<kSubNorm>(s, nullptr, 0, s->d_r.p, s->d_h.p + m + 1, st);
    if (rc) return rc;
    SCK(s, cudaMemcpyAsync(hb, s->d_h.p + m + 1, sizeof(double), cudaMemcpyDeviceToHost, st), "residual norm");
    SCK(s, cudaStreamSynchronize(st), "residual");
    beta = hb[0];
    r = s->d_r.p;
    if (est_conv && beta <= p.rel_res_tol * bnorm) converged = true;
  }
  if (!x_dev) {
    SCK(s, cudaMemcpyAsync(x, dx, n * sizeof(double), cudaMemcpyDeviceToHost, st), "copy x");
    SCK(s, cudaStreamSynchronize(st), "copy x");
  }
  if (prec) {  // a substitution wait that ran out (not expected on a working device)
    unsigned int w[2];
    rc = read_status(s, st, w);
    if (rc) return rc;
    if (w[1]) return sfail(s, GALES_ERR_TIMEOUT, "a substitution wait ran out");
  }
  if (res) {
    res->iterations = iters;
    res->abs_res = beta;
    res->rel_res = bnorm > 0.0 ? beta / bnorm : 0.0;
    res->converged = converged ? 1 : 0;
    res->cycles = cycles;
    res->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
  }
  return 0;
}

int gales_solver_correct(gales_solver* s, double* I, const double* dx, int32_t trim_first, int32_t trim_last,
                         double lo, double hi, void* stream) {
  if (!s || !I || !dx || !dev_ptr(I) || !dev_ptr(dx)) return GALES_ERR_BAD_INPUT;
  SCK(s, cudaSetDevice(s->device), "cudaSetDevice");
  cudaStream_t st = (cudaStream_t)stream;
  correct_kernel<<<stream_grid(s->n_rows, s->sms), 256, 0, st>>>(I, dx, s->n_rows, s->nd, trim_first, trim_last, lo,
                                                                  hi);
  ++s->launches;
  SCK(s, cudaGetLastError(), "correct");
  return 0;
}

int64_t gales_solver_launches(gales_solver* s) { return s ? s->launches : 0; }

const char* gales_solver_last_error(gales_solver* s) { return s ? s->err.c_str() : "null handle"; }

void gales_solver_destroy(gales_solver* s) {
  if (!s) return;
  cudaSetDevice(s->device);
  if (s->prec_graph) cudaGraphExecDestroy(s->prec_graph);
  if (s->cap) cudaStreamDestroy(s->cap);
  if (s->h_buf) cudaFreeHost(s->h_buf);
  for (auto* b : {&s->d_node_rp, &s->d_f_rp, &s->d_f_diag, &s->d_a2f}) b->release();
  for (auto* b : {&s->d_node_col, &s->d_f_col, &s->d_rows_f, &s->d_rows_b}) b->release();
  s->d_Ff.release();
  for (auto* b : {&s->d_F, &s->d_V, &s->d_Z, &s->d_w, &s->d_r, &s->d_x, &s->d_part, &s->d_h, &s->d_h2, &s->d_y,
                  &s->d_vals, &s->d_b})
    b->release();
  s->d_j.release();
  s->d_ready.release();
  s->d_sweep.release();
  s->d_udiag.release();
  s->d_scaled.release();
  s->d_status.release();
  s->d_count.release();
  delete s;
}

}  // extern "C"
