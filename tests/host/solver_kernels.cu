// The solver's bounded waits: each kernel with the rows it waits for left out of its list, and how
// a wait that ran out reaches the caller.  The solver's source is compiled here over a node graph
// of its own (a band), without an assembly.
#include "../../gales-multi-fluid_gb300/csrc/gales_solver.cu"

namespace {
constexpr int kNodes = 40, kBand = 8, kNd = 8;
std::vector<int64_t> g_rp;
std::vector<int32_t> g_col;
}  // namespace

extern "C" int gales_asm_node_graph(gales_asm*, int64_t* n, int64_t* nnz, const int64_t** rp, const int32_t** col) {
  g_rp.assign(1, 0);
  g_col.clear();
  for (int i = 0; i < kNodes; ++i) {
    for (int j = std::max(0, i - kBand); j < std::min(kNodes, i + kBand + 1); ++j) g_col.push_back(j);
    g_rp.push_back((int64_t)g_col.size());
  }
  *n = kNodes;
  *nnz = (int64_t)g_col.size();
  *rp = g_rp.data();
  *col = g_col.data();
  return 0;
}
extern "C" int gales_asm_pattern(gales_asm*, int64_t* n_rows, int64_t* nnz, const int64_t**, const int32_t**) {
  *n_rows = kNodes * kNd;
  *nnz = (int64_t)g_col.size() * kNd * kNd;
  return 0;
}

namespace {
struct System {
  gales_solver* s = nullptr;
  double *v = nullptr, *z = nullptr;
  std::vector<double> vals;
  System() {
    gales_solver_params p;
    gales_solver_default(&p);
    p.fill = 0;
    if (gales_solver_create(reinterpret_cast<gales_asm*>(&p), &p, &s)) return;
    for (int i = 0; i < kNodes; ++i) {
      const int64_t t0 = g_rp[i], len = (g_rp[i + 1] - t0) * kNd;
      for (int k = 0; k < kNd; ++k)
        for (int64_t e = 0; e < len; ++e)
          vals.push_back(g_col[t0 + e / kNd] == i && e % kNd == k ? 100.0 : 0.1);
    }
    cudaMalloc(&v, kNodes * kNd * sizeof(double));
    cudaMalloc(&z, kNodes * kNd * sizeof(double));
    cudaMemset(v, 0, kNodes * kNd * sizeof(double));
  }
  ~System() {
    gales_solver_destroy(s);
    cudaFree(v);
    cudaFree(z);
  }
  void set_word() {
    const unsigned int bit = GALES_ERR_TIMEOUT;
    cudaMemcpy(s->d_status.p + 1, &bit, sizeof(bit), cudaMemcpyHostToDevice);
  }
};
}  // namespace

// out: the codes of sync, sync, factorize, factorize, solve, solve after each pair's first call
// finds the substitutions' word set
extern "C" int solver_reports(int* out) {
  System y;
  if (!y.s || gales_solver_factorize(y.s, y.vals.data(), nullptr)) return 1;
  std::vector<double> b(kNodes * kNd, 1.0), x(b.size());
  for (int i = 0; i < 6; ++i) {
    if (i % 2 == 0) y.set_word();
    out[i] = i < 2   ? gales_solver_sync(y.s, nullptr)
             : i < 4 ? gales_solver_factorize(y.s, y.vals.data(), nullptr)
                     : gales_solver_solve(y.s, y.vals.data(), b.data(), x.data(), nullptr, nullptr);
  }
  return cudaGetLastError() != cudaSuccess;
}

// kernel 0: factorisation, 1: lower substitution through L2, 2: in a cluster, with the first kBand
// rows never taken; returns the status word's value, -1 on a CUDA error
extern "C" int solver_wait_runs_out(int kernel) {
  using K = Kernels<kNd, double>;
  System y;
  gales_solver* s = y.s;
  if (!s || gales_solver_factorize(s, y.vals.data(), nullptr)) return -1;
  const int64_t n = kNodes - kBand;
  const int32_t* rows = s->d_rows_f.p + kBand;   // a band's levels are its rows
  double* t = reinterpret_cast<double*>(s->d_sweep.p);
  cudaMemset(s->d_sweep.p, 0xff, s->d_sweep.n);
  if (kernel == 0) {
    if (!s->factor_smem) return -1;
    cudaMemset(s->d_ready.p, 0, s->d_ready.n * sizeof(int));
    ilu_factor_rows_kernel<kNd, double><<<4, kFactorThreads, s->factor_smem>>>(
        s->d_F.p, s->d_f_rp.p, s->d_f_col.p, s->d_f_diag.p, rows, n, reinterpret_cast<unsigned int*>(s->d_ready.p),
        s->d_ready.p + 1, s->d_status.p + 1, s->max_row, s->max_u);
  } else if (kernel == 1) {
    unsigned int* tk = reinterpret_cast<unsigned int*>(t + 2 * s->n_rows);
    ilu_sweep_kernel<kNd, double, true><<<2, 32 * kSweepWarps>>>(
        s->d_F.p, s->d_f_rp.p, s->d_f_col.p, s->d_f_diag.p, nullptr, rows, n, y.v, nullptr, t, nullptr, nullptr, 0, tk,
        s->d_status.p + 1);
  } else {
    int size = 8;
    if (K::prepare_cluster<true>(s, size) != cudaSuccess || !size) return -1;
    // the kernel polls n nd words of its shared memory: the whole vector, rows from kBand on
    const K::ClusterLaunch l((unsigned)size, K::cluster_smem(s), nullptr);
    std::vector<int32_t> order(kNodes, kNodes - 1);   // the last row again for the rows left out
    for (int i = 0; i < n; ++i) order[i] = kBand + i;
    cudaMemcpy(s->d_rows_f.p, order.data(), order.size() * sizeof(int32_t), cudaMemcpyHostToDevice);
    cudaLaunchKernelEx(&l.cfg, ilu_sweep_cluster_kernel<kNd, double, true>, (const double*)s->d_F.p,
                       (const int64_t*)s->d_f_rp.p, (const int32_t*)s->d_f_col.p, (const int64_t*)s->d_f_diag.p,
                       (const double*)s->d_F.p, (const int32_t*)s->d_rows_f.p, s->n_nodes, (const double*)y.v, t,
                       (double*)nullptr, (const int*)nullptr, (int64_t)0, s->d_status.p + 1);
  }
  unsigned int w = 0;
  if (cudaMemcpy(&w, s->d_status.p + 1, sizeof(w), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  return (int)w;
}

// The three Arnoldi passes over nv columns of n rows (V column-major): out_h = V^T w, then w,
// out_h2 and out_h of kSubDots, then w and the norm of kSubNorm; 0 or a CUDA error.
extern "C" int solver_arnoldi(const double* V, int64_t n, int nv, double* w, double* h, double* h1, double* h2, double* w1,
                              double* hn) {
  const int blocks = (int)((n + kTile - 1) / kTile);
  double *dV, *dw, *dh, *dh2, *dn, *part;
  unsigned int* count;
  cudaMalloc(&dV, (size_t)n * nv * 8);
  cudaMalloc(&dw, n * 8);
  cudaMalloc(&dh, nv * 8);
  cudaMalloc(&dh2, nv * 8);
  cudaMalloc(&dn, 8);
  cudaMalloc(&part, (size_t)blocks * nv * 8);
  cudaMalloc(&count, sizeof(unsigned int));
  cudaMemset(count, 0, sizeof(unsigned int));
  cudaMemcpy(dV, V, (size_t)n * nv * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(dw, w, n * 8, cudaMemcpyHostToDevice);
  arnoldi_kernel<kDots><<<blocks, kDotThreads>>>(dV, n, nv, dw, n, dh, dh2, nullptr, part, count);
  cudaMemcpy(h, dh, nv * 8, cudaMemcpyDeviceToHost);
  arnoldi_kernel<kSubDots><<<blocks, kDotThreads>>>(dV, n, nv, dw, n, dh, dh2, nullptr, part, count);
  cudaMemcpy(h1, dh, nv * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(h2, dh2, nv * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(w1, dw, n * 8, cudaMemcpyDeviceToHost);
  arnoldi_kernel<kSubNorm><<<blocks, kDotThreads>>>(dV, n, nv, dw, n, dh, dh2, dn, part, count);
  cudaMemcpy(w, dw, n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(hn, dn, 8, cudaMemcpyDeviceToHost);
  for (void* p : {(void*)dV, (void*)dw, (void*)dh, (void*)dh2, (void*)dn, (void*)part, (void*)count}) cudaFree(p);
  return (int)cudaGetLastError();
}
