// Host build of the assembly's form of the magma mixture (gales_magma_fast.cuh) beside the
// property code it rearranges (gales_magma.cuh), for the CPU tests.
#include <cstdint>
#include <vector>

#include "../../gales-multi-fluid_gb300/csrc/gales_magma_fast.cuh"

using namespace magma_mix;

// which 0: mix_point, 1: fast::mix_point, 2: fast::mix_rho_cv (out rows 0 and 3); st[i] the
// status bits of point i
extern "C" void magma_fast_host(const gales_magma_desc* comps, int32_t nc, const double* p, const double* T,
                                const double* Y, const double* shear, int64_t n, int which, double* out, double* comp,
                                int32_t* st) {
  std::vector<DevMagma> mg(nc);
  for (int c = 0; c < nc; ++c) {
    build_constants(comps[c], mg[c]);
    mg[c].p_tab = comps[c].p_table;
    mg[c].T_tab = comps[c].n_T > 0 ? comps[c].T_table : nullptr;
    mg[c].h2o_tab = comps[c].wf_l_h2o;
    mg[c].co2_tab = comps[c].wf_l_co2;
  }
  for (int64_t i = 0; i < n; ++i) {
    double f[8] = {}, cc[GALES_MAX_COMP][4] = {};
    const double* y = Y + i * nc;
    st[i] = (int32_t)(which == 0   ? mix_point(mg.data(), nc, p[i], T[i], y, shear[i], f, cc)
                      : which == 1 ? fast::mix_point(mg.data(), nc, p[i], T[i], y, shear[i], f, cc)
                                   : fast::mix_rho_cv(mg.data(), nc, p[i], T[i], y, f[0], f[3]));
    for (int k = 0; k < 8; ++k) out[k * n + i] = f[k];
    for (int c = 0; c < nc; ++c)
      for (int k = 0; k < 4; ++k) comp[(c * 4 + k) * n + i] = cc[c][k];
  }
}
