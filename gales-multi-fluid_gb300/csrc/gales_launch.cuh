// Kernel dispatch for one element type (DIM, NEN): picks the template instance for
// the number of components and the numerical form.  Each (element type, form)
// pair lives in its own translation unit (gales_<type>_<form>.cu) so the library
// builds in parallel; the boundary kernels are in the FP64 unit.
#pragma once

#include <type_traits>

#include "gales_fp64.cuh"
#include "gales_rows32.cuh"

namespace gales {

struct LaunchResult {
  cudaError_t err;
  int launches;
};

// Whether some node flag blocks a dof.
inline bool any_dirichlet(const KParams& k) {
  uint32_t any = 0u;
  for (int f = 0; f < GALES_MAX_FLAGS; ++f) any |= k.dirichlet_mask[f];
  return any != 0u;
}

// The mixed form (gales_kernels.cuh, gales_rows32.cuh).
template <int DIM, int NEN, int NC, int NQ, int EOS = kEosChemicals>
struct InteriorInst {
  using S = float;
  using Rec = QP<DIM, NEN, NC, S>;
  using RB = RecBlock<DIM, NEN, NC>;
  using T = Rows32<DIM, NEN, NC>;
  // record bytes per element and elements per block of records: a chunk of n elements needs
  // at most (n + rec_block()) rec_bytes()
  static size_t rec_bytes() { return RB::BYTES / RB::EB; }
  static int rec_block() { return RB::EB; }
  static LaunchResult point(const KParams& k, bool, void* buf, long long first, long long n, cudaStream_t st) {
    if (n <= 0) return {cudaSuccess, 0};
    const long long threads = n * NQ;
    point_kernel<DIM, NEN, NC, NQ, S, EOS><<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(
        k, reinterpret_cast<Rec*>(buf), first, n);
    return {cudaGetLastError(), 1};
  }
  static cudaError_t prepare() { return cudaSuccess; }
  static LaunchResult matrix(const KParams& k, bool want_m, void* buf, long long first, long long n,
                             cudaStream_t st) {
    if (n <= 0) return {cudaSuccess, 0};
    const unsigned ctas = (unsigned)((n + RB::EB - 1) / RB::EB * T::ND);
    unsigned char* in = reinterpret_cast<unsigned char*>(buf);
    if (!want_m) {
      rows32_kernel<DIM, NEN, NC, false><<<ctas, T::THREADS, 0, st>>>(k, in, first, n);
      return {cudaGetLastError(), 1};
    }
    rows32_kernel<DIM, NEN, NC, true><<<ctas, T::THREADS, 0, st>>>(k, in, first, n);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !any_dirichlet(k) || k.local_r) return {e, 1};
    dirichlet32_kernel<DIM, NEN, NC><<<(unsigned)((n + RB::EB - 1) / RB::EB), 32 * NEN, 0, st>>>(k, in, n);
    return {cudaGetLastError(), 2};
  }
};

// The blocked rows' diagonal after the FP64 matrix stage, where some flag blocks a dof and the
// blocks are scattered or contracted; counts the matrix launch too.
template <int DIM, int NEN, int NC>
LaunchResult dirichlet64(const KParams& k, const double* in, long long n, cudaStream_t st) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !any_dirichlet(k) || k.local_r) return {e, 1};
  dirichlet64_kernel<DIM, NEN, NC><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(k, in, n);
  return {cudaGetLastError(), 2};
}

// The FP64 form of a simplex (gales_fp64.cuh).
template <int DIM, int NC, int EOS>
struct Simplex64Inst {
  static constexpr int NEN = DIM + 1;
  using R = Rec64<DIM, NEN, NC>;
  static constexpr size_t kSmem = sizeof(Rows64Smem<DIM, NC>);
  static size_t rec_bytes() { return R::ELEM_BYTES; }
  static int rec_block() { return R::EB; }
  static cudaError_t prepare() {
    return cudaFuncSetAttribute(rows64_kernel<DIM, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kRows64Warps * kSmem));
  }
  static LaunchResult point(const KParams& k, bool want_m, void* buf, long long first, long long n, cudaStream_t st) {
    if (n <= 0) return {cudaSuccess, 0};
    const unsigned blocks = (unsigned)((n * NEN + 127) / 128);
    double* out = reinterpret_cast<double*>(buf);
    if (want_m) point64_kernel<DIM, NEN, NC, EOS, true><<<blocks, 128, 0, st>>>(k, out, first, n);
    else point64_kernel<DIM, NEN, NC, EOS, false><<<blocks, 128, 0, st>>>(k, out, first, n);
    return {cudaGetLastError(), 1};
  }
  static LaunchResult matrix(const KParams& k, bool want_m, void* buf, long long first, long long n, cudaStream_t st) {
    if (n <= 0) return {cudaSuccess, 0};
    double* in = reinterpret_cast<double*>(buf);
    const long long tasks = (n + R::EB - 1) / R::EB * R::ND;   // a warp each
    if (!want_m) {
      residual64_kernel<DIM, NEN, NC><<<(unsigned)((tasks + 3) / 4), 128, 0, st>>>(k, in, first, n);
      return {cudaGetLastError(), 1};
    }
    const int w = tasks < 16ll * k.sms ? 1 : kRows64Warps;   // see rows64_kernel
    const long long nblk = (n + R::EB - 1) / R::EB, ncta = (nblk + w - 1) / w * R::ND;
    rows64_kernel<DIM, NC><<<(unsigned)ncta, 32 * w, w * kSmem, st>>>(k, in, first, n);
    return dirichlet64<DIM, NEN, NC>(k, in, n, st);
  }
};

// The FP64 form of a quadrilateral or hexahedron (gales_fp64.cuh).
template <int DIM, int NC, int EOS>
struct Tensor64Inst {
  using T = Tensor64<DIM, NC>;
  using R = typename T::R;
  static constexpr int NEN = T::NEN;
  static constexpr size_t kSmem = sizeof(typename T::Smem);
  static size_t rec_bytes() { return R::ELEM_BYTES; }
  static int rec_block() { return R::EB; }
  static cudaError_t prepare() {
    return cudaFuncSetAttribute(tensor64_kernel<DIM, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  }
  static LaunchResult point(const KParams& k, bool want_m, void* buf, long long first, long long n, cudaStream_t st) {
    if (n <= 0) return {cudaSuccess, 0};
    const unsigned blocks = (unsigned)((n * NEN + 127) / 128);
    double* out = reinterpret_cast<double*>(buf);
    if (want_m) point64_kernel<DIM, NEN, NC, EOS, true><<<blocks, 128, 0, st>>>(k, out, first, n);
    else point64_kernel<DIM, NEN, NC, EOS, false><<<blocks, 128, 0, st>>>(k, out, first, n);
    return {cudaGetLastError(), 1};
  }
  static LaunchResult matrix(const KParams& k, bool want_m, void* buf, long long first, long long n, cudaStream_t st) {
    if (n <= 0) return {cudaSuccess, 0};
    double* in = reinterpret_cast<double*>(buf);
    if (!want_m) {
      const long long threads = (n + R::EB - 1) / R::EB * R::ND * R::EB;
      residual64_kernel<DIM, NEN, NC><<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(k, in, first, n);
      return {cudaGetLastError(), 1};
    }
    tensor64_kernel<DIM, NC><<<(unsigned)n, T::THREADS, kSmem, st>>>(k, in, first, n);
    return dirichlet64<DIM, NEN, NC>(k, in, n, st);
  }
};

template <int DIM, int NEN, int NC, int NS, int NSQ, typename S, int EOS = kEosChemicals>
cudaError_t prepare_boundary_nc() {
  return cudaFuncSetAttribute(boundary_kernel<DIM, NEN, NC, NS, NSQ, S, EOS>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sizeof(BoundarySmem<DIM, NEN, NC, NS, NSQ, S>));
}

// Boundary pass: with point records (k.bpt_rec) the point stage runs first, one thread
// per flagged side point; the element stage then reads the records.  k.bd_stage 1 launches the
// point stage alone, 2 the element stage alone.
template <int DIM, int NEN, int NC, int NS, int NSQ, typename S, int EOS = kEosChemicals>
LaunchResult launch_boundary_nc(const KParams& k, long long n_items, cudaStream_t st) {
  if (n_items == 0) return {cudaSuccess, 0};
  int launches = 0;
  if (k.bpt_rec && k.n_bpt > 0 && k.bd_stage != 2) {
    bpoint_kernel<DIM, NEN, NC, NS, NSQ, S, EOS><<<(unsigned)((k.n_bpt + 127) / 128), 128, 0, st>>>(k);
    ++launches;
  }
  if (k.bd_stage == 1) return {cudaGetLastError(), launches};
  const size_t smem = k.bpt_rec ? 0 : sizeof(BoundarySmem<DIM, NEN, NC, NS, NSQ, S>);
  boundary_kernel<DIM, NEN, NC, NS, NSQ, S, EOS><<<(unsigned)n_items, boundary_threads<NC, DIM>(), smem, st>>>(k);
  return {cudaGetLastError(), launches + 1};
}

// Interior operations of one (element type, form): record bytes per element, point
// stage and matrix stage, for 1..4 components.
struct InteriorOps {
  cudaError_t (*prepare)(int nc);
  size_t (*rec_bytes)(int nc);
  int (*rec_block)(int nc);
  LaunchResult (*point)(const KParams&, int nc, bool want_m, void* buf, long long first, long long n, cudaStream_t);
  LaunchResult (*matrix)(const KParams&, int nc, bool want_m, void* buf, long long first, long long n, cudaStream_t);
};

#define GALES_NC_SWITCH(expr_nc, CALL) \
  switch (expr_nc) {                   \
    case 1: CALL(1);                   \
    case 2: CALL(2);                   \
    case 3: CALL(3);                   \
    case 4: CALL(4);                   \
    default: break;                    \
  }

template <int DIM, int NEN, int NC, int NQ, int FORM, int EOS>
using InteriorOf = typename std::conditional<
    FORM == GALES_FORM_MIXED, InteriorInst<DIM, NEN, NC, NQ, EOS>,
    typename std::conditional<NEN == DIM + 1, Simplex64Inst<DIM, NC, EOS>, Tensor64Inst<DIM, NC, EOS>>::type>::type;

template <int DIM, int NEN, int NQ, int FORM, int EOS = kEosChemicals>
struct InteriorDispatch {
  template <int NC>
  using I = InteriorOf<DIM, NEN, NC, NQ, FORM, EOS>;
  static cudaError_t prepare(int nc) {
#define GALES_C(NC) return I<NC>::prepare()
    GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
    return cudaErrorInvalidValue;
  }
  static size_t rec_bytes(int nc) {
#define GALES_C(NC) return I<NC>::rec_bytes()
    GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
    return 0;
  }
  static int rec_block(int nc) {
#define GALES_C(NC) return I<NC>::rec_block()
    GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
    return 4;
  }
  static LaunchResult point(const KParams& k, int nc, bool want_m, void* buf, long long first, long long n,
                            cudaStream_t st) {
#define GALES_C(NC) return I<NC>::point(k, want_m, buf, first, n, st)
    GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
    return {cudaErrorInvalidValue, 0};
  }
  static LaunchResult matrix(const KParams& k, int nc, bool want_m, void* buf, long long first, long long n,
                             cudaStream_t st) {
#define GALES_C(NC) return I<NC>::matrix(k, want_m, buf, first, n, st)
    GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
    return {cudaErrorInvalidValue, 0};
  }
  static InteriorOps ops() { return {&prepare, &rec_bytes, &rec_block, &point, &matrix}; }
};

// Boundary pass of one element type; S is the matrix arithmetic type of the form.
// n < 0 only prepares the kernel (shared-memory limit) and launches nothing.
template <int DIM, int NEN, int NS, int NSQ, typename S, int EOS = kEosChemicals>
LaunchResult boundary_dispatch(const KParams& k, int nc, long long n, cudaStream_t st) {
  if (n < 0) {
#define GALES_C(NC) return {prepare_boundary_nc<DIM, NEN, NC, NS, NSQ, S, EOS>(), 0}
    GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
    return {cudaErrorInvalidValue, 0};
  }
#define GALES_C(NC) return launch_boundary_nc<DIM, NEN, NC, NS, NSQ, S, EOS>(k, n, st)
  GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
  return {cudaErrorInvalidValue, 0};
}

// Adaptive time step (f_mc) per element of one element type.
template <int DIM, int NEN, int NQ, int EOS = kEosChemicals>
LaunchResult adaptive_dt_dispatch(const KParams& k, int nc, double cfl, double* dt_el, long long n, cudaStream_t st) {
  if (n <= 0) return {cudaSuccess, 0};
  const unsigned blocks = (unsigned)((n + 127) / 128);
#define GALES_C(NC)                                                                       \
  adaptive_dt_kernel<DIM, NEN, NC, NQ, EOS><<<blocks, 128, 0, st>>>(k, cfl, dt_el, n); \
  return {cudaGetLastError(), 1}
  GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
  return {cudaErrorInvalidValue, 0};
}

// Secondary variables at the nodes (any element type of the dimension).
template <int DIM, int EOS = kEosChemicals>
LaunchResult secondary_dofs_dispatch(const KParams& k, int nc, double* out, long long n, cudaStream_t st) {
  if (n <= 0) return {cudaSuccess, 0};
  const unsigned blocks = (unsigned)((n + 127) / 128);
#define GALES_C(NC)                                                            \
  secondary_dofs_kernel<DIM, NC, EOS><<<blocks, 128, 0, st>>>(k, out, n); \
  return {cudaGetLastError(), 1}
  GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
  return {cudaErrorInvalidValue, 0};
}

// Magma gas fractions at the nodes (pp_vf_g).
template <int DIM>
LaunchResult magma_fractions_dispatch(const KParams& k, int nc, double* out, long long n, cudaStream_t st) {
  if (n <= 0) return {cudaSuccess, 0};
  const unsigned blocks = (unsigned)((n + 127) / 128);
#define GALES_C(NC)                                                            \
  magma_fractions_kernel<DIM, NC><<<blocks, 128, 0, st>>>(k, out, n); \
  return {cudaGetLastError(), 1}
  GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
  return {cudaErrorInvalidValue, 0};
}

// Every kernel of one element type compiled with the magma EOS (gales_<type>_magma.cu).
struct MagmaOps {
  InteriorOps interior[2];   // per form (FP64, mixed)
  LaunchResult (*boundary)(const KParams&, int nc, int form, long long n, cudaStream_t);
  LaunchResult (*adaptive_dt)(const KParams&, int nc, double cfl, double* dt_el, long long n, cudaStream_t);
  LaunchResult (*secondary_dofs)(const KParams&, int nc, double* out, long long n, cudaStream_t);
  LaunchResult (*fractions)(const KParams&, int nc, double* out, long long n, cudaStream_t);
};

// Boundary side-point geometry (handle creation) and record sizes.
struct BoundaryInfo {
  size_t bgeo_bytes;
  size_t rec_bytes[2];   // per form (FP64, mixed)
  LaunchResult (*geometry)(const KParams& k, void* out, cudaStream_t st);
};

template <int DIM, int NEN, int NS, int NSQ>
struct BoundaryInfoDispatch {
  static LaunchResult geometry(const KParams& k, void* out, cudaStream_t st) {
    if (k.n_bpt <= 0) return {cudaSuccess, 0};
    bgeo_kernel<DIM, NEN, NS, NSQ><<<(unsigned)((k.n_bpt + 127) / 128), 128, 0, st>>>(
        k, reinterpret_cast<BGeo<DIM, NEN>*>(out));
    return {cudaGetLastError(), 1};
  }
  static BoundaryInfo info(int nc) {
    BoundaryInfo b{sizeof(BGeo<DIM, NEN>), {0, 0}, &geometry};
#define GALES_C(NC)                                                      \
  b.rec_bytes[0] = sizeof(BPointRec<DIM, NEN, NC, double>);            \
  b.rec_bytes[1] = sizeof(BPointRec<DIM, NEN, NC, float>);             \
  break
    GALES_NC_SWITCH(nc, GALES_C)
#undef GALES_C
    return b;
  }
};

// Element geometry precompute (handle creation).
struct GeometryOps {
  size_t bytes_per_element;
  LaunchResult (*launch)(const double* coords, const int32_t* conn, const KParams& k, void* out, long long n_el,
                         cudaStream_t st);
};

template <int DIM, int NEN, int NQ>
struct GeometryDispatch {
  static constexpr int NG = geo_per_element<DIM, NEN>(NQ);
  static LaunchResult launch(const double* coords, const int32_t* conn, const KParams& k, void* out, long long n_el,
                             cudaStream_t st) {
    if (n_el <= 0) return {cudaSuccess, 0};
    const long long threads = n_el * NG;
    geometry_kernel<DIM, NEN, NQ><<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(
        coords, conn, k, reinterpret_cast<ElemGeo<DIM, NEN>*>(out), n_el);
    return {cudaGetLastError(), 1};
  }
  static GeometryOps ops() { return {sizeof(ElemGeo<DIM, NEN>) * NG, &launch}; }
};

// Entry points defined by the per-element translation units.
InteriorOps interior_ops_tri3_fp64();
InteriorOps interior_ops_tri3_mixed();
LaunchResult boundary_tri3(const KParams&, int nc, int form, long long n, cudaStream_t);
LaunchResult boundary_tri3_mixed(const KParams&, int nc, long long n, cudaStream_t);
GeometryOps geometry_ops_tri3();
BoundaryInfo boundary_info_tri3(int nc);
LaunchResult adaptive_dt_tri3(const KParams&, int nc, double cfl, double* dt_el, long long n, cudaStream_t);
LaunchResult secondary_dofs_2d(const KParams&, int nc, double* out, long long n, cudaStream_t);
InteriorOps interior_ops_quad4_fp64();
InteriorOps interior_ops_quad4_mixed();
LaunchResult boundary_quad4(const KParams&, int nc, int form, long long n, cudaStream_t);
LaunchResult boundary_quad4_mixed(const KParams&, int nc, long long n, cudaStream_t);
GeometryOps geometry_ops_quad4();
BoundaryInfo boundary_info_quad4(int nc);
LaunchResult adaptive_dt_quad4(const KParams&, int nc, double cfl, double* dt_el, long long n, cudaStream_t);
InteriorOps interior_ops_tet4_fp64();
InteriorOps interior_ops_tet4_mixed();
LaunchResult boundary_tet4(const KParams&, int nc, int form, long long n, cudaStream_t);
LaunchResult boundary_tet4_mixed(const KParams&, int nc, long long n, cudaStream_t);
GeometryOps geometry_ops_tet4();
BoundaryInfo boundary_info_tet4(int nc);
LaunchResult adaptive_dt_tet4(const KParams&, int nc, double cfl, double* dt_el, long long n, cudaStream_t);
LaunchResult secondary_dofs_3d(const KParams&, int nc, double* out, long long n, cudaStream_t);
InteriorOps interior_ops_hex8_fp64();
InteriorOps interior_ops_hex8_mixed();
LaunchResult boundary_hex8(const KParams&, int nc, int form, long long n, cudaStream_t);
// exact VJP kernels (gales_vjp_<type>.cu)
LaunchResult vjp_interior_tri3(const KParams&, int nc, long long n, cudaStream_t);
LaunchResult vjp_boundary_tri3(const KParams&, int nc, long long n, cudaStream_t);
LaunchResult vjp_interior_quad4(const KParams&, int nc, long long n, cudaStream_t);
LaunchResult vjp_boundary_quad4(const KParams&, int nc, long long n, cudaStream_t);
LaunchResult vjp_interior_tet4(const KParams&, int nc, long long n, cudaStream_t);
LaunchResult vjp_boundary_tet4(const KParams&, int nc, long long n, cudaStream_t);
LaunchResult vjp_interior_hex8(const KParams&, int nc, long long n, cudaStream_t);
LaunchResult vjp_boundary_hex8(const KParams&, int nc, long long n, cudaStream_t);
LaunchResult boundary_hex8_mixed(const KParams&, int nc, long long n, cudaStream_t);
GeometryOps geometry_ops_hex8();
BoundaryInfo boundary_info_hex8(int nc);
LaunchResult adaptive_dt_hex8(const KParams&, int nc, double cfl, double* dt_el, long long n, cudaStream_t);
// The device array of a magma material's sub-mixtures, its count and its device
// (gales_magma.cu).
const magma_mix::DevMagma* magma_device_table(const gales_magma* m, int* nc, int* device);
MagmaOps magma_ops_tri3();
MagmaOps magma_ops_quad4();
MagmaOps magma_ops_tet4();
MagmaOps magma_ops_hex8();

}  // namespace gales
