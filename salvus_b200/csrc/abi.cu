// abi.cu -- extern "C" entry points (include/salvus_b200.h): mesh flattening,
// device residency, and the per-step launch sequence
//   stiffness (element-local residual) -> node gather with the sources +
//   inverse mass + Newmark -> receivers.
#include <cuda_runtime.h>

#include <unistd.h>

#include <atomic>
#include <cmath>
#include <condition_variable>
#include <functional>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <random>
#include <thread>
#include <vector>

#include "internal.h"
#include "once_per_device.h"
#include "kernels_setup.cuh"
#include "kernels_stiffness.cuh"
#include "kernels_step.cuh"
#include "kernels_hex_v2.cuh"
#include "kernels_hex_affine.cuh"
#include "kernels_batch.cuh"
#include "kernels_simplex.cuh"
#include "kernels_simplex_tc.cuh"
#include "kernels_tri_tc.cuh"
#include "kernels_elastic2d.cuh"
#include "kernels_quad_col.cuh"
#include "kernels_group.cuh"
#include <algorithm>
#include <cstdlib>
#include <type_traits>

namespace salvus {
const char *last_error();
int flatten_mesh(salvus_mesh *m, const int64_t *cells, int64_t n_vertices);
int locate_point(const salvus_mesh *m, const double *x, int64_t *elem, double *ref);
int boundary_nodes(const salvus_mesh *m, std::vector<int64_t> &out);
int setup_coupled(salvus_mesh *m, const int64_t *cells);

static std::atomic<int64_t> g_launches{0};

enum Kind { K_STIFF = 0, K_SRC, K_UPDATE, K_REC, K_GATHER, K_MINV, K_NEWMARK, K_GRAPH, K_NKINDS };
static const char *kKindNames[K_NKINDS] = {"stiffness", "source",        "gather_update",
                                           "receivers", "gather",        "inverse_mass",
                                           "newmark",   "graph_replay"};

struct ProfScope {
  salvus_problem *p;
  int kind;
  cudaEvent_t a = nullptr, b = nullptr;
  ProfScope(salvus_problem *p_, int k) : p(p_), kind(k) {
    if (p && p->profiling) {
      cudaEventCreate(&a);
      cudaEventCreate(&b);
      cudaEventRecord(a, p->stream);
    }
  }
  ~ProfScope() {
    if (a) {
      cudaEventRecord(b, p->stream);
      p->events.push_back({kind, a, b});
    }
  }
};

static inline unsigned blocks_for(int64_t n, int threads) {
  return (unsigned)((n + threads - 1) / threads);
}

template <typename real>
static DMatrix<real> dmatrix(const Basis &b) {
  DMatrix<real> d{};
  for (int i = 0; i < b.n * b.n; ++i) d.d[i] = (real)b.D[i];
  return d;
}

static int check_launch(const char *what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(SALVUS_E_CUDA, "%s launch failed: %s", what, cudaGetErrorString(e));
  return SALVUS_OK;
}

// Calls fn(std::integral_constant<int, C>) for the field's component count
// (1 acoustic, 2 elastic 2-D, 3 elastic 3-D).
template <typename Fn>
static int by_components(int c, Fn &&fn) {
  switch (c) {
    case 1: return fn(std::integral_constant<int, 1>{});
    case 2: return fn(std::integral_constant<int, 2>{});
    case 3: return fn(std::integral_constant<int, 3>{});
  }
  return fail(SALVUS_E_UNSUPPORTED, "no kernels for %d field components", c);
}

// ---------------------------------------------------------------------------
// stiffness dispatch
template <int DIM, int N, typename real>
static int launch_acoustic(const salvus_mesh *m, const real *rec, const real *u, real *r,
                           cudaStream_t st) {
  using S = AcousticShape<DIM, N>;
  const unsigned grid = blocks_for(m->E, S::EPB);
  acoustic_stiffness_kernel<DIM, N, real><<<grid, S::THREADS, 0, st>>>(
      m->E, rec, m->d_conn.as<int32_t>(), u, r, dmatrix<real>(m->basis));
  g_launches++;
  return check_launch("acoustic stiffness");
}

// FP32 elastic hexahedra: the column-threaded kernel with 32-bit shared
// planes and 128-thread CTAs (whole warps: 5 order-4 elements) by default;
// SALVUS_HEX_KERNEL=classic selects the register / shared-memory kernel that
// also serves FP64 general hexahedra of order 3 (read at every launch).
static bool hex_classic() {
  const char *s = std::getenv("SALVUS_HEX_KERNEL");
  return s && std::strcmp(s, "classic") == 0;
}

// Lets a kernel's launches on the mesh's device, which is the current one, use
// `bytes` of dynamic shared memory (more than 48 KB has to be asked for).
template <typename Kern>
static int dynamic_smem(OncePerDevice &once, const salvus_mesh *m, Kern kern, size_t bytes) {
  const int e = once(m->device, [&] {
    return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  });
  if (e == 0) return SALVUS_OK;
  return fail(SALVUS_E_CUDA, "%zu bytes of shared memory refused: %s", bytes,
              cudaGetErrorString((cudaError_t)e));
}

template <int N, bool TI>
static int launch_elastic_v2(const salvus_mesh *m, const float *rec, const float *u, float *r,
                             cudaStream_t st) {
  constexpr int n2 = (N + 1) * (N + 1), EPB = 128 / n2 > 0 ? 128 / n2 : 1;
  using T = ElasticV2Shape<N, EPB, TI>;
  static OncePerDevice attr;
  if (int rc = dynamic_smem(attr, m, elastic_hex_stiffness_v2_kernel<N, EPB, TI>, T::SMEM)) return rc;
  elastic_hex_stiffness_v2_kernel<N, EPB, TI><<<blocks_for(m->E, EPB), T::THREADS, T::SMEM, st>>>(
      m->E, rec, u, r, dmatrix<float>(m->basis));
  g_launches++;
  return check_launch("elastic stiffness");
}

template <int N, typename real, bool TI>
static int launch_elastic_classic(const salvus_mesh *m, const real *rec, const real *u, real *r,
                                  cudaStream_t st) {
  using S = ElasticShape<N, real>;
  static OncePerDevice attr;
  if (int rc = dynamic_smem(attr, m, elastic_hex_stiffness_kernel<N, real, TI>, S::SMEM)) return rc;
  elastic_hex_stiffness_kernel<N, real, TI><<<blocks_for(m->E, S::EPB), S::THREADS, S::SMEM, st>>>(
      m->E, rec, m->d_conn.as<int32_t>(), u, r, dmatrix<real>(m->basis));
  g_launches++;
  return check_launch("elastic stiffness");
}

// Parallelepiped meshes (m->affine): per-element inverse Jacobian, material
// planes; kFuse also advances the interior nodes (kernels_hex_affine.cuh).
// CTAs hold EPB elements: 128 / (N+1)^2 or, when the hexahedron autotuner
// found it faster on this mesh (m->hex_wide), twice as many.
template <int N, int EPB, bool TI, bool kFuse>
static int launch_elastic_affine_epb(const salvus_mesh *m, const float *mat, float *u, float *r,
                                     cudaStream_t st, const HexInteriorUpdate &iu) {
  using T = HexAffineShape<N, EPB, TI>;
  auto kern = kFuse ? elastic_hex_affine_fused_kernel<N, EPB, TI>
                    : elastic_hex_affine_kernel<N, EPB, TI>;
  static OncePerDevice attr;
  if (int rc = dynamic_smem(attr, m, kern, T::SMEM)) return rc;
  kern<<<blocks_for(m->E, EPB), T::THREADS, T::SMEM, st>>>(
      m->E, m->d_jac32.as<float>(), mat, m->d_conn.as<int32_t>(), u, r, dmatrix<float>(m->basis),
      iu);
  g_launches++;
  return check_launch(kFuse ? "elastic stiffness (fused interior)" : "elastic stiffness");
}
template <int N, bool TI, bool kFuse>
static int launch_elastic_affine(const salvus_mesh *m, const float *mat, float *u, float *r,
                                 cudaStream_t st, const HexInteriorUpdate &iu) {
  constexpr int n2 = (N + 1) * (N + 1), EPB = 128 / n2 > 0 ? 128 / n2 : 1;
  return m->hex_wide ? launch_elastic_affine_epb<N, 2 * EPB, TI, kFuse>(m, mat, u, r, st, iu)
                     : launch_elastic_affine_epb<N, EPB, TI, kFuse>(m, mat, u, r, st, iu);
}

template <int N, bool TI, bool kAffine>
static int launch_elastic_col64(const salvus_mesh *m, const double *rec, const double *u, double *r,
                                cudaStream_t st) {
  constexpr int EPB = HexCol64<N, TI, kAffine>::EPB;
  using T = HexColShape<N, EPB, double>;
  static OncePerDevice attr;
  if (int rc = dynamic_smem(attr, m, elastic_hex_col64_kernel<N, TI, kAffine>, T::SMEM)) return rc;
  elastic_hex_col64_kernel<N, TI, kAffine><<<blocks_for(m->E, EPB), T::THREADS, T::SMEM, st>>>(
      m->E, m->d_jac64.as<double>(), rec, m->d_conn.as<int32_t>(), const_cast<double *>(u), r,
      dmatrix<double>(m->basis));
  g_launches++;
  return check_launch("elastic stiffness");
}

template <int N, typename real>
static int launch_elastic(const salvus_mesh *m, const real *rec, const real *u, real *r,
                          cudaStream_t st) {
  if constexpr (std::is_same<real, float>::value) {
    if (m->affine) {
      HexInteriorUpdate none{};
      return m->ti ? launch_elastic_affine<N, true, false>(m, rec, const_cast<float *>(u), r, st, none)
                   : launch_elastic_affine<N, false, false>(m, rec, const_cast<float *>(u), r, st, none);
    }
    if (!hex_classic())
      return m->ti ? launch_elastic_v2<N, true>(m, rec, u, r, st)
                   : launch_elastic_v2<N, false>(m, rec, u, r, st);
  } else {
    if (m->affine64)
      return m->ti ? launch_elastic_col64<N, true, true>(m, rec, u, r, st)
                   : launch_elastic_col64<N, false, true>(m, rec, u, r, st);
    if constexpr (HexCol64<N, false, false>::kUse)
      return m->ti ? launch_elastic_col64<N, true, false>(m, rec, u, r, st)
                   : launch_elastic_col64<N, false, false>(m, rec, u, r, st);
  }
  if constexpr (sizeof(real) == 4 || !HexCol64<N, false, false>::kUse)
    return m->ti ? launch_elastic_classic<N, real, true>(m, rec, u, r, st)
                 : launch_elastic_classic<N, real, false>(m, rec, u, r, st);
}

// Quadrilateral stiffness: column-threaded kernels (kernels_quad_col.cuh) by
// default; SALVUS_QUAD_KERNEL=point selects the point-threaded ones (read at
// every launch).
static bool quad_point_kernels() {
  const char *v = std::getenv("SALVUS_QUAD_KERNEL");
  return v && std::strcmp(v, "point") == 0;
}
template <int N, typename real>
static int acoustic2(const salvus_mesh *m, const real *rec, const real *u, real *r, cudaStream_t s) {
  // (FP64 elastic columns of order 9-10 exceed the register file: point kernels)
  if (!quad_point_kernels() && (sizeof(real) == 4 || N <= 8)) {
    constexpr int EPB = quad_col_epb<N>();
    using S = QuadColShape<N, EPB>;
    const DMatrix<real> D = dmatrix<real>(m->basis);
    const int32_t *cn = m->d_conn.as<int32_t>();
    if constexpr (std::is_same<real, float>::value) {
      if (m->qscalar) {
        acoustic_quad_square_kernel<N, EPB><<<blocks_for(m->E, EPB), S::THREADS, 0, s>>>(
            m->E, m->d_qs32.as<float>(), cn, u, r, D);
        g_launches++;
        return check_launch("acoustic quad stiffness");
      }
    }
    if (m->physics == SALVUS_ACOUSTIC) {
      acoustic_quad_col_kernel<N, EPB, real><<<blocks_for(m->E, EPB), S::THREADS, 0, s>>>(
          m->E, rec, cn, u, r, D);
      g_launches++;
      return check_launch("acoustic quad stiffness");
    }
    if (m->physics == SALVUS_ELASTIC2D) {
      elastic2d_col_kernel<N, EPB, real, 2, 0><<<blocks_for(m->E, EPB), S::THREADS, 0, s>>>(
          m->E, nullptr, rec, cn, u, r, D);
      g_launches++;
      return check_launch("elastic 2-D stiffness");
    }
    // fluid elements (u) then solid elements (ux, uy), class-compact records
    const int64_t Ef = m->n_fluid, Es = m->E - m->n_fluid;
    const int32_t *el = m->d_elist.as<int32_t>();
    if (Ef > 0) {
      acoustic_quad_col_list_kernel<N, EPB, real><<<blocks_for(Ef, EPB), S::THREADS, 0, s>>>(
          Ef, el, rec, cn, u, r, D);
      g_launches++;
      int rc = check_launch("fluid stiffness");
      if (rc) return rc;
    }
    if (Es > 0) {
      const real *rs = rec + Ef * m->P * (sizeof(real) == 4 ? 4 : 3);
      elastic2d_col_kernel<N, EPB, real, 3, 1><<<blocks_for(Es, EPB), S::THREADS, 0, s>>>(
          Es, el + Ef, rs, cn, u, r, D);
      g_launches++;
      return check_launch("solid stiffness");
    }
    return SALVUS_OK;
  }
  if (m->physics == SALVUS_COUPLED2D) {
    // fluid elements (u) then solid elements (ux, uy), class-compact records
    const int64_t Ef = m->n_fluid, Es = m->E - m->n_fluid;
    const int32_t *el = m->d_elist.as<int32_t>();
    if (Ef > 0) {
      using S = AcousticShape<2, N>;
      acoustic_list_kernel<N, real><<<blocks_for(Ef, S::EPB), S::THREADS, 0, s>>>(
          Ef, el, rec, m->d_conn.as<int32_t>(), u, r, dmatrix<real>(m->basis));
      g_launches++;
      int rc = check_launch("fluid stiffness");
      if (rc) return rc;
    }
    if (Es > 0) {
      using S = Elastic2DShape<N>;
      const real *rs = rec + Ef * m->P * (sizeof(real) == 4 ? 4 : 3);
      elastic2d_stiffness_kernel<N, real, 3, 1><<<blocks_for(Es, S::EPB), S::THREADS, 0, s>>>(
          Es, el + Ef, rs, m->d_conn.as<int32_t>(), u, r, dmatrix<real>(m->basis));
      g_launches++;
      return check_launch("solid stiffness");
    }
    return SALVUS_OK;
  }
  if (m->physics == SALVUS_ELASTIC2D) {
    // CTA shape: SALVUS_E2D_EPB elements per CTA (read at every launch; 0 or
    // unset: as many as fit 256 threads)
    const char *ev = std::getenv("SALVUS_E2D_EPB");
    const int epb = ev ? std::atoi(ev) : 0;
    auto go = [&](auto tag) {
      constexpr int EPB = decltype(tag)::value;
      using S = Elastic2DShape<N, EPB>;
      elastic2d_stiffness_kernel<N, real, 2, 0, EPB><<<blocks_for(m->E, S::EPB), S::THREADS, 0, s>>>(
          m->E, nullptr, rec, m->d_conn.as<int32_t>(), u, r, dmatrix<real>(m->basis));
      g_launches++;
      return check_launch("elastic 2-D stiffness");
    };
    switch (epb) {
      case 2: return go(std::integral_constant<int, 2>{});
      case 4: return go(std::integral_constant<int, 4>{});
      case 5: return go(std::integral_constant<int, 5>{});
      case 8: return go(std::integral_constant<int, 8>{});
      default: return go(std::integral_constant<int, 0>{});
    }
  }
  return launch_acoustic<2, N, real>(m, rec, u, r, s);
}
template <int N, typename real>
static int acoustic3(const salvus_mesh *m, const real *rec, const real *u, real *r, cudaStream_t s) {
  // order 1: one thread per point (60^3: FP32 16.7 us a step against 16.9, FP64
  // 30.7 against 41.4)
  if constexpr (N >= 2) {
    using T = AcousticHexCol<N, real>;
    acoustic_hex_col_kernel<N, real><<<blocks_for(m->E, T::EPB), T::Shape::THREADS, 0, s>>>(
        m->E, rec, m->d_conn.as<int32_t>(), u, r, dmatrix<real>(m->basis));
    g_launches++;
    return check_launch("acoustic stiffness");
  } else {
    return launch_acoustic<3, N, real>(m, rec, u, r, s);
  }
}

// P3 simplices on CUDA cores
template <typename real>
static const real *simplex_tables(const salvus_mesh *m) {
  return sizeof(real) == 4 ? (const real *)m->d_sd32.ptr : (const real *)m->d_sd64.ptr;
}

template <typename real, int C, bool TI = false>
static int launch_tet(const salvus_mesh *m, const real *rec, const real *u, real *r,
                      cudaStream_t st) {
  using S = TetShape<real, C, TI>;
  static OncePerDevice attr;
  if (int rc = dynamic_smem(attr, m, tet_stiffness_kernel<real, C, TI>, S::SMEM)) return rc;
  tet_stiffness_kernel<real, C, TI><<<blocks_for(m->E, S::EPB), S::THREADS, S::SMEM, st>>>(
      m->E, rec, m->d_conn.as<int32_t>(), simplex_tables<real>(m), u, r);
  g_launches++;
  return check_launch("tetrahedron stiffness");
}

// FP32 tetrahedra on the tensor cores (tcgen05, split TF32)
template <int C>
static int launch_tet_tc(const salvus_mesh *m, const float *rec, const float *u, float *r,
                         cudaStream_t st, int *err, long long wlim, int hold) {
  using S = TetTcShape<C>;
  static OncePerDevice attr;
  if (int rc = dynamic_smem(attr, m, tet_tc_kernel<C>, S::SMEM)) return rc;
  const int64_t tiles = (m->E + S::NE - 1) / S::NE;
  const unsigned grid = (unsigned)(tiles < m->sm_count ? tiles : m->sm_count);
  tet_tc_kernel<C><<<grid, S::THREADS, S::SMEM, st>>>(
      m->E, rec, m->d_conn.as<int32_t>(), m->d_tc_tab.as<uint4>(), u, r, err, wlim, hold);
  g_launches++;
  return check_launch("tetrahedron stiffness (tensor cores)");
}

static int launch_tri_tc(const salvus_mesh *m, const float *rec, const float *u, float *r,
                         cudaStream_t st, int *err, long long wlim, int hold) {
  using S = TriTcShape;
  static OncePerDevice attr;
  if (int rc = dynamic_smem(attr, m, tri_tc_kernel, S::SMEM)) return rc;
  static std::atomic<int> resident{0};  // CTAs per SM, the same on every device this runs on
  int per_sm = resident.load();
  if (per_sm == 0) {
    SALVUS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tri_tc_kernel, S::THREADS,
                                                              S::SMEM));
    if (per_sm < 1) per_sm = 1;
    resident = per_sm;
  }
  const int64_t tiles = (m->E + S::NE - 1) / S::NE;
  const int64_t slots = (int64_t)per_sm * m->sm_count;
  const unsigned grid = (unsigned)(tiles < slots ? tiles : slots);
  tri_tc_kernel<<<grid, S::THREADS, S::SMEM, st>>>(m->E, rec, m->d_conn.as<int32_t>(),
                                                   m->d_tc_tab.as<uint4>(), u, r, err, wlim, hold);
  g_launches++;
  return check_launch("triangle stiffness (tensor cores)");
}

template <typename real>
static int launch_simplex(const salvus_mesh *m, const real *rec, const real *u, real *r,
                          cudaStream_t st, int *err, long long wlim, int hold) {
  if constexpr (std::is_same<real, float>::value) {
    if (m->shape == SALVUS_TRI && m->tri_kernel == 0)
      return launch_tri_tc(m, rec, u, r, st, err, wlim, hold);
    if (m->shape == SALVUS_TET && m->tet_kernel == 0) {
      if (m->physics == SALVUS_ELASTIC3D)
        return launch_tet_tc<3>(m, rec, u, r, st, err, wlim, hold);
      return launch_tet_tc<1>(m, rec, u, r, st, err, wlim, hold);
    }
  }
  if (m->shape == SALVUS_TRI) {
    if (m->tri_kernel == 2)
      tri_acoustic_kernel<real><<<blocks_for(m->E, 128), 128, 0, st>>>(
          m->E, rec, m->d_conn.as<int32_t>(), simplex_tables<real>(m), u, r);
    else
      tri_acoustic_const_kernel<real><<<blocks_for(m->E, 128), 128, 0, st>>>(
          m->E, rec, m->d_conn.as<int32_t>(), u, r);
    g_launches++;
    return check_launch("triangle stiffness");
  }
  if (m->physics == SALVUS_ELASTIC3D)
    return m->ti ? launch_tet<real, 3, true>(m, rec, u, r, st) : launch_tet<real, 3>(m, rec, u, r, st);
  return launch_tet<real, 1>(m, rec, u, r, st);
}

template <typename real>
static int launch_stiffness(const salvus_mesh *m, const real *rec, const real *u, real *r,
                            cudaStream_t st, int *err = nullptr,
                            long long wlim = salvus::kDefaultWaitLimit, int hold = 0) {
  if (is_simplex(m->shape)) return launch_simplex<real>(m, rec, u, r, st, err, wlim, hold);
  if (m->physics == SALVUS_ELASTIC3D) {
    switch (m->order) {
      case 1: return launch_elastic<1, real>(m, rec, u, r, st);
      case 2: return launch_elastic<2, real>(m, rec, u, r, st);
      case 3: return launch_elastic<3, real>(m, rec, u, r, st);
      case 4: return launch_elastic<4, real>(m, rec, u, r, st);
      case 5: return launch_elastic<5, real>(m, rec, u, r, st);
      case 6: return launch_elastic<6, real>(m, rec, u, r, st);
    }
  } else if (m->shape == SALVUS_QUAD) {
    switch (m->order) {
      case 1: return acoustic2<1, real>(m, rec, u, r, st);
      case 2: return acoustic2<2, real>(m, rec, u, r, st);
      case 3: return acoustic2<3, real>(m, rec, u, r, st);
      case 4: return acoustic2<4, real>(m, rec, u, r, st);
      case 5: return acoustic2<5, real>(m, rec, u, r, st);
      case 6: return acoustic2<6, real>(m, rec, u, r, st);
      case 7: return acoustic2<7, real>(m, rec, u, r, st);
      case 8: return acoustic2<8, real>(m, rec, u, r, st);
      case 9: return acoustic2<9, real>(m, rec, u, r, st);
      case 10: return acoustic2<10, real>(m, rec, u, r, st);
    }
  } else {
    switch (m->order) {
      case 1: return acoustic3<1, real>(m, rec, u, r, st);
      case 2: return acoustic3<2, real>(m, rec, u, r, st);
      case 3: return acoustic3<3, real>(m, rec, u, r, st);
      case 4: return acoustic3<4, real>(m, rec, u, r, st);
      case 5: return acoustic3<5, real>(m, rec, u, r, st);
      case 6: return acoustic3<6, real>(m, rec, u, r, st);
    }
  }
  return fail(SALVUS_E_UNSUPPORTED, "no stiffness kernel for shape %d order %d", m->shape, m->order);
}

// ---------------------------------------------------------------------------
// mesh setup
template <typename real>
static int build_simplex_records(salvus_mesh *m, DeviceBuffer &out, DeviceBuffer &sd,
                                 DeviceBuffer &mass_local) {
  const int rw = record_words(m->shape, m->physics, sizeof(real) == 8, m->ti);
  int rc = out.alloc(sizeof(real) * (size_t)m->E * rw);
  if (rc) return rc;
  SimplexTable tab{};
  for (int q = 0; q < m->P; ++q) {
    for (int a = 0; a < 3; ++a) tab.x[q][a] = m->basis.nodes[(size_t)q * 3 + a];
    tab.w[q] = m->basis.sw[q];
  }
  simplex_geometry_kernel<real><<<blocks_for(m->E, 128), 128, 0, m->stream>>>(
      m->E, m->shape, m->physics, m->P, rw, m->d_vtx.as<double>(), m->d_par.as<double>(), tab,
      out.as<real>(), mass_local.as<double>(), m->ti);
  g_launches++;
  if ((rc = check_launch("simplex geometry"))) return rc;
  std::vector<real> t(m->basis.SD.size());
  for (size_t i = 0; i < t.size(); ++i) t[i] = (real)m->basis.SD[i];
  if ((rc = sd.alloc(sizeof(real) * t.size()))) return rc;
  SALVUS_CUDA(cudaMemcpyAsync(sd.ptr, t.data(), sizeof(real) * t.size(), cudaMemcpyHostToDevice,
                              m->stream));
  if (m->shape == SALVUS_TRI) {
    // the reference triangle's table, identical for every mesh: constant
    // memory of this device (tri_acoustic_const_kernel)
    if (sizeof(real) == 4)
      SALVUS_CUDA(cudaMemcpyToSymbolAsync(c_tri_sd32, t.data(), sizeof(real) * t.size(), 0,
                                          cudaMemcpyHostToDevice, m->stream));
    else
      SALVUS_CUDA(cudaMemcpyToSymbolAsync(c_tri_sd64, t.data(), sizeof(real) * t.size(), 0,
                                          cudaMemcpyHostToDevice, m->stream));
  }
  if (sizeof(real) == 4 && m->shape == SALVUS_TRI) {
    // tensor-core operand images (kernels_tri_tc.cuh), K-major no-swizzle
    // core-matrix order, TF32 hi part and FP32 remainder, zero padding:
    //   B1[kappa = 16 k + q][j] = dphi_j/dxi_k (x_q)   32 x 16
    //   B2[i][kappa = 16 k + q] = dphi_i/dxi_k (x_q)    16 x 32
    constexpr int P = 12;
    constexpr size_t B = 32 * 16;
    std::vector<float> img(4 * B, 0.f);
    auto off = [](int row, int k, int kdim) {
      return (size_t)(((row >> 3) * (kdim / 4) * 128 + (k >> 2) * 128 + (row & 7) * 16 + (k & 3) * 4) / 4);
    };
    for (int k = 0; k < 2; ++k)
      for (int q = 0; q < P; ++q)
        for (int j = 0; j < P; ++j) {
          const double v = m->basis.SD[((size_t)k * P + j) * P + q];
          const float f = (float)v;
          uint32_t bits;
          std::memcpy(&bits, &f, 4);
          bits = (bits + 0x1000u) & 0xFFFFE000u;  // nearest TF32 (ties away from zero)
          float hi, lo;
          std::memcpy(&hi, &bits, 4);
          lo = (float)(v - (double)hi);
          const int kap = 16 * k + q;
          img[off(kap, j, 16)] = hi;
          img[B + off(kap, j, 16)] = lo;
          img[2 * B + off(j, kap, 32)] = hi;
          img[3 * B + off(j, kap, 32)] = lo;
        }
    if ((rc = m->d_tc_tab.alloc(sizeof(float) * img.size()))) return rc;
    SALVUS_CUDA(cudaMemcpyAsync(m->d_tc_tab.ptr, img.data(), sizeof(float) * img.size(),
                                cudaMemcpyHostToDevice, m->stream));
  }
  if (sizeof(real) == 4 && m->shape == SALVUS_TET) {
    // tensor-core operand images, K-major no-swizzle core-matrix order, each
    // as a TF32 hi part and an FP32 remainder:
    //   B1[kappa = 56 k + q][j] = dphi_j/dxi_k (x_q)   176 x 56
    //   B2[i][kappa = 56 k + q] = dphi_i/dxi_k (x_q)    64 x 168
    constexpr int P = 50;
    constexpr size_t B1 = 176 * 56, B2 = 64 * 168;
    std::vector<float> img(2 * B1 + 2 * B2, 0.f);
    auto off = [](int row, int k, int kdim) {
      return (size_t)(((row >> 3) * (kdim / 4) * 128 + (k >> 2) * 128 + (row & 7) * 16 + (k & 3) * 4) / 4);
    };
    auto split = [](double v, float &hi, float &lo) {
      // nearest TF32 value (round half away from zero on the 13 dropped bits)
      const float f = (float)v;
      uint32_t bits;
      std::memcpy(&bits, &f, 4);
      bits = (bits + 0x1000u) & 0xFFFFE000u;
      std::memcpy(&hi, &bits, 4);
      lo = (float)(v - (double)hi);
    };
    for (int k = 0; k < 3; ++k)
      for (int q = 0; q < P; ++q)
        for (int j = 0; j < P; ++j) {
          float hi, lo;
          split(m->basis.SD[((size_t)k * P + j) * P + q], hi, lo);
          const int kap = 56 * k + q;
          img[off(kap, j, 56)] = hi;
          img[B1 + off(kap, j, 56)] = lo;
          img[2 * B1 + off(j, kap, 168)] = hi;
          img[2 * B1 + B2 + off(j, kap, 168)] = lo;
        }
    if ((rc = m->d_tc_tab.alloc(sizeof(float) * img.size()))) return rc;
    SALVUS_CUDA(cudaMemcpyAsync(m->d_tc_tab.ptr, img.data(), sizeof(float) * img.size(),
                                cudaMemcpyHostToDevice, m->stream));
  }
  SALVUS_CUDA(cudaStreamSynchronize(m->stream));
  return SALVUS_OK;
}

template <typename real, bool kPack>
static int build_records(salvus_mesh *m, DeviceBuffer &out, DeviceBuffer &mass_local) {
  if (is_simplex(m->shape))
    return build_simplex_records<real>(m, out, sizeof(real) == 4 ? m->d_sd32 : m->d_sd64,
                                       mass_local);
  const int rw = record_words(m->shape, m->physics, sizeof(real) == 8, m->ti);
  int rc = out.alloc(sizeof(real) * (size_t)(m->E * m->P) * rw);
  if (rc) return rc;
  GllTable gll{};
  for (int i = 0; i < m->n; ++i) {
    gll.xi[i] = m->basis.xi[i];
    gll.w[i] = m->basis.w[i];
  }
  const int64_t total = m->E * m->P;
  geometry_kernel<real, kPack><<<blocks_for(total, 128), 128, 0, m->stream>>>(
      m->E, m->dim, m->n, m->P, m->physics, rw, m->d_vtx.as<double>(), m->d_par.as<double>(),
      m->d_conn.as<int32_t>(), gll, out.as<real>(), mass_local.as<double>(),
      m->d_cls_k.as<int32_t>(), m->n_fluid, m->ti, m->qsquare);
  g_launches++;
  return check_launch("geometry");
}

// Nodes the fused step (parallelepiped elastic hexahedra) and the fused
// batched step (acoustic quadrilaterals) gather: all but the element-interior
// ones (every local index in 1..N-1), which those steps advance in the
// stiffness kernel.  Host-side, ascending node ids.
static void interior_free_nodes(salvus_mesh *m) {
  m->gnodes.clear();
  m->n_gnodes = 0;
  const bool quad = m->shape == SALVUS_QUAD && m->physics == SALVUS_ACOUSTIC;
  if (m->order < 2 || !(m->affine || quad)) return;
  const int n = m->n;
  std::vector<char> interior((size_t)m->G, 0);
  for (int64_t e = 0; e < m->E; ++e) {
    const int32_t *cn = m->conn.data() + e * m->P;
    if (m->dim == 2) {
      for (int j = 1; j < n - 1; ++j)
        for (int i = 1; i < n - 1; ++i) interior[(size_t)cn[i + n * j]] = 1;
    } else {
      for (int k = 1; k < n - 1; ++k)
        for (int j = 1; j < n - 1; ++j)
          for (int i = 1; i < n - 1; ++i) interior[(size_t)cn[i + n * j + n * n * k]] = 1;
    }
  }
  m->gnodes.reserve((size_t)m->G);
  for (int64_t g = 0; g < m->G; ++g)
    if (!interior[(size_t)g]) m->gnodes.push_back((int32_t)g);
  m->n_gnodes = (int64_t)m->gnodes.size();
}

static bool acoustic_quads(const salvus_mesh *m) {
  return m->shape == SALVUS_QUAD && m->physics == SALVUS_ACOUSTIC;
}
static Incidence incidence(const salvus_mesh *m) {
  return {m->d_inc_head.as<int2>(), m->d_inc_rest.as<int32_t>()};
}
// Two nodes per thread (gather_pair_kernel): acoustic quadrilaterals with six
// CTAs of nodes per SM (227 k nodes) or more; fewer leave SMs without enough
// warps to hide the chain (40 k-116 k nodes: 5.3-5.5 us a step with one node
// per thread, 5.4-6.0 with two; 361 k: 8.1 against 7.2-7.6).  Orders 1 and 2
// are mostly vertices, whose lists take the longer way (500^2 order 1: 8.3
// against 9.1 us).
static bool gather_pairs(const salvus_mesh *m, int64_t nodes) {
  return acoustic_quads(m) && m->order >= 3 && nodes >= 6 * (int64_t)kPairTile * m->sm_count;
}

// The pairs of Incidence on the device, from the offsets and the index there;
// the host only counts where each CTA's part of `rest` begins (building and
// uploading both here took 3 ms of the 44 that a 200^2 order-4 mesh takes).
static int incidence_pairs(salvus_mesh *m) {
  std::vector<int32_t> base;
  int32_t total = 0;
  for (int64_t g0 = 0; g0 < m->G; g0 += kHeadTile) {
    base.push_back(total);
    const int64_t g1 = std::min(m->G, g0 + kHeadTile);
    for (int64_t g = g0; g < g1; ++g) {
      const int32_t n = m->inc_off[(size_t)g + 1] - m->inc_off[(size_t)g];
      total += n > 2 ? n : 0;
    }
  }
  // base lies behind the lists: freeing a buffer of its own would wait for
  // everything that other problems have on the device
  int rc;
  if ((rc = m->d_inc_head.alloc(sizeof(int2) * (size_t)m->G)) ||
      (rc = m->d_inc_rest.alloc(sizeof(int32_t) * ((size_t)total + base.size()))))
    return rc;
  int32_t *rest = m->d_inc_rest.as<int32_t>();
  SALVUS_CUDA(cudaMemcpyAsync(rest + total, base.data(), sizeof(int32_t) * base.size(),
                              cudaMemcpyHostToDevice, m->stream));
  incidence_pairs_kernel<<<(unsigned)base.size(), kHeadTile, 0, m->stream>>>(
      m->G, m->d_inc_off.as<int32_t>(), m->d_inc_idx.as<int32_t>(), rest + total,
      m->d_inc_head.as<int2>(), rest);
  g_launches++;
  if ((rc = check_launch("incidence pairs"))) return rc;
  SALVUS_CUDA(cudaStreamSynchronize(m->stream));  // base ends here
  return SALVUS_OK;
}

static int mesh_setup_device(salvus_mesh *m) {
  int rc;
  SALVUS_CUDA(cudaSetDevice(m->device));
  SALVUS_CUDA(cudaDeviceGetAttribute(&m->sm_count, cudaDevAttrMultiProcessorCount, m->device));
  SALVUS_CUDA(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
  const int64_t EP = m->E * m->P;
  if ((rc = m->d_conn.alloc(sizeof(int32_t) * EP))) return rc;
  if ((rc = m->d_inc_off.alloc(sizeof(int32_t) * (m->G + 1)))) return rc;
  if ((rc = m->d_inc_idx.alloc(sizeof(int32_t) * EP))) return rc;
  if ((rc = m->d_vtx.alloc(sizeof(double) * m->vtx.size()))) return rc;
  if ((rc = m->d_par.alloc(sizeof(double) * m->par.size()))) return rc;
  if ((rc = m->d_mi64.alloc(sizeof(double) * m->G))) return rc;
  if ((rc = m->d_mi32.alloc(sizeof(float) * m->G))) return rc;
  SALVUS_CUDA(cudaMemcpyAsync(m->d_conn.ptr, m->conn.data(), sizeof(int32_t) * EP,
                              cudaMemcpyHostToDevice, m->stream));
  SALVUS_CUDA(cudaMemcpyAsync(m->d_inc_off.ptr, m->inc_off.data(), sizeof(int32_t) * (m->G + 1),
                              cudaMemcpyHostToDevice, m->stream));
  SALVUS_CUDA(cudaMemcpyAsync(m->d_inc_idx.ptr, m->inc_idx.data(), sizeof(int32_t) * EP,
                              cudaMemcpyHostToDevice, m->stream));
  SALVUS_CUDA(cudaMemcpyAsync(m->d_vtx.ptr, m->vtx.data(), sizeof(double) * m->vtx.size(),
                              cudaMemcpyHostToDevice, m->stream));
  SALVUS_CUDA(cudaMemcpyAsync(m->d_par.ptr, m->par.data(), sizeof(double) * m->par.size(),
                              cudaMemcpyHostToDevice, m->stream));
  if (m->physics == SALVUS_COUPLED2D) {
    const size_t nc = (size_t)m->n_cpl;
    std::vector<float> c32(m->cpl_coef.begin(), m->cpl_coef.end());
    if ((rc = m->d_elist.alloc(sizeof(int32_t) * m->E)) ||
        (rc = m->d_cls_k.alloc(sizeof(int32_t) * m->E)) ||
        (rc = m->d_cpl_pts.alloc(sizeof(int32_t) * 2 * nc)) ||
        (rc = m->d_cpl32.alloc(sizeof(float) * 2 * nc)) ||
        (rc = m->d_cpl64.alloc(sizeof(double) * 2 * nc)))
      return rc;
    SALVUS_CUDA(cudaMemcpyAsync(m->d_elist.ptr, m->elist.data(), sizeof(int32_t) * m->E,
                                cudaMemcpyHostToDevice, m->stream));
    SALVUS_CUDA(cudaMemcpyAsync(m->d_cls_k.ptr, m->cls_k.data(), sizeof(int32_t) * m->E,
                                cudaMemcpyHostToDevice, m->stream));
    if (nc) {
      SALVUS_CUDA(cudaMemcpyAsync(m->d_cpl_pts.ptr, m->cpl_pts.data(), sizeof(int32_t) * 2 * nc,
                                  cudaMemcpyHostToDevice, m->stream));
      SALVUS_CUDA(cudaMemcpyAsync(m->d_cpl32.ptr, c32.data(), sizeof(float) * 2 * nc,
                                  cudaMemcpyHostToDevice, m->stream));
      SALVUS_CUDA(cudaMemcpyAsync(m->d_cpl64.ptr, m->cpl_coef.data(), sizeof(double) * 2 * nc,
                                  cudaMemcpyHostToDevice, m->stream));
    }
    SALVUS_CUDA(cudaStreamSynchronize(m->stream));
  }
  if (acoustic_quads(m) && (rc = incidence_pairs(m))) return rc;
  DeviceBuffer mass_local;
  if ((rc = mass_local.alloc(sizeof(double) * EP))) return rc;
  if (m->affine) {
    // parallelepiped elastic hexahedra: material planes + per-element invJ
    const int nm = m->ti ? 5 : 2;
    if ((rc = m->d_rec32.alloc(sizeof(float) * (size_t)nm * EP)) ||
        (rc = m->d_jac32.alloc(sizeof(float) * 9 * (size_t)m->E)))
      return rc;
    GllTable gll{};
    for (int i = 0; i < m->n; ++i) {
      gll.xi[i] = m->basis.xi[i];
      gll.w[i] = m->basis.w[i];
    }
    affine_hex_records_kernel<float><<<blocks_for(EP, 128), 128, 0, m->stream>>>(
        m->E, m->n, m->P, m->ti, m->d_vtx.as<double>(), m->d_par.as<double>(), gll,
        m->d_rec32.as<float>(), m->d_jac32.as<float>(), mass_local.as<double>());
    g_launches++;
    if (m->affine64 && !m->fp32_only) {
      if ((rc = m->d_rec64.alloc(sizeof(double) * (size_t)nm * EP)) ||
          (rc = m->d_jac64.alloc(sizeof(double) * 9 * (size_t)m->E)))
        return rc;
      affine_hex_records_kernel<double><<<blocks_for(EP, 128), 128, 0, m->stream>>>(
          m->E, m->n, m->P, m->ti, m->d_vtx.as<double>(), m->d_par.as<double>(), gll,
          m->d_rec64.as<double>(), m->d_jac64.as<double>(), mass_local.as<double>());
      g_launches++;
    }
    if ((rc = check_launch("affine records"))) return rc;
  } else if ((rc = build_records<float, true>(m, m->d_rec32, mass_local))) {
    return rc;
  }
  if (m->qscalar) {
    if ((rc = m->d_qs32.alloc(sizeof(float) * EP))) return rc;
    GllTable gll{};
    for (int i = 0; i < m->n; ++i) {
      gll.xi[i] = m->basis.xi[i];
      gll.w[i] = m->basis.w[i];
    }
    quad_square_kernel<<<blocks_for(EP, 128), 128, 0, m->stream>>>(
        m->E, m->n, m->P, m->d_vtx.as<double>(), m->d_par.as<double>(), gll, m->d_qs32.as<float>());
    g_launches++;
    if ((rc = check_launch("squares"))) return rc;
  }
  // the node list of the fused steps (interior_free_nodes, at creation)
  if (m->n_gnodes > 0) {
    if ((rc = m->d_gnodes.alloc(sizeof(int32_t) * (size_t)m->n_gnodes))) return rc;
    SALVUS_CUDA(cudaMemcpyAsync(m->d_gnodes.ptr, m->gnodes.data(), sizeof(int32_t) * m->gnodes.size(),
                                cudaMemcpyHostToDevice, m->stream));
    SALVUS_CUDA(cudaStreamSynchronize(m->stream));
  }
  if (!m->fp32_only && !m->affine64 &&
      (rc = build_records<double, false>(m, m->d_rec64, mass_local)))
    return rc;
  mass_gather_kernel<<<blocks_for(m->G, 256), 256, 0, m->stream>>>(
      m->G, m->d_inc_off.as<int32_t>(), m->d_inc_idx.as<int32_t>(), mass_local.as<double>(),
      m->d_mi64.as<double>(), m->d_mi32.as<float>());
  g_launches++;
  if ((rc = check_launch("mass"))) return rc;
  m->mi.resize(m->G);
  SALVUS_CUDA(cudaMemcpyAsync(m->mi.data(), m->d_mi64.ptr, sizeof(double) * m->G,
                              cudaMemcpyDeviceToHost, m->stream));
  SALVUS_CUDA(cudaStreamSynchronize(m->stream));
  return SALVUS_OK;
}

// ---------------------------------------------------------------------------
// problem helpers
template <typename real>
static real *F(const DeviceBuffer &b) { return b.as<real>(); }

// The node gather's view of the sources (SourceTerms).  el: the sources'
// elements, ascending (an element's sources adjacent).
static void source_tiles(const salvus_mesh *m, const std::vector<int64_t> &el,
                         std::vector<int32_t> &tile, std::vector<int4> &node) {
  const int4 none{0, 0, 0, -1};
  tile.assign((size_t)((m->G + kSrcTile - 1) / kSrcTile), -1);
  size_t tiles = 0;
  for (size_t s = 0; s < el.size(); ++s)
    for (int q = 0; q < m->P; ++q) {
      int32_t &t = tile[(size_t)(m->conn[(size_t)(el[s] * m->P + q)] / kSrcTile)];
      if (t < 0) t = (int32_t)(kSrcTile * tiles++);
    }
  node.assign(kSrcTile * tiles, none);
  for (size_t s = 0; s < el.size();) {
    size_t t = s;
    while (t < el.size() && el[t] == el[s]) ++t;
    for (int q = 0; q < m->P; ++q) {
      const int32_t g = m->conn[(size_t)(el[s] * m->P + q)];
      size_t at = (size_t)(tile[(size_t)(g / kSrcTile)] + g % kSrcTile);
      if (node[at].z > 0) {  // a node of another source element too: append
        while (node[at].w >= 0) at = (size_t)node[at].w;
        node[at].w = (int32_t)node.size();
        at = node.size();
        node.push_back(none);
      }
      node[at] = int4{(int32_t)(s * m->P + q), (int32_t)s, (int32_t)(t - s), -1};
    }
    s = t;
  }
}

static SourceTerms source_terms(const salvus_problem *p) {
  SourceTerms s;
  if (p->srcs.empty()) return s;
  s.tile = p->src_tile;
  s.node = p->src_node;
  s.wts = p->src_wts;
  s.stf = p->stf;
  s.P = p->mesh->P;
  return s;
}

static int upload_sources(salvus_problem *p) {
  if (!p->src_dirty) return SALVUS_OK;
  const salvus_mesh *m = p->mesh;
  const size_t ns = p->srcs.size();
  p->n_src_uelem = 0;
  if (ns) {
    // batched problems group sources by shot, single-shot ones by element
    // (attach order kept within each)
    std::vector<size_t> order(ns);
    for (size_t s = 0; s < ns; ++s) order[s] = s;
    std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) {
      return p->shots > 1 ? p->srcs[a].desc.shot < p->srcs[b].desc.shot
                          : p->srcs[a].elem < p->srcs[b].elem;
    });
    std::vector<int64_t> el(ns), ue;
    std::vector<double> par(3 * ns), w(ns * m->P * p->c);
    std::vector<int32_t> shot_off(p->shots_pad + 1, 0), tile;
    std::vector<int4> node;
    std::vector<uint8_t> has(p->shots > 1 ? (size_t)m->E : 0, 0);
    for (size_t k = 0; k < ns; ++k) {
      const auto &src = p->srcs[order[k]];
      el[k] = src.elem;
      par[3 * k] = src.desc.center_freq;
      par[3 * k + 1] = src.desc.time_delay;
      par[3 * k + 2] = src.desc.amplitude;
      std::memcpy(&w[k * m->P * p->c], src.wts.data(), sizeof(double) * m->P * p->c);
      shot_off[src.desc.shot + 1]++;
      // distinct source elements (fused hexahedron step)
      if (p->shots == 1 && (ue.empty() || ue.back() != src.elem)) ue.push_back(src.elem);
      if (p->shots > 1) has[(size_t)src.elem] = 1;
    }
    for (int s = 0; s < p->shots_pad; ++s) shot_off[s + 1] += shot_off[s];
    if (p->shots == 1) source_tiles(m, el, tile, node);
    // one host image, one allocation and one copy
    std::vector<char> img;
    auto put = [&](const void *data, size_t bytes) {
      const size_t at = (img.size() + 15) & ~size_t(15);
      img.resize(at + bytes);
      if (data) std::memcpy(img.data() + at, data, bytes);
      return at;
    };
    const size_t o_el = put(el.data(), sizeof(int64_t) * ns);
    const size_t o_ue = put(ue.data(), sizeof(int64_t) * ue.size());
    const size_t o_par = put(par.data(), sizeof(double) * par.size());
    const size_t o_w = put(w.data(), sizeof(double) * w.size());
    const size_t o_so = put(shot_off.data(), sizeof(int32_t) * shot_off.size());
    const size_t o_t = put(tile.data(), sizeof(int32_t) * tile.size());
    const size_t o_n = put(node.data(), sizeof(int4) * node.size());
    const size_t o_h = put(has.data(), has.size());
    const size_t o_stf = put(nullptr, sizeof(double) * ns);
    int rc = p->d_src.alloc(img.size());
    if (rc) return rc;
    char *d = p->d_src.as<char>();
    p->src_elem = (const int64_t *)(d + o_el);
    p->src_uelem = (const int64_t *)(d + o_ue);
    p->src_par = (const double *)(d + o_par);
    p->src_wts = (const double *)(d + o_w);
    p->shot_off = (const int32_t *)(d + o_so);
    p->src_tile = (const int32_t *)(d + o_t);
    p->src_node = (const int4 *)(d + o_n);
    p->has_src = (const uint8_t *)(d + o_h);
    p->stf = (double *)(d + o_stf);
    p->n_src_uelem = (int)ue.size();
    SALVUS_CUDA(cudaMemcpyAsync(d, img.data(), img.size(), cudaMemcpyHostToDevice, p->stream));
    SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  }
  p->src_dirty = false;
  p->stf_ready = false;
  return SALVUS_OK;
}

static int upload_receivers(salvus_problem *p) {
  if (!p->rec_dirty) return SALVUS_OK;
  const salvus_mesh *m = p->mesh;
  const size_t nr = p->recs.size();
  int rc;
  std::vector<int64_t> el(nr ? nr : 1, 0);
  std::vector<double> l(nr ? nr * m->P : 1, 0.0);
  for (size_t r = 0; r < nr; ++r) {
    el[r] = p->recs[r].elem;
    std::memcpy(&l[r * m->P], p->recs[r].l.data(), sizeof(double) * m->P);
  }
  if ((rc = p->d_rec_elem.alloc(sizeof(int64_t) * el.size()))) return rc;
  if ((rc = p->d_rec_l.alloc(sizeof(double) * l.size()))) return rc;
  size_t sz = sizeof(double) * (size_t)(nr ? nr : 1) * p->c * p->seis_cap * p->shots_pad;
  if ((rc = p->d_seis.alloc(sz))) return rc;
  SALVUS_CUDA(cudaMemsetAsync(p->d_seis.ptr, 0, sz, p->stream));
  SALVUS_CUDA(cudaMemcpyAsync(p->d_rec_elem.ptr, el.data(), sizeof(int64_t) * el.size(),
                              cudaMemcpyHostToDevice, p->stream));
  SALVUS_CUDA(cudaMemcpyAsync(p->d_rec_l.ptr, l.data(), sizeof(double) * l.size(),
                              cudaMemcpyHostToDevice, p->stream));
  SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  p->rec_dirty = false;
  return SALVUS_OK;
}

static void drop_graph(salvus_problem *p) {
  if (p->graph_exec) cudaGraphExecDestroy(p->graph_exec);
  p->graph_exec = nullptr;
  p->graph_steps = 0;
  if (p->tail_exec) cudaGraphExecDestroy(p->tail_exec);
  p->tail_exec = nullptr;
  p->tail_steps = 0;
}

// fluid-solid coupling integrals (meshes of fluid and solid quadrilaterals);
// half_step: what d_v holds when the launch runs (which, captured, is later)
template <typename real>
static int launch_coupling(salvus_problem *p, bool half_step) {
  const salvus_mesh *m = p->mesh;
  if (m->physics != SALVUS_COUPLED2D || m->n_cpl == 0) return SALVUS_OK;
  const real *coef = sizeof(real) == 4 ? (const real *)m->d_cpl32.ptr : (const real *)m->d_cpl64.ptr;
  coupling_kernel<real><<<blocks_for(m->n_cpl, 256), 256, 0, p->stream>>>(
      m->n_cpl_fluid, m->n_cpl, m->d_cpl_pts.as<int32_t>(), coef, F<real>(p->d_v),
      F<real>(p->d_ap), half_step ? (real)(0.5 * p->dt) : real(0), F<real>(p->d_r));
  g_launches++;
  return check_launch("coupling");
}

template <typename real, int C>
static int launch_dirichlet(salvus_problem *p) {
  if (p->n_dir_pts == 0) return SALVUS_OK;
  dirichlet_zero_kernel<real, C><<<blocks_for(p->n_dir_pts, 256), 256, 0, p->stream>>>(
      p->n_dir_pts, p->d_dir_pts.as<int32_t>(), F<real>(p->d_r));
  g_launches++;
  return check_launch("dirichlet");
}

// The tail of step n (step_tail_kernel) samples its receivers, which read u
// after its update, and evaluates the sources of step n + 1, whose stiffness
// launch only reads u.  In the steps a graph run captures (rec_overlap) it
// therefore runs on a second stream, forked after the node update, and step
// n + 1 joins it after its stiffness launch, before its node update (which
// writes u and advances the step counter): off the critical path, which is
// two launches.  The captured sequence ends joined, so every later operation
// on the problem's stream is ordered after it.  Host-launched and profiled
// steps keep it on the problem's stream.
static int join_receivers(salvus_problem *p) {
  if (!p->rec_pending) return SALVUS_OK;
  p->rec_pending = false;
  SALVUS_CUDA(cudaStreamWaitEvent(p->stream, p->ev_recorded, 0));
  return SALVUS_OK;
}

template <typename real, int C>
static int launch_step_tail(salvus_problem *p, int nrec, cudaStream_t st) {
  const int nsrc = (int)p->srcs.size(), blocks = nrec + (nsrc > 0 ? 1 : 0);
  if (blocks == 0) return SALVUS_OK;
  step_tail_kernel<real, C><<<blocks, kRecThreads, 0, st>>>(
      nrec, p->mesh->P, p->d_rec_elem.as<int64_t>(), p->d_rec_l.as<double>(),
      p->mesh->d_conn.as<int32_t>(), F<real>(p->d_u), p->d_seis.as<double>(), p->seis_cap,
      p->d_step.as<int64_t>(), nsrc, p->src_par, p->dt, p->stf);
  g_launches++;
  return check_launch("receivers");
}

template <typename real, int C>
static int launch_receivers(salvus_problem *p) {
  ProfScope ps(p, K_REC);
  const int nrec = (int)p->recs.size();
  if (nrec == 0 && p->srcs.empty()) return SALVUS_OK;
  const bool fork = p->rec_overlap && !p->profiling && p->rec_stream;
  if (!fork) return launch_step_tail<real, C>(p, nrec, p->stream);
  SALVUS_CUDA(cudaEventRecord(p->ev_updated, p->stream));
  SALVUS_CUDA(cudaStreamWaitEvent(p->rec_stream, p->ev_updated, 0));
  int rc = launch_step_tail<real, C>(p, nrec, p->rec_stream);
  SALVUS_CUDA(cudaEventRecord(p->ev_recorded, p->rec_stream));
  p->rec_pending = true;
  return rc;
}

// The source-time functions of the step that the device counter stands at,
// where no tail has evaluated them (new sources, a new time step, steps of a
// single-launch group).  Never inside a graph capture: the entry points call
// it before they step or capture.
static int sources_ready(salvus_problem *p) {
  if (p->stf_ready || p->srcs.empty() || p->shots > 1) return SALVUS_OK;
  ProfScope ps(p, K_SRC);
  p->stf_ready = true;
  return launch_step_tail<float, 1>(p, 0, p->stream);  // no receiver: the type does not matter
}

template <typename real>
static const real *records(const salvus_problem *p) {
  return sizeof(real) == 4 ? (const real *)p->mesh->d_rec32.ptr : (const real *)p->mesh->d_rec64.ptr;
}
template <typename real>
static const real *inv_mass(const salvus_problem *p) {
  return sizeof(real) == 4 ? (const real *)p->mesh->d_mi32.ptr : (const real *)p->mesh->d_mi64.ptr;
}

// The fused FP32 step of parallelepiped elastic hexahedra advances the
// element-interior nodes inside the stiffness kernel and gathers the rest
// (kernels_hex_affine.cuh).  Measured on the 64^3 order-4 workload it is
// slower than the plain sequence on the same records (the interior update
// costs the stiffness kernel more than the shorter gather saves, figures at
// tune_hex), so it runs only where SALVUS_HEX_STEP=fused (read at every step)
// or SALVUS_HEX_CONFIG asks for it.  It is
// admissible for problems without Dirichlet points and with at most
// kFuseMaxSources sources (each interior column scans their elements).
constexpr int kFuseMaxSources = 16;
static bool hex_fusion_admissible(const salvus_problem *p) {
  const salvus_mesh *m = p->mesh;
  return m->affine && m->n_gnodes > 0 && p->prec == SALVUS_FP32 && p->shots == 1 &&
         p->n_dir_pts == 0 && (int)p->srcs.size() <= kFuseMaxSources;
}
static bool hex_interior_fusion(const salvus_problem *p) {
  if (!hex_fusion_admissible(p)) return false;
  const char *s = std::getenv("SALVUS_HEX_STEP");
  if (s && std::strcmp(s, "fused") == 0) return true;
  if (s && std::strcmp(s, "plain") == 0) return false;
  return p->hex_form == 1;
}

template <bool TI>
static int launch_fused_interior(salvus_problem *p, const HexInteriorUpdate &iu) {
  const salvus_mesh *m = p->mesh;
  const float *mat = m->d_rec32.as<float>();
  float *u = F<float>(p->d_u), *r = F<float>(p->d_r);
  switch (m->order) {
    case 2: return launch_elastic_affine<2, TI, true>(m, mat, u, r, p->stream, iu);
    case 3: return launch_elastic_affine<3, TI, true>(m, mat, u, r, p->stream, iu);
    case 4: return launch_elastic_affine<4, TI, true>(m, mat, u, r, p->stream, iu);
    case 5: return launch_elastic_affine<5, TI, true>(m, mat, u, r, p->stream, iu);
    case 6: return launch_elastic_affine<6, TI, true>(m, mat, u, r, p->stream, iu);
  }
  return fail(SALVUS_E_UNSUPPORTED, "fused hexahedron step: order %d", m->order);
}

static int step_fused_hex_interior(salvus_problem *p, bool store_a) {
  const salvus_mesh *m = p->mesh;
  int rc;
  // this stiffness launch writes u (interior nodes): the previous step's
  // receivers, which read u, finish first
  if ((rc = join_receivers(p))) return rc;
  {
    ProfScope ps(p, K_STIFF);
    HexInteriorUpdate iu{};
    iu.mi = m->d_mi32.as<float>();
    iu.w = F<float>(p->d_v);
    iu.ap = store_a ? F<float>(p->d_ap) : nullptr;
    iu.dt = (float)p->dt;
    iu.nsrc_elem = p->n_src_uelem;
    iu.src_elem = p->src_uelem;
    if ((rc = m->ti ? launch_fused_interior<true>(p, iu) : launch_fused_interior<false>(p, iu)))
      return rc;
  }
  // sources, then the source elements' interior nodes
  if (!p->srcs.empty()) {
    ProfScope ps(p, K_SRC);
    auto go = [&](auto nt) {
      constexpr int N = decltype(nt)::value;
      source_fused_hex_kernel<N><<<1, 256, 0, p->stream>>>(
          m->P, F<float>(p->d_r), p->n_src_uelem, p->src_uelem,
          m->d_conn.as<int32_t>(), m->d_mi32.as<float>(), F<float>(p->d_u), F<float>(p->d_v),
          store_a ? F<float>(p->d_ap) : nullptr, (float)p->dt, source_terms(p));
    };
    switch (m->order) {
      case 2: go(std::integral_constant<int, 2>{}); break;
      case 3: go(std::integral_constant<int, 3>{}); break;
      case 4: go(std::integral_constant<int, 4>{}); break;
      case 5: go(std::integral_constant<int, 5>{}); break;
      case 6: go(std::integral_constant<int, 6>{}); break;
      default: return fail(SALVUS_E_UNSUPPORTED, "fused hexahedron step: order %d", m->order);
    }
    g_launches++;
    if ((rc = check_launch("source (fused step)"))) return rc;
  }
  {
    ProfScope ps(p, K_UPDATE);
    gather_list_kernel<float, 3, 0><<<blocks_for(m->n_gnodes, 256), 256, 0, p->stream>>>(
        m->n_gnodes, m->d_gnodes.as<int32_t>(), m->d_inc_off.as<int32_t>(),
        m->d_inc_idx.as<int32_t>(), F<float>(p->d_r), m->d_mi32.as<float>(), F<float>(p->d_u),
        F<float>(p->d_v), store_a ? F<float>(p->d_ap) : nullptr, nullptr, (float)p->dt,
        source_terms(p), p->d_step.as<int64_t>());
    g_launches++;
    if ((rc = check_launch("gather update (shared nodes)"))) return rc;
  }
  return launch_receivers<float, 3>(p);
}

// store_a: keep this step's a in a_ (every step that a caller can see; the
// steps inside a run only where the fluid-solid coupling reads v)
template <typename real, int C>
static int step_fused_t(salvus_problem *p, bool store_a) {
  const salvus_mesh *m = p->mesh;
  int rc;
  if constexpr (std::is_same<real, float>::value && C == 3) {
    if (hex_interior_fusion(p)) return step_fused_hex_interior(p, store_a);
  }
  {
    ProfScope ps(p, K_STIFF);
    if ((rc = launch_stiffness<real>(m, records<real>(p), F<real>(p->d_u), F<real>(p->d_r), p->stream,
                                       p->d_err.as<int>(), p->wait_limit, p->hold_waits)))
      return rc;
  }
  if ((rc = join_receivers(p))) return rc;  // the previous step's receivers
  if ((rc = launch_dirichlet<real, C>(p))) return rc;
  if ((rc = launch_coupling<real>(p, true))) return rc;
  {
    ProfScope ps(p, K_UPDATE);
    if (C == 1 && gather_pairs(m, m->G))
      gather_pair_kernel<real><<<blocks_for(m->G, kPairTile), kGatherThreads, 0, p->stream>>>(
          m->G, incidence(m), F<real>(p->d_r), inv_mass<real>(p), F<real>(p->d_u), F<real>(p->d_v),
          store_a ? F<real>(p->d_ap) : nullptr, (real)p->dt, source_terms(p),
          p->d_step.as<int64_t>());
    else
      gather_kernel<real, C, 0><<<blocks_for(m->G, kGatherThreads), kGatherThreads, 0, p->stream>>>(
          m->G, m->d_inc_off.as<int32_t>(), m->d_inc_idx.as<int32_t>(), F<real>(p->d_r),
          inv_mass<real>(p), F<real>(p->d_u), F<real>(p->d_v),
          store_a || m->physics == SALVUS_COUPLED2D ? F<real>(p->d_ap) : nullptr, nullptr,
          (real)p->dt, source_terms(p), p->d_step.as<int64_t>());
    g_launches++;
    if ((rc = check_launch("gather update"))) return rc;
  }
  return launch_receivers<real, C>(p);
}

// ---------------------------------------------------------------------------
// shot-batched step (FP32 acoustic quads)
struct BatchCfg {
  int sc, epc, npt;  // shots, elements / node groups per CTA, nodes per thread
  bool timed = false;  // a candidate of the autotuner; the others run where they are pinned
};
// The places in these lists are what SALVUS_BATCH_CONFIG names: new shapes go to
// the end.  Stiffness: the third number is the shots per thread; {0, 1, 2} takes
// CTAs of pair_shots.  Below 64 shots its CTAs would be less than a warp.
static const BatchCfg kStiffCfg[] = {{32, 1, 1, true}, {32, 2, 1, true}, {32, 4, 1, true},
                                     {64, 1, 1, true}, {64, 2, 1},       {128, 1, 1, true},
                                     {128, 2, 1},      {256, 1, 1},      {0, 1, 2, true}};
// shots per CTA of {0, 1, 2}: the most 32-shot groups, up to eight, that
// divide the padded shots
static int pair_shots(int shots_pad) {
  for (int k = 8; k > 1; --k)
    if (shots_pad % (32 * k) == 0) return 32 * k;
  return 32;
}
static bool stiff_cfg_fits(int cfg, int shots_pad) {
  const int sc = kStiffCfg[cfg].sc;
  return sc ? shots_pad % sc == 0 : pair_shots(shots_pad) >= 64;
}
// Gather: 32 to 64 threads in the first twelve (four shots a thread), 128 to 256
// in the others, which the autotuner times.
static const BatchCfg kGatherCfg[] = {
    {32, 4, 1},         {32, 8, 1},         {64, 2, 1},         {64, 4, 1},
    {128, 1, 1},        {128, 2, 1},        {256, 1, 1},        {32, 4, 2},
    {64, 2, 2},         {128, 1, 2},        {128, 1, 4},        {256, 1, 2},
    {32, 16, 1, true},  {32, 32, 1, true},  {64, 8, 1, true},   {64, 16, 1, true},
    {128, 4, 1, true},  {128, 8, 1, true},  {256, 2, 1, true},  {256, 4, 1, true},
    {32, 16, 2, true},  {64, 8, 2, true},   {128, 4, 2, true},  {256, 2, 2, true}};
constexpr int kNumStiffCfg = sizeof(kStiffCfg) / sizeof(kStiffCfg[0]);
constexpr int kNumGatherCfg = sizeof(kGatherCfg) / sizeof(kGatherCfg[0]);

// Fused batched step (kernels_batch.cuh, kFuse): interior nodes advanced in
// the stiffness kernel, edge nodes by the node-list gather.  Used when the
// mesh has interior nodes (order >= 2); SALVUS_BATCH_STEP=unfused selects
// the plain sequence (read at every step).
static bool batch_fusion(const salvus_problem *p) {
  if (p->mesh->n_gnodes <= 0) return false;
  const char *s = std::getenv("SALVUS_BATCH_STEP");
  return !(s && std::strcmp(s, "unfused") == 0);
}

template <int N, int SC, int EPC, int V>
static void launch_qb(const salvus_problem *p, cudaStream_t st, bool fuse) {
  const salvus_mesh *m = p->mesh;
  const int sc = SC ? SC : pair_shots(p->shots_pad);
  dim3 grid((unsigned)((m->E + EPC - 1) / EPC), (unsigned)(p->shots_pad / sc));
  BatchInterior bi{};
  if (fuse) {
    bi.mi = m->d_mi32.as<float>();
    bi.w = F<float>(p->d_v);
    bi.dt = (float)p->dt;
    bi.shot_off = p->shot_off;
    bi.src_elem = p->src_elem;
    bi.has_src = p->srcs.empty() ? nullptr : p->has_src;
    quad_acoustic_batched_kernel<N, SC, EPC, V, true><<<grid, sc / V * EPC, 0, st>>>(
        m->E, p->shots_pad, m->d_rec32.as<float>(), F<float>(p->d_u), F<float>(p->d_r),
        dmatrix<float>(m->basis), bi);
  } else {
    quad_acoustic_batched_kernel<N, SC, EPC, V, false><<<grid, sc / V * EPC, 0, st>>>(
        m->E, p->shots_pad, m->d_rec32.as<float>(), F<float>(p->d_u), F<float>(p->d_r),
        dmatrix<float>(m->basis), bi);
  }
}

template <int N>
static int launch_qb_cfg(const salvus_problem *p, int cfg, cudaStream_t st, bool fuse) {
  switch (cfg) {
    case 0: launch_qb<N, 32, 1, 1>(p, st, fuse); break;
    case 1: launch_qb<N, 32, 2, 1>(p, st, fuse); break;
    case 2: launch_qb<N, 32, 4, 1>(p, st, fuse); break;
    case 3: launch_qb<N, 64, 1, 1>(p, st, fuse); break;
    case 4: launch_qb<N, 64, 2, 1>(p, st, fuse); break;
    case 5: launch_qb<N, 128, 1, 1>(p, st, fuse); break;
    case 6: launch_qb<N, 128, 2, 1>(p, st, fuse); break;
    case 7: launch_qb<N, 256, 1, 1>(p, st, fuse); break;
    case 8: launch_qb<N, 0, 1, 2>(p, st, fuse); break;
    default: return fail(SALVUS_E_INVALID, "bad batch config %d", cfg);
  }
  g_launches++;
  return check_launch("batched stiffness");
}

static int batched_stiffness(const salvus_problem *p, int cfg, cudaStream_t st, bool fuse) {
  switch (p->mesh->order) {
    case 1: return launch_qb_cfg<1>(p, cfg, st, false);  // no interior nodes
    case 2: return launch_qb_cfg<2>(p, cfg, st, fuse);
    case 3: return launch_qb_cfg<3>(p, cfg, st, fuse);
    case 4: return launch_qb_cfg<4>(p, cfg, st, fuse);
    case 5: return launch_qb_cfg<5>(p, cfg, st, fuse);
    case 6: return launch_qb_cfg<6>(p, cfg, st, fuse);
  }
  return fail(SALVUS_E_UNSUPPORTED, "batched quads support orders 1..6");
}

template <int SC, int NPB, int NPT = 1>
static void launch_bg(const salvus_problem *p, cudaStream_t st, bool fuse, int64_t *step) {
  const salvus_mesh *m = p->mesh;
  const int64_t n = fuse ? m->n_gnodes : m->G;
  dim3 grid((unsigned)((n + NPB * NPT - 1) / (NPB * NPT)), (unsigned)(p->shots_pad / SC));
  batched_gather_update_kernel<SC, NPB, NPT><<<grid, SC / 4 * NPB, 0, st>>>(
      n, p->shots_pad, incidence(m),
      F<float>(p->d_r), m->d_mi32.as<float>(), F<float>(p->d_u), F<float>(p->d_v), (float)p->dt,
      fuse ? m->d_gnodes.as<int32_t>() : nullptr, step);
}

// step: the device step counter to advance (null: a timing run of the autotuner)
static int batched_gather(const salvus_problem *p, int cfg, cudaStream_t st, bool fuse,
                          int64_t *step) {
  switch (cfg) {
    case 0: launch_bg<32, 4>(p, st, fuse, step); break;
    case 1: launch_bg<32, 8>(p, st, fuse, step); break;
    case 2: launch_bg<64, 2>(p, st, fuse, step); break;
    case 3: launch_bg<64, 4>(p, st, fuse, step); break;
    case 4: launch_bg<128, 1>(p, st, fuse, step); break;
    case 5: launch_bg<128, 2>(p, st, fuse, step); break;
    case 6: launch_bg<256, 1>(p, st, fuse, step); break;
    case 7: launch_bg<32, 4, 2>(p, st, fuse, step); break;
    case 8: launch_bg<64, 2, 2>(p, st, fuse, step); break;
    case 9: launch_bg<128, 1, 2>(p, st, fuse, step); break;
    case 10: launch_bg<128, 1, 4>(p, st, fuse, step); break;
    case 11: launch_bg<256, 1, 2>(p, st, fuse, step); break;
    case 12: launch_bg<32, 16>(p, st, fuse, step); break;
    case 13: launch_bg<32, 32>(p, st, fuse, step); break;
    case 14: launch_bg<64, 8>(p, st, fuse, step); break;
    case 15: launch_bg<64, 16>(p, st, fuse, step); break;
    case 16: launch_bg<128, 4>(p, st, fuse, step); break;
    case 17: launch_bg<128, 8>(p, st, fuse, step); break;
    case 18: launch_bg<256, 2>(p, st, fuse, step); break;
    case 19: launch_bg<256, 4>(p, st, fuse, step); break;
    case 20: launch_bg<32, 16, 2>(p, st, fuse, step); break;
    case 21: launch_bg<64, 8, 2>(p, st, fuse, step); break;
    case 22: launch_bg<128, 4, 2>(p, st, fuse, step); break;
    case 23: launch_bg<256, 2, 2>(p, st, fuse, step); break;
    default: return fail(SALVUS_E_INVALID, "bad gather config %d", cfg);
  }
  g_launches++;
  return check_launch("batched gather");
}

// Times every admissible configuration of the batched stiffness and gather
// kernels on this problem and keeps the fastest.  The stiffness timing writes
// only the residual scratch; the gather timing runs on copies of u and w, so
// the problem's state is untouched.  Results are cached per (order, padded
// shots, elements, device, step form) for the process.
static int autotune(salvus_problem *p) {
  if (p->tune_stiff >= 0 && p->tune_gather >= 0) return SALVUS_OK;
  // "stiff,gather" fixes the choice, whatever other problems of this size were
  // tuned to
  const char *env = std::getenv("SALVUS_BATCH_CONFIG");
  if (env) {
    int a = -1, b = -1;
    if (std::sscanf(env, "%d,%d", &a, &b) == 2 && a >= 0 && a < kNumStiffCfg && b >= 0 &&
        b < kNumGatherCfg && stiff_cfg_fits(a, p->shots_pad) && p->shots_pad % kGatherCfg[b].sc == 0) {
      p->tune_stiff = a;
      p->tune_gather = b;
      return SALVUS_OK;
    }
  }
  struct Key {
    int order, shots;
    int64_t E;
    int dev;
    bool fuse;  // the two forms of the step move different work
  };
  const bool fuse = batch_fusion(p);
  static std::mutex cache_mu;
  static std::vector<std::pair<Key, std::pair<int, int>>> cache;
  {
    std::lock_guard<std::mutex> lk(cache_mu);
    for (auto &c : cache)
      if (c.first.order == p->mesh->order && c.first.shots == p->shots_pad &&
          c.first.E == p->mesh->E && c.first.dev == p->mesh->device && c.first.fuse == fuse) {
        p->tune_stiff = c.second.first;
        p->tune_gather = c.second.second;
        return SALVUS_OK;
      }
  }
  cudaEvent_t e0, e1;
  SALVUS_CUDA(cudaEventCreate(&e0));
  SALVUS_CUDA(cudaEventCreate(&e1));
  int rc = SALVUS_OK;
  auto time_it = [&](auto &&fn) -> float {
    float best = 1e30f;
    for (int rep = 0; rep < 3; ++rep) {
      cudaEventRecord(e0, p->stream);
      if ((rc = fn())) return 1e30f;
      cudaEventRecord(e1, p->stream);
      cudaEventSynchronize(e1);
      float ms = 0;
      cudaEventElapsedTime(&ms, e0, e1);
      best = std::min(best, ms);
    }
    return best;
  };
  // both kernels are timed on zeroed scratch copies of u and w (the fused
  // stiffness kernel also advances interior nodes), so the problem's state
  // is untouched
  const size_t nf = (size_t)p->mesh->G * p->shots_pad * sizeof(float);
  DeviceBuffer su, sw;
  float bs = 1e30f;
  int cs = -1;
  if (rc == SALVUS_OK && ((rc = su.alloc(nf)) == SALVUS_OK) && ((rc = sw.alloc(nf)) == SALVUS_OK)) {
    std::swap(p->d_u.ptr, su.ptr);
    std::swap(p->d_v.ptr, sw.ptr);
    cudaMemsetAsync(p->d_u.ptr, 0, nf, p->stream);
    cudaMemsetAsync(p->d_v.ptr, 0, nf, p->stream);
    for (int c = 0; c < kNumStiffCfg && rc == SALVUS_OK; ++c) {
      if (!kStiffCfg[c].timed || !stiff_cfg_fits(c, p->shots_pad)) continue;
      float t = time_it([&] { return batched_stiffness(p, c, p->stream, fuse); });
      if (t < bs) { bs = t; cs = c; }
    }
    float bg = 1e30f;
    int cg = -1;
    for (int c = 0; c < kNumGatherCfg && rc == SALVUS_OK; ++c) {
      if (!kGatherCfg[c].timed || p->shots_pad % kGatherCfg[c].sc) continue;
      float t = time_it([&] { return batched_gather(p, c, p->stream, fuse, nullptr); });
      if (t < bg) { bg = t; cg = c; }
    }
    std::swap(p->d_u.ptr, su.ptr);
    std::swap(p->d_v.ptr, sw.ptr);
    p->tune_gather = cg;
  }
  cudaStreamSynchronize(p->stream);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  if (cs < 0 || p->tune_gather < 0) return fail(SALVUS_E_INVALID, "no admissible batch configuration");
  p->tune_stiff = cs;
  std::lock_guard<std::mutex> lk(cache_mu);
  cache.push_back({{p->mesh->order, p->shots_pad, p->mesh->E, p->mesh->device, fuse},
                   {p->tune_stiff, p->tune_gather}});
  return SALVUS_OK;
}

static int step_batched(salvus_problem *p) {
  const salvus_mesh *m = p->mesh;
  int rc;
  {
    ProfScope ps(p, K_STIFF);
    if ((rc = batched_stiffness(p, p->tune_stiff, p->stream, batch_fusion(p)))) return rc;
  }
  if (!p->srcs.empty()) {
    ProfScope ps(p, K_SRC);
    const int threads = 256, total = p->shots_pad * m->P;
    // fused step: the source elements' interior nodes are finished here
    const bool fuse = batch_fusion(p) && m->order >= 2;
    batched_source_kernel<<<(total + threads - 1) / threads, threads, 0, p->stream>>>(
        p->shots_pad, m->P, p->shot_off, p->src_elem,
        p->src_par, p->src_wts, p->d_step.as<int64_t>(), p->dt,
        F<float>(p->d_r), fuse ? m->n : 0, m->d_conn.as<int32_t>(), m->d_mi32.as<float>(),
        F<float>(p->d_u), F<float>(p->d_v), (float)p->dt);
    g_launches++;
    if ((rc = check_launch("batched sources"))) return rc;
  }
  {
    ProfScope ps(p, K_UPDATE);
    if ((rc = batched_gather(p, p->tune_gather, p->stream, batch_fusion(p),
                             p->d_step.as<int64_t>()))) return rc;
  }
  ProfScope ps(p, K_REC);
  if (!p->recs.empty()) {
    const int threads = p->shots_pad < 256 ? p->shots_pad : 256;
    batched_receiver_kernel<<<(unsigned)p->recs.size(), threads, 0, p->stream>>>(
        p->shots_pad, (int)p->recs.size(), m->P, p->d_rec_elem.as<int64_t>(),
        p->d_rec_l.as<double>(), m->d_conn.as<int32_t>(), F<float>(p->d_u),
        p->d_seis.as<double>(), p->seis_cap, p->d_step.as<int64_t>());
    g_launches++;
  }
  return check_launch("batched receivers");
}

static int step_fused(salvus_problem *p, bool store_a) {
  if (p->shots > 1) return step_batched(p);
  return by_components(p->c, [&](auto cc) {
    constexpr int C = decltype(cc)::value;
    return p->prec == SALVUS_FP32 ? step_fused_t<float, C>(p, store_a)
                                  : step_fused_t<double, C>(p, store_a);
  });
}

// Puts d_v into the form the caller needs: half = true before steps (w = v +
// dt/2 a_), false before v or a_ is overwritten or dt changes.  One pass over
// the field, and only when the form changes: a run after a run converts
// nothing.  Batched problems hold w throughout.
static int velocity_form(salvus_problem *p, bool half) {
  if (p->shots > 1 || p->half_step == half) return SALVUS_OK;
  const int64_t N = p->mesh->G * p->c;
  const double s = (half ? 0.5 : -0.5) * p->dt;
  if (p->prec == SALVUS_FP32)
    axpy_kernel<float><<<blocks_for(N, 256), 256, 0, p->stream>>>(N, (float)s, F<float>(p->d_ap),
                                                                  F<float>(p->d_v));
  else
    axpy_kernel<double><<<blocks_for(N, 256), 256, 0, p->stream>>>(N, s, F<double>(p->d_ap),
                                                                   F<double>(p->d_v));
  g_launches++;
  p->half_step = half;
  return check_launch("velocity form");
}

template <typename real, int C>
static int assemble_t(salvus_problem *p) {
  const salvus_mesh *m = p->mesh;
  int rc;
  {
    ProfScope ps(p, K_STIFF);
    if ((rc = launch_stiffness<real>(m, records<real>(p), F<real>(p->d_u), F<real>(p->d_r), p->stream,
                                       p->d_err.as<int>(), p->wait_limit, p->hold_waits)))
      return rc;
  }
  if ((rc = launch_dirichlet<real, C>(p))) return rc;
  if ((rc = launch_coupling<real>(p, p->half_step))) return rc;
  ProfScope ps(p, K_GATHER);
  gather_kernel<real, C, 1><<<blocks_for(m->G, 256), 256, 0, p->stream>>>(
      m->G, m->d_inc_off.as<int32_t>(), m->d_inc_idx.as<int32_t>(), F<real>(p->d_r), nullptr,
      nullptr, nullptr, nullptr, F<real>(p->d_a), (real)0, source_terms(p));
  g_launches++;
  return check_launch("gather");
}

template <typename real, int C>
static int minv_t(salvus_problem *p) {
  ProfScope ps(p, K_MINV);
  const int64_t N = p->mesh->G * C;
  inverse_mass_kernel<real, C><<<blocks_for(N, 256), 256, 0, p->stream>>>(
      p->mesh->G, inv_mass<real>(p), F<real>(p->d_a));
  g_launches++;
  return check_launch("inverse mass");
}

template <typename real, int C>
static int newmark_t(salvus_problem *p) {
  int rc;
  {
    ProfScope ps(p, K_NEWMARK);
    const int64_t N = p->mesh->G * C;
    newmark_kernel<real><<<blocks_for(N, 256), 256, 0, p->stream>>>(
        N, F<real>(p->d_a), F<real>(p->d_u), F<real>(p->d_v), F<real>(p->d_ap), (real)p->dt,
        p->d_step.as<int64_t>());
    g_launches++;
    if ((rc = check_launch("newmark"))) return rc;
  }
  return launch_receivers<real, C>(p);
}

// True when the FP32 stiffness launch of this mesh runs a kernel whose
// bounded waits report a timeout through the error word (tensor-core
// simplices); mirrors launch_stiffness.
bool stiffness_reports_errors(const salvus_mesh *m, int precision) {
  if (precision != SALVUS_FP32) return false;
  if (m->shape == SALVUS_TET) return m->tet_kernel == 0;
  if (m->shape == SALVUS_TRI) return m->tri_kernel == 0;
  return false;
}

// a = -K u for caller-owned device buffers, with the element-local residual
// in caller-provided scratch and timeouts of bounded device waits recorded in
// the caller-provided device word `err` (used by
// salvus_apply_stiffness_noalloc).
template <typename real>
static int apply_stiffness_into_t(const salvus_mesh *m, const real *rec, const real *u, real *a,
                                  real *scratch, int *err, cudaStream_t st) {
  int rc = launch_stiffness<real>(m, rec, u, scratch, st, err);
  if (rc) return rc;
  return by_components(m->c, [&](auto cc) {
    gather_kernel<real, decltype(cc)::value, 1><<<blocks_for(m->G, 256), 256, 0, st>>>(
        m->G, m->d_inc_off.as<int32_t>(), m->d_inc_idx.as<int32_t>(), scratch, nullptr, nullptr,
        nullptr, nullptr, a, (real)0);
    g_launches++;
    return check_launch("allocation-free gather");
  });
}

int apply_stiffness_into(const salvus_mesh *m, int precision, const void *u, void *a,
                         void *scratch, int *err, cudaStream_t st) {
  if (precision == SALVUS_FP32)
    return apply_stiffness_into_t<float>(m, m->d_rec32.as<float>(), (const float *)u, (float *)a,
                                         (float *)scratch, err, st);
  if (!m->d_rec64.ptr)
    return fail(SALVUS_E_STATE, "mesh holds no FP64 records (created with SALVUS_MESH_FP32_ONLY)");
  return apply_stiffness_into_t<double>(m, m->d_rec64.as<double>(), (const double *)u,
                                        (double *)a, (double *)scratch, err, st);
}

// Reads the device status word: set by kernels whose bounded waits ran out
// (the wait's code) or by the finite check (kNonFiniteCode).
int status_error(const salvus_problem *p, int h) {
  if (h == kNonFiniteCode)
    return fail(SALVUS_E_NONFINITE,
                "the wavefield became non-finite (NaN / Inf) by step %lld: the time step is "
                "unstable or an input field is not finite",
                (long long)p->step);
  if (h) return fail(SALVUS_E_TIMEOUT, "a bounded device wait gave up (code %d); results invalid", h);
  return SALVUS_OK;
}

static int device_status(salvus_problem *p) {
  int h = 0;
  SALVUS_CUDA(cudaMemcpyAsync(&h, p->d_err.ptr, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
  SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  return status_error(p, h);
}

int enqueue_seis_copy(salvus_problem *p, double *ring, int *status) {
  if (!p || !ring || !status) return fail(SALVUS_E_INVALID, "null argument");
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  const int64_t rows = (int64_t)p->shots * p->recs.size() * p->c;
  if (rows > 0 && p->d_seis.ptr)
    SALVUS_CUDA(cudaMemcpyAsync(ring, p->d_seis.ptr, sizeof(double) * rows * p->seis_cap,
                                cudaMemcpyDeviceToHost, p->stream));
  SALVUS_CUDA(cudaMemcpyAsync(status, p->d_err.ptr, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
  return SALVUS_OK;
}

void seis_ring_shape(const salvus_problem *p, int64_t *rows, int64_t *capacity) {
  if (rows) *rows = (int64_t)p->shots * p->recs.size() * p->c;
  if (capacity) *capacity = p->seis_cap;
}

// Finite check of u (all shots) into the status word; part of every 32-step
// chunk (kFiniteEvery) of salvus_run and of the single-step entry points.
constexpr int kFiniteEvery = 32;
static int launch_finite_check(salvus_problem *p) {
  const int64_t n = p->mesh->G * p->c * p->shots_pad;
  const int64_t want = (n + 255) / 256, cap = (int64_t)p->mesh->sm_count * 8;
  const unsigned grid = (unsigned)std::max<int64_t>(1, std::min(want, cap));
  if (p->prec == SALVUS_FP32)
    finite_check_kernel<float><<<grid, 256, 0, p->stream>>>(n, F<float>(p->d_u), p->d_err.as<int>());
  else
    finite_check_kernel<double><<<grid, 256, 0, p->stream>>>(n, F<double>(p->d_u), p->d_err.as<int>());
  g_launches++;
  return check_launch("finite check");
}

// Hexahedron autotuner (FP32 elastic meshes of parallelepipeds of orders 1-3,
// one shot): times the plain step (stiffness, node gather/update) with CTAs of 128 /
// (N+1)^2 elements and with twice as many, on zeroed scratch copies of u and
// w, and keeps the faster.  Both give bitwise the same wavefield (the same
// arithmetic per element and per node, in the same order), so the choice
// changes only the time.  Results are cached per (order, elements, nodes,
// anisotropy, device) for the process; the CTA width belongs to the mesh.
// The fused interior form is not among the candidates: it lost on every mesh
// measured (per step, plain against fused: 64^3 order 4 0.73 / 0.84 ms, 16^3
// order 4 15.1 / 19.4 us, 18^3 order 5 anisotropic 35.6 / 52.1 us) and its
// source launch and receivers stay on the critical path.
// SALVUS_HEX_CONFIG="form,wide" fixes form and width; SALVUS_HEX_STEP forces
// the form.  Without room for the scratch fields the default width is kept.
static int tune_hex(salvus_problem *p) {
  if (p->hex_form >= 0) return SALVUS_OK;
  salvus_mesh *m = p->mesh;
  if (!(m->shape == SALVUS_HEX && m->affine && m->physics == SALVUS_ELASTIC3D &&
        p->prec == SALVUS_FP32 && p->shots == 1 && !m->host_only)) {
    p->hex_form = 0;
    return SALVUS_OK;
  }
  struct Key {
    int order;
    int64_t E, G;
    bool ti;
    int dev;
  };
  if (const char *env = std::getenv("SALVUS_HEX_CONFIG")) {
    const bool fusable = hex_fusion_admissible(p) && m->order >= 2 && m->order <= 6;
    int a = -1, b = -1;
    if (std::sscanf(env, "%d,%d", &a, &b) == 2 && (a == 0 || (a == 1 && fusable)) &&
        (b == 0 || b == 1)) {
      p->hex_form = a;
      m->hex_wide = b;
      return SALVUS_OK;
    }
  }
  // line-exchange kernels (orders 4 and up): the narrow CTA was the faster one
  // on every mesh measured (64^3 order 4: 0.377 against 0.434 ms), and on
  // small ones a few timed launches picked the slower (16^3: 15.4 against 13.9
  // us a step)
  if (m->order >= 4) {
    p->hex_form = 0;
    m->hex_wide = 0;  // an earlier problem may have pinned the other
    return SALVUS_OK;
  }
  // problems are prepared on several threads (the job server)
  static std::mutex cache_mu;
  static std::vector<std::pair<Key, int>> cache;
  {
    std::lock_guard<std::mutex> lk(cache_mu);
    for (auto &c : cache)
      if (c.first.order == m->order && c.first.E == m->E && c.first.G == m->G &&
          c.first.ti == m->ti && c.first.dev == m->device) {
        p->hex_form = 0;
        m->hex_wide = c.second;
        return SALVUS_OK;
      }
  }
  p->hex_form = 0;
  const size_t nf = (size_t)m->G * 3 * sizeof(float);
  DeviceBuffer su, sv;
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || free_b < 2 * nf + (size_t(1) << 30) ||
      su.alloc(nf) || sv.alloc(nf)) {
    cudaGetLastError();
    return SALVUS_OK;
  }
  SALVUS_CUDA(cudaMemsetAsync(su.ptr, 0, nf, p->stream));
  SALVUS_CUDA(cudaMemsetAsync(sv.ptr, 0, nf, p->stream));
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  int rc = SALVUS_OK;
  // one step without sources and receivers (the same for both widths)
  auto sequence = [&]() -> int {
    int r;
    if ((r = launch_stiffness<float>(m, records<float>(p), su.as<float>(), F<float>(p->d_r),
                                     p->stream, p->d_err.as<int>(), p->wait_limit, 0)))
      return r;
    gather_kernel<float, 3, 0><<<blocks_for(m->G, kGatherThreads), kGatherThreads, 0, p->stream>>>(
        m->G, m->d_inc_off.as<int32_t>(), m->d_inc_idx.as<int32_t>(), F<float>(p->d_r),
        m->d_mi32.as<float>(), su.as<float>(), sv.as<float>(), nullptr, nullptr, (float)p->dt);
    g_launches++;
    return check_launch("hexahedron autotuner");
  };
  float best = 1e30f;
  int bw = 0;
  for (int w = 0; w < 2 && rc == SALVUS_OK; ++w) {
    m->hex_wide = w;
    if ((rc = sequence())) break;  // first launch (attributes, caches)
    float t = 1e30f;
    for (int rep = 0; rep < 3 && rc == SALVUS_OK; ++rep) {
      cudaEventRecord(e0, p->stream);
      for (int k = 0; k < 4 && rc == SALVUS_OK; ++k) rc = sequence();
      cudaEventRecord(e1, p->stream);
      cudaEventSynchronize(e1);
      float ms = 0;
      cudaEventElapsedTime(&ms, e0, e1);
      t = std::min(t, ms);
    }
    if (rc == SALVUS_OK && t < best) {
      best = t;
      bw = w;
    }
  }
  cudaStreamSynchronize(p->stream);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  m->hex_wide = bw;
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(cache_mu);
  cache.push_back({{m->order, m->E, m->G, m->ti, m->device}, bw});
  return SALVUS_OK;
}

static int ready(salvus_problem *p) {
  if (!p) return fail(SALVUS_E_INVALID, "null problem");
  if (!p->dt_set) return fail(SALVUS_E_STATE, "time step not set (salvus_problem_set_dt)");
  int rc;
  if ((rc = upload_sources(p))) return rc;
  if ((rc = upload_receivers(p))) return rc;
  if (p->shots > 1 && (rc = autotune(p))) return rc;
  if ((rc = tune_hex(p))) return rc;
  return SALVUS_OK;
}

// ---------------------------------------------------------------------------
// problem groups: FP32 single-shot problems of one element class advance with
// one launch per stage (kernels_group.cuh)
template <int N>
static int group_stiffness_t(const salvus_mesh *m0, const GroupSlot *slots, const int32_t *owner,
                             int64_t blocks, cudaStream_t st) {
  if (m0->shape == SALVUS_QUAD) {
    group_quad_acoustic_stiffness<N><<<(unsigned)blocks, QuadColShape<N, quad_col_epb<N>()>::THREADS,
                                        0, st>>>(slots, owner, dmatrix<float>(m0->basis));
  } else if constexpr (N <= kMaxHexOrder) {
    constexpr int n2 = (N + 1) * (N + 1), EPB = 128 / n2 > 0 ? 128 / n2 : 1;
    using T = ElasticV2Shape<N, EPB, false>;
    static OncePerDevice attr;
    if (int rc = dynamic_smem(attr, m0, group_hex_elastic_stiffness<N, EPB>, T::SMEM)) return rc;
    group_hex_elastic_stiffness<N, EPB><<<(unsigned)blocks, T::THREADS, T::SMEM, st>>>(
        slots, owner, dmatrix<float>(m0->basis));
  }
  g_launches++;
  return check_launch("group stiffness");
}

static int group_stiffness(const salvus_mesh *m0, const GroupSlot *slots, const int32_t *owner,
                           int64_t blocks, cudaStream_t st) {
  switch (m0->order) {
    case 1: return group_stiffness_t<1>(m0, slots, owner, blocks, st);
    case 2: return group_stiffness_t<2>(m0, slots, owner, blocks, st);
    case 3: return group_stiffness_t<3>(m0, slots, owner, blocks, st);
    case 4: return group_stiffness_t<4>(m0, slots, owner, blocks, st);
    case 5: return group_stiffness_t<5>(m0, slots, owner, blocks, st);
    case 6: return group_stiffness_t<6>(m0, slots, owner, blocks, st);
    case 7: return group_stiffness_t<7>(m0, slots, owner, blocks, st);
    case 8: return group_stiffness_t<8>(m0, slots, owner, blocks, st);
    case 9: return group_stiffness_t<9>(m0, slots, owner, blocks, st);
    case 10: return group_stiffness_t<10>(m0, slots, owner, blocks, st);
  }
  return fail(SALVUS_E_UNSUPPORTED, "no grouped stiffness for order %d", m0->order);
}

// stiffness CTAs per member (the single-problem kernel's element groups)
static int64_t group_stiff_blocks(const salvus_mesh *m) {
  const int n2 = m->n * m->n;
  if (m->shape == SALVUS_QUAD) {
    const int epb = 128 / m->n > 0 ? 128 / m->n : 1;  // quad_col_epb<N>()
    return (m->E + epb - 1) / epb;
  }
  const int epb = 128 / n2 > 0 ? 128 / n2 : 1;  // v2 with 128-thread CTAs
  return (m->E + epb - 1) / epb;
}

}  // namespace salvus

struct salvus_group {
  std::vector<salvus_problem *> members;
  const salvus_mesh *m0 = nullptr;
  int c = 1;
  bool stages = true;  // one launch per stage; SALVUS_GROUP_STEP=persistent: one queue launch per step
  bool partitioned = false;  // SALVUS_GROUP_STEP=partitioned: one cooperative launch per step
  std::vector<salvus::GroupPart> parts;
  salvus::DeviceBuffer d_parts, d_bars;
  int coop_slots = 0;  // co-resident CTAs of the partitioned kernel
  std::vector<salvus::GroupSlot> slots;
  salvus::DeviceBuffer d_slots;
  // per-stage CTA -> member tables of the per-stage launches, one after the
  // other: stiffness (n_stiff), gather (n_gather), receivers (n_rec)
  std::vector<int32_t> owner;
  salvus::DeviceBuffer d_owner;
  int64_t n_stiff = 0, n_gather = 0, n_rec = 0;
  bool pairs = false;  // two nodes per thread in the gather
  // persistent single-launch step: work-item queue
  std::vector<salvus::GroupCounts> counts;
  std::vector<salvus::GroupWork> work;
  int64_t total = 0;
  int grid = 0;
  salvus::DeviceBuffer d_counts, d_work, d_done, d_sync;
  long long wait_limit = salvus::kDefaultWaitLimit;  // bound of the device waits, SM cycles
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev = nullptr;
  std::vector<cudaEvent_t> member_ev;
  cudaGraphExec_t graph = nullptr;
  int graph_steps = 0;
  int64_t sig[3] = {-1, -1, -1};
};

namespace salvus {

static int group_upload(salvus::DeviceBuffer &b, const void *src, size_t bytes, cudaStream_t st) {
  if (b.bytes < bytes) {
    int rc = b.alloc(bytes);
    if (rc) return rc;
  }
  SALVUS_CUDA(cudaMemcpyAsync(b.ptr, src, bytes, cudaMemcpyHostToDevice, st));
  return SALVUS_OK;
}

static int group_partitioned(salvus_group *g, bool launch, bool store_a);

static int group_fill(salvus_group *g) {
  int64_t bs = 0, bg = 0, br = 0;
  g->slots.resize(g->members.size());
  for (size_t k = 0; k < g->members.size(); ++k) {
    salvus_problem *p = g->members[k];
    const salvus_mesh *m = p->mesh;
    int rc = ready(p);
    if (rc) return rc;
    GroupSlot &s = g->slots[k];
    s.rec = m->qscalar ? m->d_qs32.as<float>() : m->d_rec32.as<float>();
    s.jac = m->affine ? m->d_jac32.as<float>() : nullptr;
    s.square = m->qscalar;
    s.conn = m->d_conn.as<int32_t>();
    s.inc_off = m->d_inc_off.as<int32_t>();
    s.inc_idx = m->d_inc_idx.as<int32_t>();
    s.inc = incidence(m);
    s.mi = m->d_mi32.as<float>();
    s.E = m->E;
    s.G = m->G;
    s.u = p->d_u.as<float>();
    s.w = p->d_v.as<float>();
    s.ap = p->d_ap.as<float>();
    s.r = p->d_r.as<float>();
    s.dt = (float)p->dt;
    s.dtd = p->dt;
    s.step = p->d_step.as<int64_t>();
    s.nsrc = (int)p->srcs.size();
    s.nrec = (int)p->recs.size();
    s.src_par = p->src_par;
    s.src = source_terms(p);
    s.stf = p->stf;
    s.rec_elem = p->d_rec_elem.as<int64_t>();
    s.rec_l = p->d_rec_l.as<double>();
    s.seis = p->d_seis.as<double>();
    s.cap = p->seis_cap;
    s.b_stiff = bs;
    s.b_gather = bg;
    s.b_rec = br;
    bs += group_stiff_blocks(m);
    bg += (m->G + 255) / 256;  // 256 nodes per CTA in both forms (kPairTile)
    br += s.nrec + (s.nsrc > 0 ? 1 : 0);
  }
  int64_t nodes = 0;
  for (auto *p : g->members) nodes += p->mesh->G;
  g->pairs = gather_pairs(g->m0, nodes);
  g->n_stiff = bs;
  g->n_gather = bg;
  g->n_rec = br;
  int rc = group_upload(g->d_slots, g->slots.data(), sizeof(GroupSlot) * g->slots.size(), g->stream);
  if (rc) return rc;
  g->owner.resize((size_t)(bs + bg + br));
  {
    int32_t *o = g->owner.data();
    for (size_t k = 0; k < g->members.size(); ++k) {
      const GroupSlot &sk = g->slots[k];
      const salvus_mesh *mk = g->members[k]->mesh;
      std::fill(o + sk.b_stiff, o + sk.b_stiff + group_stiff_blocks(mk), (int32_t)k);
      std::fill(o + bs + sk.b_gather, o + bs + sk.b_gather + (mk->G + 255) / 256, (int32_t)k);
      std::fill(o + bs + bg + sk.b_rec, o + bs + bg + sk.b_rec + sk.nrec + (sk.nsrc > 0 ? 1 : 0),
                (int32_t)k);
    }
  }
  if ((rc = group_upload(g->d_owner, g->owner.data(), sizeof(int32_t) * g->owner.size(), g->stream)))
    return rc;
  // work-item queue of the persistent step: every member's stiffness items
  // (kStiffPer element groups each), then per member source (1), gather items
  // (kGatherPer CTA-wide node tiles each), receivers (1 each), advance (1)
  constexpr int kStiffPer = 2, kGatherPer = 8;
  const int J = (int)g->members.size();
  const int tile = 128;  // CTA width of the persistent kernel
  g->counts.assign(J, GroupCounts{0, 0, 0});
  g->work.clear();
  auto add = [&](int type, int j, int64_t tiles, int per) -> int32_t {
    int32_t items = 0;
    for (int64_t f = 0; f < tiles; f += per, ++items)
      g->work.push_back(GroupWork{type, j, (int)f, (int)std::min<int64_t>(per, tiles - f)});
    return items;
  };
  for (int j = 0; j < J; ++j)
    g->counts[j].stiff = add(GI_STIFF, j, group_stiff_blocks(g->members[j]->mesh), kStiffPer);
  for (int j = 0; j < J; ++j) {
    add(GI_SRC, j, 1, 1);
    g->counts[j].gather = add(GI_GATHER, j, (g->members[j]->mesh->G + tile - 1) / tile, kGatherPer);
    g->counts[j].rec = add(GI_REC, j, (int64_t)g->members[j]->recs.size(), 1);
    add(GI_ADV, j, 1, 1);
  }
  g->total = (int64_t)g->work.size();
  if ((rc = group_upload(g->d_counts, g->counts.data(), sizeof(GroupCounts) * J, g->stream))) return rc;
  if ((rc = group_upload(g->d_work, g->work.data(), sizeof(GroupWork) * g->work.size(), g->stream)))
    return rc;
  if (g->d_done.bytes < sizeof(int32_t) * 4 * J) {
    if ((rc = g->d_done.alloc(sizeof(int32_t) * 4 * J))) return rc;
    SALVUS_CUDA(cudaMemsetAsync(g->d_done.ptr, 0, sizeof(int32_t) * 4 * J, g->stream));
  }
  if (!g->d_sync.ptr) {
    if ((rc = g->d_sync.alloc(sizeof(GroupSync)))) return rc;
    SALVUS_CUDA(cudaMemsetAsync(g->d_sync.ptr, 0, sizeof(GroupSync), g->stream));
  }
  // the partitioned step's CTA ranges and counters (allocated here, before any capture)
  if (g->partitioned) return group_partitioned(g, false, false);
  return SALVUS_OK;
}

template <int N, bool kHex, int C>
static int group_persistent_t(salvus_group *g, bool store_a) {
  constexpr int threads = 128;
  size_t smem = 0;
  if constexpr (kHex) {
    constexpr int n2 = (N + 1) * (N + 1), EPB = 128 / n2 > 0 ? 128 / n2 : 1;
    smem = ElasticV2Shape<N, EPB, false>::SMEM;
  }
  auto kern = group_persistent_step<N, kHex, C>;
  if (g->grid == 0) {
    if (smem) SALVUS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    SALVUS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
    g->grid = (per_sm > 0 ? per_sm : 1) * g->m0->sm_count;
  }
  const int grid = (int)std::min<int64_t>(g->grid, g->total);
  kern<<<grid, threads, smem, g->stream>>>(
      g->d_slots.as<GroupSlot>(), g->d_counts.as<GroupCounts>(), (int)g->members.size(),
      g->d_work.as<GroupWork>(), g->total, g->d_done.as<int32_t>(), g->d_sync.as<GroupSync>(),
      dmatrix<float>(g->m0->basis), g->m0->P, g->wait_limit, store_a);
  g_launches++;
  return check_launch("group persistent step");
}

static int group_persistent(salvus_group *g, bool store_a) {
  const salvus_mesh *m = g->m0;
  if (m->shape == SALVUS_HEX) {
    switch (m->order) {
      case 1: return group_persistent_t<1, true, 3>(g, store_a);
      case 2: return group_persistent_t<2, true, 3>(g, store_a);
      case 3: return group_persistent_t<3, true, 3>(g, store_a);
      case 4: return group_persistent_t<4, true, 3>(g, store_a);
      case 5: return group_persistent_t<5, true, 3>(g, store_a);
      case 6: return group_persistent_t<6, true, 3>(g, store_a);
    }
  } else {
    switch (m->order) {
      case 1: return group_persistent_t<1, false, 1>(g, store_a);
      case 2: return group_persistent_t<2, false, 1>(g, store_a);
      case 3: return group_persistent_t<3, false, 1>(g, store_a);
      case 4: return group_persistent_t<4, false, 1>(g, store_a);
      case 5: return group_persistent_t<5, false, 1>(g, store_a);
      case 6: return group_persistent_t<6, false, 1>(g, store_a);
      case 7: return group_persistent_t<7, false, 1>(g, store_a);
      case 8: return group_persistent_t<8, false, 1>(g, store_a);
      case 9: return group_persistent_t<9, false, 1>(g, store_a);
      case 10: return group_persistent_t<10, false, 1>(g, store_a);
    }
  }
  return fail(SALVUS_E_UNSUPPORTED, "no grouped step for order %d", m->order);
}

// launch=false: size the member CTA ranges (once) and allocate their counters;
// launch=true: one cooperative launch of the step
template <int N, bool kHex, int C>
static int group_partitioned_t(salvus_group *g, bool launch, bool store_a) {
  constexpr int threads = 128;
  size_t smem = 0;
  if constexpr (kHex) {
    constexpr int n2 = (N + 1) * (N + 1), EPB = 128 / n2 > 0 ? 128 / n2 : 1;
    smem = ElasticV2Shape<N, EPB, false>::SMEM;
  }
  auto kern = group_partitioned_step<N, kHex, C>;
  const int J = (int)g->members.size();
  if (!launch) {
    if (g->coop_slots == 0) {
      if (smem) SALVUS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      int per_sm = 0;
      SALVUS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
      g->coop_slots = (per_sm > 0 ? per_sm : 1) * g->m0->sm_count;
    }
    if (g->parts.size() == (size_t)J) return SALVUS_OK;
    // CTAs per member in proportion to its work (element points + nodes), at least one
    if (J > g->coop_slots)
      return fail(SALVUS_E_UNSUPPORTED, "%d members exceed the %d co-resident CTAs", J, g->coop_slots);
    const int tile = 128;
    std::vector<double> w(J);
    double wsum = 0;
    for (int j = 0; j < J; ++j) {
      const salvus_mesh *m = g->members[j]->mesh;
      w[j] = (double)m->E * m->P + (double)m->G;
      wsum += w[j];
    }
    std::vector<GroupPart> parts(J);
    const int spare = g->coop_slots - J;
    int first = 0;
    for (int j = 0; j < J; ++j) {
      const salvus_mesh *m = g->members[j]->mesh;
      GroupPart &pt = parts[j];
      pt.cta_first = first;
      pt.cta_count = 1 + (int)std::floor((double)spare * w[j] / wsum);
      pt.n_stiff = (int32_t)group_stiff_blocks(m);
      pt.n_gather = (int32_t)((m->G + tile - 1) / tile);
      first += pt.cta_count;
    }
    int rc = group_upload(g->d_parts, parts.data(), sizeof(GroupPart) * J, g->stream);
    if (rc) return rc;
    if ((rc = g->d_bars.alloc(sizeof(GroupBar) * J))) return rc;
    SALVUS_CUDA(cudaMemsetAsync(g->d_bars.ptr, 0, sizeof(GroupBar) * J, g->stream));
    g->parts = std::move(parts);
    return SALVUS_OK;
  }
  if (g->parts.size() != (size_t)J) return fail(SALVUS_E_INVALID, "partitioned group not set up");
  const int grid = g->parts.back().cta_first + g->parts.back().cta_count;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = g->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SALVUS_CUDA(cudaLaunchKernelEx(&cfg, kern, (const GroupSlot *)g->d_slots.as<GroupSlot>(),
                                 (const GroupPart *)g->d_parts.as<GroupPart>(), J,
                                 g->d_bars.as<GroupBar>(), g->d_sync.as<GroupSync>(),
                                 dmatrix<float>(g->m0->basis), g->m0->P,
                                 (long long)g->wait_limit, store_a));
  g_launches++;
  return check_launch("group partitioned step");
}

static int group_partitioned(salvus_group *g, bool launch, bool store_a) {
  const salvus_mesh *m = g->m0;
  if (m->shape == SALVUS_HEX) {
    switch (m->order) {
      case 1: return group_partitioned_t<1, true, 3>(g, launch, store_a);
      case 2: return group_partitioned_t<2, true, 3>(g, launch, store_a);
      case 3: return group_partitioned_t<3, true, 3>(g, launch, store_a);
      case 4: return group_partitioned_t<4, true, 3>(g, launch, store_a);
      case 5: return group_partitioned_t<5, true, 3>(g, launch, store_a);
      case 6: return group_partitioned_t<6, true, 3>(g, launch, store_a);
    }
  } else {
    switch (m->order) {
      case 1: return group_partitioned_t<1, false, 1>(g, launch, store_a);
      case 2: return group_partitioned_t<2, false, 1>(g, launch, store_a);
      case 3: return group_partitioned_t<3, false, 1>(g, launch, store_a);
      case 4: return group_partitioned_t<4, false, 1>(g, launch, store_a);
      case 5: return group_partitioned_t<5, false, 1>(g, launch, store_a);
      case 6: return group_partitioned_t<6, false, 1>(g, launch, store_a);
      case 7: return group_partitioned_t<7, false, 1>(g, launch, store_a);
      case 8: return group_partitioned_t<8, false, 1>(g, launch, store_a);
      case 9: return group_partitioned_t<9, false, 1>(g, launch, store_a);
      case 10: return group_partitioned_t<10, false, 1>(g, launch, store_a);
    }
  }
  return fail(SALVUS_E_UNSUPPORTED, "no grouped step for order %d", m->order);
}

// store_a: keep a_ (the last step of a run, see step_fused_t)
static int group_step(salvus_group *g, bool store_a) {
  if (g->partitioned) return group_partitioned(g, true, store_a);
  if (!g->stages) return group_persistent(g, store_a);
  const int P = g->m0->P;
  const GroupSlot *slots = g->d_slots.as<GroupSlot>();
  int rc;
  const int32_t *own = g->d_owner.as<int32_t>();
  if ((rc = group_stiffness(g->m0, slots, own, g->n_stiff, g->stream))) return rc;
  if (g->pairs)
    group_gather_pairs<<<(unsigned)g->n_gather, kGatherThreads, 0, g->stream>>>(slots, own + g->n_stiff, store_a);
  else if (g->c == 1) group_gather_update<1><<<(unsigned)g->n_gather, 256, 0, g->stream>>>(slots, own + g->n_stiff, store_a);
  else group_gather_update<3><<<(unsigned)g->n_gather, 256, 0, g->stream>>>(slots, own + g->n_stiff, store_a);
  if (g->n_rec > 0) {
    const int32_t *own_rec = own + g->n_stiff + g->n_gather;
    if (g->c == 1) group_step_tail<1><<<(unsigned)g->n_rec, kRecThreads, 0, g->stream>>>(slots, own_rec, P);
    else group_step_tail<3><<<(unsigned)g->n_rec, kRecThreads, 0, g->stream>>>(slots, own_rec, P);
  }
  g_launches += g->n_rec > 0 ? 2 : 1;
  return check_launch("group step");
}

}  // namespace salvus

using namespace salvus;

// ===========================================================================
extern "C" {

const char *salvus_last_error(void) { return salvus::last_error(); }

const char *salvus_version(void) {
  return "salvus_b200 0.1 (sm_100a; FP32/FP64 tensor-product SEM; deterministic gather assembly)";
}

int64_t salvus_launch_count(void) { return g_launches.load(); }

int salvus_element_tables(int32_t shape, int32_t order, int32_t *n_points, double *points,
                          double *weights, double *dphi) {
  Basis b;
  int rc = make_basis(shape, order, &b);
  if (rc) return rc;
  const int P = b.P, dim = b.dim;
  if (n_points) *n_points = P;
  std::vector<double> phi(P), dp((size_t)P * 3);
  for (int q = 0; q < P; ++q) {
    double ref[3];
    point_ref(b, q, ref);
    if (points)
      for (int a = 0; a < dim; ++a) points[(size_t)q * dim + a] = ref[a];
    if (weights) weights[q] = point_weight(b, q);
    if (dphi) {
      if (b.simplex) {
        for (int k = 0; k < dim; ++k)
          for (int i = 0; i < P; ++i) dphi[((size_t)k * P + i) * P + q] = b.SD[((size_t)k * P + i) * P + q];
      } else {
        basis_at(b, ref, phi.data(), dp.data());
        for (int k = 0; k < dim; ++k)
          for (int i = 0; i < P; ++i) dphi[((size_t)k * P + i) * P + q] = dp[(size_t)i * 3 + k];
      }
    }
  }
  return SALVUS_OK;
}

int salvus_mesh_create(const salvus_mesh_desc *d, int device, salvus_mesh **out) {
  if (!d || !out) return fail(SALVUS_E_INVALID, "null argument");
  *out = nullptr;
  if (d->shape < SALVUS_QUAD || d->shape > SALVUS_TET)
    return fail(SALVUS_E_UNSUPPORTED, "unknown element shape %d", d->shape);
  if (d->physics == SALVUS_ELASTIC3D && d->shape != SALVUS_HEX && d->shape != SALVUS_TET)
    return fail(SALVUS_E_UNSUPPORTED, "elastic 3-D physics needs hexahedra or tetrahedra");
  if ((d->physics == SALVUS_ELASTIC2D || d->physics == SALVUS_COUPLED2D) && d->shape != SALVUS_QUAD)
    return fail(SALVUS_E_UNSUPPORTED, "elastic 2-D and coupled physics need quadrilaterals");
  if (d->physics < SALVUS_ACOUSTIC || d->physics > SALVUS_COUPLED2D)
    return fail(SALVUS_E_INVALID, "unknown physics %d", d->physics);
  if (d->n_elements <= 0 || d->n_vertices <= 0 || !d->vertices || !d->cells || !d->params)
    return fail(SALVUS_E_INVALID, "empty mesh");
  std::unique_ptr<salvus_mesh> m(new salvus_mesh());
  m->device = device;
  m->fp32_only = (d->reserved & SALVUS_MESH_FP32_ONLY) != 0;
  {
    // FP32 tetrahedra: tensor cores by default; SALVUS_TET_KERNEL=cuda selects
    // the CUDA-core kernel (read when the mesh is created)
    const char *s = std::getenv("SALVUS_TET_KERNEL");
    m->tet_kernel = (s && std::strcmp(s, "cuda") == 0) ? 1 : 0;
    // triangles: CUDA cores with the derivative table in constant memory by
    // default; SALVUS_TRI_KERNEL=tc selects the tensor-core kernel (FP32),
    // =shared the shared-memory-table kernel (read when the mesh is created)
    const char *t = std::getenv("SALVUS_TRI_KERNEL");
    m->tri_kernel = (t && std::strcmp(t, "tc") == 0) ? 0 : (t && std::strcmp(t, "shared") == 0) ? 2 : 1;
  }
  m->shape = d->shape;
  m->order = d->order;
  m->physics = d->physics;
  int rc = make_basis(d->shape, d->order, &m->basis);
  if (rc) return rc;
  m->dim = m->basis.dim;
  m->nv = m->basis.nv;
  m->n = m->basis.n;
  m->P = m->basis.P;
  m->c = physics_components(d->physics);
  m->npar = physics_params(d->physics, d->reserved);
  m->E = d->n_elements;
  m->vtx.resize((size_t)(m->E * m->nv * m->dim));
  for (int64_t e = 0; e < m->E; ++e)
    for (int k = 0; k < m->nv; ++k) {
      int64_t vi = d->cells[e * m->nv + k];
      if (vi < 0 || vi >= d->n_vertices)
        return fail(SALVUS_E_INVALID, "element %lld references vertex %lld out of range",
                    (long long)e, (long long)vi);
      for (int a = 0; a < m->dim; ++a)
        m->vtx[(size_t)((e * m->nv + k) * m->dim + a)] = d->vertices[vi * m->dim + a];
    }
  for (int64_t e = 0; e < m->E; ++e) {
    // right-hand rule check (QuadP1::checkHull / HexP1::checkHull): detJ > 0
    // at every corner (simplices: the constant detJ)
    const double *v = m->vtx.data() + e * m->nv * m->dim;
    const int ncheck = is_simplex(m->shape) ? 1 : (m->dim == 2 ? 4 : 8);
    for (int q = 0; q < ncheck; ++q) {
      double ref[3] = {0, 0, 0};
      if (!is_simplex(m->shape))
        for (int a = 0; a < m->dim; ++a) ref[a] = ((q >> a) & 1) ? 1.0 : -1.0;
      double det;
      p1_jacobian(m->shape, v, ref, &det, nullptr);
      if (!(det > 0))
        return fail(SALVUS_E_INVALID, "element %lld is inverted or degenerate (detJ <= 0)",
                    (long long)e);
    }
  }
  const size_t npar_total = (size_t)m->npar * m->E * m->nv;
  m->par.assign(d->params, d->params + npar_total);
  for (size_t i = 0; i < npar_total; ++i)
    if (!std::isfinite(m->par[i])) return fail(SALVUS_E_INVALID, "non-finite material parameter");
  if (m->npar == 6) {
    // RHO VPV VPH VSV VSH ETA (Elastic3D.cpp:33-54).  An isotropic model
    // (VPH = VPV, VSH = VSV, ETA = 1 everywhere) keeps the two-constant
    // records and kernels; anything else gets the five-constant ones.
    const size_t K = (size_t)m->E * m->nv;
    const double *pr = m->par.data();
    bool iso = true;
    for (size_t i = 0; i < K && iso; ++i)
      iso = pr[2 * K + i] == pr[K + i] && pr[4 * K + i] == pr[3 * K + i] && pr[5 * K + i] == 1.0;
    if (iso) {
      std::vector<double> p3(3 * K);
      std::copy(pr, pr + K, p3.begin());                    // RHO
      std::copy(pr + K, pr + 2 * K, p3.begin() + K);        // VP = VPV
      std::copy(pr + 3 * K, pr + 4 * K, p3.begin() + 2 * K);  // VS = VSV
      m->par.swap(p3);
      m->npar = 3;
    } else {
      m->ti = true;
      m->tet_kernel = 1;  // tetrahedra: the CUDA-core kernel has the five-constant stress
    }
  }
  if (m->shape == SALVUS_HEX && m->physics == SALVUS_ELASTIC3D &&
      !(d->reserved & SALVUS_MESH_PER_POINT_GEOMETRY)) {
    // every element a parallelepiped: the inverse Jacobian at the eight
    // corners equals the element's (to 1e-12 relative).  FP64 takes the one
    // Jacobian only where they agree to eps |x| / (2 h) relative, the rounding of
    // the sums that form a point's own: boxes always, three in four sheared or
    // turned lattices of rounded coordinates.  At twice that the one Jacobian is
    // up to 2.8 times further from extended precision than the points', below
    // it at most 0.96 (rms over the GLL points)
    bool affine = true, affine64 = true;
    for (int64_t e = 0; e < m->E && affine; ++e) {
      const double *v = m->vtx.data() + e * 24;
      double det0, J0[9];
      p1_jacobian_edges(v, &det0, J0);
      double scale = 0, far = 0;
      for (int a = 0; a < 9; ++a) scale = std::max(scale, std::fabs(J0[a]));
      for (int a = 0; a < 24; ++a) far = std::max(far, std::fabs(v[a]));
      const double tol64 = 0.5 * 2.220446049250313e-16 * far * scale;
      for (int q = 0; q < 8 && affine; ++q) {
        double ref[3], det, J[9];
        for (int a = 0; a < 3; ++a) ref[a] = ((q >> a) & 1) ? 1.0 : -1.0;
        p1_jacobian(m->shape, v, ref, &det, J);
        for (int a = 0; a < 9; ++a) {
          if (std::fabs(J[a] - J0[a]) > 1e-12 * scale) affine = false;
          if (std::fabs(J[a] - J0[a]) > tol64 * scale) affine64 = false;
        }
      }
    }
    m->affine = affine;
    m->affine64 = affine && affine64;
  }
  if (m->shape == SALVUS_QUAD && m->physics != SALVUS_ELASTIC2D) {
    // every element a square (opposite edges equal, adjacent ones equal and at a
    // right angle) to 1e-10 of the edge: G then differs from a multiple of the
    // identity by less than a hundredth of an FP32 rounding (6e-8)
    m->qsquare = true;
    for (int64_t e = 0; e < m->E && m->qsquare; ++e) {
      const double *v = m->vtx.data() + e * 8;
      const double a[2] = {v[2] - v[0], v[3] - v[1]}, b[2] = {v[6] - v[0], v[7] - v[1]};
      const double off = std::hypot((v[0] - v[2]) + (v[4] - v[6]), (v[1] - v[3]) + (v[5] - v[7]));
      const double aa = a[0] * a[0] + a[1] * a[1], bb = b[0] * b[0] + b[1] * b[1];
      m->qsquare = off <= 1e-10 * std::sqrt(aa) && std::fabs(aa - bb) <= 1e-10 * aa &&
                   std::fabs(a[0] * b[0] + a[1] * b[1]) <= 1e-10 * aa;
    }
    m->qscalar = m->qsquare && m->physics == SALVUS_ACOUSTIC &&
                 !(d->reserved & SALVUS_MESH_PER_POINT_GEOMETRY);
  }
  if ((rc = flatten_mesh(m.get(), d->cells, d->n_vertices))) return rc;
  if (m->physics == SALVUS_COUPLED2D && (rc = setup_coupled(m.get(), d->cells))) return rc;
  interior_free_nodes(m.get());
  if (device >= 0) {
    if ((rc = mesh_setup_device(m.get()))) return rc;
  } else {
    m->host_only = true;  // numbering and coordinates only; no GPU residency
  }
  *out = m.release();
  return SALVUS_OK;
}

int salvus_mesh_destroy(salvus_mesh *m) {
  if (!m) return SALVUS_OK;
  if (m->host_only) {
    delete m;
    return SALVUS_OK;
  }
  cudaSetDevice(m->device);
  if (m->stream) cudaStreamSynchronize(m->stream);
  cudaStream_t s = m->stream;
  delete m;
  if (s) cudaStreamDestroy(s);
  return SALVUS_OK;
}

int salvus_mesh_info(const salvus_mesh *m, int64_t *G, int32_t *c, int32_t *P) {
  if (!m) return fail(SALVUS_E_INVALID, "null mesh");
  if (G) *G = m->G;
  if (c) *c = m->c;
  if (P) *P = m->P;
  return SALVUS_OK;
}

int salvus_mesh_layout(const salvus_mesh *m, int32_t *per_element_jacobian,
                       int64_t *gathered_nodes) {
  if (!m) return fail(SALVUS_E_INVALID, "null mesh");
  if (per_element_jacobian) *per_element_jacobian = m->affine ? 1 : 0;
  if (gathered_nodes) *gathered_nodes = m->n_gnodes > 0 ? m->n_gnodes : m->G;
  return SALVUS_OK;
}

int salvus_mesh_node_coords(const salvus_mesh *m, double *xyz) {
  if (!m || !xyz) return fail(SALVUS_E_INVALID, "null argument");
  std::memcpy(xyz, m->xyz.data(), sizeof(double) * m->xyz.size());
  return SALVUS_OK;
}

int salvus_mesh_connectivity(const salvus_mesh *m, int64_t *conn) {
  if (!m || !conn) return fail(SALVUS_E_INVALID, "null argument");
  for (size_t i = 0; i < m->conn.size(); ++i) conn[i] = m->conn[i];
  return SALVUS_OK;
}

int salvus_mesh_locate_point(const salvus_mesh *m, const double *xyz, int64_t *elem, double *ref) {
  if (!m || !xyz || !elem || !ref) return fail(SALVUS_E_INVALID, "null argument");
  double x[3] = {xyz[0], xyz[1], m->dim == 3 ? xyz[2] : 0.0}, r[3] = {0, 0, 0};
  int rc = locate_point(m, x, elem, r);
  if (rc) return rc;
  for (int a = 0; a < m->dim; ++a) ref[a] = r[a];
  return SALVUS_OK;
}

int salvus_mesh_inverse_mass(const salvus_mesh *m, double *mi) {
  if (!m || !mi) return fail(SALVUS_E_INVALID, "null argument");
  if (m->host_only) return fail(SALVUS_E_STATE, "host-only mesh has no mass matrix");
  std::memcpy(mi, m->mi.data(), sizeof(double) * m->G);
  return SALVUS_OK;
}

int salvus_mesh_max_eigenvalue(salvus_mesh *m, int32_t iters, uint64_t seed, double *lam_out) {
  if (!m || !lam_out) return fail(SALVUS_E_INVALID, "null argument");
  if (m->host_only) return fail(SALVUS_E_STATE, "host-only mesh");
  if (m->fp32_only) return fail(SALVUS_E_STATE, "the eigenvalue estimate needs the FP64 records");
  SALVUS_CUDA(cudaSetDevice(m->device));
  const int64_t N = m->G * m->c;
  // partial sums of the three dot products, then the estimate
  DeviceBuffer x, y, r, part;
  int rc;
  if ((rc = x.alloc(8 * N)) || (rc = y.alloc(8 * N)) || (rc = r.alloc(8 * m->E * m->P * m->c)) ||
      (rc = part.alloc(sizeof(double) * (3 * kEigBlocks + 1))))
    return rc;
  std::vector<double> h(N);
  std::mt19937_64 rng(seed ? seed : 1);
  std::uniform_real_distribution<double> U(-0.5, 0.5);
  for (auto &v : h) v = U(rng);
  SALVUS_CUDA(cudaMemcpyAsync(x.ptr, h.data(), 8 * N, cudaMemcpyHostToDevice, m->stream));
  double *lam = part.as<double>() + 3 * kEigBlocks;
  SALVUS_CUDA(cudaMemsetAsync(lam, 0, sizeof(double), m->stream));
  // Nothing of an iteration comes back to the host: four launches, where three
  // dot products each copied and summed 512 partials there
  for (int it = 0; it < iters; ++it) {
    if ((rc = launch_stiffness<double>(m, m->d_rec64.as<double>(), x.as<double>(), r.as<double>(),
                                       m->stream)))
      return rc;
    rc = by_components(m->c, [&](auto cc) {
      constexpr int C = decltype(cc)::value;
      gather_kernel<double, C, 1><<<blocks_for(m->G, 256), 256, 0, m->stream>>>(
          m->G, m->d_inc_off.as<int32_t>(), m->d_inc_idx.as<int32_t>(), r.as<double>(), nullptr,
          nullptr, nullptr, nullptr, y.as<double>(), 0.0);
      eig_dots_kernel<C><<<kEigBlocks, kEigThreads, 0, m->stream>>>(
          N, m->d_mi64.as<double>(), x.as<double>(), y.as<double>(), part.as<double>());
      return SALVUS_OK;
    });
    if (rc) return rc;
    eig_scale_kernel<<<kEigBlocks, kEigThreads, 0, m->stream>>>(N, part.as<double>(),
                                                                y.as<double>(), lam);
    g_launches += 3;
    if ((rc = check_launch("eigenvalue iteration"))) return rc;
    std::swap(x.ptr, y.ptr);
  }
  SALVUS_CUDA(cudaMemcpyAsync(lam_out, lam, sizeof(double), cudaMemcpyDeviceToHost, m->stream));
  SALVUS_CUDA(cudaStreamSynchronize(m->stream));
  return SALVUS_OK;
}

int salvus_problem_create(salvus_mesh *m, int32_t precision, int32_t n_shots, salvus_problem **out) {
  if (!m || !out) return fail(SALVUS_E_INVALID, "null argument");
  *out = nullptr;
  if (m->host_only) return fail(SALVUS_E_STATE, "mesh was created host-only (device < 0)");
  if (precision != SALVUS_FP32 && precision != SALVUS_FP64)
    return fail(SALVUS_E_INVALID, "unknown precision %d", precision);
  if (n_shots < 1) return fail(SALVUS_E_INVALID, "n_shots must be >= 1");
  if (precision == SALVUS_FP64 && m->fp32_only)
    return fail(SALVUS_E_STATE, "mesh was created with SALVUS_MESH_FP32_ONLY");
  if (n_shots > 1 && (precision != SALVUS_FP32 || m->shape != SALVUS_QUAD ||
                      m->physics != SALVUS_ACOUSTIC || m->order > 6))
    return fail(SALVUS_E_UNSUPPORTED,
                "shot batching is built for FP32 acoustic quads of order 1..6 (got shape %d, "
                "order %d, precision %d)", m->shape, m->order, precision);
  SALVUS_CUDA(cudaSetDevice(m->device));
  std::unique_ptr<salvus_problem> p(new salvus_problem());
  p->mesh = m;
  p->device = m->device;
  p->prec = precision;
  p->shots = n_shots;
  p->shots_pad = n_shots == 1 ? 1 : (n_shots + 31) / 32 * 32;
  p->c = m->c;
  p->rsize = precision == SALVUS_FP32 ? 4 : 8;
  SALVUS_CUDA(cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking));
  const size_t nf = (size_t)m->G * p->c * p->rsize * p->shots_pad;
  const size_t na = n_shots == 1 ? nf : 16;  // batched problems keep no a / a_ fields
  int rc;
  if ((rc = p->d_u.alloc(nf)) || (rc = p->d_v.alloc(nf)) || (rc = p->d_a.alloc(na)) ||
      (rc = p->d_ap.alloc(na)) ||
      (rc = p->d_r.alloc((size_t)m->E * m->P * p->c * p->rsize * p->shots_pad)) ||
      (rc = p->d_step.alloc(sizeof(int64_t))) || (rc = p->d_err.alloc(sizeof(int))))
    return rc;
  SALVUS_CUDA(cudaMemsetAsync(p->d_err.ptr, 0, sizeof(int), p->stream));
  SALVUS_CUDA(cudaMemsetAsync(p->d_u.ptr, 0, nf, p->stream));
  SALVUS_CUDA(cudaMemsetAsync(p->d_v.ptr, 0, nf, p->stream));
  SALVUS_CUDA(cudaMemsetAsync(p->d_a.ptr, 0, na, p->stream));
  SALVUS_CUDA(cudaMemsetAsync(p->d_ap.ptr, 0, na, p->stream));
  SALVUS_CUDA(cudaMemsetAsync(p->d_step.ptr, 0, sizeof(int64_t), p->stream));
  SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  p->prof_ms.assign(K_NKINDS, 0.0);
  p->prof_n.assign(K_NKINDS, 0);
  *out = p.release();
  return SALVUS_OK;
}

int salvus_problem_destroy(salvus_problem *p) {
  if (!p) return SALVUS_OK;
  // the problem's own device: its mesh may already be gone
  cudaSetDevice(p->device);
  cudaStreamSynchronize(p->stream);
  drop_graph(p);
  for (auto &e : p->events) {
    cudaEventDestroy(e.a);
    cudaEventDestroy(e.b);
  }
  for (int b = 0; b < 2; ++b) {
    if (p->h_pin[b]) cudaFreeHost(p->h_pin[b]);
    if (p->pin_ev[b]) cudaEventDestroy(p->pin_ev[b]);
  }
  if (p->rec_stream) {
    cudaStreamSynchronize(p->rec_stream);
    cudaStreamDestroy(p->rec_stream);
    cudaEventDestroy(p->ev_updated);
    cudaEventDestroy(p->ev_recorded);
  }
  cudaStream_t s = p->stream;
  delete p;
  if (s) cudaStreamDestroy(s);
  return SALVUS_OK;
}

int salvus_problem_set_dt(salvus_problem *p, double dt) {
  if (!p) return fail(SALVUS_E_INVALID, "null problem");
  if (!(dt > 0) || !std::isfinite(dt)) return fail(SALVUS_E_INVALID, "dt must be positive");
  if (p->dt != dt) {
    drop_graph(p);
    SALVUS_CUDA(cudaSetDevice(p->mesh->device));
    if (int rc = velocity_form(p, false)) return rc;  // w belongs to the old step
    p->stf_ready = false;
  }
  p->dt = dt;
  p->dt_set = true;
  return SALVUS_OK;
}

int salvus_problem_add_source(salvus_problem *p, const salvus_source *s) {
  if (!p || !s) return fail(SALVUS_E_INVALID, "null argument");
  const salvus_mesh *m = p->mesh;
  if (s->shot < 0 || s->shot >= p->shots)
    return fail(SALVUS_E_INVALID, "shot index %d out of range", s->shot);
  if (s->kind == SALVUS_SOURCE_MOMENT_TENSOR && m->physics == SALVUS_ACOUSTIC)
    return fail(SALVUS_E_INVALID, "moment-tensor sources need elastic physics");
  if (s->kind != SALVUS_SOURCE_FORCE && s->kind != SALVUS_SOURCE_MOMENT_TENSOR)
    return fail(SALVUS_E_INVALID, "unknown source kind %d", s->kind);
  salvus_problem::Src src;
  src.desc = *s;
  int rc = locate_point(m, s->location, &src.elem, src.ref);
  if (rc) return rc;
  const int P = m->P, c = p->c;
  // components the owning element pushes: all, or on meshes of fluid and
  // solid elements u (fluid) / ux, uy (solid)
  int k0 = 0, k1 = c;
  if (m->physics == SALVUS_COUPLED2D) {
    const bool fl = m->par[(size_t)src.elem * 4] == 1.0;
    k0 = fl ? 0 : 1;
    k1 = fl ? 1 : 3;
    if (fl && s->kind == SALVUS_SOURCE_MOMENT_TENSOR)
      return fail(SALVUS_E_INVALID, "moment-tensor source inside a fluid element");
  }
  // delta-function coefficients phi_q(x_s) / (w_q detJ_q), times w_q detJ_q
  // by applyTestAndIntegrate (Scalar.cpp:87): phi_q(x_s) per unit force
  std::vector<double> phi(P), dphi((size_t)P * 3);
  basis_at(m->basis, src.ref, phi.data(), dphi.data());
  src.wts.assign((size_t)P * c, 0.0);
  if (s->kind == SALVUS_SOURCE_FORCE) {
    for (int q = 0; q < P; ++q)
      for (int a = k0; a < k1; ++a) src.wts[(size_t)q * c + a] = phi[q] * s->comp[a];
  } else {
    // 3-D comp = [Mxx Myy Mzz Myz Mxz Mxy]; 2-D comp = [Mxx Myy Mxy]
    const int d = m->dim;
    double det, iJ[9];
    p1_jacobian(m->shape, m->vtx.data() + src.elem * m->nv * d, src.ref, &det, iJ);
    double M[3][3] = {{s->comp[0], s->comp[5], s->comp[4]},
                      {s->comp[5], s->comp[1], s->comp[3]},
                      {s->comp[4], s->comp[3], s->comp[2]}};
    if (d == 2) {
      M[0][0] = s->comp[0];
      M[1][1] = s->comp[1];
      M[0][1] = M[1][0] = s->comp[2];
    }
    for (int q = 0; q < P; ++q) {
      const double *gref = &dphi[(size_t)q * 3];
      double gx[3] = {0, 0, 0};
      for (int a = 0; a < d; ++a)
        for (int k = 0; k < d; ++k) gx[a] += iJ[a * d + k] * gref[k];
      for (int a = 0; a < d; ++a) {
        double f = 0;
        for (int k = 0; k < d; ++k) f += M[a][k] * gx[k];
        src.wts[(size_t)q * c + k0 + a] = f;
      }
    }
  }
  p->srcs.push_back(std::move(src));
  p->src_dirty = true;
  drop_graph(p);
  return SALVUS_OK;
}

int salvus_problem_add_receiver(salvus_problem *p, const double *xyz) {
  if (!p || !xyz) return fail(SALVUS_E_INVALID, "null argument");
  const salvus_mesh *m = p->mesh;
  salvus_problem::Rec r;
  for (int a = 0; a < 3; ++a) r.xyz[a] = a < m->dim ? xyz[a] : 0.0;
  int rc = locate_point(m, r.xyz, &r.elem, r.ref);
  if (rc) return rc;
  r.l.resize(m->P);
  basis_at(m->basis, r.ref, r.l.data(), nullptr);
  p->recs.push_back(std::move(r));
  p->rec_dirty = true;
  drop_graph(p);
  return SALVUS_OK;
}

int salvus_problem_set_seismogram_capacity(salvus_problem *p, int64_t steps) {
  if (!p || steps <= 0) return fail(SALVUS_E_INVALID, "bad capacity");
  p->seis_cap = steps;
  p->rec_dirty = true;
  drop_graph(p);
  return SALVUS_OK;
}

// Host <-> device copies of whole fields through two pinned bounce chunks:
// the host copy into (out of) one chunk overlaps the DMA of the other, which
// runs at pinned-memory speed instead of the staged pageable path.  Small
// copies go directly.
static constexpr size_t kPinChunk = size_t(32) << 20;
// Host work on one chunk, split over the host threads (one thread's memcpy
// or conversion is slower than the DMA it feeds): fn(lo, hi) on [0, n).
static int host_threads() {
  static const int n = std::max(1, std::min(16, (int)std::thread::hardware_concurrency()));
  return n;
}
// Persistent host workers for those copies: a field of the 64^3 workload
// is 13 chunks, and creating and joining a fresh set of threads for every
// chunk cost about as much as the conversion itself.  One parallel job runs
// at a time (callers serialise on run_mu); the calling thread takes part 0.
// The pool is created on first use and never destroyed (its threads are
// detached and end with the process); a process forked after that has no
// workers, so it runs the parts itself.
extern "C++" {
class HostPool {
 public:
  static HostPool &get() {
    static HostPool *pool = new HostPool(host_threads());
    return *pool;
  }
  int threads() const { return T_; }
  void run(size_t n, size_t part, const std::function<void(size_t, size_t)> &fn) {
    if (getpid() != pid_ || T_ == 1) {
      for (size_t lo = 0; lo < n; lo += part) fn(lo, std::min(n, lo + part));
      return;
    }
    std::lock_guard<std::mutex> rl(run_mu_);
    {
      std::lock_guard<std::mutex> lk(mu_);
      fn_ = &fn;
      n_ = n;
      part_ = part;
      remaining_ = T_ - 1;
      ++gen_;
    }
    cv_work_.notify_all();
    fn(0, std::min(part, n));
    std::unique_lock<std::mutex> lk(mu_);
    cv_done_.wait(lk, [&] { return remaining_ == 0; });
    fn_ = nullptr;
  }

 private:
  explicit HostPool(int T) : T_(T), pid_(getpid()) {
    for (int t = 1; t < T_; ++t) std::thread([this, t] { loop(t); }).detach();
  }
  void loop(int t) {
    uint64_t seen = 0;
    for (;;) {
      const std::function<void(size_t, size_t)> *fn;
      size_t lo, hi;
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_work_.wait(lk, [&] { return gen_ != seen; });
        seen = gen_;
        fn = fn_;
        lo = std::min(n_, (size_t)t * part_);
        hi = std::min(n_, lo + part_);
      }
      if (lo < hi) (*fn)(lo, hi);
      std::lock_guard<std::mutex> lk(mu_);
      if (--remaining_ == 0) cv_done_.notify_one();
    }
  }
  const int T_;
  const pid_t pid_;
  std::mutex run_mu_, mu_;
  std::condition_variable cv_work_, cv_done_;
  const std::function<void(size_t, size_t)> *fn_ = nullptr;
  size_t n_ = 0, part_ = 0;
  uint64_t gen_ = 0;
  int remaining_ = 0;
};

template <typename Fn>
static void par_range(size_t n, Fn fn) {
  if (n < 32768) return fn(size_t(0), n);  // less work than waking the pool
  HostPool &pool = HostPool::get();
  const int T = pool.threads();
  const size_t part = ((n + T - 1) / T + 63) & ~size_t(63);
  const std::function<void(size_t, size_t)> f = fn;
  pool.run(n, part, f);
}
}  // extern "C++"
static void par_memcpy(void *dst, const void *src, size_t n) {
  par_range(n, [=](size_t lo, size_t hi) {
    std::memcpy((char *)dst + lo, (const char *)src + lo, hi - lo);
  });
}
// FP64 -> FP32 with round-to-nearest-even, the rounding of the device's
// conversion (cvt.rn.f32.f64), so both give the same bits.
static void par_convert(float *dst, const double *src, size_t n) {
  par_range(n, [=](size_t lo, size_t hi) {
    for (size_t i = lo; i < hi; ++i) dst[i] = (float)src[i];
  });
}
static int pin_ready(salvus_problem *p) {
  for (int b = 0; b < 2; ++b) {
    if (!p->h_pin[b]) SALVUS_CUDA(cudaMallocHost(&p->h_pin[b], kPinChunk));
    if (!p->pin_ev[b]) SALVUS_CUDA(cudaEventCreateWithFlags(&p->pin_ev[b], cudaEventDisableTiming));
  }
  return SALVUS_OK;
}
static int copy_h2d(salvus_problem *p, void *dst, const void *src, size_t bytes) {
  if (bytes < 2 * kPinChunk) {
    SALVUS_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, p->stream));
    return SALVUS_OK;
  }
  int rc = pin_ready(p);
  if (rc) return rc;
  size_t off = 0;
  for (int k = 0; off < bytes; ++k) {
    const int b = k & 1;
    const size_t n = std::min(kPinChunk, bytes - off);
    if (k >= 2) SALVUS_CUDA(cudaEventSynchronize(p->pin_ev[b]));  // chunk free again
    par_memcpy(p->h_pin[b], (const char *)src + off, n);
    SALVUS_CUDA(cudaMemcpyAsync((char *)dst + off, p->h_pin[b], n, cudaMemcpyHostToDevice, p->stream));
    SALVUS_CUDA(cudaEventRecord(p->pin_ev[b], p->stream));
    off += n;
  }
  return SALVUS_OK;
}
// FP64 host array -> FP32 device field: the host threads convert each chunk
// into a pinned buffer while the previous chunk's DMA runs (half the bytes
// of an FP64 transfer cross PCIe).  Smaller fields go through a plain buffer:
// page-locking the two chunks takes 30-60 ms (B200 host), the pageable copy
// of the most it replaces about 6.
static int copy_h2d_f32(salvus_problem *p, float *dst, const double *src, size_t n) {
  if (n * sizeof(float) < 2 * kPinChunk) {
    const std::unique_ptr<float[]> h(new (std::nothrow) float[n]);
    if (!h) return fail(SALVUS_E_OOM, "no host memory for a field of %zu values", n);
    par_convert(h.get(), src, n);
    SALVUS_CUDA(cudaMemcpyAsync(dst, h.get(), n * sizeof(float), cudaMemcpyHostToDevice, p->stream));
    SALVUS_CUDA(cudaStreamSynchronize(p->stream));  // the buffer ends here
    return SALVUS_OK;
  }
  int rc = pin_ready(p);
  if (rc) return rc;
  const size_t per = kPinChunk / sizeof(float);
  size_t off = 0;
  for (int k = 0; off < n; ++k) {
    const int b = k & 1;
    const size_t m = std::min(per, n - off);
    if (k >= 2) SALVUS_CUDA(cudaEventSynchronize(p->pin_ev[b]));  // chunk free again
    par_convert(static_cast<float *>(p->h_pin[b]), src + off, m);
    SALVUS_CUDA(cudaMemcpyAsync(dst + off, p->h_pin[b], m * sizeof(float), cudaMemcpyHostToDevice,
                                p->stream));
    SALVUS_CUDA(cudaEventRecord(p->pin_ev[b], p->stream));
    off += m;
  }
  return SALVUS_OK;
}
static int copy_d2h(salvus_problem *p, void *dst, const void *src, size_t bytes) {
  if (bytes < 2 * kPinChunk) {
    SALVUS_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, p->stream));
    return SALVUS_OK;
  }
  int rc = pin_ready(p);
  if (rc) return rc;
  const size_t nchunks = (bytes + kPinChunk - 1) / kPinChunk;
  auto issue = [&](size_t k) -> int {
    const size_t off = k * kPinChunk, n = std::min(kPinChunk, bytes - off);
    SALVUS_CUDA(cudaMemcpyAsync(p->h_pin[k & 1], (const char *)src + off, n, cudaMemcpyDeviceToHost,
                                p->stream));
    SALVUS_CUDA(cudaEventRecord(p->pin_ev[k & 1], p->stream));
    return SALVUS_OK;
  };
  if ((rc = issue(0))) return rc;
  for (size_t k = 0; k < nchunks; ++k) {
    // chunk (k + 1) & 1 was drained to the host in the previous iteration
    if (k + 1 < nchunks && (rc = issue(k + 1))) return rc;
    SALVUS_CUDA(cudaEventSynchronize(p->pin_ev[k & 1]));
    const size_t off = k * kPinChunk, n = std::min(kPinChunk, bytes - off);
    par_memcpy((char *)dst + off, p->h_pin[k & 1], n);
  }
  return SALVUS_OK;
}

static salvus::DeviceBuffer *field_buffer(salvus_problem *p, int32_t f) {
  switch (f) {
    case SALVUS_FIELD_U: return &p->d_u;
    case SALVUS_FIELD_V: return &p->d_v;
    case SALVUS_FIELD_A: return &p->d_a;
    case SALVUS_FIELD_A_PREV: return &p->d_ap;
  }
  return nullptr;
}

// One shot's column of a shot-batched field (u, or the half-step velocity w
// for SALVUS_FIELD_V; with a_ = 0 at the start, w = v there).
static int batched_field(salvus_problem *p, int32_t f, int32_t shot, double *vals, bool set) {
  if (f != SALVUS_FIELD_U && f != SALVUS_FIELD_V)
    return fail(SALVUS_E_UNSUPPORTED, "batched problems hold u and the half-step velocity only");
  if (shot < 0 || shot >= p->shots) return fail(SALVUS_E_INVALID, "shot %d out of range", shot);
  DeviceBuffer *b = f == SALVUS_FIELD_U ? &p->d_u : &p->d_v;
  const int64_t G = p->mesh->G;
  int rc;
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  if (p->d_stage.bytes < (size_t)(8 * G) && (rc = p->d_stage.alloc(8 * G))) return rc;
  if (set) {
    SALVUS_CUDA(cudaMemcpyAsync(p->d_stage.ptr, vals, 8 * G, cudaMemcpyHostToDevice, p->stream));
    shot_scatter_kernel<<<blocks_for(G, 256), 256, 0, p->stream>>>(G, p->shots_pad, shot,
                                                                   p->d_stage.as<double>(), b->as<float>());
  } else {
    shot_gather_kernel<<<blocks_for(G, 256), 256, 0, p->stream>>>(G, p->shots_pad, shot, b->as<float>(),
                                                                  p->d_stage.as<double>());
    SALVUS_CUDA(cudaMemcpyAsync(vals, p->d_stage.ptr, 8 * G, cudaMemcpyDeviceToHost, p->stream));
  }
  g_launches++;
  if ((rc = check_launch("shot field copy"))) return rc;
  SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  return SALVUS_OK;
}

int salvus_problem_set_field(salvus_problem *p, int32_t f, int32_t shot, const double *vals) {
  if (!p || !vals) return fail(SALVUS_E_INVALID, "null argument");
  if (p->shots > 1) return batched_field(p, f, shot, const_cast<double *>(vals), true);
  DeviceBuffer *b = field_buffer(p, f);
  if (!b || shot != 0) return fail(SALVUS_E_INVALID, "bad field %d / shot %d", f, shot);
  const size_t N = (size_t)p->mesh->G * p->c;
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  if (f == SALVUS_FIELD_A_PREV) {
    if (int rc = velocity_form(p, false)) return rc;  // v does not change with a_
  }
  if (p->prec == SALVUS_FP64) {
    int rc = copy_h2d(p, b->ptr, vals, 8 * N);
    if (rc) return rc;
  } else {
    // FP64 host array -> FP32 on the host threads -> FP32 field
    int rc = copy_h2d_f32(p, b->as<float>(), vals, N);
    if (rc) return rc;
  }
  if (f == SALVUS_FIELD_V) p->half_step = false;  // v as given; w is formed before the next step
  SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  return SALVUS_OK;
}

int salvus_problem_get_field(salvus_problem *p, int32_t f, int32_t shot, double *vals) {
  if (!p || !vals) return fail(SALVUS_E_INVALID, "null argument");
  if (p->shots > 1) return batched_field(p, f, shot, vals, false);
  DeviceBuffer *b = field_buffer(p, f);
  if (!b || shot != 0) return fail(SALVUS_E_INVALID, "bad field %d / shot %d", f, shot);
  const size_t N = (size_t)p->mesh->G * p->c;
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  const bool from_w = f == SALVUS_FIELD_V && p->half_step;
  if (p->prec == SALVUS_FP64 && !from_w) {
    int rc = copy_d2h(p, vals, b->ptr, 8 * N);
    if (rc) return rc;
  } else {
    int rc;
    // FP64 takes no memory to read v: the residual is scratch between calls and
    // as large as a field (every node is some element's point)
    const bool spare = p->prec == SALVUS_FP64 && p->d_r.bytes >= 8 * N;
    DeviceBuffer &stage = spare ? p->d_r : p->d_stage;
    if (stage.bytes < 8 * N && (rc = stage.alloc(8 * N))) return rc;
    const unsigned grid = blocks_for((int64_t)N, 256);
    if (!from_w)
      convert_kernel<float, double><<<grid, 256, 0, p->stream>>>((int64_t)N, b->as<float>(),
                                                                 stage.as<double>());
    else if (p->prec == SALVUS_FP32)
      velocity_kernel<float><<<grid, 256, 0, p->stream>>>((int64_t)N, b->as<float>(),
                                                          p->d_ap.as<float>(), (float)(0.5 * p->dt),
                                                          stage.as<double>());
    else
      velocity_kernel<double><<<grid, 256, 0, p->stream>>>((int64_t)N, b->as<double>(),
                                                           p->d_ap.as<double>(), 0.5 * p->dt,
                                                           stage.as<double>());
    g_launches++;
    if ((rc = check_launch("convert"))) return rc;
    if ((rc = copy_d2h(p, vals, stage.ptr, 8 * N))) return rc;
  }
  SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  return device_status(p);
}

static int single_shot_only(salvus_problem *p) {
  if (p && p->shots > 1)
    return fail(SALVUS_E_UNSUPPORTED,
                "the three-call form is single-shot; batched problems use salvus_step / salvus_run");
  return SALVUS_OK;
}

int salvus_assemble(salvus_problem *p) {
  int rc = single_shot_only(p);
  if (rc) return rc;
  rc = ready(p);
  if (rc) return rc;
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  if ((rc = sources_ready(p))) return rc;
  return by_components(p->c, [&](auto cc) {
    constexpr int C = decltype(cc)::value;
    return p->prec == SALVUS_FP32 ? assemble_t<float, C>(p) : assemble_t<double, C>(p);
  });
}

int salvus_apply_inverse_mass(salvus_problem *p) {
  int rc = single_shot_only(p);
  if (rc) return rc;
  rc = ready(p);
  if (rc) return rc;
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  return by_components(p->c, [&](auto cc) {
    constexpr int C = decltype(cc)::value;
    return p->prec == SALVUS_FP32 ? minv_t<float, C>(p) : minv_t<double, C>(p);
  });
}

int salvus_take_time_step(salvus_problem *p) {
  int rc = single_shot_only(p);
  if (rc) return rc;
  rc = ready(p);
  if (rc) return rc;
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  if ((rc = velocity_form(p, true))) return rc;
  rc = by_components(p->c, [&](auto cc) {
    constexpr int C = decltype(cc)::value;
    return p->prec == SALVUS_FP32 ? newmark_t<float, C>(p) : newmark_t<double, C>(p);
  });
  if (rc == SALVUS_OK) p->step++;
  if (rc == SALVUS_OK && p->step % kFiniteEvery == 0) rc = launch_finite_check(p);
  return rc;
}

int salvus_step(salvus_problem *p) {
  int rc = ready(p);
  if (rc) return rc;
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  if ((rc = velocity_form(p, true)) || (rc = sources_ready(p))) return rc;
  rc = step_fused(p, true);
  if (rc == SALVUS_OK) p->step++;
  if (rc == SALVUS_OK && p->step % kFiniteEvery == 0) rc = launch_finite_check(p);
  return rc;
}

int salvus_problem_set_wait_limit(salvus_problem *p, int64_t cycles) {
  if (!p) return fail(SALVUS_E_INVALID, "null problem");
  p->wait_limit = cycles > 0 ? (long long)cycles : salvus::kDefaultWaitLimit;
  drop_graph(p);  // captured launches hold the old bound
  return SALVUS_OK;
}

int salvus_problem_hold_device_waits(salvus_problem *p, int32_t enable) {
  if (!p) return fail(SALVUS_E_INVALID, "null problem");
  p->hold_waits = enable ? 1 : 0;
  drop_graph(p);  // captured launches hold the old setting
  return SALVUS_OK;
}

int salvus_problem_status(salvus_problem *p, int32_t clear) {
  if (!p) return fail(SALVUS_E_INVALID, "null problem");
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  const int rc = device_status(p);
  if (clear) {
    SALVUS_CUDA(cudaMemsetAsync(p->d_err.ptr, 0, sizeof(int), p->stream));
    SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  }
  return rc;
}

// Time loops replay CUDA graphs of captured fused steps: a run of n steps
// replays the 32-step graph n / 32 times and a graph of the remainder (the
// last remainder length is kept) when it is at least 8 steps, else launches
// those steps from the host.  Each graph ends with a finite check of u (the
// 32-step graph at every 32nd step, as host-launched runs do; a remainder
// graph at its end).
constexpr int kGraphChunk = 32, kGraphMin = 8;

static int capture_steps(salvus_problem *p, int steps, cudaGraphExec_t *exec, int64_t *launches) {
  const bool prof = p->profiling;
  p->profiling = false;
  // receivers forked onto the second stream in the captured steps only (in
  // host-launched steps the extra event calls would cost more host time
  // than the overlap saves on small meshes)
  p->rec_overlap = p->shots == 1 && p->rec_stream;
  cudaGraph_t graph;
  SALVUS_CUDA(cudaStreamBeginCapture(p->stream, cudaStreamCaptureModeThreadLocal));
  int crc = SALVUS_OK;
  const int64_t l0 = g_launches.load();
  for (int s = 0; s < steps && crc == SALVUS_OK; ++s) crc = step_fused(p, s == steps - 1);
  if (crc == SALVUS_OK) crc = launch_finite_check(p);
  // the captured sequence ends joined (a forked stream must rejoin the
  // capture), so every replay is self-contained
  const int jrc = join_receivers(p);
  if (crc == SALVUS_OK) crc = jrc;
  p->rec_overlap = false;
  cudaError_t ce = cudaStreamEndCapture(p->stream, &graph);
  // captured launches run only when the graph is replayed: count them there
  *launches = g_launches.load() - l0;
  g_launches -= *launches;
  p->profiling = prof;
  if (crc) {
    if (ce == cudaSuccess) cudaGraphDestroy(graph);
    return crc;
  }
  if (ce != cudaSuccess) return fail(SALVUS_E_CUDA, "graph capture failed: %s", cudaGetErrorString(ce));
  ce = cudaGraphInstantiate(exec, graph, 0);
  cudaGraphDestroy(graph);
  if (ce != cudaSuccess) return fail(SALVUS_E_CUDA, "graph instantiate failed: %s", cudaGetErrorString(ce));
  return SALVUS_OK;
}

// the graphs a graph run of n_steps replays, captured if missing
static int prepare_graphs(salvus_problem *p, int64_t n_steps) {
  int rc;
  if (n_steps >= kGraphChunk && !p->graph_exec) {
    if ((rc = capture_steps(p, kGraphChunk, &p->graph_exec, &p->graph_launches))) return rc;
    p->graph_steps = kGraphChunk;
  }
  const int rem = (int)(n_steps % kGraphChunk);
  if (rem >= kGraphMin && p->tail_steps != rem) {
    if (p->tail_exec) cudaGraphExecDestroy(p->tail_exec);
    p->tail_exec = nullptr;
    p->tail_steps = 0;
    if ((rc = capture_steps(p, rem, &p->tail_exec, &p->tail_launches))) return rc;
    p->tail_steps = rem;
  }
  return SALVUS_OK;
}

static int rec_stream_ready(salvus_problem *p) {
  if (p->shots == 1 && !p->rec_stream) {  // created outside any graph capture
    SALVUS_CUDA(cudaStreamCreateWithFlags(&p->rec_stream, cudaStreamNonBlocking));
    SALVUS_CUDA(cudaEventCreateWithFlags(&p->ev_updated, cudaEventDisableTiming));
    SALVUS_CUDA(cudaEventCreateWithFlags(&p->ev_recorded, cudaEventDisableTiming));
  }
  return SALVUS_OK;
}

static int run_steps(salvus_problem *p, int64_t n_steps, int32_t mode);
int salvus_run(salvus_problem *p, int64_t n_steps, int32_t mode) {
  int rc = ready(p);
  if (rc) return rc;
  if (n_steps < 0) return fail(SALVUS_E_INVALID, "negative step count");
  if (mode != SALVUS_RUN_PLAIN && mode != SALVUS_RUN_GRAPH)
    return fail(SALVUS_E_INVALID, "unknown run mode %d", mode);
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  if ((rc = rec_stream_ready(p))) return rc;
  if (n_steps > 0 && ((rc = velocity_form(p, true)) || (rc = sources_ready(p)))) return rc;
  return run_steps(p, n_steps, mode);
}

int salvus_problem_prepare_run(salvus_problem *p, int64_t n_steps) {
  int rc = ready(p);
  if (rc) return rc;
  if (n_steps < 0) return fail(SALVUS_E_INVALID, "negative step count");
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  if ((rc = rec_stream_ready(p))) return rc;
  return prepare_graphs(p, n_steps);
}

static int plain_steps(salvus_problem *p, int64_t n) {
  int rc;
  for (int64_t s = 0; s < n; ++s) {
    if ((rc = step_fused(p, s == n - 1))) return rc;
    p->step++;
    if (p->step % kFiniteEvery == 0 && (rc = launch_finite_check(p))) return rc;
  }
  return SALVUS_OK;
}

static int run_steps(salvus_problem *p, int64_t n_steps, int32_t mode) {
  if (mode == SALVUS_RUN_PLAIN || n_steps < kGraphMin) return plain_steps(p, n_steps);
  int rc = prepare_graphs(p, n_steps);
  if (rc) return rc;
  int64_t done = 0;
  while (n_steps - done >= p->graph_steps && p->graph_exec) {
    ProfScope ps(p, K_GRAPH);
    SALVUS_CUDA(cudaGraphLaunch(p->graph_exec, p->stream));
    g_launches += p->graph_launches;
    done += p->graph_steps;
    p->step += p->graph_steps;
  }
  if (p->tail_exec && n_steps - done == p->tail_steps) {
    ProfScope ps(p, K_GRAPH);
    SALVUS_CUDA(cudaGraphLaunch(p->tail_exec, p->stream));
    g_launches += p->tail_launches;
    done += p->tail_steps;
    p->step += p->tail_steps;
  }
  return plain_steps(p, n_steps - done);
}

// Energy of the current state: -K u into a scratch field (stiffness and
// Dirichlet zeroing, then the gather), then the compensated FP64 sums.
extern "C++" {
template <typename real, int C>
static int energy_t(salvus_problem *p, double *kinetic, double *strain) {
  const salvus_mesh *m = p->mesh;
  const size_t N = (size_t)m->G * C;
  int rc;
  if (p->d_escr.bytes < N * sizeof(real) && (rc = p->d_escr.alloc(N * sizeof(real)))) return rc;
  constexpr int kBlocks = 1024;
  if (p->d_epart.bytes < 2 * kBlocks * sizeof(double) &&
      (rc = p->d_epart.alloc(2 * kBlocks * sizeof(double))))
    return rc;
  if ((rc = launch_stiffness<real>(m, records<real>(p), F<real>(p->d_u), F<real>(p->d_r), p->stream,
                                   p->d_err.as<int>(), p->wait_limit, p->hold_waits)))
    return rc;
  if ((rc = launch_dirichlet<real, C>(p))) return rc;
  gather_kernel<real, C, 1><<<blocks_for(m->G, 256), 256, 0, p->stream>>>(
      m->G, m->d_inc_off.as<int32_t>(), m->d_inc_idx.as<int32_t>(), F<real>(p->d_r), nullptr,
      nullptr, nullptr, nullptr, p->d_escr.as<real>(), (real)0);
  g_launches++;
  if ((rc = check_launch("energy gather"))) return rc;
  energy_kernel<real, C><<<kBlocks, 256, 0, p->stream>>>(
      m->G, F<real>(p->d_u), F<real>(p->d_v), F<real>(p->d_ap),
      p->half_step ? (real)(0.5 * p->dt) : real(0), p->d_escr.as<real>(), m->d_mi64.as<double>(),
      p->d_epart.as<double>());
  g_launches++;
  if ((rc = check_launch("energy"))) return rc;
  std::vector<double> h(2 * kBlocks);
  SALVUS_CUDA(cudaMemcpyAsync(h.data(), p->d_epart.ptr, sizeof(double) * h.size(),
                              cudaMemcpyDeviceToHost, p->stream));
  SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  // Kahan over the block partials, in block order
  double sk = 0, ck = 0, ss = 0, cs = 0;
  for (int b = 0; b < kBlocks; ++b) {
    const double yk = h[2 * b] - ck, tk = sk + yk;
    ck = (tk - sk) - yk;
    sk = tk;
    const double ys = h[2 * b + 1] - cs, ts = ss + ys;
    cs = (ts - ss) - ys;
    ss = ts;
  }
  if (kinetic) *kinetic = sk;
  if (strain) *strain = ss;
  return device_status(p);
}
}  // extern "C++"

int salvus_problem_energy(salvus_problem *p, double *kinetic, double *strain) {
  if (!p) return fail(SALVUS_E_INVALID, "null problem");
  if (p->shots > 1)
    return fail(SALVUS_E_UNSUPPORTED, "energy is computed for single-shot problems");
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  return by_components(p->c, [&](auto cc) {
    constexpr int C = decltype(cc)::value;
    return p->prec == SALVUS_FP32 ? energy_t<float, C>(p, kinetic, strain)
                                  : energy_t<double, C>(p, kinetic, strain);
  });
}

int salvus_synchronize(salvus_problem *p) {
  if (!p) return fail(SALVUS_E_INVALID, "null problem");
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  return device_status(p);
}

int64_t salvus_problem_step_index(const salvus_problem *p) { return p ? p->step : -1; }

int salvus_problem_autotune(salvus_problem *p, int32_t *stiff_shot_lanes, int32_t *stiff_elements,
                            int32_t *gather_shot_lanes, int32_t *gather_nodes) {
  int rc = ready(p);
  if (rc) return rc;
  if (p->shots == 1) {
    if (stiff_shot_lanes) *stiff_shot_lanes = 1;
    if (stiff_elements) *stiff_elements = 0;
    if (gather_shot_lanes) *gather_shot_lanes = 1;
    if (gather_nodes) *gather_nodes = 256;
    return SALVUS_OK;
  }
  if (stiff_shot_lanes)
    *stiff_shot_lanes = kStiffCfg[p->tune_stiff].sc ? kStiffCfg[p->tune_stiff].sc
                                                    : pair_shots(p->shots_pad);
  if (stiff_elements) *stiff_elements = kStiffCfg[p->tune_stiff].epc;
  if (gather_shot_lanes) *gather_shot_lanes = kGatherCfg[p->tune_gather].sc;
  if (gather_nodes) *gather_nodes = kGatherCfg[p->tune_gather].epc * kGatherCfg[p->tune_gather].npt;
  return SALVUS_OK;
}

int salvus_problem_step_config(salvus_problem *p, int32_t *form, int32_t *elements_per_cta) {
  int rc = ready(p);
  if (rc) return rc;
  const salvus_mesh *m = p->mesh;
  int32_t f = SALVUS_STEP_PLAIN, epc = 0;
  if (p->shots > 1) {
    f = batch_fusion(p) && m->order >= 2 ? SALVUS_STEP_FUSED_INTERIOR : SALVUS_STEP_PLAIN;
    epc = kStiffCfg[p->tune_stiff].epc;
  } else if (m->shape == SALVUS_HEX && m->affine && p->prec == SALVUS_FP32 &&
             m->physics == SALVUS_ELASTIC3D) {
    f = hex_interior_fusion(p) ? SALVUS_STEP_FUSED_INTERIOR : SALVUS_STEP_PLAIN;
    const int n2 = (m->order + 1) * (m->order + 1), e1 = 128 / n2 > 0 ? 128 / n2 : 1;
    epc = e1 * (m->hex_wide ? 2 : 1);
  }
  if (form) *form = f;
  if (elements_per_cta) *elements_per_cta = epc;
  return SALVUS_OK;
}

int salvus_problem_stream(const salvus_problem *p, void **stream) {
  if (!p || !stream) return fail(SALVUS_E_INVALID, "null argument");
  *stream = (void *)p->stream;
  return SALVUS_OK;
}

int salvus_problem_info(const salvus_problem *p, int32_t *shots, int32_t *nrec, int32_t *c) {
  if (!p) return fail(SALVUS_E_INVALID, "null problem");
  if (shots) *shots = p->shots;
  if (nrec) *nrec = (int32_t)p->recs.size();
  if (c) *c = p->c;
  return SALVUS_OK;
}

int salvus_get_seismograms(salvus_problem *p, int64_t first, int64_t count, double *out) {
  if (!p || !out) return fail(SALVUS_E_INVALID, "null argument");
  if (count < 0 || first < 0 || first + count > p->step || first < p->step - p->seis_cap)
    return fail(SALVUS_E_INVALID, "steps [%lld, %lld) not held (step %lld, capacity %lld)",
                (long long)first, (long long)(first + count), (long long)p->step,
                (long long)p->seis_cap);
  if (p->recs.empty() || count == 0) return SALVUS_OK;
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  // The columns asked for (one piece, two where the window wraps), not the whole
  // ring: copying 4096 steps and picking from them took 0.1-1.5 ms for what is
  // 10-50 us (16 to 4096 rows of 16-100 steps, B200).  The caller's array is
  // written only if the status is good: windows of up to 128 KB come with the
  // status word, in one wait, by way of a local buffer; before larger ones the
  // status is read first (a wait more, 7 us on B200, about what the host takes to
  // copy 128 KB).
  constexpr size_t kLocal = 16384;
  const size_t rows = (size_t)p->shots * p->recs.size() * p->c;
  const int64_t c0 = first % p->seis_cap, n0 = std::min(count, p->seis_cap - c0);
  auto piece = [&](int64_t col, int64_t n, double *to) -> int {
    SALVUS_CUDA(cudaMemcpy2DAsync(to, sizeof(double) * count, p->d_seis.as<double>() + col,
                                  sizeof(double) * p->seis_cap, sizeof(double) * n, rows,
                                  cudaMemcpyDeviceToHost, p->stream));
    return SALVUS_OK;
  };
  auto window = [&](double *to) -> int {
    int rc = piece(c0, n0, to);
    if (rc == SALVUS_OK && n0 < count) rc = piece(0, count - n0, to + n0);
    return rc;
  };
  int rc;
  if (rows * (size_t)count <= kLocal) {
    double local[kLocal];
    rc = window(local);
    const int done = device_status(p);  // waits for the copies into local too
    if (rc == SALVUS_OK) rc = done;
    if (rc == SALVUS_OK) std::memcpy(out, local, sizeof(double) * rows * (size_t)count);
    return rc;
  }
  if ((rc = device_status(p)) || (rc = window(out))) return rc;
  SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  return SALVUS_OK;
}

int salvus_profile_enable(salvus_problem *p, int32_t enable) {
  if (!p) return fail(SALVUS_E_INVALID, "null problem");
  p->profiling = enable != 0;
  return SALVUS_OK;
}

int salvus_profile_read(salvus_problem *p, int32_t max_entries, const char **names, double *ms,
                        int64_t *launches, int32_t *n_entries) {
  if (!p) return fail(SALVUS_E_INVALID, "null problem");
  SALVUS_CUDA(cudaSetDevice(p->mesh->device));
  SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  for (auto &e : p->events) {
    float t = 0.f;
    cudaEventElapsedTime(&t, e.a, e.b);
    p->prof_ms[e.kind] += t;
    p->prof_n[e.kind] += 1;
    cudaEventDestroy(e.a);
    cudaEventDestroy(e.b);
  }
  p->events.clear();
  int k = 0;
  for (int i = 0; i < K_NKINDS && k < max_entries; ++i) {
    if (!p->prof_n[i]) continue;
    if (names) names[k] = kKindNames[i];
    if (ms) ms[k] = p->prof_ms[i];
    if (launches) launches[k] = p->prof_n[i];
    ++k;
  }
  if (n_entries) *n_entries = k;
  std::fill(p->prof_ms.begin(), p->prof_ms.end(), 0.0);
  std::fill(p->prof_n.begin(), p->prof_n.end(), 0);
  return SALVUS_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// problem groups
int salvus_group_create(salvus_problem *const *members, int32_t n, salvus_group **out) {
  if (!members || !out || n < 1) return fail(SALVUS_E_INVALID, "empty group");
  *out = nullptr;
  const salvus_mesh *m0 = members[0] ? members[0]->mesh : nullptr;
  if (!m0) return fail(SALVUS_E_INVALID, "null problem in group");
  const bool quad_ac = m0->shape == SALVUS_QUAD && m0->physics == SALVUS_ACOUSTIC;
  const bool hex_el = m0->shape == SALVUS_HEX && m0->physics == SALVUS_ELASTIC3D;
  if (!quad_ac && !hex_el)
    return fail(SALVUS_E_UNSUPPORTED, "groups are built for acoustic quads and elastic hexahedra");
  for (int32_t k = 0; k < n; ++k) {
    const salvus_problem *p = members[k];
    if (!p) return fail(SALVUS_E_INVALID, "null problem in group");
    const salvus_mesh *m = p->mesh;
    if (p->prec != SALVUS_FP32 || p->shots != 1)
      return fail(SALVUS_E_UNSUPPORTED, "group members must be FP32 single-shot problems");
    if (p->n_dir_pts > 0)
      return fail(SALVUS_E_UNSUPPORTED, "group members cannot carry Dirichlet boundaries");
    if (m->ti)
      return fail(SALVUS_E_UNSUPPORTED,
                  "group members must have isotropic material (transversely isotropic meshes "
                  "run as single problems)");
    if (m->shape != m0->shape || m->order != m0->order || m->physics != m0->physics ||
        m->device != m0->device)
      return fail(SALVUS_E_INVALID, "group members must share shape, order, physics and device");
    for (int32_t q = 0; q < k; ++q)
      if (members[q] == p) return fail(SALVUS_E_INVALID, "problem listed twice in a group");
  }
  std::unique_ptr<salvus_group> g(new salvus_group());
  g->members.assign(members, members + n);
  g->m0 = m0;
  g->device = m0->device;
  g->c = m0->physics == SALVUS_ELASTIC3D ? 3 : 1;
  {
    // measured: one launch per stage beats both single-launch forms (the
    // work-queue and the member-partitioned kernel, whose combined bodies
    // run the latency-bound gather at the occupancy of the heaviest body),
    // so it is the default
    const char *s = std::getenv("SALVUS_GROUP_STEP");
    g->partitioned = s && std::strcmp(s, "partitioned") == 0;
    g->stages = !(s && (std::strcmp(s, "persistent") == 0 || g->partitioned));
  }
  SALVUS_CUDA(cudaSetDevice(m0->device));
  SALVUS_CUDA(cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
  SALVUS_CUDA(cudaEventCreateWithFlags(&g->ev, cudaEventDisableTiming));
  g->member_ev.resize(n, nullptr);
  for (auto &e : g->member_ev) SALVUS_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  *out = g.release();
  return SALVUS_OK;
}

int salvus_group_run(salvus_group *g, int64_t n_steps) {
  if (!g) return fail(SALVUS_E_INVALID, "null group");
  if (n_steps < 0) return fail(SALVUS_E_INVALID, "negative step count");
  SALVUS_CUDA(cudaSetDevice(g->m0->device));
  for (auto *p : g->members) {
    int rc = ready(p);
    if (rc) return rc;
    if (n_steps == 0) continue;
    if ((rc = velocity_form(p, true)) || (rc = sources_ready(p))) return rc;
    if (!g->stages) p->stf_ready = false;  // these forms have no tail
  }
  // order the group after every member's pending work
  for (size_t k = 0; k < g->members.size(); ++k) {
    SALVUS_CUDA(cudaEventRecord(g->member_ev[k], g->members[k]->stream));
    SALVUS_CUDA(cudaStreamWaitEvent(g->stream, g->member_ev[k], 0));
  }
  int rc = group_fill(g);
  if (rc) return rc;
  const int chunk = 32;
  const int64_t sig[3] = {g->n_stiff, g->n_gather, g->n_rec};
  if (g->graph && (sig[0] != g->sig[0] || sig[1] != g->sig[1] || sig[2] != g->sig[2])) {
    cudaGraphExecDestroy(g->graph);
    g->graph = nullptr;
  }
  if (!g->graph && n_steps >= chunk) {
    cudaGraph_t graph;
    SALVUS_CUDA(cudaStreamBeginCapture(g->stream, cudaStreamCaptureModeThreadLocal));
    int crc = SALVUS_OK;
    for (int s = 0; s < chunk && crc == SALVUS_OK; ++s) crc = group_step(g, s == chunk - 1);
    cudaError_t ce = cudaStreamEndCapture(g->stream, &graph);
    if (crc) return crc;
    if (ce != cudaSuccess) return fail(SALVUS_E_CUDA, "graph capture failed: %s", cudaGetErrorString(ce));
    ce = cudaGraphInstantiate(&g->graph, graph, 0);
    cudaGraphDestroy(graph);
    if (ce != cudaSuccess) return fail(SALVUS_E_CUDA, "graph instantiate failed: %s", cudaGetErrorString(ce));
    g->graph_steps = chunk;
    for (int a = 0; a < 3; ++a) g->sig[a] = sig[a];
  }
  int64_t done = 0;
  while (g->graph && n_steps - done >= g->graph_steps) {
    SALVUS_CUDA(cudaGraphLaunch(g->graph, g->stream));
    g_launches += (int64_t)g->graph_steps * (g->stages ? (g->n_rec > 0 ? 3 : 2) : 1);
    done += g->graph_steps;
  }
  for (; done < n_steps; ++done)
    if ((rc = group_step(g, done == n_steps - 1))) return rc;
  for (auto *p : g->members) p->step += n_steps;
  // members' later work waits for the group; then each member's finite check
  // on its own stream
  SALVUS_CUDA(cudaEventRecord(g->ev, g->stream));
  for (auto *p : g->members) {
    SALVUS_CUDA(cudaStreamWaitEvent(p->stream, g->ev, 0));
    if (n_steps > 0 && (rc = launch_finite_check(p))) return rc;
  }
  return SALVUS_OK;
}

int salvus_group_set_wait_limit(salvus_group *g, int64_t cycles) {
  if (!g) return fail(SALVUS_E_INVALID, "null group");
  g->wait_limit = cycles > 0 ? (long long)cycles : salvus::kDefaultWaitLimit;
  if (g->graph) cudaGraphExecDestroy(g->graph);  // captured launches hold the old bound
  g->graph = nullptr;
  return SALVUS_OK;
}

int salvus_group_clear_status(salvus_group *g) {
  if (!g) return fail(SALVUS_E_INVALID, "null group");
  SALVUS_CUDA(cudaSetDevice(g->m0->device));
  SALVUS_CUDA(cudaStreamSynchronize(g->stream));
  if (g->d_sync.ptr) SALVUS_CUDA(cudaMemset(g->d_sync.ptr, 0, sizeof(GroupSync)));
  for (auto *p : g->members) {
    SALVUS_CUDA(cudaMemsetAsync(p->d_err.ptr, 0, sizeof(int), p->stream));
    SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  }
  return SALVUS_OK;
}

int salvus_group_synchronize(salvus_group *g) {
  if (!g) return fail(SALVUS_E_INVALID, "null group");
  SALVUS_CUDA(cudaSetDevice(g->m0->device));
  SALVUS_CUDA(cudaStreamSynchronize(g->stream));
  if (g->d_sync.ptr) {
    GroupSync s{};
    SALVUS_CUDA(cudaMemcpy(&s, g->d_sync.ptr, sizeof(s), cudaMemcpyDeviceToHost));
    if (s.err) return fail(SALVUS_E_TIMEOUT, "a bounded wait of the grouped step gave up; results invalid");
  }
  for (auto *p : g->members)
    if (int rc = device_status(p)) return rc;
  return SALVUS_OK;
}

cudaStream_t salvus_group_stream_internal(const salvus_group *g) { return g ? g->stream : nullptr; }

int salvus_group_destroy(salvus_group *g) {
  if (!g) return SALVUS_OK;
  // the group's own device: its members' meshes may already be gone
  cudaSetDevice(g->device);
  if (g->stream) cudaStreamSynchronize(g->stream);
  if (g->graph) cudaGraphExecDestroy(g->graph);
  for (auto e : g->member_ev)
    if (e) cudaEventDestroy(e);
  if (g->ev) cudaEventDestroy(g->ev);
  g->d_slots.release();
  g->d_counts.release();
  g->d_work.release();
  g->d_done.release();
  g->d_sync.release();
  if (g->stream) cudaStreamDestroy(g->stream);
  delete g;
  return SALVUS_OK;
}

// ---------------------------------------------------------------------------
// homogeneous Dirichlet boundaries
int salvus_mesh_boundary_nodes(const salvus_mesh *m, int64_t *count, int64_t *nodes) {
  if (!m || !count) return fail(SALVUS_E_INVALID, "null argument");
  std::vector<int64_t> b;
  int rc = boundary_nodes(m, b);
  if (rc) return rc;
  if (nodes) std::memcpy(nodes, b.data(), sizeof(int64_t) * b.size());
  *count = (int64_t)b.size();
  return SALVUS_OK;
}

int salvus_problem_set_dirichlet(salvus_problem *p, int64_t n, const int64_t *nodes) {
  if (!p || (n > 0 && !nodes) || n < 0) return fail(SALVUS_E_INVALID, "bad arguments");
  const salvus_mesh *m = p->mesh;
  if (p->shots > 1)
    return fail(SALVUS_E_UNSUPPORTED, "Dirichlet boundaries are not built for shot-batched problems");
  std::vector<char> flag((size_t)m->G, 0);
  for (int64_t k = 0; k < n; ++k) {
    if (nodes[k] < 0 || nodes[k] >= m->G) return fail(SALVUS_E_INVALID, "node %lld out of range",
                                                      (long long)nodes[k]);
    flag[(size_t)nodes[k]] = 1;
  }
  // every element point on a flagged node, ascending (element, point)
  std::vector<int32_t> pts;
  for (int64_t i = 0; i < m->E * m->P; ++i)
    if (flag[(size_t)m->conn[(size_t)i]]) pts.push_back((int32_t)i);
  SALVUS_CUDA(cudaSetDevice(m->device));
  if (!pts.empty()) {
    int rc = p->d_dir_pts.alloc(sizeof(int32_t) * pts.size());
    if (rc) return rc;
    SALVUS_CUDA(cudaMemcpyAsync(p->d_dir_pts.ptr, pts.data(), sizeof(int32_t) * pts.size(),
                                cudaMemcpyHostToDevice, p->stream));
    SALVUS_CUDA(cudaStreamSynchronize(p->stream));
  }
  p->n_dir_pts = (int64_t)pts.size();
  drop_graph(p);
  return SALVUS_OK;
}
