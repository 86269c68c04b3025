// kernels_step.cuh -- assembly by node gather, inverse mass, explicit
// Newmark update, Ricker source injection and receiver sampling.
//
// Reference arithmetic restated:
//   assembly        Problem::assembleIntoGlobalDof (Problem.cpp:143-214) with
//                   the scatter-add of addFieldOnElement (Problem.cpp:271-284),
//                   done here as a gather over each node's incident element
//                   points in ascending element order (deterministic);
//   inverse mass    Order2Newmark::applyInverseMassMatrix (Order2Newmark.cpp:68-83);
//   Newmark         Order2Newmark::takeTimeStep (Order2Newmark.cpp:85-114):
//                   v += dt/2 (a + a_), u += dt v + dt^2/2 a, a_ = a, kept in
//                   the half-step velocity w = v + dt/2 a_ (newmark_point);
//   source          Scalar::computeSourceTerm (Scalar.cpp:79-88),
//                   Elastic3D::computeSourceTerm (Elastic3D.cpp:126-133),
//                   Ricker::fire (Ricker.cpp:27-33), evaluated at t_n = n dt;
//   receivers       Lagrange interpolation (TensorQuad.cpp:145-174,
//                   Hexahedra.cpp:494-532) of u at the receiver point,
//                   accumulated in FP64 with Kahan compensation.
#pragma once

#include <cstdint>

namespace salvus {

// Explicitly rounded operations for the update, so that the fused
// gather/update kernel and the three-call path (gather, inverse mass,
// Newmark) produce bitwise identical wavefields whatever the compiler's
// contraction choices.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// One Newmark update on the half-step velocity w = v + dt/2 a_.  The
// reference's v += dt/2 (a + a_), u += dt v + dt^2/2 a, a_ = a
// (Order2Newmark.cpp:104-108) is, with w, the two operations below: v after
// the step is w - dt/2 a with the step's a, which is needed only when a
// caller asks for v (half_step_velocity).  A step therefore reads and writes
// u and w alone: 4 field streams instead of 6 (u, v and a_ both ways), which
// is what bounds the node gather (DRAM).  On 17 M nodes x 3 components that
// is 48 instead of 72 bytes per node: 32 steps of the 64^3 order-4 elastic
// mesh went from 26.7 to 23.9 ms by this alone (B200).
template <typename real>
__device__ __forceinline__ void newmark_point(real an, real &w, real &u, real dt) {
  w = fma_rn(dt, an, w);
  u = fma_rn(dt, w, u);
}

// The velocity at a whole step from the stored pair (hdt = dt/2), and back.
template <typename real>
__device__ __forceinline__ real half_step_velocity(real w, real ap, real hdt) {
  return fma_rn(-hdt, ap, w);
}
// x <- x + s y: v -> w (s = dt/2) and w -> v (s = -dt/2) in place.
template <typename real>
__global__ void axpy_kernel(int64_t N, real s, const real *__restrict__ y, real *__restrict__ x) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) x[i] = fma_rn(s, y[i], x[i]);
}
// out = w - dt/2 a_ in FP64, the velocity field a caller reads.
template <typename real>
__global__ void velocity_kernel(int64_t N, const real *__restrict__ w, const real *__restrict__ ap,
                                real hdt, double *__restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) out[i] = (double)half_step_velocity<real>(w[i], ap[i], hdt);
}

// Source terms of a single-shot problem: added by the node gather to a
// node's assembled residual (Problem.cpp:188-200: a = f - K u).  A kernel of
// its own between the stiffness and the gather is a few threads' work at the
// price of a launch and of its latency on the critical path: about 2 of the
// 7.5 us that a step of a 40 x 40 order-4 quadrilateral mesh took (B200).
// The gather finds the few nodes concerned through a table by tile of
// kSrcTile nodes: tile[b] is -1, or where the tile's kSrcTile entries begin
// in `node`: {x, y, z, w} = weights of source y at this node (index into
// wts / C), first source y, z sources (0: none; an element's sources are
// adjacent, in attach order, their weights P apart), w: the node's entry for
// another source element or -1.  Two loads lead to the weights, as two lead
// to the residual, and the sum needs no residual slot: adding the terms to
// the incident residual of their element instead kept all eight points'
// indices and residuals live (48 -> 72 registers for 3 components).
// stf holds the source-time functions of the coming step, which the receiver
// launch of the step before evaluates (step_tail_kernel).
constexpr int kSrcTile = 128;
struct SourceTerms {
  const int32_t *tile = nullptr;  // null: no sources
  const int4 *node;
  const double *wts;  // [source][P][C]
  const double *stf;  // [source]
  int P;
};

// kInKernel: stf was written earlier in the same launch (coherent loads).
template <typename real, int C, bool kInKernel>
__device__ __forceinline__ void add_sources(int4 at, const SourceTerms &src, real (&acc)[C]) {
  for (;;) {
    for (int32_t s = 0; s < at.z; ++s) {
      const double *sp = src.stf + at.y + s;
      const double stf = kInKernel ? __ldca(sp) : *sp;
#pragma unroll
      for (int c = 0; c < C; ++c)
        acc[c] = add_rn(acc[c], (real)__dmul_rn(src.wts[(at.x + (int64_t)s * src.P) * C + c], stf));
    }
    if (at.w < 0) return;
    at = src.node[at.w];
  }
}

// mode 0: fused  a = mi * sum(r); Newmark update of (u, w); a_ = a is stored
//         when ap is not null (the last step of a run: later steps never read
//         it, only callers do)
// mode 1: gather a = sum(r)
// kInKernelR: r was written earlier in the same launch (fused group steps)
// and is read with coherent loads (ld.global.ca), not ld.global.nc.
template <typename real, int C, int MODE, bool kInKernelR = false>
__device__ __forceinline__ void gather_body(int64_t g, int64_t G, const int32_t *__restrict__ off,
                                            const int32_t *__restrict__ idx,
                                            const real *__restrict__ r,
                                            const real *__restrict__ mi, real *__restrict__ u,
                                            real *__restrict__ w, real *__restrict__ ap,
                                            real *__restrict__ a, real dt,
                                            const SourceTerms &src = SourceTerms()) {
  if (g >= G) return;
  // Newmark operands first: they do not depend on the gather, so their loads
  // overlap the dependent index -> residual chain below.
  real m = 0, uo[C], wo[C];
  if (MODE == 0) {
    m = mi[g];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      uo[c] = u[g * C + c];
      wo[c] = w[g * C + c];
    }
  }
  real acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c) acc[c] = 0;
  const int32_t q0 = off[g], q1 = off[g + 1];
  const int32_t src_at = src.tile ? src.tile[g / kSrcTile] : -1;
  const int cnt = q1 - q0;
  constexpr int kFast = 8;  // hexahedral / quadrilateral valence bound
  if (cnt <= kFast) {
    int32_t ep[kFast];
#pragma unroll
    for (int q = 0; q < kFast; ++q) ep[q] = q < cnt ? idx[q0 + q] : 0;
    real rv[kFast][C];
#pragma unroll
    for (int q = 0; q < kFast; ++q)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const real *rp = r + (int64_t)ep[q] * C + c;
        rv[q][c] = q < cnt ? (kInKernelR ? __ldca(rp) : *rp) : real(0);
      }
    // ascending element order, as in the general loop
#pragma unroll
    for (int q = 0; q < kFast; ++q)
      if (q < cnt) {
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c] += rv[q][c];
      }
  } else {
    // high-valence nodes (tetrahedron vertices: about two dozen incident
    // points): batches of kBatch independent loads, summed in the same
    // ascending order as one at a time
    constexpr int kBatch = 4;
    for (int32_t qb = q0; qb < q1; qb += kBatch) {
      const int nq = q1 - qb < kBatch ? q1 - qb : kBatch;
      int32_t ep[kBatch];
#pragma unroll
      for (int q = 0; q < kBatch; ++q) ep[q] = q < nq ? idx[qb + q] : 0;
      real rv[kBatch][C];
#pragma unroll
      for (int q = 0; q < kBatch; ++q)
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const real *rp = r + (int64_t)ep[q] * C + c;
          rv[q][c] = q < nq ? (kInKernelR ? __ldca(rp) : *rp) : real(0);
        }
#pragma unroll
      for (int q = 0; q < kBatch; ++q)
        if (q < nq) {
#pragma unroll
          for (int c = 0; c < C; ++c) acc[c] += rv[q][c];
        }
    }
  }
  if (src_at >= 0)
    add_sources<real, C, kInKernelR>(src.node[src_at + g % kSrcTile], src, acc);
  if constexpr (MODE == 1) {
#pragma unroll
    for (int c = 0; c < C; ++c) a[g * C + c] = acc[c];
  } else {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int64_t i = g * C + c;
      const real an = mul_rn(acc[c], m);
      newmark_point<real>(an, wo[c], uo[c], dt);
      u[i] = uo[c];
      w[i] = wo[c];
      if (ap) ap[i] = an;
    }
  }
}

template <typename real, int C, int MODE>
__global__ void gather_kernel(int64_t G, const int32_t *__restrict__ off,
                              const int32_t *__restrict__ idx, const real *__restrict__ r,
                              const real *__restrict__ mi, real *__restrict__ u,
                              real *__restrict__ w, real *__restrict__ ap, real *__restrict__ a,
                              real dt, SourceTerms src = SourceTerms(),
                              int64_t *__restrict__ step = nullptr) {
  // step counter (steps completed): nothing else of the launch reads it
  if (step && blockIdx.x == 0 && threadIdx.x == 0) *step += 1;
  gather_body<real, C, MODE>((int64_t)blockIdx.x * blockDim.x + threadIdx.x, G, off, idx, r, mi, u,
                             w, ap, a, dt, src);
}

// Incidence of quadrilateral meshes, as the kernels below and the batched
// gather read it: one pair per node holds the whole list of element points
// e*P + p where it has one entry (x, -1) or two (x, y) -- 94 % of the nodes of
// an order-4 mesh -- so that the residual loads depend on one load, not on an
// offset and then an index; longer lists (vertices) are rest[x, x - y) with
// y = -length.  rest holds those lists alone, in node order: read from the mesh's
// incidence index, where 25 other entries lie between two of them, the 400^2 step
// took 34.9 instead of 32.2 us (B200).
struct Incidence {
  const int2 *head;
  const int32_t *rest;
};
// base: where the lists of each CTA's kHeadTile nodes begin in rest
constexpr int kHeadTile = 256;
__global__ void __launch_bounds__(kHeadTile)
incidence_pairs_kernel(int64_t G, const int32_t *__restrict__ off, const int32_t *__restrict__ idx,
                       const int32_t *base, int2 *__restrict__ head, int32_t *rest) {
  __shared__ int32_t sum[kHeadTile];
  const int t = threadIdx.x;
  const int64_t g = (int64_t)blockIdx.x * kHeadTile + t;
  const int32_t q0 = g < G ? off[g] : 0, n = g < G ? off[g + 1] - q0 : 0;
  sum[t] = n > 2 ? n : 0;
  __syncthreads();
  for (int o = 1; o < kHeadTile; o *= 2) {  // running sums
    const int32_t before = t >= o ? sum[t - o] : 0;
    __syncthreads();
    sum[t] += before;
    __syncthreads();
  }
  if (g >= G) return;
  if (n > 2) {
    const int32_t at = base[blockIdx.x] + sum[t] - n;
    for (int32_t q = 0; q < n; ++q) rest[at + q] = idx[q0 + q];
    head[g] = int2{at, -n};
  } else {
    head[g] = int2{idx[q0], n == 2 ? idx[q0 + 1] : -1};
  }
}

// Gather and update (mode 0 of gather_body, the same arithmetic) of two
// adjacent nodes of a 1-component quadrilateral mesh, g even: every stream is
// one 64- or 128-bit access for both nodes.  Half the threads and two thirds
// of the instructions of one node per thread; what remains is DRAM traffic
// and the chain head -> residual.  Per step, order 4: 400^2 41.2 -> 37.4 us,
// 700^2 121 -> 112, 16 grouped meshes of 10^2-90^2 22.2 -> 18.3; FP64 150^2
// order 7 29.6 -> 25.1 (B200).  Other element classes keep one node per
// thread: on triangles (six-element vertices) 19.5 us became 21.1, and on
// 3-component fields pairs or heads changed a step by -1 to +8 %.
template <typename real, bool kInKernelR = false>
__device__ __forceinline__ void gather_pair_body(int64_t g, int64_t G, const Incidence &inc,
                                                 const real *__restrict__ r,
                                                 const real *__restrict__ mi, real *__restrict__ u,
                                                 real *__restrict__ w, real *__restrict__ ap,
                                                 real dt, const SourceTerms &src) {
  if (g >= G) return;
  struct alignas(2 * sizeof(real)) Pair {
    real v[2];
  };
  const bool two = g + 1 < G;
  int2 h[2];
  Pair m, uo, wo;
  if (two) {
    const int4 hh = *reinterpret_cast<const int4 *>(inc.head + g);
    h[0] = {hh.x, hh.y};
    h[1] = {hh.z, hh.w};
    m = *reinterpret_cast<const Pair *>(mi + g);
    uo = *reinterpret_cast<const Pair *>(u + g);
    wo = *reinterpret_cast<const Pair *>(w + g);
  } else {
    h[0] = inc.head[g];
    h[1] = {h[0].x, -1};
    m.v[0] = m.v[1] = mi[g];
    uo.v[0] = uo.v[1] = u[g];
    wo.v[0] = wo.v[1] = w[g];
  }
  const int32_t src_at = src.tile ? src.tile[g / kSrcTile] : -1;
  auto load = [&](int32_t ep) -> real { return kInKernelR ? __ldca(r + ep) : r[ep]; };
  real acc[2], second[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    acc[q] = h[q].y >= -1 ? load(h[q].x) : real(0);
    second[q] = h[q].y >= 0 ? load(h[q].y) : real(0);
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    acc[q] = add_rn(real(0), acc[q]);  // the general gather's first addition
    if (h[q].y >= 0) {
      acc[q] += second[q];
    } else if (h[q].y < -1) {
      constexpr int kBatch = 4;  // the usual valence of a quadrilateral vertex
      const int32_t q1 = h[q].x - h[q].y;
      for (int32_t qb = h[q].x; qb < q1; qb += kBatch) {
        int32_t ep[kBatch];
        real rv[kBatch];
#pragma unroll
        for (int z = 0; z < kBatch; ++z) ep[z] = qb + z < q1 ? inc.rest[qb + z] : 0;
#pragma unroll
        for (int z = 0; z < kBatch; ++z) rv[z] = qb + z < q1 ? load(ep[z]) : real(0);
#pragma unroll
        for (int z = 0; z < kBatch; ++z)
          if (qb + z < q1) acc[q] += rv[z];
      }
    }
  }
  if (src_at >= 0) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      real aq[1] = {acc[q]};
      if (q == 0 || two)
        add_sources<real, 1, kInKernelR>(src.node[src_at + (g + q) % kSrcTile], src, aq);
      acc[q] = aq[0];
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    acc[q] = mul_rn(acc[q], m.v[q]);
    newmark_point<real>(acc[q], wo.v[q], uo.v[q], dt);
  }
  if (two) {
    *reinterpret_cast<Pair *>(u + g) = uo;
    *reinterpret_cast<Pair *>(w + g) = wo;
    if (ap) *reinterpret_cast<Pair *>(ap + g) = Pair{acc[0], acc[1]};
  } else {
    u[g] = uo.v[0];
    w[g] = wo.v[0];
    if (ap) ap[g] = acc[0];
  }
}

// 128-thread CTAs of the step's node gathers: measured against 64 / 256 / 512
// on the benchmark meshes, 1 % (hexahedra) to 5 % (tetrahedra) faster than 256
constexpr int kGatherThreads = 128;
constexpr int kPairTile = 2 * kGatherThreads;  // nodes per CTA

// CTAs per SM asked of the compiler: FP32 12 (10: 38.7 us on 400^2, 118 on
// 700^2), FP64 10 (12: 28.8 on 150^2 order 7).
template <typename real>
__global__ void __launch_bounds__(kGatherThreads, sizeof(real) == 4 ? 12 : 10)
gather_pair_kernel(int64_t G, Incidence inc, const real *__restrict__ r,
                   const real *__restrict__ mi, real *__restrict__ u, real *__restrict__ w,
                   real *__restrict__ ap, real dt, SourceTerms src, int64_t *__restrict__ step) {
  const int64_t t = (int64_t)blockIdx.x * kGatherThreads + threadIdx.x;
  if (t == 0) *step += 1;  // nothing else of the launch reads it
  gather_pair_body<real>(2 * t, G, inc, r, mi, u, w, ap, dt, src);
}

// The gather / update over a list of nodes (the shared nodes of a fused
// hexahedron step, whose interior nodes the stiffness kernel advanced).
template <typename real, int C, int MODE>
__global__ void gather_list_kernel(int64_t n, const int32_t *__restrict__ nodes,
                                   const int32_t *__restrict__ off,
                                   const int32_t *__restrict__ idx, const real *__restrict__ r,
                                   const real *__restrict__ mi, real *__restrict__ u,
                                   real *__restrict__ w, real *__restrict__ ap,
                                   real *__restrict__ a, real dt,
                                   SourceTerms src = SourceTerms(),
                                   int64_t *__restrict__ step = nullptr) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (step && t == 0) *step += 1;
  if (t >= n) return;
  gather_body<real, C, MODE>(nodes[t], INT64_MAX, off, idx, r, mi, u, w, ap, a, dt, src);
}

// Blow-up detection: any NaN / Inf among n values sets the problem's device
// status word to kNonFiniteCode (unless a wait timeout code is already
// there).  Launched after every 32 steps on the displacement field: an
// unstable explicit step grows without bound and reaches Inf / NaN in u.
constexpr int kNonFiniteCode = 0x4e614e;  // distinct from the wait codes (1000-1099)
template <typename real>
__global__ void finite_check_kernel(int64_t n, const real *__restrict__ x, int *__restrict__ err) {
  bool bad = false;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    bad |= !isfinite(x[i]);
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicCAS(err, 0, kNonFiniteCode);
}

// Homogeneous Dirichlet (HomogeneousDirichlet.cpp:65-73): zero the stiffness
// rows of the listed element-local points (before sources are added).
template <typename real, int C>
__global__ void dirichlet_zero_kernel(int64_t n, const int32_t *__restrict__ pts,
                                      real *__restrict__ r) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t ep = pts[i];
#pragma unroll
  for (int c = 0; c < C; ++c) r[ep * C + c] = real(0);
}

// Fluid-solid coupling surface integrals on meshes of fluid and solid quads
// (ElasticToAcoustic.cpp:26-41, AcousticToElastic2D.cpp:48-60), fields
// [u, ux, uy]: one thread per coupled element point with its coefficients
// summed over the element's coupled edges; the first n_fluid points belong to
// fluid elements (u += cx vx + cy vy), the rest to solid elements
// (ux += cx v, uy += cy v).  Runs after the stiffness (and Dirichlet zeroing)
// and before the sources, on the velocity field v = w - dt/2 a_ (these meshes
// store a_ at every step for it); hdt = 0: w holds v itself.
template <typename real>
__global__ void coupling_kernel(int64_t n_fluid, int64_t n, const int32_t *__restrict__ pts,
                                const real *__restrict__ coef, const real *__restrict__ w,
                                const real *__restrict__ ap, real hdt, real *__restrict__ r) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t ep = pts[2 * i], g = pts[2 * i + 1];
  const real cx = coef[2 * i], cy = coef[2 * i + 1];
  auto v = [&](int64_t x) { return hdt != 0 ? half_step_velocity<real>(w[x], ap[x], hdt) : w[x]; };
  if (i < n_fluid) {
    r[ep * 3] += cx * v(g * 3 + 1) + cy * v(g * 3 + 2);
  } else {
    const real vf = v(g * 3);
    r[ep * 3 + 1] += cx * vf;
    r[ep * 3 + 2] += cy * vf;
  }
}

template <typename real, int C>
__global__ void inverse_mass_kernel(int64_t G, const real *__restrict__ mi, real *__restrict__ a) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= G * C) return;
  a[i] = mul_rn(a[i], mi[i / C]);
}

template <typename real>
__global__ void newmark_kernel(int64_t N, const real *__restrict__ a, real *__restrict__ u,
                               real *__restrict__ w, real *__restrict__ ap, real dt,
                               int64_t *__restrict__ step) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *step += 1;
  if (i >= N) return;
  const real an = a[i];
  real wv = w[i], uv = u[i];
  newmark_point<real>(an, wv, uv, dt);
  u[i] = uv;
  w[i] = wv;
  ap[i] = an;
}

__device__ __forceinline__ double ricker_dev(double t, double f0, double t0, double amp) {
  const double pi = 3.14159265358979323846;
  const double factor = pi * pi * f0 * f0 * (t - t0) * (t - t0);
  return amp * ((1 - 2 * factor) * exp(-1 * factor));
}

// Source-time functions of step n into stf, by the threads of one CTA.
// par = [f0, t0, amplitude] of each source.
__device__ __forceinline__ void source_times(int nsrc, const double *__restrict__ par, int64_t n,
                                             double dt, double *__restrict__ stf) {
  for (int s = threadIdx.x; s < nsrc; s += blockDim.x)
    stf[s] = ricker_dev((double)n * dt, par[3 * s], par[3 * s + 1], par[3 * s + 2]);
}

// Receivers: one CTA per receiver, one thread per element point (strided);
// each thread keeps a Kahan-compensated FP64 partial per component, then a
// fixed-order tree combines the partials (deterministic): across each warp
// by shuffles, then the warps' sums in order.
// seis[(rec*C + c)*cap + n % cap] = sum_p l_p u_p after step n.
// kInKernelU: u was written earlier in the same launch (fused group steps),
// so it is read with a coherent load (ld.global.ca, ordered by the waits'
// fences), never through the non-coherent read-only path (ld.global.nc),
// which is only defined for data that no thread writes during the launch.
constexpr int kRecThreads = 128;
template <typename real, int C, bool kInKernelU = false>
__device__ __forceinline__ void receiver_body(int rc, int P, const int64_t *__restrict__ elem,
                                              const double *__restrict__ lw,
                                              const int32_t *__restrict__ conn,
                                              const real *__restrict__ u,
                                              double *__restrict__ seis, int64_t cap, int64_t n) {
  constexpr int kWarps = kRecThreads / 32;
  __shared__ double part[C][kWarps];
  const int t = threadIdx.x;
  const int64_t e = elem[rc], col = t < C ? n % cap : 0;
  double s[C], comp[C];
#pragma unroll
  for (int c = 0; c < C; ++c) s[c] = comp[c] = 0.0;
  for (int p = t; p < P; p += kRecThreads) {
    const double l = lw[(int64_t)rc * P + p];
    const int64_t node = conn[e * P + p];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const real uc = kInKernelU ? __ldca(u + node * C + c) : u[node * C + c];
      const double y = l * (double)uc - comp[c];
      const double tt = s[c] + y;
      comp[c] = (tt - s[c]) - y;
      s[c] = tt;
    }
  }
#pragma unroll
  for (int c = 0; c < C; ++c)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[c] += __shfl_down_sync(0xffffffffu, s[c], o);
  __syncthreads();  // part may still be read by an earlier call's threads
  if ((t & 31) == 0)
#pragma unroll
    for (int c = 0; c < C; ++c) part[c][t >> 5] = s[c];
  __syncthreads();
  if (t < C) {
    double sum = part[t][0];
#pragma unroll
    for (int k = 1; k < kWarps; ++k) sum += part[t][k];
    seis[((int64_t)rc * C + t) * cap + col] = sum;
  }
}

// What follows a step's update, in one launch: CTA b < nrec samples receiver
// b after the step just completed (number *step - 1); the last CTA evaluates
// the source-time functions of the step to come (SourceTerms::stf).  With
// nrec = 0 it is the evaluation alone, before a first step.
template <typename real, int C>
__global__ void __launch_bounds__(kRecThreads)
step_tail_kernel(int nrec, int P, const int64_t *__restrict__ elem, const double *__restrict__ lw,
                 const int32_t *__restrict__ conn, const real *__restrict__ u,
                 double *__restrict__ seis, int64_t cap, const int64_t *__restrict__ step, int nsrc,
                 const double *__restrict__ par, double dt, double *__restrict__ stf) {
  const int64_t n = *step;
  if ((int)blockIdx.x < nrec) {
    receiver_body<real, C>(blockIdx.x, P, elem, lw, conn, u, seis, cap, n - 1);
    return;
  }
  source_times(nsrc, par, n, dt, stf);
}

// One power iteration's vector work (salvus_mesh_max_eigenvalue).  y holds the
// gathered -K x; it becomes M^-1 K x, and each CTA writes its partial sums of
// x.y, x.x and y.y in the mass product (M = 1 / mi), summed in a fixed order.
// One pass over x and y: the inverse mass, the sign and three dot products
// were six launches with three copies to the host and three waits; an
// iteration on 22^3 order-4 hexahedra took 189 us and takes 77 (B200; 6^3: 80 and
// 18).
constexpr int kEigBlocks = 512, kEigThreads = 256;
template <int K>
__device__ __forceinline__ void block_sums(double (&s)[K], double *sh /* [K][kEigThreads] */) {
  const int t = threadIdx.x;
#pragma unroll
  for (int k = 0; k < K; ++k) sh[k * kEigThreads + t] = s[k];
  __syncthreads();
  for (int o = kEigThreads / 2; o > 0; o >>= 1) {
    if (t < o)
#pragma unroll
      for (int k = 0; k < K; ++k) sh[k * kEigThreads + t] += sh[k * kEigThreads + t + o];
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < K; ++k) s[k] = sh[k * kEigThreads];
}
template <int C>
__global__ void __launch_bounds__(kEigThreads)
eig_dots_kernel(int64_t N, const double *__restrict__ mi, const double *__restrict__ x,
                double *__restrict__ y, double *__restrict__ partial) {
  __shared__ double sh[3 * kEigThreads];
  double s[3] = {0.0, 0.0, 0.0};
  for (int64_t i = (int64_t)blockIdx.x * kEigThreads + threadIdx.x; i < N;
       i += (int64_t)kEigBlocks * kEigThreads) {
    const double m = mi[i / C], w = 1.0 / m, xv = x[i], yv = -mul_rn(y[i], m);
    y[i] = yv;
    s[0] += xv * yv * w;
    s[1] += xv * xv * w;
    s[2] += yv * yv * w;
  }
  block_sums<3>(s, sh);
  if (threadIdx.x < 3) partial[threadIdx.x * kEigBlocks + blockIdx.x] = sh[threadIdx.x * kEigThreads];
}
// y /= sqrt(y.y); *lam = x.y / x.x.  Every CTA adds up the partials itself.
__global__ void __launch_bounds__(kEigThreads)
eig_scale_kernel(int64_t N, const double *__restrict__ partial, double *__restrict__ y,
                 double *__restrict__ lam) {
  __shared__ double sh[3 * kEigThreads];
  double s[3] = {0.0, 0.0, 0.0};
  for (int b = threadIdx.x; b < kEigBlocks; b += kEigThreads)
#pragma unroll
    for (int k = 0; k < 3; ++k) s[k] += partial[k * kEigBlocks + b];
  block_sums<3>(s, sh);
  if (blockIdx.x == 0 && threadIdx.x == 0) *lam = s[0] / s[1];
  const double f = 1.0 / sqrt(s[2]);
  for (int64_t i = (int64_t)blockIdx.x * kEigThreads + threadIdx.x; i < N;
       i += (int64_t)kEigBlocks * kEigThreads)
    y[i] *= f;
}

// Energy 1/2 v^T M v and 1/2 u^T K u with FP64 compensated (Kahan) sums:
// each thread accumulates its grid-stride share of the nodes with a running
// compensation, the CTA adds the threads' sums in a fixed tree order, and
// partial[2 * block] / [2 * block + 1] (kinetic, strain) are summed on the
// host in block order -- the same bits on every run for a given grid.
// ku = -K u (the gathered stiffness action); v = w - dt/2 a_; M = 1 / mi per
// node, nodes without mass (mi = 0) carry none; hdt = 0: w holds v itself.
template <typename real, int C>
__global__ void __launch_bounds__(256)
energy_kernel(int64_t G, const real *__restrict__ u, const real *__restrict__ w,
              const real *__restrict__ ap, real hdt, const real *__restrict__ ku,
              const double *__restrict__ mi, double *__restrict__ partial) {
  __shared__ double sk[256], ss[256];
  double ek = 0.0, ck = 0.0, es = 0.0, cs = 0.0;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < G;
       g += (int64_t)gridDim.x * blockDim.x) {
    const double m = mi[g] != 0.0 ? 1.0 / mi[g] : 0.0;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const real wv = w[g * C + c];
      const double vv = hdt != 0 ? (double)half_step_velocity<real>(wv, ap[g * C + c], hdt) : (double)wv;
      const double uu = (double)u[g * C + c];
      const double yk = 0.5 * m * vv * vv - ck;
      const double tk = ek + yk;
      ck = (tk - ek) - yk;
      ek = tk;
      const double ys = -0.5 * uu * (double)ku[g * C + c] - cs;
      const double ts = es + ys;
      cs = (ts - es) - ys;
      es = ts;
    }
  }
  sk[threadIdx.x] = ek;
  ss[threadIdx.x] = es;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      sk[threadIdx.x] += sk[threadIdx.x + o];
      ss[threadIdx.x] += ss[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = sk[0];
    partial[2 * blockIdx.x + 1] = ss[0];
  }
}

template <typename A, typename B>
__global__ void convert_kernel(int64_t N, const A *__restrict__ a, B *__restrict__ b) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) b[i] = (B)a[i];
}

}  // namespace salvus
