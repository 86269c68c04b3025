// kernels_hex_affine.cuh -- FP32 elastic hexahedra whose elements are all
// parallelepipeds (affine maps): the inverse Jacobian is one 3x3 matrix per
// element, so the per-point record shrinks to the folded material constants
// (plus the connectivity, read from the [E][P] map).
//
// Orders 4 and up run the line-exchange body of kernels_hex_col.cuh on these
// records.  Same arithmetic as the column-threaded kernel of kernels_hex_v2.cuh
// (Elastic3D.cpp:70-118 via Hexahedra.cpp:580-632 / 689-754) with J taken
// from the element instead of the point.  Global arrays:
//   jac  [E][9]    invJ (row-major [x_a][xi_b]) of each element
//   mat  [NM][E*P] material planes: lambda', mu' (isotropic) or A', C', F',
//                  L', N' (transversely isotropic), w detJ folded in
//   conn [E][P]    element point -> global node
//
// Fused step form (kFuse): the interior GLL points of an element (all three
// local indices in 1..N-1) are nodes that no other element touches, so the
// kernel finishes them itself -- the one-term assembly 0 + r (the node
// gather's first addition), the inverse mass and the Newmark update
// (newmark_point) -- and writes element-local residuals only for the points
// on the element's faces, which the node gather then assembles over the
// shared nodes alone.  In the few elements that hold a source the interior
// residuals are written too; the source kernel adds the source terms and
// finishes those nodes (source_fused_hex_kernel).  Every operation and its order is the one of the
// unfused sequence (stiffness, sources, gather, update), so the two forms
// give bitwise the same wavefield.  In the fused form u is written for
// interior nodes during the launch, so u is read with coherent loads (the
// read-only path is for data no thread writes during the launch); each
// interior node is read and then written by the one thread that owns it.
#pragma once

#include <cstdint>

#include "kernels_hex_v2.cuh"
#include "kernels_material.cuh"
#include "kernels_step.cuh"

namespace salvus {

template <int N, int EPB_, bool TI>
struct HexAffineShape {
  using V2 = ElasticV2Shape<N, EPB_, TI>;
  static constexpr int n = V2::n, n2 = V2::n2, P = V2::P, EPB = V2::EPB;
  static constexpr int THREADS = V2::THREADS;
  static constexpr int NM = ElasticMat<TI>::kWords;
  static constexpr int US = V2::US, FS = V2::FS;
  static constexpr bool LINES = V2::LINES;
  static constexpr size_t SMEM = V2::SMEM;
};

// One group of EPB elements (bid), all threads of the CTA (contains
// __syncthreads); also the body of the grouped hexahedron steps.
template <int N, int EPB_, bool TI, bool kFuse>
__device__ __forceinline__ void elastic_hex_affine_body(
    int64_t bid, int64_t E, const float *__restrict__ jac, const float *__restrict__ mat,
    const int32_t *__restrict__ conn, float *__restrict__ u, float *__restrict__ r,
    const DMatrix<float> &Dm, const HexInteriorUpdate &iu) {
  using S = HexAffineShape<N, EPB_, TI>;
  if constexpr (S::LINES) {
    elastic_hex_col_body<N, EPB_, float, TI, true, kFuse>(bid, E, jac, mat, conn, u, r, Dm, iu);
    return;
  }
  constexpr int n = S::n, n2 = S::n2, P = S::P, EPB = S::EPB, NM = S::NM;
  extern __shared__ __align__(16) float smem_af[];
  const int t = threadIdx.x;
  const int le = t / n2, ij = t - le * n2;
  const int i = ij % n, j = ij / n;
  const int64_t e = bid * EPB + le;
  const bool ok = le < EPB && e < E;
  float *su = smem_af + (size_t)(ok ? le : 0) * S::US;                      // [3][P]
  float *sF = smem_af + (size_t)EPB * S::US + (size_t)(ok ? le : 0) * S::FS;  // [3][2][P]

  float Dri[n], Dsj[n], DTi[n], DTj[n];
#pragma unroll
  for (int l = 0; l < n; ++l) {
    Dri[l] = Dm.d[i * n + l];
    Dsj[l] = Dm.d[j * n + l];
    DTi[l] = Dm.d[l * n + i];
    DTj[l] = Dm.d[l * n + j];
  }
  int32_t node[n];
  float ux[n], uy[n], uz[n];
  if (ok) {
#pragma unroll
    for (int k = 0; k < n; ++k) node[k] = __ldg(conn + e * P + ij + n2 * k);
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const float *up = u + 3 * (int64_t)node[k];
      if constexpr (kFuse) {
        ux[k] = up[0];
        uy[k] = up[1];
        uz[k] = up[2];
      } else {
        ux[k] = __ldg(up + 0);
        uy[k] = __ldg(up + 1);
        uz[k] = __ldg(up + 2);
      }
    }
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const int p = ij + n2 * k;
      su[0 * P + p] = ux[k];
      su[1 * P + p] = uy[k];
      su[2 * P + p] = uz[k];
    }
  }
  float J[9];
#pragma unroll
  for (int a = 0; a < 9; ++a) J[a] = ok ? __ldg(jac + e * 9 + a) : 0.f;
  __syncthreads();
  float Ftx[n], Fty[n], Ftz[n];
  if (ok) {
    const int64_t P_E = (int64_t)P * E;
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const int p = ij + n2 * k;
      float m[NM];
#pragma unroll
      for (int q = 0; q < NM; ++q) m[q] = __ldg(mat + q * P_E + e * P + p);
      float d[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float *sc = su + c * P;
        const float *uc = c == 0 ? ux : (c == 1 ? uy : uz);
        float dr = 0, ds = 0, dt = 0;
#pragma unroll
        for (int l = 0; l < n; ++l) {
          dr += Dri[l] * sc[l + n * j + n2 * k];
          ds += Dsj[l] * sc[i + n * l + n2 * k];
          dt += Dm.d[k * n + l] * uc[l];
        }
        d[c][0] = dr; d[c][1] = ds; d[c][2] = dt;
      }
      float g[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int a = 0; a < 3; ++a)
          g[c][a] = J[a * 3 + 0] * d[c][0] + J[a * 3 + 1] * d[c][1] + J[a * 3 + 2] * d[c][2];
      float sig[3][3];
      if constexpr (TI) stress_ti<float>(g, m, sig);
      else stress_iso<float>(g, m[0], m[1], sig);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float F0 = J[0] * sig[c][0] + J[3] * sig[c][1] + J[6] * sig[c][2];
        const float F1 = J[1] * sig[c][0] + J[4] * sig[c][1] + J[7] * sig[c][2];
        const float F2 = J[2] * sig[c][0] + J[5] * sig[c][1] + J[8] * sig[c][2];
        sF[(c * 2 + 0) * P + p] = F0;
        sF[(c * 2 + 1) * P + p] = F1;
        if (c == 0) Ftx[k] = F2;
        else if (c == 1) Fty[k] = F2;
        else Ftz[k] = F2;
      }
    }
  }
  __syncthreads();
  if (!ok) return;
  // Elements holding a source keep the unfused form for their interior
  // points (residuals written; the source kernel adds the source terms and
  // finishes those nodes).  For the others, the interior operands (w)
  // are loaded here, before the divergence, so that their latency overlaps
  // it (after the stores below the compiler could not reorder them: the
  // pointers may alias as far as it knows).
  const bool fuse_here = kFuse && fuse_column<n>(i, j, e, iu);
  float wpre[n][3];
  if constexpr (kFuse) {
    if (fuse_here) {
      const float *__restrict__ ww = iu.w;
#pragma unroll
      for (int k = 1; k < n - 1; ++k) {
        const int64_t g = node[k];
#pragma unroll
        for (int c = 0; c < 3; ++c) wpre[k][c] = ww[g * 3 + c];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < n; ++k) {
    const int p = ij + n2 * k;
    float o[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float *Fr = sF + (c * 2 + 0) * P, *Fs = sF + (c * 2 + 1) * P;
      const float *Ft = c == 0 ? Ftx : (c == 1 ? Fty : Ftz);
      float acc = 0;
#pragma unroll
      for (int l = 0; l < n; ++l) {
        acc += DTi[l] * Fr[l + n * j + n2 * k];
        acc += DTj[l] * Fs[i + n * l + n2 * k];
        acc += Dm.d[l * n + k] * Ft[l];
      }
      o[c] = -acc;
    }
    const bool interior = fuse_here && k >= 1 && k <= n - 2;
    if (!interior) {
#pragma unroll
      for (int c = 0; c < 3; ++c) r[(e * P + p) * 3 + c] = o[c];
      continue;
    }
    if constexpr (kFuse) {
      // assembly (one incident point: 0 + r), inverse mass, Newmark
      const int64_t g = node[k];
      const float mm = __ldg(iu.mi + g);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int64_t x = g * 3 + c;
        float uo = c == 0 ? ux[k] : (c == 1 ? uy[k] : uz[k]);
        float wo = wpre[k][c];
        const float an = mul_rn(add_rn(0.f, o[c]), mm);
        newmark_point<float>(an, wo, uo, iu.dt);
        u[x] = uo;
        iu.w[x] = wo;
        if (iu.ap) iu.ap[x] = an;
      }
    }
  }
}

// Source kernel of the fused step (one CTA): the interior nodes of the
// source elements -- which the fused stiffness kernel left to it -- with the
// one-term assembly 0 + r, the source terms (add_sources), the inverse mass
// and the Newmark update: the arithmetic of the node gather, so the result is
// the unfused sequence's.
template <int N>
__global__ void source_fused_hex_kernel(int P, const float *__restrict__ r, int nse,
                                       const int64_t *__restrict__ src_elems,
                                       const int32_t *__restrict__ conn,
                                       const float *__restrict__ mi, float *__restrict__ u,
                                       float *__restrict__ w, float *__restrict__ ap, float dt,
                                       SourceTerms src) {
  constexpr int n = N + 1, m = N - 1, NI = m * m * m;
  for (int t = threadIdx.x; t < nse * NI; t += blockDim.x) {
    const int se = t / NI, q = t - se * NI;
    const int i = 1 + q % m, j = 1 + (q / m) % m, k = 1 + q / (m * m);
    const int64_t e = src_elems[se];
    const int pt = i + n * j + n * n * k;
    const int32_t g = conn[e * P + pt];
    float acc[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[c] = add_rn(0.f, r[(e * P + pt) * 3 + c]);
    add_sources<float, 3, false>(src.node[src.tile[g / kSrcTile] + g % kSrcTile], src, acc);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t x = (int64_t)g * 3 + c;
      float uo = u[x], wo = w[x];
      const float an = mul_rn(acc[c], mi[g]);
      newmark_point<float>(an, wo, uo, dt);
      u[x] = uo;
      w[x] = wo;
      if (ap) ap[x] = an;
    }
  }
}

// CTAs per SM asked of the compiler for the isotropic line-exchange kernels:
// what their registers allow anyway, but it schedules for it (order 4, 64^3:
// 373 -> 367 us; order 5, 18^3: 20.5 -> 18.9 us).
template <int N, int EPB_, bool TI>
constexpr int affine_min_blocks() {
  constexpr int nominal = 128 / ((N + 1) * (N + 1)) > 0 ? 128 / ((N + 1) * (N + 1)) : 1;
  if (TI || EPB_ != nominal) return 1;
  return N == 4 ? 8 : N == 5 ? 7 : N == 6 ? 6 : 1;
}
template <int N, int EPB_, bool TI>
__global__ void __launch_bounds__(HexAffineShape<N, EPB_, TI>::THREADS,
                                  affine_min_blocks<N, EPB_, TI>())
elastic_hex_affine_kernel(int64_t E, const float *__restrict__ jac, const float *__restrict__ mat,
                          const int32_t *__restrict__ conn, float *__restrict__ u,
                          float *__restrict__ r, DMatrix<float> Dm, HexInteriorUpdate iu) {
  elastic_hex_affine_body<N, EPB_, TI, false>(blockIdx.x, E, jac, mat, conn, u, r, Dm, iu);
}

// The fused form asks for 768 resident threads per SM (six 128-thread CTAs,
// a register cap): its interior-update registers would otherwise cost two
// CTAs per SM.
template <int THREADS>
constexpr int fuse_min_blocks() {
  return 768 / THREADS > 0 ? 768 / THREADS : 1;
}
template <int N, int EPB_, bool TI>
__global__ void __launch_bounds__(HexAffineShape<N, EPB_, TI>::THREADS,
                                  fuse_min_blocks<HexAffineShape<N, EPB_, TI>::THREADS>())
elastic_hex_affine_fused_kernel(int64_t E, const float *__restrict__ jac,
                                const float *__restrict__ mat, const int32_t *__restrict__ conn,
                                float *__restrict__ u, float *__restrict__ r, DMatrix<float> Dm,
                                HexInteriorUpdate iu) {
  elastic_hex_affine_body<N, EPB_, TI, true>(blockIdx.x, E, jac, mat, conn, u, r, Dm, iu);
}

}  // namespace salvus
