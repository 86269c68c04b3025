// kernels_hex_col.cuh -- elastic hexahedron stiffness of orders 4 and up (FP64:
// of every order, see HexCol64), r_e = -K_e u_e, by column threads and line exchange (Elastic3D.cpp:70-118 via
// Hexahedra.cpp:580-632 / 689-754).
//
// What bounds the kernel is the shared-memory pipe: a shared load delivers 32
// words per wavefront whatever its width and however many lanes share an
// address, so the words that the contractions read are what counts.  One
// thread per (i, j) column that reads the n points of its r- and s-line for
// each of its own n points (the order <= 3 kernels) reads 4 n words per point
// and component for gradient and divergence: 8.6 k words per order-4 element
// with the writes.  Here the r- and s-derivatives are taken line by line
// instead: a thread reads the n words of one line, forms all n outputs with
// compile-time D entries and writes them back for the column threads, which
// keep the t direction in registers.  Each direction then costs 3 words per
// point and component (read, write, read): 5.6 k words.  No thread holds rows
// of D any more (64 registers instead of 72 at order 4, 8 CTAs per SM).
// Parallelepipeds: 64^3 order 4 0.435 -> 0.367 ms, 18^3 order 5 25.0 -> 18.9
// us, 24^3 order 6 98.7 -> 67.9 us; per-point records: 64^3 order 4 0.517 ->
// 0.426 ms, 78 % of the measured copy bandwidth (B200).  At orders 1-3 the two
// added barriers cost more than the words save (order 3: 48.5 -> 51.5 us on
// 40^3), so those keep the column kernels.
#pragma once

#include <cstdint>

#include "kernels_material.cuh"
#include "kernels_step.cuh"
#include "kernels_stiffness.cuh"

namespace salvus {

// Shared-memory layout of one component of one element: point (i, j, k) at
// word i + A j + B k, elements of a CTA at a stride congruent to R mod 32.
// (A, B, R) were searched, with the line order of HexLines, for the fewest
// bank conflicts over the seven column and eight line accesses of a step
// (wavefronts per access: 1.27, 1.07, 1.00, 1.00 for n = 4..7; with the plain
// layout and the lines in element order 1.5 for n = 5).
template <int n>
struct HexColPad;
template <> struct HexColPad<2> { static constexpr int A = 2, B = 5, R = 4; };
template <> struct HexColPad<3> { static constexpr int A = 3, B = 11, R = 9; };
template <> struct HexColPad<4> { static constexpr int A = 4, B = 19, R = 16; };
template <> struct HexColPad<5> { static constexpr int A = 5, B = 29, R = 25; };
template <> struct HexColPad<6> { static constexpr int A = 6, B = 37, R = 4; };
template <> struct HexColPad<7> { static constexpr int A = 7, B = 52, R = 17; };

// NC components per node.
template <int N, int EPB_, typename real, int NC = 3>
struct HexColShape {
  static constexpr int n = N + 1, n2 = n * n, P = n2 * n;
  static constexpr int EPB = EPB_;
  static constexpr int THREADS = ((EPB * n2 + 31) / 32) * 32;
  static constexpr int A = HexColPad<n>::A, B = HexColPad<n>::B;
  static constexpr int PL = (n - 1) * (1 + A + B) + 1;  // words of one component
  static constexpr int ES = NC * PL + ((HexColPad<n>::R - NC * PL % 32) + 32) % 32;
  static constexpr int ARR = EPB * ES;  // words of one array (all components)
  static constexpr size_t SMEM = sizeof(real) * (size_t)3 * ARR;
};

// Which r-line and s-line each thread of a CTA works on, as the offset of the
// line's first point (kNone: none).  The EPB n^2 lines of a direction are
// dealt to the warps in turn so that as few lanes of a warp as possible start
// in the same bank: a warp takes one line of each bank, the banks with the
// most lines left first, and a second one only where the warps after it could
// not hold what is left.
template <int N, int EPB, int NC = 3>
struct HexLines {
  using S = HexColShape<N, EPB, float, NC>;
  static constexpr uint16_t kNone = 0xffff;
  uint16_t r[S::THREADS], s[S::THREADS];
};
template <int N, int EPB, int NC = 3>
constexpr HexLines<N, EPB, NC> make_hex_lines() {
  using S = HexColShape<N, EPB, float, NC>;
  constexpr int n = S::n, W = S::THREADS / 32, L = EPB * S::n2;
  HexLines<N, EPB, NC> h{};
  for (int dir = 0; dir < 2; ++dir) {
    uint16_t *out = dir == 0 ? h.r : h.s;
    for (int t = 0; t < S::THREADS; ++t) out[t] = HexLines<N, EPB>::kNone;
    uint16_t by[32][L] = {};  // the lines that start in each bank
    int cnt[32] = {};
    for (int x = 0; x < L; ++x) {
      const int le = x / S::n2, a = x % n, b = (x / n) % n;
      const int at = le * S::ES + (dir == 0 ? S::A * a : a) + S::B * b;
      by[at % 32][cnt[at % 32]++] = (uint16_t)at;
    }
    int left = L;
    for (int w = 0; w < W; ++w) {
      const int must = left - 32 * (W - 1 - w);
      int took = 0;
      for (int depth = 0; took < 32 && left > 0 && (depth == 0 || took < must); ++depth) {
        bool done[32] = {};
        for (int pick = 0; pick < 32 && took < 32 && (depth == 0 || took < must); ++pick) {
          int best = -1;
          for (int q = 0; q < 32; ++q)
            if (!done[q] && cnt[q] > 0 && (best < 0 || cnt[q] > cnt[best])) best = q;
          if (best < 0) break;
          done[best] = true;
          out[32 * w + took++] = by[best][--cnt[best]];
          --left;
        }
      }
    }
  }
  return h;
}
template <int N, int EPB, int NC = 3>
__device__ const HexLines<N, EPB, NC> kHexLines = make_hex_lines<N, EPB, NC>();

// The NC components' lines: out[m] = sum_l D[m][l] in[l] (kT: D[l][m]),
// every load before the first store (they may alias for the compiler, and in
// the divergence they do).
template <int n, int stride, int PL, bool kT, int NC = 3, typename real>
__device__ __forceinline__ void line_apply(const real *in, real *out, const DMatrix<real> &Dm) {
  real v[NC][n];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int l = 0; l < n; ++l) v[c][l] = in[c * PL + l * stride];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int m = 0; m < n; ++m) {
      real acc = 0;
#pragma unroll
      for (int l = 0; l < n; ++l) acc += (kT ? Dm.d[l * n + m] : Dm.d[m * n + l]) * v[c][l];
      out[c * PL + m * stride] = acc;
    }
}

// Interior-node update of the fused step: Newmark state, inverse mass, and
// the elements that hold a source (their interior nodes are finished by the
// source kernel, which adds the source terms).
struct HexInteriorUpdate {
  const float *mi;
  float *w, *ap;  // ap: null unless this step stores a_
  float dt;
  int nsrc_elem;
  const int64_t *src_elem;  // distinct source elements
};

// Finishes an interior column (fused step): see kernels_hex_affine.cuh.
template <int n>
__device__ __forceinline__ bool fuse_column(int i, int j, int64_t e, const HexInteriorUpdate &iu) {
  bool fuse = i >= 1 && i <= n - 2 && j >= 1 && j <= n - 2;
  for (int s = 0; s < iu.nsrc_elem && fuse; ++s) fuse = __ldg(iu.src_elem + s) != e;
  return fuse;
}

// One group of EPB elements (bid), all threads of the CTA (contains
// __syncthreads).  Geometry and material, as the kernels of the lower orders:
//   kAffine  jac [E][9], rec = material planes [NM][E*P], conn [E][P]
//   FP32     rec = float4 planes [E][3|4][P] (connectivity inside)
//   FP64     rec [E][P][9 + NM], conn [E][P]
template <int N, int EPB_, typename real, bool TI, bool kAffine, bool kFuse>
__device__ __forceinline__ void elastic_hex_col_body(
    int64_t bid, int64_t E, const real *__restrict__ jac, const real *__restrict__ rec,
    const int32_t *__restrict__ conn, real *__restrict__ u, real *__restrict__ r,
    const DMatrix<real> &Dm, const HexInteriorUpdate &iu) {
  using S = HexColShape<N, EPB_, real>;
  constexpr int n = S::n, n2 = S::n2, P = S::P, EPB = S::EPB, A = S::A, B = S::B, PL = S::PL;
  constexpr int NM = ElasticMat<TI>::kWords;
  constexpr bool kPacked = !kAffine && sizeof(real) == 4;  // connectivity in the record
  extern __shared__ __align__(16) unsigned char smem_hc[];
  real *su = reinterpret_cast<real *>(smem_hc), *sR = su + S::ARR, *sS = sR + S::ARR;
  const int t = threadIdx.x;
  const int le = t / n2, ij = t - le * n2;
  const int i = ij % n, j = ij / n;
  const int64_t e = bid * EPB + le;
  const bool ok = le < EPB && e < E;
  const int at = le * S::ES + i + A * j;
  const uint32_t lr = kHexLines<N, EPB_>.r[t], ls = kHexLines<N, EPB_>.s[t];
  constexpr uint32_t kNone = HexLines<N, EPB_>::kNone;

  real uc[3][n], mat[n][NM], J[9];
  int32_t node[n];
  // packed records: planes (invJ 0-3), (invJ 4-7), (invJ 8, m0, m1, node)
  const float4 *rq = reinterpret_cast<const float4 *>(rec) + e * (TI ? 4 : 3) * P + ij;
  float4 ra[n], rb[n], rc[n];
  if (ok) {
    if constexpr (kPacked) {
#pragma unroll
      for (int k = 0; k < n; ++k) {
        rc[k] = __ldg(rq + 2 * P + n2 * k);
        node[k] = __float_as_int(rc[k].w);
      }
    } else {
#pragma unroll
      for (int k = 0; k < n; ++k) node[k] = __ldg(conn + e * P + ij + n2 * k);
    }
#pragma unroll
    for (int k = 0; k < n; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const real *up = u + 3 * (int64_t)node[k] + c;
        uc[c][k] = kFuse ? *up : __ldg(up);  // the fused form writes u during the launch
      }
    if constexpr (kAffine) {
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int q = 0; q < NM; ++q)
          mat[k][q] = __ldg(rec + (int64_t)q * P * E + e * P + ij + n2 * k);
#pragma unroll
      for (int a = 0; a < 9; ++a) J[a] = __ldg(jac + e * 9 + a);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int k = 0; k < n; ++k) su[at + c * PL + B * k] = uc[c][k];
  }
  __syncthreads();
  if constexpr (kPacked) {
    // the geometry of the whole column, in flight during the line phase (read
    // point by point behind the barrier it held the 27^3 order-4 kernel at 55
    // instead of 39 us)
    if (ok)
#pragma unroll
      for (int k = 0; k < n; ++k) {
        ra[k] = __ldg(rq + n2 * k);
        rb[k] = __ldg(rq + P + n2 * k);
      }
  }
  if (lr != kNone) line_apply<n, 1, PL, false>(su + lr, sR + lr, Dm);
  if (ls != kNone) line_apply<n, A, PL, false>(su + ls, sS + ls, Dm);
  __syncthreads();
  real o[3][n];  // t part of the divergence
  if (ok) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int k = 0; k < n; ++k) o[c][k] = 0;
#pragma unroll
    for (int k = 0; k < n; ++k) {
      if constexpr (kPacked) {
        J[0] = ra[k].x, J[1] = ra[k].y, J[2] = ra[k].z, J[3] = ra[k].w;
        J[4] = rb[k].x, J[5] = rb[k].y, J[6] = rb[k].z, J[7] = rb[k].w;
        J[8] = rc[k].x, mat[k][0] = rc[k].y, mat[k][1] = rc[k].z;
        if constexpr (TI) {
          const float4 rt = __ldg(rq + 3 * P + n2 * k);
          mat[k][2] = rt.x, mat[k][3] = rt.y, mat[k][4] = rt.z;
        }
      } else if constexpr (!kAffine) {
        load_elastic_rec<TI>(rec, e, ij + n2 * k, P, J, mat[k]);
      }
      real d[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        d[c][0] = sR[at + c * PL + B * k];
        d[c][1] = sS[at + c * PL + B * k];
        real dt = 0;
#pragma unroll
        for (int l = 0; l < n; ++l) dt += Dm.d[k * n + l] * uc[c][l];
        d[c][2] = dt;
      }
      real g[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int a = 0; a < 3; ++a)
          g[c][a] = J[a * 3 + 0] * d[c][0] + J[a * 3 + 1] * d[c][1] + J[a * 3 + 2] * d[c][2];
      real sig[3][3];
      if constexpr (TI) stress_ti<real>(g, mat[k], sig);
      else stress_iso<real>(g, mat[k][0], mat[k][1], sig);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        sR[at + c * PL + B * k] = J[0] * sig[c][0] + J[3] * sig[c][1] + J[6] * sig[c][2];
        sS[at + c * PL + B * k] = J[1] * sig[c][0] + J[4] * sig[c][1] + J[7] * sig[c][2];
        const real F2 = J[2] * sig[c][0] + J[5] * sig[c][1] + J[8] * sig[c][2];
#pragma unroll
        for (int m = 0; m < n; ++m) o[c][m] += Dm.d[k * n + m] * F2;
      }
    }
  }
  __syncthreads();
  if (lr != kNone) line_apply<n, 1, PL, true>(sR + lr, sR + lr, Dm);
  if (ls != kNone) line_apply<n, A, PL, true>(sS + ls, sS + ls, Dm);
  // interior operand of the fused form, loaded under the barrier
  bool fuse = false;
  real wp[3][n];
  if constexpr (kFuse) {
    fuse = ok && fuse_column<n>(i, j, e, iu);
    if (fuse)
#pragma unroll
      for (int k = 1; k < n - 1; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) wp[c][k] = iu.w[(int64_t)node[k] * 3 + c];
  }
  __syncthreads();
  if (!ok) return;
#pragma unroll
  for (int k = 0; k < n; ++k) {
    real out[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
      out[c] = -(o[c][k] + sR[at + c * PL + B * k] + sS[at + c * PL + B * k]);
    if (kFuse && fuse && k >= 1 && k <= n - 2) {
      if constexpr (kFuse) {
        const real mm = __ldg(iu.mi + node[k]);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int64_t x = (int64_t)node[k] * 3 + c;
          const real an = mul_rn(add_rn(0.f, out[c]), mm);
          newmark_point<real>(an, wp[c][k], uc[c][k], iu.dt);
          u[x] = uc[c][k];
          iu.w[x] = wp[c][k];
          if (iu.ap) iu.ap[x] = an;
        }
      }
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) r[(e * P + ij + n2 * k) * 3 + c] = out[c];
    }
  }
}

// FP64 kernels.  The FP64 column kernel (elastic_hex_stiffness_kernel) reads
// 88-byte records point by point; on meshes of parallelepipeds this body reads
// 16 bytes of material per point and one Jacobian per element instead, and
// runs at every order.  Elements per CTA and CTAs per SM by measurement (B200,
// us, FP64 column kernel -> here): 22^3 order 4 57.4 -> 33.2 (4 CTAs asked;
// 35.3 without), 18^3 order 5 83.7 -> 37.2, 12^3 order 6 29.1 -> 20.8, 28^3
// order 3 45.2 -> 31.0 (64-thread CTAs; 33.0 with 128), 36^3 order 2 53.6 ->
// 33.1, 50^3 order 1 43.2 -> 24.9.  General hexahedra keep their records:
// order 4 51.6, order 5 53.8 (4 CTAs asked; 59.7), order 6 24.8 (one element
// per CTA), order 2 49.3, order 1 39.2; order 3 stays on the column kernel
// (45.2 against 49.6).
template <int N, bool TI, bool kAffine>
struct HexCol64 {
  static constexpr int n2 = (N + 1) * (N + 1);
  static constexpr int kThreads = N >= 4 && !(N == 6 && !kAffine) ? 128 : 64;
  static constexpr int EPB = kThreads / n2 > 0 ? kThreads / n2 : 1;
  static constexpr int CTAS = !TI && N == (kAffine ? 4 : 5) ? 4 : 1;
  static constexpr bool kUse = kAffine || N != 3;
};
template <int N, bool TI, bool kAffine>
__global__ void __launch_bounds__(HexColShape<N, HexCol64<N, TI, kAffine>::EPB, double>::THREADS,
                                  HexCol64<N, TI, kAffine>::CTAS)
elastic_hex_col64_kernel(int64_t E, const double *__restrict__ jac, const double *__restrict__ rec,
                         const int32_t *__restrict__ conn, double *__restrict__ u,
                         double *__restrict__ r, DMatrix<double> Dm) {
  elastic_hex_col_body<N, HexCol64<N, TI, kAffine>::EPB, double, TI, kAffine, false>(
      blockIdx.x, E, jac, rec, conn, u, r, Dm, HexInteriorUpdate{});
}

// Acoustic hexahedra of orders 2 and up (Scalar.cpp:58-71) by the same line
// exchange: G = w detJ vp^2 invJ^T invJ (six products) per point, records as in
// load_acoustic_rec.  One thread per point read 6 n shared words per point,
// here 13 and the t direction in registers.  Per step, FP32 / FP64 (B200, us):
// 24^3 order 4 28.4 -> 20.1 / 53.1 -> 37.4, 15^3 order 6 24.3 -> 15.7 / 42.9 ->
// 26.8, 40^3 order 2 23.4 -> 18.0 / 42.6 -> 34.7.
template <int N, typename real>
struct AcousticHexCol {
  static constexpr int n2 = (N + 1) * (N + 1);
  static constexpr int EPB = 128 / n2 > 0 ? 128 / n2 : 1;
  using Shape = HexColShape<N, EPB, real, 1>;
};
template <int N, typename real>
__global__ void __launch_bounds__(AcousticHexCol<N, real>::Shape::THREADS)
acoustic_hex_col_kernel(int64_t E, const real *__restrict__ rec, const int32_t *__restrict__ conn,
                        const real *__restrict__ u, real *__restrict__ r, DMatrix<real> Dm) {
  constexpr int EPB = AcousticHexCol<N, real>::EPB;
  using S = typename AcousticHexCol<N, real>::Shape;
  constexpr int n = S::n, n2 = S::n2, P = S::P, A = S::A, B = S::B, PL = S::PL;
  __shared__ real su[S::ARR], sR[S::ARR], sS[S::ARR];
  const int t = threadIdx.x;
  const int le = t / n2, ij = t - le * n2;
  const int64_t e = (int64_t)blockIdx.x * EPB + le;
  const bool ok = le < EPB && e < E;
  const int at = le * S::ES + ij % n + A * (ij / n);
  const uint32_t lr = kHexLines<N, EPB, 1>.r[t], ls = kHexLines<N, EPB, 1>.s[t];
  constexpr uint32_t kNone = HexLines<N, EPB, 1>::kNone;
  real uc[n], g[n][6];
  if (ok) {
    int32_t node[n];
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const int64_t ep = e * P + ij + n2 * k;
      load_acoustic_rec<3>(rec, conn, ep, ep, g[k], &node[k]);
    }
#pragma unroll
    for (int k = 0; k < n; ++k) uc[k] = __ldg(u + node[k]);
#pragma unroll
    for (int k = 0; k < n; ++k) su[at + B * k] = uc[k];
  }
  __syncthreads();
  if (lr != kNone) line_apply<n, 1, PL, false, 1>(su + lr, sR + lr, Dm);
  if (ls != kNone) line_apply<n, A, PL, false, 1>(su + ls, sS + ls, Dm);
  __syncthreads();
  real o[n];
  if (ok) {
#pragma unroll
    for (int k = 0; k < n; ++k) o[k] = 0;
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const real dr = sR[at + B * k], ds = sS[at + B * k];
      real dt = 0;
#pragma unroll
      for (int l = 0; l < n; ++l) dt += Dm.d[k * n + l] * uc[l];
      // G00 G01 G02 G11 G12 G22
      sR[at + B * k] = g[k][0] * dr + g[k][1] * ds + g[k][2] * dt;
      sS[at + B * k] = g[k][1] * dr + g[k][3] * ds + g[k][4] * dt;
      const real Ft = g[k][2] * dr + g[k][4] * ds + g[k][5] * dt;
#pragma unroll
      for (int m = 0; m < n; ++m) o[m] += Dm.d[k * n + m] * Ft;
    }
  }
  __syncthreads();
  if (lr != kNone) line_apply<n, 1, PL, true, 1>(sR + lr, sR + lr, Dm);
  if (ls != kNone) line_apply<n, A, PL, true, 1>(sS + ls, sS + ls, Dm);
  __syncthreads();
  if (!ok) return;
#pragma unroll
  for (int k = 0; k < n; ++k)
    r[e * P + ij + n2 * k] = -(o[k] + sR[at + B * k] + sS[at + B * k]);
}

}  // namespace salvus
