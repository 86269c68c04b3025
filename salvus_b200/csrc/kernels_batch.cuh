// kernels_batch.cuh -- shot-batched kernels: S shots on one mesh advance
// together.  Fields are shot-interleaved, f[node][S] (S padded to a multiple
// of 32), so a warp's lanes are consecutive shots: every field load and store
// is coalesced and each geometry / connectivity word is read once for all
// shots of a CTA.
//
// The arithmetic per shot is the reference's (Scalar::computeStiffnessTerm,
// Scalar.cpp:58-71; Ricker::fire, Ricker.cpp:27-33); the time update uses the
// velocity-at-half-step form of the reference's Newmark scheme
// (Order2Newmark.cpp:99-108): with w = v + dt/2 a_ the pair
//   v += dt/2 (a + a_);  u += dt v + dt^2/2 a
// is exactly  w += dt a;  u += dt w  (one fewer field to stream).
#pragma once

#include <cstdint>

namespace salvus {

// Interior-node update of the fused batched step (kFuse): the points with
// both local indices in 1..N-1 are nodes of this element alone, so the
// stiffness thread of (element, shot) finishes them -- the one-term assembly
// 0 + r, the inverse mass and the half-step-velocity update
// (batched_gather_update_kernel's arithmetic) -- and writes residuals only
// for the element's edge points.  Where the shot has a source in the element
// the interior residuals are written too, and batched_source_kernel adds the
// source terms and then finishes those nodes.  Same operations in the same
// order as the unfused sequence, so both forms give bitwise the same
// wavefields.
struct BatchInterior {
  const float *mi;
  float *w;
  float dt;
  const int32_t *shot_off;  // sources of shot s: [shot_off[s], shot_off[s + 1])
  const int64_t *src_elem;
  const uint8_t *has_src;  // per element: any shot has a source in it (null: no sources)
};

// half-step-velocity update of one node (one shot): w += dt a; u += dt w,
// with explicitly rounded operations so that every kernel applying it gives
// the same bits
__device__ __forceinline__ void half_step_update(float acc, float m, float dt, float &w, float &u) {
  w = __fmaf_rn(dt, __fmul_rn(acc, m), w);
  u = __fmaf_rn(dt, w, u);
}

// One thread = V consecutive shots of one quad element; the element's n^2
// values of those shots live in registers, so the tensor-product contractions
// need no shared memory.  CTA = EPC elements x SC shots, SC / V * EPC threads
// (SC = 0: one element, V shots for each thread of the launch).
// The element is walked row by row: a row's fluxes are formed, spread over the
// outputs of their columns and dropped, so that values and outputs (2 n^2 a
// shot) are all that lives throughout; with both flux fields kept the kernel
// could not take two shots.  Two shots per thread make every access 8 bytes
// and halve the address and record work; the register caps below keep enough
// warps per SM.  200^2 order 4 x 256 shots, fused launch: 564 us with one shot
// per thread and both flux fields, 446 with two (512 threads per SM; without
// the cap 533, 163 registers); 130^2 order 3, a step: 234 -> 217 us (768
// threads per SM; 512: 231).
template <int N, int SC, int EPC, int V>
constexpr int batched_ctas_per_sm() {
  constexpr int threads = SC ? SC / V * EPC : 128;
  constexpr int pair = N <= 2 ? 1024 : N == 3 ? 768 : N == 4 ? 512 : 256;
  constexpr int one = N <= 2 ? 1536 : N == 3 ? 1024 : N == 4 ? 896 : N == 5 ? 512 : 384;
  constexpr int resident = V == 2 ? pair : one;  // threads per SM
  constexpr int ctas = resident / threads > 0 ? resident / threads : 1;
  return ctas < 32 ? ctas : 32;
}
template <int N, int SC, int EPC, int V, bool kFuse = false>
__global__ void __launch_bounds__(SC ? SC / V * EPC : 128, batched_ctas_per_sm<N, SC, EPC, V>())
quad_acoustic_batched_kernel(int64_t E, int S, const float *__restrict__ rec,
                             float *__restrict__ u, float *__restrict__ r,
                             DMatrix<float> Dm, BatchInterior bi) {
  constexpr int n = N + 1, P = n * n;
  const int LN = SC ? SC / V : (int)blockDim.x;
  __shared__ float4 sg[EPC * P];  // G00 G01 G11 conn of the CTA's elements
  const int64_t e0 = (int64_t)blockIdx.x * EPC;
  for (int q = threadIdx.x; q < EPC * P; q += blockDim.x) {
    const int64_t ee = e0 + q / P;
    sg[q] = ee < E ? __ldg(reinterpret_cast<const float4 *>(rec) + e0 * P + q)
                   : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  const int ey = threadIdx.x / LN, lane = threadIdx.x - ey * LN;
  const int64_t e = e0 + ey;
  const int s = (blockIdx.y * LN + lane) * V;
  if (e >= E || s >= S) return;
  const float4 *g = sg + ey * P;
  struct alignas(4 * V) Shots {
    float v[V];
  };
  auto at = [&](float *field, int p) -> Shots & {
    return *reinterpret_cast<Shots *>(field + (int64_t)__float_as_int(g[p].w) * S + s);
  };
  auto interior = [](int p) {
    const int i = p % n, j = p / n;
    return i >= 1 && i <= n - 2 && j >= 1 && j <= n - 2;
  };
  // plain (coherent) loads: the fused form writes u of interior nodes
  Shots uu[P];
#pragma unroll
  for (int p = 0; p < P; ++p) uu[p] = at(u, p);
  // fused form: the interior nodes' w, and whether one of a shot's sources
  // sits in this element (then the unfused form for its interior points).
  // Nearly no element holds a source of any shot, and one byte says so; with
  // the shots' source lists searched by every thread the order-4 launch on
  // 200^2 x 256 shots took 535 us
  Shots wpre[P];
  bool fuse[V], all = kFuse;
  if constexpr (kFuse) {
#pragma unroll
    for (int p = 0; p < P; ++p)
      if (interior(p)) wpre[p] = at(bi.w, p);
    const bool search = bi.has_src && __ldg(bi.has_src + e);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      fuse[v] = true;
      if (search)
        for (int k = bi.shot_off[s + v]; k < bi.shot_off[s + v + 1] && fuse[v]; ++k)
          fuse[v] = __ldg(bi.src_elem + k) != e;
      all = all && fuse[v];
    }
  }
  float o[V][P];
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int p = 0; p < P; ++p) o[v][p] = 0.f;
#pragma unroll
  for (int j = 0; j < n; ++j)
#pragma unroll
    for (int v = 0; v < V; ++v) {
      float Fr[n];
#pragma unroll
      for (int i = 0; i < n; ++i) {
        float gr = 0.f, gs = 0.f;
#pragma unroll
        for (int l = 0; l < n; ++l) {
          gr += Dm.d[i * n + l] * uu[l + n * j].v[v];
          gs += Dm.d[j * n + l] * uu[i + n * l].v[v];
        }
        const float4 G = g[i + n * j];
        Fr[i] = G.x * gr + G.y * gs;
        const float Fs = G.y * gr + G.z * gs;
#pragma unroll
        for (int m = 0; m < n; ++m) o[v][i + n * m] += Dm.d[j * n + m] * Fs;
      }
#pragma unroll
      for (int i = 0; i < n; ++i)
#pragma unroll
        for (int l = 0; l < n; ++l) o[v][i + n * j] += Dm.d[l * n + i] * Fr[l];
    }
  float *out = r + (e * P) * S + s;
#pragma unroll
  for (int p = 0; p < P; ++p) {
    if (!interior(p) || !all) {
      Shots x;
#pragma unroll
      for (int v = 0; v < V; ++v) x.v[v] = -o[v][p];
      *reinterpret_cast<Shots *>(out + (int64_t)p * S) = x;
    }
    if constexpr (kFuse) {
      if (interior(p)) {
        // a shot left to the source kernel keeps its u and w
        Shots wv = wpre[p], uv = uu[p];
        const float m = __ldg(bi.mi + __float_as_int(g[p].w));
#pragma unroll
        for (int v = 0; v < V; ++v)
          if (fuse[v])
            half_step_update(__fadd_rn(0.f, -o[v][p]), m, bi.dt, wv.v[v], uv.v[v]);
        at(bi.w, p) = wv;
        at(u, p) = uv;
      }
    }
  }
}

// Ricker sources of every shot into the element-local residual.  Thread =
// (shot, point); a shot's sources are applied in attach order.  Fused step
// (n > 0, the element's points per line): afterwards the thread of an
// interior point finishes that node of each distinct source element of its
// shot -- the node the fused stiffness kernel left to it -- with the
// gather's arithmetic (one-term assembly 0 + r, inverse mass, update).
__global__ void batched_source_kernel(int S, int P, const int32_t *__restrict__ shot_off,
                                      const int64_t *__restrict__ elem,
                                      const double *__restrict__ par,
                                      const double *__restrict__ wts,
                                      const int64_t *__restrict__ step, double dt,
                                      float *__restrict__ r, int n = 0,
                                      const int32_t *__restrict__ conn = nullptr,
                                      const float *__restrict__ mi = nullptr,
                                      float *__restrict__ u = nullptr,
                                      float *__restrict__ w = nullptr, float dtf = 0.f) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= S * P) return;
  const int p = q % P, s = q / P;
  const double t = (double)(*step) * dt;
  for (int k = shot_off[s]; k < shot_off[s + 1]; ++k) {
    const double stf = ricker_dev(t, par[3 * k], par[3 * k + 1], par[3 * k + 2]);
    r[(elem[k] * P + p) * S + s] += (float)(wts[(int64_t)k * P + p] * stf);
  }
  if (n == 0) return;
  const int i = p % n, j = p / n;
  if (i < 1 || i > n - 2 || j < 1 || j > n - 2) return;
  for (int k = shot_off[s]; k < shot_off[s + 1]; ++k) {
    bool first = true;  // each distinct source element once
    for (int k2 = shot_off[s]; k2 < k && first; ++k2) first = elem[k2] != elem[k];
    if (!first) continue;
    const int64_t e = elem[k];
    const int32_t node = conn[e * P + p];
    const int64_t x = (int64_t)node * S + s;
    float wv = w[x], uv = u[x];
    half_step_update(__fadd_rn(0.f, r[(e * P + p) * S + s]), mi[node], dtf, wv, uv);
    w[x] = wv;
    u[x] = uv;
  }
}

// Node gather + inverse mass + half-step-velocity update, thread = (NPT
// consecutive nodes, four consecutive shots): every field and residual access
// is 16 bytes per thread, which is what keeps enough bytes in flight behind
// the dependent chain incidence -> residual.  CTA = NPB node groups x SC
// shots, SC / 4 * NPB threads.  The NPT nodes' chains are issued side by
// side.  One shot per thread moved 3.7 of 6.5 TB/s on the edge nodes of 200^2
// order-4 quads x 256 shots; four took the step from 1075 to 875 us (B200).
// The per-node arithmetic and summation order do not depend on the split.
// nodes != nullptr: thread slot t handles node nodes[t] (the edge nodes of
// the fused form), G is then the list's length.
template <int SC, int NPB, int NPT>
__global__ void __launch_bounds__(SC / 4 * NPB)
batched_gather_update_kernel(int64_t G, int S, Incidence inc, const float *__restrict__ r,
                             const float *__restrict__ mi, float *__restrict__ u,
                             float *__restrict__ w, float dt,
                             const int32_t *__restrict__ nodes, int64_t *__restrict__ step) {
  if (step && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *step += 1;
  constexpr int LN = SC / 4;
  const int ny = threadIdx.x / LN, lane = threadIdx.x - ny * LN;
  const int64_t g0 = ((int64_t)blockIdx.x * NPB + ny) * NPT;
  const int s = blockIdx.y * SC + 4 * lane;
  if (g0 >= G || s >= S) return;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto add = [](float4 &x, const float4 &y) { x.x += y.x, x.y += y.y, x.z += y.z, x.w += y.w; };
  float4 uo[NPT], wo[NPT];
  float m[NPT];
  int2 h[NPT];
  int64_t gk[NPT];
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    const bool live = g0 + k < G;
    const int64_t g = !live ? 0 : nodes ? (int64_t)__ldg(nodes + g0 + k) : g0 + k;
    gk[k] = g;
    h[k] = live ? __ldg(inc.head + g) : int2{0, -1};
    uo[k] = live ? *reinterpret_cast<const float4 *>(u + g * S + s) : zero;
    wo[k] = live ? *reinterpret_cast<const float4 *>(w + g * S + s) : zero;
    m[k] = live ? __ldg(mi + g) : 0.f;
  }
  auto load = [&](int32_t ep) {
    return __ldg(reinterpret_cast<const float4 *>(r + (int64_t)ep * S + s));
  };
  // summed in ascending element order
  float4 acc[NPT], second[NPT];
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    const bool live = g0 + k < G;
    acc[k] = live && h[k].y >= -1 ? load(h[k].x) : zero;
    second[k] = live && h[k].y >= 0 ? load(h[k].y) : zero;
  }
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    if (g0 + k >= G) break;
    float4 sum = zero;
    add(sum, acc[k]);
    if (h[k].y >= 0) {
      add(sum, second[k]);
    } else if (h[k].y < -1) {
      constexpr int kBatch = 4;  // the usual valence of a quadrilateral vertex
      const int32_t q1 = h[k].x - h[k].y;
      for (int32_t qb = h[k].x; qb < q1; qb += kBatch) {
        int32_t ep[kBatch];
        float4 rv[kBatch];
#pragma unroll
        for (int z = 0; z < kBatch; ++z) ep[z] = qb + z < q1 ? __ldg(inc.rest + qb + z) : 0;
#pragma unroll
        for (int z = 0; z < kBatch; ++z) rv[z] = qb + z < q1 ? load(ep[z]) : zero;
#pragma unroll
        for (int z = 0; z < kBatch; ++z)
          if (qb + z < q1) add(sum, rv[z]);
      }
    }
    half_step_update(sum.x, m[k], dt, wo[k].x, uo[k].x);
    half_step_update(sum.y, m[k], dt, wo[k].y, uo[k].y);
    half_step_update(sum.z, m[k], dt, wo[k].z, uo[k].z);
    half_step_update(sum.w, m[k], dt, wo[k].w, uo[k].w);
    const int64_t i = gk[k] * S + s;
    *reinterpret_cast<float4 *>(w + i) = wo[k];
    *reinterpret_cast<float4 *>(u + i) = uo[k];
  }
}

// Receivers of every shot: block = receiver, thread = shot; FP64 Kahan over
// the element points.  seis[(s * R + rec) * cap + n % cap] after step n, the
// one just completed (*step - 1).
__global__ void batched_receiver_kernel(int S, int R, int P, const int64_t *__restrict__ elem,
                                        const double *__restrict__ lw,
                                        const int32_t *__restrict__ conn,
                                        const float *__restrict__ u, double *__restrict__ seis,
                                        int64_t cap, const int64_t *__restrict__ step) {
  const int rc = blockIdx.x;
  const int64_t e = elem[rc];
  const int64_t slot = (*step - 1) % cap;
  for (int s = threadIdx.x; s < S; s += blockDim.x) {
    double acc = 0.0, comp = 0.0;
    for (int p = 0; p < P; ++p) {
      const double y = lw[(int64_t)rc * P + p] * (double)u[(int64_t)conn[e * P + p] * S + s] - comp;
      const double tt = acc + y;
      comp = (tt - acc) - y;
      acc = tt;
    }
    seis[((int64_t)s * R + rc) * cap + slot] = acc;
  }
}

// Column k of a shot-interleaved field <-> a contiguous FP64 array.
__global__ void shot_scatter_kernel(int64_t G, int S, int k, const double *__restrict__ src,
                                    float *__restrict__ f) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < G) f[g * S + k] = (float)src[g];
}
__global__ void shot_gather_kernel(int64_t G, int S, int k, const float *__restrict__ f,
                                   double *__restrict__ dst) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < G) dst[g] = (double)f[g * S + k];
}

}  // namespace salvus
