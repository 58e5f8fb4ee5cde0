// Gradient surrogate network: a small MLP d_in -> h1 -> h2 -> d_out with
// exact (erf) GELU after the two hidden layers, trained online by the
// sampler on (position, gradient) pairs.  No counterpart in the reference,
// whose samplers always evaluate the exact gradient.
//
// Parameters are one flat FP32 master vector
//   [W1 (h1 x d_in), b1 (h1), W2 (h2 x h1), b2 (h2), W3 (d_out x h2), b3 (d_out)]
// with a bf16 copy of the same layout; forward passes multiply by the bf16
// weights with FP32 accumulation and FP32 biases.  The layer products run on
// the CUDA cores: they are a few hundred MFLOP per step, small beside the exact
// HLR pass.  An output is one chain of multiply-adds in k order in
// mlp_gemm_kernel and mlp_rows_kernel; mlp_cluster_kernel splits it over up to 32
// lanes and adds their parts in a tree.  So a prediction's last bits depend on
// whether its batch is one for clusters, and a forward pass's on whether it
// keeps the activations; each repeats bit for bit.
//
//   forward   P1 = X W1^T + b1, A1 = gelu(P1), P2 = A1 W2^T + b2,
//             A2 = gelu(P2), Y = A2 W3^T + b3 — a product per layer when the
//             activations are kept for the backward pass, otherwise one fused
//             launch, a few rows per cluster or block with the activations in
//             shared memory
//   loss      mean squared error against a target, dY = 2 (Y - T) / (B d_out)
//   backward  dW3 = dY^T A2, db3 = colsum dY, dP2 = (dY W3) . gelu'(P2), ...
//   Adam      on the master vector, refreshing the bf16 copy.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <math.h>

#include "common.cuh"

namespace ab {
namespace {

constexpr int TM = 32, TN = 32, TK = 32;       // output tile and K slice of mlp_gemm_kernel
constexpr int GEMM_THREADS = 128;
constexpr int GROUPS = TK * TM / 4 / GEMM_THREADS;   // four-element groups of a slice a thread loads

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

enum { EPI_STORE = 0, EPI_GELU = 1, EPI_GELU_GRAD = 2 };

// C[m][n] = sum_k A(m, k) B(k, n) (+ bias[n]) with A(m, k) = A[m*sam + k*sak]
// and B(k, n) = B[k*sbk + n*sbn].  EPI_GELU also stores P (pre-activation)
// to C and gelu(P) to C2; EPI_GELU_GRAD multiplies by gelu'(P[m][n]).
// `colsum`, when given, receives sum_k A(m, k) for every m.
struct GemmJob {
  int M, N, K, epi;
  const float* A;
  int sam, sak;
  const void* B;   // float, or bf16 (b_bf16)
  int b_bf16, sbk, sbn;
  const float* bias;
  float* C;
  int ldc;
  float* C2;
  const float* P;
  int ldp;
  float* colsum;
  int a_vec, b_vec;   // set by gemm(): 16-byte (bf16: 8-byte) loads along the unit-stride dimension
};

// Up to two independent products in one launch (a layer's weight gradient
// beside the gradient handed to the layer below).
struct GemmJobs {
  GemmJob j[2];
  int tiles0;      // 32 x 32 output tiles of j[0]
};

// A group of four elements of one operand as loaded (raw bits, so that a
// prefetched group waits for its load only when it is stored).
__device__ __forceinline__ uint4 ld4(const float* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ uint4 ld4(const __nv_bfloat16* p) {
  const uint2 r = *reinterpret_cast<const uint2*>(p);
  return make_uint4(r.x, r.y, 0u, 0u);
}
__device__ __forceinline__ uint4 pack4(const float* p, size_t su, int n) {
  return make_uint4(__float_as_uint(p[0]), n > 1 ? __float_as_uint(p[su]) : 0u, n > 2 ? __float_as_uint(p[2 * su]) : 0u,
                    n > 3 ? __float_as_uint(p[3 * su]) : 0u);
}
__device__ __forceinline__ uint4 pack4(const __nv_bfloat16* p, size_t su, int n) {
  const unsigned short* h = reinterpret_cast<const unsigned short*>(p);
  const uint32_t a = h[0], b = n > 1 ? h[su] : 0u, c = n > 2 ? h[2 * su] : 0u, d = n > 3 ? h[3 * su] : 0u;
  return make_uint4(a | (b << 16), c | (d << 16), 0u, 0u);
}
template <bool BF16>
__device__ __forceinline__ float4 to_f32(const uint4& r) {
  if (BF16)
    return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16),
                       __uint_as_float(r.y & 0xffff0000u));
  return make_float4(__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z), __uint_as_float(r.w));
}

// A staged K slice is [TK][32] floats; the float4 holding rows (m or n)
// 4g..4g+3 of k lies at group g ^ ((k >> 2) & 7), which keeps both kinds of
// store below and the reads free of bank conflicts.
__device__ __forceinline__ int slot(int k, int r) { return k * 32 + ((((r >> 2) ^ (k >> 2)) & 7) << 2) + (r & 3); }

// The next K slice of one operand into registers, GROUPS groups of four
// elements along its unit-stride dimension a thread.  (r, k) is an element's
// row (m or n) and K index; rows at or past R and k at or past K are zero.
// `vec`: whole groups are in or out of range and aligned, one load each.
template <typename T>
__device__ __forceinline__ void fetch_slice(uint4 (&v)[GROUPS], const T* __restrict__ X, bool vec, int r0, int R,
                                            int sr, int k0, int K, int sk) {
  const bool k_unit = sk == 1;
  const int u = 4 * (threadIdx.x & 7), o = threadIdx.x >> 3;   // along, across the unit-stride dimension
  const int u_left = (k_unit ? K - k0 : R - r0) - u, o_left = (k_unit ? R - r0 : K - k0) - o;
  const size_t so = k_unit ? sr : sk, su = k_unit ? sk : sr;
  const T* p = X + (size_t)r0 * sr + (size_t)k0 * sk + (size_t)o * so + (size_t)u * su;
#pragma unroll
  for (int i = 0; i < GROUPS; ++i, p += (GEMM_THREADS / 8) * so) {
    v[i] = make_uint4(0u, 0u, 0u, 0u);
    if (o_left > (GEMM_THREADS / 8) * i && u_left > 0) v[i] = vec ? ld4(p) : pack4(p, su, u_left);
  }
}

template <bool BF16>
__device__ __forceinline__ void put_slice(float* S, const uint4 (&v)[GROUPS], bool k_unit) {
  const int u = 4 * (threadIdx.x & 7), o = threadIdx.x >> 3;
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int oo = o + (GEMM_THREADS / 8) * i;
    const float4 f = to_f32<BF16>(v[i]);
    if (k_unit) {
      S[slot(u, oo)] = f.x;
      S[slot(u + 1, oo)] = f.y;
      S[slot(u + 2, oo)] = f.z;
      S[slot(u + 3, oo)] = f.w;
    } else {
      *reinterpret_cast<float4*>(S + slot(oo, u)) = f;
    }
  }
}

// One 32 x 32 output tile per CTA of 128 threads, 4 x 2 outputs a thread, so
// that the layers of a 512-256-256-512 network and a batch of 512 give 64 to
// 256 CTAs a launch (64 x 64 tiles gave 16 to 32 and left most SMs idle).  Each
// output is one chain of fused multiply-adds in k order, whatever the tile:
// the K slices are only fetched ahead, into registers, while the current one
// is multiplied out of shared memory (two buffers, one barrier a slice).
// Bound: the serial walk over K with one or two warps a scheduler (issue
// 29-40 %): 1340 us for ten training steps of batch 512 through
// 512-256-256-512, 5030 before.  64 threads with 4 x 4 outputs measured 1660,
// 256 threads with 2 x 2 outputs 1410, and three slices in flight 1370.
__global__ void __launch_bounds__(GEMM_THREADS) mlp_gemm_kernel(const __grid_constant__ GemmJobs jobs) {
  __shared__ __align__(16) float As[2][TK * TM];
  __shared__ __align__(16) float Bs[2][TK * TN];
  const bool second = (int)blockIdx.x >= jobs.tiles0;
  const GemmJob& q = jobs.j[second ? 1 : 0];
  const int tile = (int)blockIdx.x - (second ? jobs.tiles0 : 0);
  const int tiles_n = (q.N + TN - 1) / TN;
  const int M = q.M, N = q.N, K = q.K;
  const int m0 = tile / tiles_n * TM, n0 = tile % tiles_n * TN;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const bool ak = q.sak == 1, bk = q.sbk == 1, av = q.a_vec, bv = q.b_vec;
  uint4 va[GROUPS], vb[GROUPS];
  auto fetch = [&](int k0) {
    fetch_slice(va, q.A, av, m0, M, q.sam, k0, K, q.sak);
    if (q.b_bf16) fetch_slice(vb, static_cast<const __nv_bfloat16*>(q.B), bv, n0, N, q.sbn, k0, K, q.sbk);
    else fetch_slice(vb, static_cast<const float*>(q.B), bv, n0, N, q.sbn, k0, K, q.sbk);
  };
  float acc[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0.0f;
  float csum = 0.0f;   // sum_k A(m0 + tid, k), threads below TM of the first column of tiles
  const bool want_sum = q.colsum != nullptr && n0 == 0 && threadIdx.x < TM;
  fetch(0);
  for (int k0 = 0, buf = 0; k0 < K; k0 += TK, buf ^= 1) {
    put_slice<false>(As[buf], va, ak);
    if (q.b_bf16) put_slice<true>(Bs[buf], vb, bk);
    else put_slice<false>(Bs[buf], vb, bk);
    __syncthreads();
    if (k0 + TK < K) fetch(k0 + TK);
    const float* as = As[buf];
    const float* bs = Bs[buf];
    // fragments of four k at a time, the next four read while these multiply
    float4 fa[2][4];
    float2 fb[2][4];
    auto frag = [&](int g, int k) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        fa[g][j] = *reinterpret_cast<const float4*>(as + slot(k + j, 4 * ty));
        fb[g][j] = *reinterpret_cast<const float2*>(bs + slot(k + j, 2 * tx));
      }
    };
    frag(0, 0);
#pragma unroll
    for (int k4 = 0; k4 < TK / 4; ++k4) {
      const int g = k4 & 1;
      if (k4 + 1 < TK / 4) frag(g ^ 1, 4 * k4 + 4);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float a[4] = {fa[g][j].x, fa[g][j].y, fa[g][j].z, fa[g][j].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[i][0] = fmaf(a[i], fb[g][j].x, acc[i][0]);
          acc[i][1] = fmaf(a[i], fb[g][j].y, acc[i][1]);
        }
      }
    }
    if (want_sum) {
      const int nk = min(TK, K - k0);
#pragma unroll 8
      for (int kk = 0; kk < nk; ++kk) csum += as[slot(kk, threadIdx.x)];
    }
  }
  if (want_sum && m0 + (int)threadIdx.x < M) q.colsum[m0 + threadIdx.x] = csum;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + 4 * ty + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int n = n0 + 2 * tx + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (q.epi != EPI_GELU_GRAD && q.bias) v += q.bias[n];
      float* out = q.C + (size_t)m * q.ldc + n;
      if (q.epi == EPI_STORE) {
        *out = v;
      } else if (q.epi == EPI_GELU) {
        *out = v;
        q.C2[(size_t)m * q.ldc + n] = gelu(v);
      } else {
        *out = v * gelu_grad(q.P[(size_t)m * q.ldp + n]);
      }
    }
  }
}

// dY = 2 (Y - T) / (B d), and the per-row squared error (FP64).
__global__ void mse_kernel(int B, int D, const float* __restrict__ Y, int ldy, const float* __restrict__ T, int ldt,
                           float* __restrict__ dY, double* __restrict__ row_sq) {
  __shared__ double red[33];
  const int b = blockIdx.x;
  const float scale = 2.0f / ((float)B * (float)D);
  double s = 0.0;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    const float e = Y[(size_t)b * ldy + d] - T[(size_t)b * ldt + d];
    dY[(size_t)b * D + d] = scale * e;
    s += (double)e * (double)e;
  }
  s = block_sum_f64(s, red);
  if (threadIdx.x == 0) row_sq[b] = s;
}

__global__ void adam_kernel(size_t n, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2,
                            __nv_bfloat16* __restrict__ wb) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    w[i] = wi;
    wb[i] = __float2bfloat16_rn(wi);
  }
}

__global__ void to_bf16_kernel(size_t n, const float* __restrict__ w, __nv_bfloat16* __restrict__ wb) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    wb[i] = __float2bfloat16_rn(w[i]);
}

// z = (theta - mu) * inv_s, per coordinate.
__global__ void sur_pre_kernel(int C, int D, const float* __restrict__ theta, const float* __restrict__ mu,
                               const float* __restrict__ inv_s, float* __restrict__ z) {
  const size_t n = (size_t)C * D;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int d = (int)(i % D);
    z[i] = (theta[i] - mu[d]) * inv_s[d];
  }
}

// g = a + h * (theta - mu) + o * out: the diagonal linear part plus the
// network's correction in output units o.
__global__ void sur_post_kernel(int C, int D, const float* __restrict__ theta, const float* __restrict__ out,
                                const float* __restrict__ mu, const float* __restrict__ a,
                                const float* __restrict__ h, const float* __restrict__ o, float* __restrict__ g) {
  const size_t n = (size_t)C * D;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int d = (int)(i % D);
    g[i] = a[d] + h[d] * (theta[i] - mu[d]) + o[d] * out[i];
  }
}

// ---- the whole network in one launch -----------------------------------------

// One dense layer for G rows held in shared memory: out[g][j] = act(b[j] +
// sum_k W[j][k] in[g][k]).  One output feature j per thread: the thread
// walks its bf16 weight row in 16-byte pieces (consecutive pieces share a
// cache line) and reads the G input rows as shared-memory broadcasts, so no
// cross-lane reduction is needed and the sum order is fixed.
template <int G>
__device__ __forceinline__ void dense_layer(const float* __restrict__ in, int din, const __nv_bfloat16* __restrict__ W,
                                            const float* __restrict__ b, int dout, float* __restrict__ out,
                                            bool gelu_act) {
  for (int j = threadIdx.x; j < dout; j += blockDim.x) {
    float acc[G];
#pragma unroll
    for (int g = 0; g < G; ++g) acc[g] = 0.0f;
    const uint4* row = reinterpret_cast<const uint4*>(W + (size_t)j * din);
    const int n8 = din >> 3;
#pragma unroll 4
    for (int k8 = 0; k8 < n8; ++k8) {
      const uint4 raw = __ldg(row + k8);
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
      float wv[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h2[i]);
        wv[2 * i] = f.x;
        wv[2 * i + 1] = f.y;
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 x0 = *reinterpret_cast<const float4*>(in + g * din + 8 * k8);
        const float4 x1 = *reinterpret_cast<const float4*>(in + g * din + 8 * k8 + 4);
        acc[g] = fmaf(wv[0], x0.x, acc[g]);
        acc[g] = fmaf(wv[1], x0.y, acc[g]);
        acc[g] = fmaf(wv[2], x0.z, acc[g]);
        acc[g] = fmaf(wv[3], x0.w, acc[g]);
        acc[g] = fmaf(wv[4], x1.x, acc[g]);
        acc[g] = fmaf(wv[5], x1.y, acc[g]);
        acc[g] = fmaf(wv[6], x1.z, acc[g]);
        acc[g] = fmaf(wv[7], x1.w, acc[g]);
      }
    }
    const float bj = b[j];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const float v = acc[g] + bj;
      out[g * dout + j] = gelu_act ? gelu(v) : v;
    }
  }
}

// The whole network for G rows per block (large batches).  SUR: input theta with the
// surrogate's input map z = (theta - mu) * inv_s, output the gradient
// estimate a + h (theta - mu) + o * y; otherwise input x, output y.
template <int G, bool SUR>
__global__ void __launch_bounds__(256) mlp_rows_kernel(int B, int din, int h1, int h2, int dout,
                                                        const float* __restrict__ x, int ldx,
                                                        const __nv_bfloat16* __restrict__ wb,
                                                        const float* __restrict__ w, float* __restrict__ y, int ldy,
                                                        const float* __restrict__ mu,
                                                        const float* __restrict__ inv_s, const float* __restrict__ sa,
                                                        const float* __restrict__ sh, const float* __restrict__ so) {
  extern __shared__ float sm[];
  float* z = sm;                       // [G][din]
  float* a1 = z + G * din;             // [G][h1]
  float* a2 = a1 + G * h1;             // [G][h2]
  float* o3 = a2 + G * h2;             // [G][dout]
  const int r0 = blockIdx.x * G;
  const size_t ow1 = 0, ob1 = (size_t)h1 * din, ow2 = ob1 + h1, ob2 = ow2 + (size_t)h2 * h1, ow3 = ob2 + h2,
               ob3 = ow3 + (size_t)dout * h2;
  for (int i = threadIdx.x; i < G * din; i += blockDim.x) {
    const int g = i / din, k = i % din, r = r0 + g;
    float v = 0.0f;
    if (r < B) {
      v = x[(size_t)r * ldx + k];
      if (SUR) v = (v - mu[k]) * inv_s[k];
    }
    z[i] = v;
  }
  __syncthreads();
  dense_layer<G>(z, din, wb + ow1, w + ob1, h1, a1, true);
  __syncthreads();
  dense_layer<G>(a1, h1, wb + ow2, w + ob2, h2, a2, true);
  __syncthreads();
  dense_layer<G>(a2, h2, wb + ow3, w + ob3, dout, o3, false);
  __syncthreads();
  for (int i = threadIdx.x; i < G * dout; i += blockDim.x) {
    const int g = i / dout, j = i % dout, r = r0 + g;
    if (r >= B) continue;
    float v = o3[i];
    if (SUR) {
      const float th = x[(size_t)r * ldx + j];
      v = sa[j] + sh[j] * (th - mu[j]) + so[j] * v;
    }
    y[(size_t)r * ldy + j] = v;
  }
}

// A small batch: a cluster of eight CTAs takes G rows through the network, each CTA an eighth of
// every layer's features.  A feature belongs to P neighbouring lanes that walk its
// weight row in turn, 16 bytes each, so that a warp reads whole sectors; the G rows'
// inputs come from shared memory, and a hidden feature's activations go to all
// eight CTAs' copies.  One CTA per four rows reads every weight row by itself, each lane
// another row: a surrogate of 512-256-256-512 with its dense linear part as a product
// of its own takes 47 us at 16 rows, 52 at 64 and 53 at 256; this kernel 13, 17 and
// 28 (graph replays).  It is bound by its shared-memory reads and weight loads
// sharing one pipe, and by the latency of three layers with a cluster barrier each;
// two features a thread halve the former and measured the same (35 us against
// 36 at 256 rows, and 17 against 15 at 16, before dense_slices).
constexpr int NET_CTAS = 8, NET_THREADS = 256;

// Lanes per feature when `dout` features of `n` pieces are spread over the cluster: as
// many as leave no thread without one, at most a warp and no more than the pieces.
__device__ __forceinline__ int net_lanes(int dout, int n) {
  const int per = (dout + NET_CTAS - 1) / NET_CTAS;
  int P = 32;
  while (P > 1 && (P * per > NET_THREADS || P > n)) P >>= 1;
  return P;
}

template <int G>
__device__ __forceinline__ void lane_sum(float (&v)[G], int P) {
  for (int o = P >> 1; o; o >>= 1)
#pragma unroll
    for (int g = 0; g < G; ++g) v[g] += __shfl_xor_sync(0xffffffffu, v[g], o);
}

// v[g] for a run-time g.
template <int G>
__device__ __forceinline__ float pick(const float (&v)[G], int g) {
  float r = v[0];
#pragma unroll
  for (int i = 1; i < G; ++i) r = i == g ? v[i] : r;
  return r;
}

// This CTA's features of one dense layer, out = b + W in: sink(j, g, value, linear)
// is called once per feature j and row g.  M (k-major, [dout][dout]) adds the
// linear = sum_k M[k][j] dt[g][k] of the surrogate; null without one.
template <int G, class Sink>
__device__ __forceinline__ void net_layer(const float* in, int din, const __nv_bfloat16* __restrict__ W,
                                          const float* __restrict__ b, int dout, int rank, const float* dt,
                                          const float* __restrict__ M, const Sink& sink) {
  const int n8 = din >> 3, P = net_lanes(dout, n8);
  const int slot = threadIdx.x / P, p = threadIdx.x & (P - 1), slots = NET_THREADS / P;
  const int per = (dout + NET_CTAS - 1) / NET_CTAS, j_end = min(dout, (rank + 1) * per);
  // lanes 4..7 of eight start with the second half of their piece: the eight
  // 16-byte reads of a row's inputs then fall into different banks
  const bool swap = (p >> 2) & 1;
  for (int base = rank * per; base < j_end; base += slots) {
    const int j = min(base + slot, dout - 1);
    float acc[G], lin[G];
#pragma unroll
    for (int g = 0; g < G; ++g) acc[g] = lin[g] = 0.0f;
    const uint4* row = reinterpret_cast<const uint4*>(W + (size_t)j * din);
#pragma unroll 4
    for (int k8 = p; k8 < n8; k8 += P) {
      const uint4 raw = __ldg(row + k8);
      const uint32_t r0 = swap ? raw.z : raw.x, r1 = swap ? raw.w : raw.y, r2 = swap ? raw.x : raw.z,
                     r3 = swap ? raw.y : raw.w;
      const float* x0 = in + 8 * k8 + (swap ? 4 : 0);
      const float* x1 = in + 8 * k8 + (swap ? 0 : 4);
      const float w0 = __uint_as_float(r0 << 16), w1 = __uint_as_float(r0 & 0xffff0000u);
      const float w2 = __uint_as_float(r1 << 16), w3 = __uint_as_float(r1 & 0xffff0000u);
      const float w4 = __uint_as_float(r2 << 16), w5 = __uint_as_float(r2 & 0xffff0000u);
      const float w6 = __uint_as_float(r3 << 16), w7 = __uint_as_float(r3 & 0xffff0000u);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 a = *reinterpret_cast<const float4*>(x0 + g * din);
        const float4 c = *reinterpret_cast<const float4*>(x1 + g * din);
        acc[g] = fmaf(w3, a.w, fmaf(w2, a.z, fmaf(w1, a.y, fmaf(w0, a.x, acc[g]))));
        acc[g] = fmaf(w7, c.w, fmaf(w6, c.z, fmaf(w5, c.y, fmaf(w4, c.x, acc[g]))));
      }
    }
    lane_sum(acc, P);
    if (M) {
#pragma unroll 8
      for (int k4 = p; k4 < (dout >> 2); k4 += P) {
        const float* m = M + (size_t)(4 * k4) * dout + j;
        const float m0 = __ldg(m), m1 = __ldg(m + dout), m2 = __ldg(m + 2 * (size_t)dout), m3 = __ldg(m + 3 * (size_t)dout);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float4 a = *reinterpret_cast<const float4*>(dt + g * dout + 4 * k4);
          lin[g] = fmaf(m3, a.w, fmaf(m2, a.z, fmaf(m1, a.y, fmaf(m0, a.x, lin[g]))));
        }
      }
      lane_sum(lin, P);
    }
    if (base + slot < j_end) {
      const float bj = b[j];
      for (int g = p; g < G; g += P) sink(j, g, pick(acc, g) + bj, M ? pick(lin, g) : 0.0f);
    }
  }
}

// The dense linear part of this CTA's features [j0, j0 + per), per a multiple of 4: a
// thread takes four neighbouring features and every nsl-th group of four rows of M,
// so that a warp reads M in whole lines and one 16-byte read of a row's dt serves
// sixteen products (four in net_layer, whose warps read M in 32-byte pieces): 36 -> 28
// us at D = 512 and 256 rows, 22.6 -> 17.0 at 64; 21.2 -> 19.9 at D = 256; 16.7 ->
// 17.4 at D = 128, where 32 and more slices are left to add, hence D >= 256.
// red[slice][g][feature] receives the slices' sums.
template <int G>
__device__ __forceinline__ void dense_slices(const float* dt, const float* __restrict__ M, int D, int j0, int per,
                                             float* red) {
  const int quads = per >> 2, nsl = NET_THREADS / quads;
  const int q = threadIdx.x % quads, slice = threadIdx.x / quads;
  if (slice >= nsl) return;
  float4 acc[G];
#pragma unroll
  for (int g = 0; g < G; ++g) acc[g] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 2
  for (int k4 = slice; k4 < (D >> 2); k4 += nsl) {
    const float4* m = reinterpret_cast<const float4*>(M + (size_t)(4 * k4) * D + j0) + q;
    const float4 m0 = __ldg(m), m1 = __ldg(m + (D >> 2)), m2 = __ldg(m + 2 * (D >> 2)), m3 = __ldg(m + 3 * (D >> 2));
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const float4 a = *reinterpret_cast<const float4*>(dt + g * D + 4 * k4);
      acc[g].x = fmaf(m3.x, a.w, fmaf(m2.x, a.z, fmaf(m1.x, a.y, fmaf(m0.x, a.x, acc[g].x))));
      acc[g].y = fmaf(m3.y, a.w, fmaf(m2.y, a.z, fmaf(m1.y, a.y, fmaf(m0.y, a.x, acc[g].y))));
      acc[g].z = fmaf(m3.z, a.w, fmaf(m2.z, a.z, fmaf(m1.z, a.y, fmaf(m0.z, a.x, acc[g].z))));
      acc[g].w = fmaf(m3.w, a.w, fmaf(m2.w, a.z, fmaf(m1.w, a.y, fmaf(m0.w, a.x, acc[g].w))));
    }
  }
#pragma unroll
  for (int g = 0; g < G; ++g) *reinterpret_cast<float4*>(red + ((size_t)slice * G + g) * per + 4 * q) = acc[g];
}

// SUR: input theta with the surrogate's input map z = (theta - mu) * inv_s, output the
// gradient estimate a + h (theta - mu) + o * y, plus (theta - mu) M when M is given;
// otherwise input x, output y.
template <int G, bool SUR>
__global__ void __cluster_dims__(NET_CTAS, 1, 1) __launch_bounds__(NET_THREADS, 2)
    mlp_cluster_kernel(int B, int din, int h1, int h2, int dout, const float* __restrict__ x, int ldx,
                     const __nv_bfloat16* __restrict__ wb, const float* __restrict__ w, float* __restrict__ y, int ldy,
                     const float* __restrict__ mu, const float* __restrict__ inv_s, const float* __restrict__ sa,
                     const float* __restrict__ sh, const float* __restrict__ so, const float* __restrict__ M) {
  const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  extern __shared__ float4 sm4[];
  float* z = reinterpret_cast<float*>(sm4);   // [G][din]
  float* a1 = z + G * din;                    // [G][h1]
  float* a2 = a1 + G * h1;                    // [G][h2]
  float* dt = a2 + G * h2;                    // [G][din] theta - mu (SUR)
  const int rank = (int)cl.block_rank(), r0 = (int)(blockIdx.x / NET_CTAS) * G;
  const size_t ob1 = (size_t)h1 * din, ow2 = ob1 + h1, ob2 = ow2 + (size_t)h2 * h1, ow3 = ob2 + h2,
               ob3 = ow3 + (size_t)dout * h2;
#pragma unroll
  for (int g = 0; g < G; ++g)
    for (int k = threadIdx.x; k < din; k += NET_THREADS) {
      float v = r0 + g < B ? x[(size_t)(r0 + g) * ldx + k] : 0.0f;
      if (SUR) {
        v = r0 + g < B ? v - mu[k] : 0.0f;
        dt[g * din + k] = v;
        v *= inv_s[k];
      }
      z[g * din + k] = v;
    }
  cl.sync();   // the peers run: their shared memory may be written
  auto hidden = [&](float* out, int h) {
    return [=](int j, int g, float v, float) {
      const float e = gelu(v);
#pragma unroll
      for (int t = 0; t < NET_CTAS; ++t)
        cooperative_groups::this_cluster().map_shared_rank(out, t)[g * h + j] = e;
    };
  };
  net_layer<G>(z, din, wb, w + ob1, h1, rank, nullptr, nullptr, hidden(a1, h1));
  cl.sync();
  net_layer<G>(a1, h1, wb + ow2, w + ob2, h2, rank, nullptr, nullptr, hidden(a2, h2));
  const int per = dout / NET_CTAS;
  const bool wide = SUR && M && dout % (4 * NET_CTAS) == 0 && dout >= 256 && (reinterpret_cast<uintptr_t>(M) & 15) == 0;
  float* red = dt + G * din;
  if (wide) dense_slices<G>(dt, M, dout, rank * per, per, red);
  cl.sync();
  net_layer<G>(a2, h2, wb + ow3, w + ob3, dout, rank, dt, SUR && !wide ? M : nullptr, [=](int j, int g, float v, float lin) {
    if (r0 + g >= B) return;
    if (wide)
      for (int t = 0; t < NET_THREADS / (per >> 2); ++t) lin += red[((size_t)t * G + g) * per + j - rank * per];
    if (SUR) v = sa[j] + sh[j] * dt[g * din + j] + so[j] * v + lin;
    y[(size_t)(r0 + g) * ldy + j] = v;
  });
}

constexpr int ROWS_G = 4;

inline size_t fused_smem(const ab_mlp_desc* d) {
  return sizeof(float) * ROWS_G * ((size_t)d->d_in + 2 * d->h1 + 2 * d->h2 + d->d_out);
}

int check_fused(const ab_mlp_desc* d) {
  AB_REQUIRE(fused_smem(d) <= 200 * 1024, AB_ERR_ARG, "mlp: layers too wide for the fused kernel");
  return AB_OK;
}

// Rows per cluster for a batch of B, 0 for the kernel without clusters.  A cluster
// kernel's batch is one that is resident at once, up to 32 clusters.  At D = 512, 512
// rows as 64 clusters of eight take 45 us against 41 of the other kernel without the
// linear part, 56 against 60 with it (the other kernel's being a product of its own);
// 256 rows as 64 clusters of four 36 against 29 as 32 of eight.
int net_rows(const ab_mlp_desc* d, int B) {
  const size_t row = sizeof(float) * (2 * (size_t)d->d_in + d->h1 + d->h2);
  for (int G : {4, 8})
    if (B <= 32 * G && G * row <= 100 * 1024) return G;
  return 0;
}

template <int G, bool SUR>
int launch_net(const ab_mlp_desc* d, int B, const float* x, int ldx, float* y, int ldy, const float* mu,
               const float* inv_s, const float* a, const float* h, const float* o, const float* M, cudaStream_t st) {
  const size_t smem = sizeof(float) * G * ((SUR ? 2 : 1) * (size_t)d->d_in + d->h1 + d->h2 +
                                           (M ? 4 * NET_THREADS : 0));
  AB_CUDA(allow_smem((const void*)mlp_cluster_kernel<G, SUR>, smem));
  mlp_cluster_kernel<G, SUR><<<NET_CTAS * ceil_div(B, G), NET_THREADS, smem, st>>>(
      B, d->d_in, d->h1, d->h2, d->d_out, x, ldx, static_cast<const __nv_bfloat16*>(d->wb), d->w, y, ldy, mu, inv_s,
      a, h, o, M);
  AB_LAUNCH_CHECK("mlp_cluster_kernel");
  return AB_OK;
}

// M: only where net_rows is not 0.
template <bool SUR>
int launch_fused(const ab_mlp_desc* d, int B, const float* x, int ldx, float* y, int ldy, const float* mu,
                 const float* inv_s, const float* a, const float* h, const float* o, const float* M, cudaStream_t st) {
  int rc = check_fused(d);
  if (rc) return rc;
  const int G = net_rows(d, B);
  if (G == 4) return launch_net<4, SUR>(d, B, x, ldx, y, ldy, mu, inv_s, a, h, o, M, st);
  if (G == 8) return launch_net<8, SUR>(d, B, x, ldx, y, ldy, mu, inv_s, a, h, o, M, st);
  const size_t smem = fused_smem(d);
  AB_CUDA(allow_smem((const void*)mlp_rows_kernel<ROWS_G, SUR>, smem));
  mlp_rows_kernel<ROWS_G, SUR><<<ceil_div(B, ROWS_G), 256, smem, st>>>(
      B, d->d_in, d->h1, d->h2, d->d_out, x, ldx, static_cast<const __nv_bfloat16*>(d->wb), d->w, y, ldy, mu, inv_s,
      a, h, o);
  AB_LAUNCH_CHECK("mlp_rows_kernel");
  return AB_OK;
}

struct Offsets {
  size_t w1, b1, w2, b2, w3, b3, total;
};

Offsets offsets(const ab_mlp_desc* d) {
  Offsets o;
  size_t k = 0;
  o.w1 = k; k += (size_t)d->h1 * d->d_in;
  o.b1 = k; k += d->h1;
  o.w2 = k; k += (size_t)d->h2 * d->h1;
  o.b2 = k; k += d->h2;
  o.w3 = k; k += (size_t)d->d_out * d->h2;
  o.b3 = k; k += d->d_out;
  o.total = k;
  return o;
}

inline int gemm_tiles(const GemmJob& q) { return (int)(ceil_div(q.M, TM) * ceil_div(q.N, TN)); }

// Whether an operand's groups of four along its unit-stride dimension (n_unit
// elements, the other dimension `stride` elements apart) can be loaded whole.
inline int can_vec(const void* p, int unit_stride, int n_unit, int stride, int elem) {
  return unit_stride == 1 && n_unit % 4 == 0 && stride % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & (4 * elem - 1)) == 0;
}

int gemm(GemmJob a, const GemmJob* b, cudaStream_t st) {
  GemmJobs jobs{{a, b ? *b : a}, gemm_tiles(a)};
  for (GemmJob& q : jobs.j) {
    q.a_vec = q.sak == 1 ? can_vec(q.A, q.sak, q.K, q.sam, 4) : can_vec(q.A, q.sam, q.M, q.sak, 4);
    const int es = q.b_bf16 ? 2 : 4;
    q.b_vec = q.sbk == 1 ? can_vec(q.B, q.sbk, q.K, q.sbn, es) : can_vec(q.B, q.sbn, q.N, q.sbk, es);
  }
  mlp_gemm_kernel<<<jobs.tiles0 + (b ? gemm_tiles(*b) : 0), GEMM_THREADS, 0, st>>>(jobs);
  AB_LAUNCH_CHECK("mlp_gemm_kernel");
  return AB_OK;
}

int check(const ab_mlp_desc* d) {
  AB_REQUIRE(d, AB_ERR_ARG, "mlp: null descriptor");
  AB_REQUIRE(d->d_in > 0 && d->h1 > 0 && d->h2 > 0 && d->d_out > 0, AB_ERR_ARG, "mlp: bad layer sizes");
  AB_REQUIRE(d->d_in % 8 == 0 && d->h1 % 8 == 0 && d->h2 % 8 == 0 && d->d_out % 8 == 0, AB_ERR_ARG,
             "mlp: layer widths must be multiples of 8");
  AB_REQUIRE((reinterpret_cast<uintptr_t>(d->wb) & 15) == 0, AB_ERR_ARG, "mlp: bf16 weights must be 16-byte aligned");
  AB_REQUIRE(d->w && d->wb, AB_ERR_ARG, "mlp: null parameters");
  return AB_OK;
}

}  // namespace
}  // namespace ab

using namespace ab;

extern "C" size_t ab_mlp_param_count(int d_in, int h1, int h2, int d_out) {
  if (d_in <= 0 || h1 <= 0 || h2 <= 0 || d_out <= 0) return 0;
  return (size_t)h1 * d_in + h1 + (size_t)h2 * h1 + h2 + (size_t)d_out * h2 + d_out;
}

extern "C" size_t ab_mlp_act_floats(int B, int h1, int h2) {
  if (B <= 0 || h1 <= 0 || h2 <= 0) return 0;
  return (size_t)B * (2 * (size_t)h1 + 2 * (size_t)h2);
}

extern "C" int ab_mlp_forward(const ab_mlp_desc* d, int B, const float* x, int ldx, float* y, int ldy, float* act,
                              void* stream) {
  int rc = check(d);
  if (rc) return rc;
  AB_REQUIRE(B > 0 && x && y && ldx >= d->d_in && ldy >= d->d_out && ldx % 4 == 0, AB_ERR_ARG,
             "ab_mlp_forward: bad arguments");
  cudaStream_t st = as_stream(stream);
  if (!act) return launch_fused<false>(d, B, x, ldx, y, ldy, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, st);
  // the activations are wanted anyway: one tiled product per layer, which
  // spreads every layer over the GPU (three launches; for a
  // batch of 512 through 512-256-256-512 47 us cold and 49 in the fused kernel,
  // whose CTAs each read every weight)
  if ((rc = check_fused(d))) return rc;
  const Offsets o = offsets(d);
  const __nv_bfloat16* wb = static_cast<const __nv_bfloat16*>(d->wb);
  const int h1 = d->h1, h2 = d->h2, din = d->d_in, dout = d->d_out;
  float* P1 = act;
  float* A1 = P1 + (size_t)B * h1;
  float* P2 = A1 + (size_t)B * h1;
  float* A2 = P2 + (size_t)B * h2;
  if ((rc = gemm(GemmJob{B, h1, din, EPI_GELU, x, ldx, 1, wb + o.w1, 1, 1, din, d->w + o.b1, P1, h1, A1, nullptr, 0,
                         nullptr}, nullptr, st)))
    return rc;
  if ((rc = gemm(GemmJob{B, h2, h1, EPI_GELU, A1, h1, 1, wb + o.w2, 1, 1, h1, d->w + o.b2, P2, h2, A2, nullptr, 0,
                         nullptr}, nullptr, st)))
    return rc;
  return gemm(GemmJob{B, dout, h2, EPI_STORE, A2, h2, 1, wb + o.w3, 1, 1, h2, d->w + o.b3, y, ldy, nullptr, nullptr, 0,
                      nullptr}, nullptr, st);
}

extern "C" int ab_sur_predict_dense(const ab_mlp_desc* d, int C, const float* theta, int ldt, const float* mu,
                                    const float* inv_s, const float* a, const float* h, const float* o, const float* M,
                                    float* g, int ldg, void* stream) {
  int rc = check(d);
  if (rc) return rc;
  AB_REQUIRE(d->d_in == d->d_out, AB_ERR_ARG, "ab_sur_predict: the network must map D to D");
  AB_REQUIRE(C > 0 && theta && mu && inv_s && a && h && o && g && ldt >= d->d_in && ldg >= d->d_out, AB_ERR_ARG,
             "ab_sur_predict: bad arguments");
  AB_REQUIRE(!M || net_rows(d, C), AB_ERR_ARG, "ab_sur_predict_dense: batch too large for the dense part in one launch");
  return launch_fused<true>(d, C, theta, ldt, g, ldg, mu, inv_s, a, h, o, M, as_stream(stream));
}

extern "C" int ab_sur_dense_fits(const ab_mlp_desc* d, int C) { return d && C > 0 && net_rows(d, C) ? 1 : 0; }

extern "C" int ab_sur_predict(const ab_mlp_desc* d, int C, const float* theta, int ldt, const float* mu,
                              const float* inv_s, const float* a, const float* h, const float* o, float* g, int ldg,
                              void* stream) {
  return ab_sur_predict_dense(d, C, theta, ldt, mu, inv_s, a, h, o, nullptr, g, ldg, stream);
}

extern "C" int ab_mlp_mse(int B, int D, const float* y, int ldy, const float* target, int ldt, float* dy,
                          double* row_sq, void* stream) {
  AB_REQUIRE(B > 0 && D > 0 && y && target && dy && row_sq && ldy >= D && ldt >= D, AB_ERR_ARG,
             "ab_mlp_mse: bad arguments");
  mse_kernel<<<B, 256, 0, as_stream(stream)>>>(B, D, y, ldy, target, ldt, dy, row_sq);
  AB_LAUNCH_CHECK("mse_kernel");
  return AB_OK;
}

extern "C" size_t ab_mlp_backward_scratch_floats(int B, int h1, int h2) {
  if (B <= 0 || h1 <= 0 || h2 <= 0) return 0;
  return (size_t)B * ((size_t)h1 + (size_t)h2);
}

extern "C" int ab_mlp_backward(const ab_mlp_desc* d, int B, const float* x, int ldx, const float* dy,
                               const float* act, float* grad, float* scratch, void* stream) {
  int rc = check(d);
  if (rc) return rc;
  AB_REQUIRE(B > 0 && x && dy && act && grad && scratch && ldx >= d->d_in, AB_ERR_ARG,
             "ab_mlp_backward: bad arguments");
  const Offsets o = offsets(d);
  const __nv_bfloat16* wb = static_cast<const __nv_bfloat16*>(d->wb);
  cudaStream_t st = as_stream(stream);
  const float* P1 = act;
  const float* A1 = P1 + (size_t)B * d->h1;
  const float* P2 = A1 + (size_t)B * d->h1;
  const float* A2 = P2 + (size_t)B * d->h2;
  float* dP2 = scratch;                        // [B][h2]
  float* dP1 = scratch + (size_t)B * d->h2;    // [B][h1]
  const int h1 = d->h1, h2 = d->h2, din = d->d_in, dout = d->d_out;
  // dW3[o][j] = sum_b dY[b][o] A2[b][j], db3 = colsum dY; beside it
  // dP2 = (dY W3) . gelu'(P2)
  const GemmJob w3{dout, h2, B, EPI_STORE, dy, 1, dout, A2, 0, h2, 1, nullptr, grad + o.w3, h2, nullptr, nullptr, 0,
                   grad + o.b3};
  const GemmJob p2{B, h2, dout, EPI_GELU_GRAD, dy, dout, 1, wb + o.w3, 1, h2, 1, nullptr, dP2, h2, nullptr, P2, h2,
                   nullptr};
  if ((rc = gemm(w3, &p2, st))) return rc;
  // dW2, db2; beside them dP1 = (dP2 W2) . gelu'(P1)
  const GemmJob w2{h2, h1, B, EPI_STORE, dP2, 1, h2, A1, 0, h1, 1, nullptr, grad + o.w2, h1, nullptr, nullptr, 0,
                   grad + o.b2};
  const GemmJob p1{B, h1, h2, EPI_GELU_GRAD, dP2, h2, 1, wb + o.w2, 1, h1, 1, nullptr, dP1, h1, nullptr, P1, h1,
                   nullptr};
  if ((rc = gemm(w2, &p1, st))) return rc;
  // dW1, db1
  const GemmJob w1{h1, din, B, EPI_STORE, dP1, 1, h1, x, 0, ldx, 1, nullptr, grad + o.w1, din, nullptr, nullptr, 0,
                   grad + o.b1};
  return gemm(w1, nullptr, st);
}

extern "C" int ab_mlp_adam(const ab_mlp_desc* d, const float* grad, float* m, float* v, int step, float lr, float b1,
                           float b2, float eps, void* stream) {
  int rc = check(d);
  if (rc) return rc;
  AB_REQUIRE(grad && m && v && step >= 1 && lr > 0.0f, AB_ERR_ARG, "ab_mlp_adam: bad arguments");
  const size_t n = ab_mlp_param_count(d->d_in, d->h1, d->h2, d->d_out);
  const float c1 = (float)(1.0 / (1.0 - pow((double)b1, step)));
  const float c2 = (float)(1.0 / (1.0 - pow((double)b2, step)));
  adam_kernel<<<ceil_div(n, 256 * 4), 256, 0, as_stream(stream)>>>(n, d->w, grad, m, v, lr, b1, b2, eps, c1, c2,
                                                                    static_cast<__nv_bfloat16*>(d->wb));
  AB_LAUNCH_CHECK("adam_kernel");
  return AB_OK;
}

extern "C" int ab_mlp_sync_bf16(const ab_mlp_desc* d, void* stream) {
  int rc = check(d);
  if (rc) return rc;
  const size_t n = ab_mlp_param_count(d->d_in, d->h1, d->h2, d->d_out);
  to_bf16_kernel<<<ceil_div(n, 256 * 4), 256, 0, as_stream(stream)>>>(n, d->w, static_cast<__nv_bfloat16*>(d->wb));
  AB_LAUNCH_CHECK("to_bf16_kernel");
  return AB_OK;
}

extern "C" int ab_sur_pre(int C, int D, const float* theta, const float* mu, const float* inv_s, float* z,
                          void* stream) {
  AB_REQUIRE(C > 0 && D > 0 && theta && mu && inv_s && z, AB_ERR_ARG, "ab_sur_pre: bad arguments");
  sur_pre_kernel<<<ceil_div((size_t)C * D, 1024), 256, 0, as_stream(stream)>>>(C, D, theta, mu, inv_s, z);
  AB_LAUNCH_CHECK("sur_pre_kernel");
  return AB_OK;
}

extern "C" int ab_sur_post(int C, int D, const float* theta, const float* out, const float* mu, const float* a,
                           const float* h, const float* o, float* g, void* stream) {
  AB_REQUIRE(C > 0 && D > 0 && theta && out && mu && a && h && o && g, AB_ERR_ARG, "ab_sur_post: bad arguments");
  sur_post_kernel<<<ceil_div((size_t)C * D, 1024), 256, 0, as_stream(stream)>>>(C, D, theta, out, mu, a, h, o, g);
  AB_LAUNCH_CHECK("sur_post_kernel");
  return AB_OK;
}
