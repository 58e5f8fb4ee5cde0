// Gaussian mixtures: the DiscGibbs assignment draw, the conjugate statistics
// and draws of ConjGibbs [pis] / [mu] / [cov], and the ESlice / MWG moves of
// the component means, for the models compiler/augur/test/mvgmm.rv (shared
// covariance, fixed weights) and hmvgmm.rv (weights ~ Dirichlet, covariances
// ~ InvWishart).
//
// Layout in HBM: Y f32 [N][d] (data), z int32 [N], pis f64 [K],
// mu f64 [K][d], cov f64 [Kc][d][d] (Kc = 1 when shared), all row-major;
// Linv f64 [Kc][d][d] and hdet f64 [Kc] are per-sweep derived tables.
//
// Arithmetic is binary64 without contraction (this file is compiled with
// -fmad=false and uses _rn intrinsics), but for the scatter matrices and the
// mean moves' gains, which are summed in another order than the reference's and
// use multiply-adds (held to 1e-12 and 1e-9 of the oracle), and the draw's
// binary32 screen.  The reference's d x d routines
// (cbits/augur_matop.c:312-420) are in-place sequential loops; the routines
// below compute every element with the same operand order, reading the values
// the in-place reference would read at that point, so their results are
// bit-identical; only the order in which independent elements are produced
// changes.  The per-point log-density uses the Cholesky inverse
// of the component covariance computed once per sweep — the same binary64
// values the reference recomputes for every (point, component).
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "dist.cuh"

namespace ab {

constexpr int GMM_MAX_D = 64;
constexpr int GMM_MAX_K = 64;
constexpr int GMM_THREADS = 256;

// ---- thread-group matrix routines -----------------------------------------
// Factorisations by a group of `nt` threads (a whole CTA, or one of
// two equal halves that factor different matrices in step), t the thread's
// index in it.  Every thread of the CTA calls them together: they use
// __syncthreads.  The lower-triangle entries (i, j) are dealt to the threads,
// NE at most each, and every entry's sum over k is carried in a register and
// extended as soon as the column (or row) k it needs is final: the same
// additions in the same order as the reference's loop, so the same values,
// but the chain is one column after another - a reciprocal root, two barriers
// and one product - instead of all of a column's products in turn.
// Their matrices have rows of pitch(d) doubles: a column is read by many
// lanes at once, and an odd pitch spreads it over the banks (with rows of d =
// 32 doubles every such read was a 32-way conflict).
__host__ __device__ __forceinline__ int pitch(int d) { return d | 1; }
#define GP(A, i, j) (A)[(i) * (d | 1) + (j)]

template <int NE>
struct Tri {
  int ij[NE];    // i << 8 | j, or -1
  __device__ __forceinline__ void deal(int t, int nt, int d) {
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const int e = t + q * nt;
      if (e >= d * (d + 1) / 2) { ij[q] = -1; continue; }
      int r = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
      while (r * (r + 1) / 2 > e) --r;
      while ((r + 1) * (r + 2) / 2 <= e) ++r;
      ij[q] = r << 8 | (e - r * (r + 1) / 2);
    }
  }
};

// Whether 2^-n <= |v| < 2^n, from the exponent field.
__device__ __forceinline__ bool within_2(double v, int n) {
  return ((unsigned)__double2hiint(v) >> 20 & 0x7ffu) - (unsigned)(1023 - n) < (unsigned)(2 * n);
}

// Whether e, the residual b - v q rounded once, shows q to be b / v correctly
// rounded: |e| < |v| times half the distance from q to its nearer neighbour.
// That bound is v with another exponent (everything in range, as |v q| is near
// |b|), and below it e is exact.  For a root, v = q and twice the bound
// (b - q^2 is a multiple of the distance's square).  Integer operations: the
// binary64 pipe is what the callers' chains wait for.
template <int HALF>
__device__ __forceinline__ bool rounds_to(double e, double v, double q) {
  const int hq = __double2hiint(q);
  const bool pow2 = ((hq & 0xfffff) | __double2loint(q)) == 0;   // the neighbour below is half as far
  const int hb = (__double2hiint(v) & 0x7fffffff) + (hq & 0x7ff00000) - ((1023 + 52 + HALF + (pow2 ? 1 : 0)) << 20);
  return (__double_as_longlong(e) & 0x7fffffffffffffffll) < __double_as_longlong(__hiloint2double(hb, __double2loint(v)));
}

// sqrt(x) and the reciprocal of that root.  CUDA's reciprocal root (within an
// ulp) gives the root by one residual step and seeds the reciprocal, which a
// second one rounds (after Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", 1990): far shorter a chain than a square
// root and a division in turn.  The steps alone do not round every value
// correctly (a root just below a power of two, for one), hence the test, whose
// result is needed only once the values have been used: it runs beside that use.
__device__ __forceinline__ void root_recip(double x, double& root, double& rec) {
  const double y = rsqrt(x);
  const double g = __dmul_rn(x, y);
  root = __fma_rn(__fma_rn(-g, g, x), __dmul_rn(0.5, y), g);
  rec = __fma_rn(__fma_rn(-root, y, 1.0), y, y);
}
__device__ __forceinline__ bool root_recip_rounded(double x, double root, double rec) {
  return __double2hiint(x) > 0 && within_2(x, 900) && rounds_to<0>(__fma_rn(-root, root, x), root, root) &&
         rounds_to<1>(__fma_rn(-root, rec, 1.0), root, rec);
}

// b / v given rec = 1 / v correctly rounded, from the quotient's residual
// (after the same paper); true if it is known to be correctly rounded.
__device__ __forceinline__ bool quotient(double b, double v, double rec, double& q) {
  q = __dmul_rn(b, rec);
  if (b == 0.0) return within_2(v, 400);
  q = __fma_rn(__fma_rn(-q, v, b), rec, q);
  return within_2(v, 400) && within_2(b, 400) && rounds_to<1>(__fma_rn(-q, v, b), v, q);
}

// augur_mat_cholesky (:312-328) of A, in place (lower triangle; the upper one
// is left as it is, as the reference leaves it) and, with INV,
// augur_mat_lower_trmi (:335-345) of the factor into O, lower triangle, in the
// same walk: once column k of the factor is final, so is row k of its inverse.
// Entry (i, j) first sums A[i][k] A[j][k] over k < j, becomes final at k = j,
// then subtracts L[i][k] O[k][j] over j <= k < i from the identity's entry and
// gives O[i][j] at k = i.  piv: [d] scratch.  A column whose root, reciprocal or
// quotients are not known to be correctly rounded is formed again with the
// square root and divisions.
template <int NE, bool INV>
__device__ __forceinline__ void g_factor(const Tri<NE>& T, double* A, double* O, double* piv, int d) {
  double acc[NE];
#pragma unroll
  for (int q = 0; q < NE; ++q) acc[q] = 0.0;
  __syncthreads();
  for (int k = 0; k < d; ++k) {
    // the pivot A[k][k] - sum, published by its owner
#pragma unroll
    for (int q = 0; q < NE; ++q)
      if (T.ij[q] == (k << 8 | k)) piv[k] = __dadd_rn(GP(A, k, k), -acc[q]);
    __syncthreads();
    double root, rec;
    root_recip(piv[k], root, rec);
    bool ok = true;
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const int i = T.ij[q] >> 8, j = T.ij[q] & 255;
      if (T.ij[q] < 0) continue;
      if (j == k) {
        acc[q] = __dadd_rn(GP(A, i, k), -acc[q]);
        GP(A, i, k) = i == k ? root : __dmul_rn(rec, acc[q]);
        if (INV && i == k) GP(O, k, k) = rec;
      } else if (INV && i == k) {
        double b;
        ok &= quotient(acc[q], root, rec, b);
        GP(O, k, j) = b;
      }
    }
    // one warp of each half of the CTA tests the values that all of them share
    if ((threadIdx.x & 96) == 0) ok &= root_recip_rounded(piv[k], root, rec);
    if (__syncthreads_or(!ok)) {
      root = __dsqrt_rn(piv[k]);
      rec = __ddiv_rn(1.0, root);
#pragma unroll
      for (int q = 0; q < NE; ++q) {
        const int i = T.ij[q] >> 8, j = T.ij[q] & 255;
        if (T.ij[q] < 0) continue;
        if (j == k) {
          GP(A, i, k) = i == k ? root : __dmul_rn(rec, acc[q]);
          if (INV && i == k) GP(O, k, k) = rec;
        } else if (INV && i == k) {
          GP(O, k, j) = __ddiv_rn(acc[q], root);
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const int i = T.ij[q] >> 8, j = T.ij[q] & 255;
      if (T.ij[q] < 0 || i <= k || (!INV && j <= k)) continue;
      const double p = __dmul_rn(GP(A, i, k), j > k ? GP(A, j, k) : GP(O, k, j));
      acc[q] = __dadd_rn(j == k ? 0.0 : acc[q], j > k ? p : -p);
    }
  }
  __syncthreads();
}

// augur_mat_lower_trmi (:335-345) of a given factor L into O, lower triangle.
template <int NE>
__device__ __forceinline__ void g_trmi(const Tri<NE>& T, const double* L, double* O, double* recs, int t, int nt,
                                       int d) {
  double b[NE];
#pragma unroll
  for (int q = 0; q < NE; ++q) b[q] = (T.ij[q] >> 8) == (T.ij[q] & 255) ? 1.0 : 0.0;
  __syncthreads();
  for (int i = t; i < d; i += nt) recs[i] = __ddiv_rn(1.0, GP(L, i, i));
  __syncthreads();
  for (int r = 0; r < d; ++r) {
#pragma unroll
    for (int q = 0; q < NE; ++q)
      if (T.ij[q] >= 0 && (T.ij[q] >> 8) == r) {
        double o;
        const bool ok = quotient(b[q], GP(L, r, r), recs[r], o);
        GP(O, r, T.ij[q] & 255) = o;
        if (!ok) GP(O, r, T.ij[q] & 255) = __ddiv_rn(b[q], GP(L, r, r));
      }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const int m = T.ij[q] >> 8, c = T.ij[q] & 255;
      if (T.ij[q] >= 0 && m > r && c <= r) b[q] = __dadd_rn(b[q], -__dmul_rn(GP(L, m, r), GP(O, r, c)));
    }
  }
  __syncthreads();
}

// The product of augur_mat_cholesky_invert (:363-375) from the inverse factor
// M (lower triangle): A[r][c] = sum_{k >= r} M[k][r] M[k][c] in k order (the
// reference's terms k < r are zero products), mirrored.
template <int NE>
__device__ __forceinline__ void g_inverse(const Tri<NE>& T, const double* M, double* A, int d) {
#pragma unroll
  for (int q = 0; q < NE; ++q) {
    if (T.ij[q] < 0) continue;
    const int r = T.ij[q] >> 8, c = T.ij[q] & 255;
    double acc = 0.0;
#pragma unroll 8
    for (int k = r; k < d; ++k) acc = __dadd_rn(acc, __dmul_rn(GP(M, k, r), GP(M, k, c)));
    GP(A, r, c) = acc;
    GP(A, c, r) = acc;
  }
  __syncthreads();
}

// augur_mat_mvm (:412-420) by threads t = 0 .. d-1 of the group.
__device__ __forceinline__ void g_mvm(double* dst, const double* A, const double* v, int t, int nt, int d) {
  for (int i = t; i < d; i += nt) {
    double s = 0.0;
#pragma unroll 8
    for (int j = 0; j < d; ++j) s = __dadd_rn(s, __dmul_rn(GP(A, i, j), v[j]));
    dst[i] = s;
  }
}

// ---- per-component tables for the assignment draw -------------------------
// Linv = lower_trmi(chol(cov_k)) and hdet = 0.5 * log((prod L_ii)^2), the
// quantities augur_mvnormal_ll (augur_dist.c:548-568) derives from cov.
template <int DT>
__global__ void __launch_bounds__(GMM_THREADS)
gmm_prep_kernel(int d, const double* __restrict__ cov, double* __restrict__ Linv, double* __restrict__ hdet) {
  constexpr int NE = (DT * (DT + 1) / 2 + GMM_THREADS - 1) / GMM_THREADS;
  extern __shared__ double sm[];
  __shared__ double piv[DT];
  const int k = blockIdx.x, tid = threadIdx.x;
  double* L = sm;
  double* O = sm + d * pitch(d);
  for (int e = tid; e < d * d; e += GMM_THREADS) GP(L, e / d, e % d) = cov[(size_t)k * d * d + e];
  Tri<NE> T;
  T.deal(tid, GMM_THREADS, d);
  g_factor<NE, true>(T, L, O, piv, d);
  for (int e = tid; e < d * d; e += GMM_THREADS)
    Linv[(size_t)k * d * d + e] = e / d >= e % d ? GP(O, e / d, e % d) : 0.0;
  if (tid == GMM_THREADS - 1) {
    double det = 1.0;
    for (int i = 0; i < d; ++i) det = __dmul_rn(det, GP(L, i, i));
    det = __dmul_rn(det, det);
    hdet[k] = __dmul_rn(0.5, log(det));
  }
}

// ---- assignment draw --------------------------------------------------------
// One thread per point.  For each component: w = y - mu_k; w' = Linv w
// (ascending j per row); expon = sum_i w'_i^2; ll = c - hdet - expon/2;
// pmf_k = (1 * pis_k) * exp(ll) (CgDisc.hs:132-139); then the unnormalised
// discrete draw of augur_dist.c:798-813 with the uniform of substream
// (n, iter, 1|comp<<8).
template <int DT, bool UNROLL>
__global__ void __launch_bounds__(GMM_THREADS, 3)   // 3 CTAs per SM: measured 6 % faster than 1 at d = 32
gmm_z_kernel(int N, int d, int K, int shared_cov, const float* __restrict__ Y, const double* __restrict__ pis,
             const double* __restrict__ mu, const double* __restrict__ Linv, const double* __restrict__ hdet,
             int* __restrict__ z, uint64_t seed, uint32_t iter, uint32_t comp) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const double c = __dmul_rn(__dmul_rn(-0.5, (double)d), log(2.0 * 3.14159265358979323846264338327950288));
  double y[DT], w[DT];
#pragma unroll
  for (int i = 0; i < DT; ++i) y[i] = i < d ? (double)Y[(size_t)n * d + i] : 0.0;
  static_assert(UNROLL || DT == GMM_MAX_D, "generic path is the widest");
  double pmf[GMM_MAX_K];
  for (int k = 0; k < K; ++k) {
    const int kc = shared_cov ? 0 : k;
    const double* Lk = Linv + (size_t)kc * d * d;
    const double* mk = mu + (size_t)k * d;
#pragma unroll
    for (int i = 0; i < DT; ++i) w[i] = i < d ? __dadd_rn(y[i], -__ldg(mk + i)) : 0.0;
    double expon = 0.0;
#pragma unroll
    for (int i = 0; i < DT; ++i) {
      if (i < d) {
        double s = 0.0;
        if (UNROLL) {
#pragma unroll
          for (int j = 0; j <= i; ++j) s = __dadd_rn(s, __dmul_rn(__ldg(Lk + (size_t)i * d + j), w[j]));
        } else {
          for (int j = 0; j <= i; ++j) s = __dadd_rn(s, __dmul_rn(__ldg(Lk + (size_t)i * d + j), w[j]));
        }
        expon = __dadd_rn(expon, __dmul_rn(s, s));
      }
    }
    const double ll = __dadd_rn(__dadd_rn(c, -__ldg(hdet + kc)), -__dmul_rn(0.5, expon));
    double prob = 1.0;
    prob = __dmul_rn(prob, __ldg(pis + k));
    prob = __dmul_rn(prob, exp(ll));
    pmf[k] = prob;
  }
  Stream s = make_stream(seed, (uint32_t)n, iter, TAG_Z | (comp << 8));
  const double u = s.uniform();
  double norm = 0.0;
  for (int k = 0; k < K; ++k) norm = __dadd_rn(norm, pmf[k]);
  double acc = __ddiv_rn(pmf[0], norm);
  int zk = K - 1;
  for (int i = 1; i < K; ++i) {
    if (u < acc) { zk = i - 1; break; }
    acc = __dadd_rn(acc, __ddiv_rn(pmf[i], norm));
  }
  z[n] = zk;
}

// ---- assignment draw screened in binary32 ----------------------------------
// The same draw as gmm_z_kernel, decided for most points in binary32:
//   gmm_zs_prep_kernel  per component (once per call): the lower triangle of
//                       Linv_k and mu_k rounded to binary32, and the constants
//                       of the error bound below; log(pis_k) + c - hdet_k;
//   gmm_zs_kernel       one or two points a thread: t_k = log p_k in binary32 with a
//                       rigorous bound eps_k on its error against the exact
//                       value, p_k / p_max = exp(t_k - t_max), the running
//                       sums, and the reference's draw when u lies outside the
//                       sums' uncertainty band; other points go to a queue;
//   gmm_zx_kernel       one CTA per queued point, a warp per component: the
//                       reference's binary64 loop (gmm_z_kernel's operations,
//                       rows of Linv w on the lanes, every sum in its order),
//                       so every draw equals gmm_z_kernel's bit for bit.
// Error bound (u = 2^-24; all quantities of component k; L~, w~ the binary32
// values; mu_j = mh_j + ml_j + r_j, two binary32 parts, |r_j| <= 2^-48 |mu_j|;
// w~_j = fl(fl(y_j - mh_j) - ml_j)):
//   |w~_j - w_j| <= 2u |w~_j| (1 + 4u) + 2^-47 |mu_j| (1 + 4u);
//   row i of Linv w (i + 1 products, fused multiply-adds in two interleaved
//   chains, then their sum; zero padding adds exact zeros): |s~_i - s_i| <=
//   delta_i = u (1 + 4u) (i + 4) A_i, A_i = sum_j |L~_ij| (|w~_j| + 2^-23 |mu_j|)
//     <= R_i W (R_i >= ||L~_i||, W >= ||w~|| + 2^-23 ||mu||);
//   expon = sum_i s_i^2: |e~ - e| <= (d + 1) u e~ + sum_i (2 |s~_i| delta_i + delta_i^2),
//     with sum_i |s~_i| a_i (a_i = (i + 4) R_i) accumulated beside the rows
//     and sum_i delta_i^2 <= u^2 (1 + 4u)^2 W^2 S_aa, S_aa = sum_i a_i^2;
//   t_k = fl(lpc_k - e~ / 2), lpc_k = fl32(log pis_k + c - hdet_k): |t_k - log p_k|
//     <= eps_k = E_k / 2 + u (|lpc_k| + |t_k|) + 2^-40 (|lpc_k| + e~ + 1) (the last
//     term covers the reference's own binary64 roundings);
//   p~_k = exp(t_k - t_max) (binary32 exp, <= 4u); the exact p_k / p_max lies
//     in [exp(dt - x), exp(dt + x)], x = eps_k + u |dt| + 4u, dt = t_k - t_max,
//     so |p~_k - p_k / p_max| <= A_k, formed with directed roundings; a
//     component far from the point has a wide band but a tiny p_k;
//   band = sum_k A_k + (K + 6) u norm~ + 2^-40 norm~ covers the running sums'
//     and u * norm's roundings, the comparisons' and the reference's running
//     quotient sums.
// A draw is decided (and equals the reference's) when u norm~ + band is below
// the first running sum that exceeds it minus band, and the previous sum plus
// band is below u norm~ - band.  Points whose largest log density is
// outside [-690, 690] (where the reference's binary64 exp could underflow or
// overflow), any non-finite value, or a call whose components have
// c - hdet_k > 700, take the exact path.
constexpr int GMM_ZS_MAXK = 32;
constexpr int GMM_ZS_THREADS = 128;
constexpr int gmm_zs_ctas(int DT, int H) { return H == 2 ? 3 : DT <= 8 ? 10 : 5; }   // per SM

// Per component, floats: L~ with row i padded to whole float4s (zeros) at
// gmm_zs_row(i), then a, mh and ml, each padded to whole float4s (zeros), then
// lpc, S_aa and 2^-23 ||mu|| (rounded up); the stride is whole float4s.
__host__ __device__ constexpr int gmm_zs_row(int i) { return 4 * (i / 4 + 1) * (2 * (i / 4) + i % 4); }
__host__ __device__ constexpr int gmm_zs_dq(int d) { return (d + 3) / 4 * 4; }
__host__ __device__ inline int gmm_zs_stride(int d) { return gmm_zs_row(d - 1) + gmm_zs_dq(d) + 3 * gmm_zs_dq(d) + 4; }

// tab: K float tables of gmm_zs_stride(d).
__global__ void __launch_bounds__(64) gmm_zs_prep_kernel(int d, int K, int shared_cov, const double* __restrict__ pis,
                                                         const double* __restrict__ mu,
                                                         const double* __restrict__ Linv,
                                                         const double* __restrict__ hdet, float* __restrict__ tab,
                                                         int* __restrict__ flag) {
  __shared__ double red[2][64];
  const int k = blockIdx.x, kc = shared_cov ? 0 : k;
  const double* Lk = Linv + (size_t)kc * d * d;
  const double* mk = mu + (size_t)k * d;
  float* t = tab + (size_t)k * gmm_zs_stride(d);
  const int dq = gmm_zs_dq(d);
  float* L32 = t;
  float* a = t + gmm_zs_row(d - 1) + dq;
  float* mh = a + dq;
  float* ml = mh + dq;
  float* sc = ml + dq;
  double saa = 0.0, mm = 0.0;
  for (int i = threadIdx.x; i < dq; i += blockDim.x) {
    if (i >= d) {
      a[i] = mh[i] = ml[i] = 0.0f;
      continue;
    }
    double r2 = 0.0;
    const int row = gmm_zs_row(i), len = (i / 4 + 1) * 4;
    for (int j = 0; j < len; ++j) {
      const float l = j <= i ? __double2float_rn(Lk[(size_t)i * d + j]) : 0.0f;
      L32[row + j] = l;
      r2 += (double)l * (double)l;
    }
    // rounded up, with a relative slack for the binary64 sums' own rounding
    a[i] = __fmul_ru((float)(i + 4), __double2float_ru(sqrt(r2) * (1.0 + 1e-12)));
    saa += (double)a[i] * a[i];
    const double m = mk[i];
    const float h = __double2float_rn(m);
    mh[i] = -h;                                             // stored negated: w = (y + mh) + ml
    ml[i] = -__double2float_rn(__dadd_rn(m, -(double)h));
    mm += m * m;
  }
  red[0][threadIdx.x] = saa;
  red[1][threadIdx.x] = mm;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < (int)blockDim.x; ++i) {
      saa += red[0][i];
      mm += red[1][i];
    }
    const double c = -0.5 * (double)d * log(2.0 * 3.14159265358979323846264338327950288);
    const double llc = c - hdet[kc];
    const double pk = pis[k];
    sc[0] = pk > 0.0 ? __double2float_rn(log(pk) + llc) : -INFINITY;
    sc[1] = __double2float_ru(saa * (1.0 + 1e-12));
    sc[2] = __double2float_ru(sqrt(mm) * (0x1p-23 * (1.0 + 0x1p-16)));
    sc[3] = 0.0f;
    if (!(pk >= 0.0) || !(llc <= 700.0) || !isfinite(llc)) atomicExch(flag, 1);
  }
}

// Two binary32 operations per instruction, each rounded as the scalar one.
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  return (unsigned long long)__float_as_uint(y) << 32 | __float_as_uint(x);
}
__device__ __forceinline__ float lo2(unsigned long long a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi2(unsigned long long a) { return __uint_as_float((unsigned)(a >> 32)); }

// H = 1: a point a thread, pairs of a row's columns in one packed multiply-add,
// five CTAs per SM: 370 -> 235 us for the whole draw at N = 200,000, K = 16, d =
// 32, where scalar operations on a binary64 y - mu took most of the time.  Up to
// d = 8 the exponentials and running sums are most of the work, and ten CTAs per
// SM faster than the registers of five (K = 30, d = 2, N = 400,000: 104 and 117 us).
// H = 2: two points a thread, so that every 16-byte read of the factor's rows
// (a shared-memory broadcast) feeds eight multiply-adds, at three CTAs per SM.
// Only in label order, where most of the work is left out: 155 us there with
// components apart, 171 with H = 1.  Without the order it is slower than H = 1 at
// every size (252 us there; 63 against 46 at N = 3,000, K = 30, d = 12).
// Warps walk the points 32 H at a time; each CTA reads the tables once.
template <int DT, int H>
__global__ void __launch_bounds__(GMM_ZS_THREADS, gmm_zs_ctas(DT, H))
gmm_zs_kernel(int N, int d, int K, int vec, const float* __restrict__ Y, const float* __restrict__ tab,
              const int* __restrict__ perm, const int* __restrict__ flag, int* __restrict__ queue, int* __restrict__ qn,
              int* __restrict__ z, uint64_t seed, uint32_t iter, uint32_t comp) {
  extern __shared__ __align__(16) float ts[];   // the K components' tables
  constexpr int DW = (DT + 3) / 4 * 4;          // whole float4s of row entries
  constexpr bool ORDERED = H == 2;              // the points in the order of their labels (perm)
  const int stride = gmm_zs_stride(d), dq = gmm_zs_dq(d);
  {
    const float4* src = reinterpret_cast<const float4*>(tab);
    float4* dst = reinterpret_cast<float4*>(ts);
    for (int e = threadIdx.x; e < K * stride / 4; e += GMM_ZS_THREADS) dst[e] = src[e];
  }
  __syncthreads();
  const float u32 = 5.9604644775390625e-8f;   // 2^-24
  const bool all_exact = *flag != 0;
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (GMM_ZS_THREADS / 32);
  for (int tile = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; tile < (N + 32 * H - 1) / (32 * H); tile += warps) {
    int n2[H];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int i = tile * 32 * H + lane + 32 * h;
      n2[h] = i < N ? (ORDERED ? perm[i] : i) : -1;
    }
    bool exact[H];
    float tk[H][GMM_ZS_MAXK], ek[H][GMM_ZS_MAXK], tmax[H];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      exact[h] = all_exact;
      tmax[h] = -INFINITY;
    }
    if (!all_exact) {
      unsigned long long y[H][DW / 2];
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const float* yr = Y + (size_t)max(n2[h], 0) * d;
        if (vec) {   // d a multiple of 4, rows 16-byte aligned
#pragma unroll
          for (int q = 0; q < DW / 4; ++q) {
            const float4 f = 4 * q < d ? reinterpret_cast<const float4*>(yr)[q] : make_float4(0.f, 0.f, 0.f, 0.f);
            y[h][2 * q] = pack2(f.x, f.y);
            y[h][2 * q + 1] = pack2(f.z, f.w);
          }
        } else {
#pragma unroll
          for (int q = 0; q < DW / 2; ++q)
            y[h][q] = pack2(2 * q < d ? yr[2 * q] : 0.0f, 2 * q + 1 < d ? yr[2 * q + 1] : 0.0f);
        }
      }
      // In label order the tile's points have few labels between them, mostly
      // their draws too: those components first, then - where a point does not
      // look like any of them - the component its first coordinates suggest,
      // so that the other components can be found far away early.
      float low[H];                            // a lower bound of log p_max so far
      bool likely[H];
#pragma unroll
      for (int h = 0; h < H; ++h) {
        low[h] = -INFINITY;
        likely[h] = n2[h] < 0;
      }
      unsigned todo = K == 32 ? 0xffffffffu : (1u << K) - 1u, pend = todo;
      bool suggest = ORDERED;
      if constexpr (ORDERED) {
        unsigned m = 0u;
#pragma unroll
        for (int h = 0; h < H; ++h) {
          const int l = n2[h] >= 0 ? z[n2[h]] : -1;
          m |= l >= 0 && l < K ? 1u << l : 0u;
        }
        pend = __reduce_or_sync(0xffffffffu, m);
      }
      for (int k0 = 0; ORDERED ? todo != 0u : k0 < K; ++k0) {
        int k = k0;
        if constexpr (ORDERED) {
          if (pend == 0u && suggest) {
            suggest = false;
            bool odd = false;
#pragma unroll
            for (int h = 0; h < H; ++h) odd = odd || !likely[h];
            if (__any_sync(0xffffffffu, odd)) {
              float best[H];
              int at[H];
#pragma unroll
              for (int h = 0; h < H; ++h) {
                best[h] = -INFINITY;
                at[h] = 0;
              }
              for (int c = 0; c < K; ++c) {
                const float* L32 = ts + c * stride;
                const float* a = L32 + gmm_zs_row(d - 1) + dq;
                const ulonglong2 mh = *reinterpret_cast<const ulonglong2*>(a + dq);
                const float lpc = a[3 * dq];
#pragma unroll
                for (int h = 0; h < H; ++h) {
                  const unsigned long long w0 = add2(y[h][0], mh.x), w1 = add2(y[h][1], mh.y);
                  float e = 0.0f;
#pragma unroll
                  for (int i = 0; i < 4; ++i) {
                    const ulonglong2 l = *reinterpret_cast<const ulonglong2*>(L32 + gmm_zs_row(i));
                    const unsigned long long sr = fma2(l.y, w1, fma2(l.x, w0, 0ull));
                    const float r = lo2(sr) + hi2(sr);
                    e += r * r;
                  }
                  if (lpc - 0.5f * e > best[h]) {
                    best[h] = lpc - 0.5f * e;
                    at[h] = c;
                  }
                }
              }
              unsigned want = 0u;
#pragma unroll
              for (int h = 0; h < H; ++h) want |= likely[h] ? 0u : 1u << at[h];
              pend = __reduce_or_sync(0xffffffffu, want) & todo;
            }
          }
          if (pend == 0u) pend = todo;
          k = __ffs(pend) - 1;
          pend &= pend - 1u;
          todo &= ~(1u << k);
        }
        const float* L32 = ts + k * stride;
        const float* a = L32 + gmm_zs_row(d - 1) + dq;
        const float4 sc = *reinterpret_cast<const float4*>(a + 3 * dq);
        const float lpc = sc.x;
        if (lpc == -INFINITY) {   // weight 0: the term is exactly 0 here and in the reference
#pragma unroll
          for (int h = 0; h < H; ++h) {
            tk[h][k] = -INFINITY;
            ek[h][k] = 0.0f;
          }
          continue;
        }
        unsigned long long w[H][DW / 2], W2[H];
        float e[H], t1[H];
#pragma unroll
        for (int h = 0; h < H; ++h) {
          W2[h] = 0ull;
          e[h] = t1[h] = 0.0f;
        }
        float4 a4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        bool far = false;
#pragma unroll
        for (int i = 0; i < DT; ++i) {
          if (i < d && !far) {
            if (i % 4 == 0) {
              // the next four coordinates of w, and of a
              const ulonglong2 mh = reinterpret_cast<const ulonglong2*>(a + dq)[i / 4];
              const ulonglong2 ml = reinterpret_cast<const ulonglong2*>(a + 2 * dq)[i / 4];
              a4 = reinterpret_cast<const float4*>(a)[i / 4];
#pragma unroll
              for (int h = 0; h < H; ++h) {
                w[h][i / 2] = add2(add2(y[h][i / 2], mh.x), ml.x);
                W2[h] = fma2(w[h][i / 2], w[h][i / 2], W2[h]);
                if (DT > 2) {
                  w[h][i / 2 + 1] = add2(add2(y[h][i / 2 + 1], mh.y), ml.y);
                  W2[h] = fma2(w[h][i / 2 + 1], w[h][i / 2 + 1], W2[h]);
                }
              }
            }
            // row i in float4s; its padding is zero (exact zero products)
            const ulonglong2* Li = reinterpret_cast<const ulonglong2*>(L32 + gmm_zs_row(i));
            unsigned long long s[H];
#pragma unroll
            for (int h = 0; h < H; ++h) s[h] = 0ull;
#pragma unroll
            for (int q = 0; q <= i / 4; ++q) {
              const ulonglong2 l = Li[q];
#pragma unroll
              for (int h = 0; h < H; ++h) s[h] = fma2(l.x, w[h][2 * q], s[h]);
#pragma unroll
              for (int h = 0; h < H; ++h)
                if (DT > 2) s[h] = fma2(l.y, w[h][2 * q + 1], s[h]);
            }
            const float ai = i % 4 == 0 ? a4.x : i % 4 == 1 ? a4.y : i % 4 == 2 ? a4.z : a4.w;
#pragma unroll
            for (int h = 0; h < H; ++h) {
              const float r = __fadd_rn(lo2(s[h]), hi2(s[h]));
              e[h] = __fmaf_rn(r, r, e[h]);
              t1[h] = __fmaf_rn(fabsf(r), ai, t1[h]);
            }
            // After 4, 8 and 16 rows: log p_k <= lpc - (1 - 2^-9) e~ / 2 + 1 (e's
            // remaining terms are nonnegative, its error far below 2^-9 e~ + 1
            // while |lpc| < 2^20 and the bound on e~'s error is below 1), so
            // a component 41 below the largest so far for all of the warp's
            // points adds less than 2^-59 of p_max to the sums - all of them
            // far less than the band's own rounding slack of 2^-38 - and its
            // remaining rows are left out.
            if ((i == 3 || i == 7 || i == 15) && ORDERED) {
              bool f = true;
#pragma unroll
              for (int h = 0; h < H; ++h) {
                const float W = __fadd_ru(__fsqrt_ru(2.0f * __fadd_ru(lo2(W2[h]), hi2(W2[h]))), sc.z);
                const float err = __fmul_ru(4.0f * u32, __fmul_ru(W, t1[h]));
                f = f && err < 0.25f + 0x1p-11f * e[h] && fabsf(lpc) < 0x1p20f &&
                    lpc - 0.4990234375f * e[h] < low[h] - 42.0f;
              }
              far = __all_sync(0xffffffffu, f);
            }
          }
        }
        if (far) {
#pragma unroll
          for (int h = 0; h < H; ++h) {
            tk[h][k] = -INFINITY;
            ek[h][k] = 0.0f;
          }
          continue;
        }
#pragma unroll
        for (int h = 0; h < H; ++h) {
          // W >= ||w~|| + 2^-23 ||mu|| (the sum of squares' rounding and the root's covered)
          const float ww = __fadd_ru(lo2(W2[h]), hi2(W2[h]));
          const float W = __fadd_ru(__fsqrt_ru(__fmul_ru(ww, 1.0f + (float)(DT + 2) * u32)), sc.z);
          const float sd2 = __fmul_ru(__fmul_ru(W, W), sc.y);
          const float E = __fmul_ru(__fadd_ru(__fadd_ru(__fmul_ru((float)(d + 1) * u32, e[h]),
                                                        __fmul_ru(2.0f * u32, __fmul_ru(W, t1[h]))),
                                              __fmul_ru(u32 * u32 * 1.01f, sd2)),
                                    1.0f + 0x1p-16f);
          const float t = __fmaf_rn(-0.5f, e[h], lpc);
          const float eps = __fadd_ru(__fadd_ru(__fmul_ru(0.5f, E), __fmul_ru(u32, fabsf(lpc) + fabsf(t))),
                                      __fmul_ru(0x1p-40f, fabsf(lpc) + e[h] + 1.0f));
          tk[h][k] = t;
          ek[h][k] = eps;
          if (!(t < INFINITY) || !(eps < INFINITY)) exact[h] = true;   // non-finite
          tmax[h] = fmaxf(tmax[h], t);
          low[h] = fmaxf(low[h], __fsub_rd(t, eps));
          likely[h] = likely[h] || e[h] < (float)(3 * d + 30);
        }
      }
    }
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int n = n2[h];
      if (n < 0) continue;
      if (!(tmax[h] >= -690.0f && tmax[h] <= 690.0f)) exact[h] = true;
      int zk = -1;
      if (!exact[h]) {
        // p~_k and an absolute bound A_k on |p~_k - p_k / p_max| (the exact value
        // lies in [exp(dt - x), exp(dt + x)], x = eps_k + u |dt| + 4u, binary32
        // exp within 4u); far components, whose bands are wide, weigh their width
        // by their tiny size
        float C[GMM_ZS_MAXK];
        float acc = 0.0f, err = 0.0f;
        for (int k = 0; k < K; ++k) {
          float p = 0.0f;
          if (tk[h][k] != -INFINITY) {
            const float dt = __fsub_rn(tk[h][k], tmax[h]);
            p = expf(dt);
            const float x = __fadd_ru(__fadd_ru(ek[h][k], __fmul_ru(u32, fabsf(dt))), 4.0f * u32);
            const float up = __fmul_ru(expf(__fadd_ru(dt, x)), 1.0f + 8.0f * u32);
            const float dn = __fmul_rd(expf(__fsub_rd(dt, x)), 1.0f - 8.0f * u32);
            err = __fadd_ru(err, fmaxf(__fsub_ru(up, p), __fsub_ru(p, dn)));
          }
          acc = __fadd_rn(acc, p);
          C[k] = acc;
        }
        // band: the terms' errors, the running sums' and u * norm's roundings,
        // the comparisons' own roundings, the reference's running quotient sums
        const float Nt = C[K - 1];
        const float band = __fmul_ru(__fadd_ru(__fadd_ru(err, __fmul_ru((float)(K + 6) * u32, Nt)),
                                               __fmul_ru(0x1p-40f, Nt)), 1.0f + 0x1p-16f);
        Stream s = make_stream(seed, (uint32_t)n, iter, TAG_Z | (comp << 8));
        const double u = s.uniform();
        const float un = __fmul_rn(__double2float_rn(u), Nt);
        int i = 0;
        while (i < K - 1 && !(un < C[i])) ++i;
        const bool above_prev = i == 0 || __fadd_ru(C[i - 1], band) < __fsub_rd(un, band);
        const bool below_this = i == K - 1 || __fadd_ru(un, band) < __fsub_rd(C[i], band);
        if (above_prev && below_this && Nt >= 1.0f && band < INFINITY) zk = i;
      }
      if (zk >= 0) {
        z[n] = zk;
      } else {
        const int slot = atomicAdd(qn, 1);
        queue[slot] = n;
      }
    }
  }
}

// The reference's binary64 draw for the queued points, one CTA of K warps
// per point (K <= 32, d <= 32): warp k takes component k, lane i forms row
// i of Linv (y - mu_k) with gmm_z_kernel's operation order and lane 0 adds
// the squares in row order, all components side by side; thread 0 then
// makes the draw from the K densities.  CTAs take queued points in turn.
__global__ void __launch_bounds__(GMM_ZS_MAXK * 32)
gmm_zx_kernel(int d, int K, int shared_cov, const float* __restrict__ Y, const double* __restrict__ pis,
              const double* __restrict__ mu, const double* __restrict__ Linv, const double* __restrict__ hdet,
              const int* __restrict__ queue, const int* __restrict__ qn, int* __restrict__ z, uint64_t seed,
              uint32_t iter, uint32_t comp) {
  __shared__ double wsh[GMM_ZS_MAXK][32], ssh[GMM_ZS_MAXK][32], pmf[GMM_ZS_MAXK];
  const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
  const int nq = *qn;
  const double c = __dmul_rn(__dmul_rn(-0.5, (double)d), log(2.0 * 3.14159265358979323846264338327950288));
  const int kc = shared_cov ? 0 : k;
  const double* Lk = Linv + (size_t)kc * d * d;
  const double* mk = mu + (size_t)k * d;
  for (int q = blockIdx.x; q < nq; q += gridDim.x) {
    const int n = queue[q];
    if (lane < d) wsh[k][lane] = __dadd_rn((double)Y[(size_t)n * d + lane], -mk[lane]);
    __syncwarp();
    if (lane < d) {
      const double* Li = Lk + (size_t)lane * d;
      double s = 0.0;
#pragma unroll 4
      for (int jj = 0; jj <= lane; ++jj) s = __dadd_rn(s, __dmul_rn(Li[jj], wsh[k][jj]));
      ssh[k][lane] = s;
    }
    __syncwarp();
    if (lane == 0) {
      double expon = 0.0;
      for (int i = 0; i < d; ++i) expon = __dadd_rn(expon, __dmul_rn(ssh[k][i], ssh[k][i]));
      const double ll = __dadd_rn(__dadd_rn(c, -hdet[kc]), -__dmul_rn(0.5, expon));
      double prob = 1.0;
      prob = __dmul_rn(prob, pis[k]);
      prob = __dmul_rn(prob, exp(ll));
      pmf[k] = prob;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      Stream st = make_stream(seed, (uint32_t)n, iter, TAG_Z | (comp << 8));
      const double u = st.uniform();
      double norm = 0.0;
      for (int i = 0; i < K; ++i) norm = __dadd_rn(norm, pmf[i]);
      double acc = __ddiv_rn(pmf[0], norm);
      int zk = K - 1;
      for (int i = 1; i < K; ++i) {
        if (u < acc) { zk = i - 1; break; }
        acc = __dadd_rn(acc, __ddiv_rn(pmf[i], norm));
      }
      z[n] = zk;
    }
    __syncthreads();
  }
}

// ---- conjugate statistics ----------------------------------------------------
// Counts, sums of y and scatter matrices sum (y - mu_k)(y - mu_k)^T (the
// reference's full-matrix update augur_mat_atm_inc_vtmt is symmetric
// elementwise) of the points of each component.  Of many points in four launches:
//   order    the points are brought in component order, stable in the point
//            index: counts per chunk of 1024 points (gmm_count_kernel), then
//            every chunk's ranks behind the counts before it
//            (gmm_place_kernel);
//   segments one CTA per segment of at most `seg` points of one component
//            (gmm_segment_kernel): all its partial sums stay in registers for
//            the whole segment, and only one row of them is written;
//   reduce   the rows of each component added in a fixed order
//            (gmm_stats_reduce_kernel).
// Of fewer (gmm_stats_share) without the order: a CTA per component and share
// of the points, then the reduction if there is more than one share.
// Deterministic; the reference adds in point order.  Before, each of 296 CTAs
// kept a table of all components over its own points, so every pass wrote and
// read back 296 K-component tables (20 MB at K = 16, d = 32) and summed them in
// a chain of 296.  Points with a label outside [0, K) are not counted.
// Sums pass 74 -> 28 us and scatter pass 157 -> 54 us at K = 16, d = 32,
// N = 200,000 (16 of either are the ordering); bound by the gathered rows' round
// trips and, for the scatter, the binary64 pipe.
constexpr int GMM_STAT_W = 2048;            // widest row of statistics (count, sums, scatter) taken
constexpr int GMM_ORDER_CHUNK = 1024;       // points of an ordering CTA
constexpr int GMM_SLAB = 1 << 20;           // points ordered at a time (bounds the scratch)
constexpr int GMM_ORDER_CHUNKS = GMM_SLAB / GMM_ORDER_CHUNK;
constexpr int GMM_SEGMENTS = 444;           // segments aimed at: three CTAs per SM
constexpr int GMM_SEG_TILE = 64;            // points of a segment staged at a time
constexpr int GMM_SEG_GROUPS = 32;          // at most: thread groups of a CTA that share a segment's points

// The ordering's buckets: labels [0, K), and those outside in bucket K
// (B = K + 1 buckets) or left out (B = K).
__device__ __forceinline__ int gmm_bucket(int label, int K, int B) {
  return label >= 0 && label < K ? label : (B == K ? -1 : K);
}

// cnt [B][GMM_ORDER_CHUNKS]: counts of chunk blockIdx.x.
__global__ void __launch_bounds__(GMM_THREADS)
gmm_count_kernel(int n, int K, int B, const int* __restrict__ z, int* __restrict__ cnt) {
  __shared__ int h[GMM_MAX_K + 1];
  for (int k = threadIdx.x; k < B; k += GMM_THREADS) h[k] = 0;
  __syncthreads();
  const int n0 = blockIdx.x * GMM_ORDER_CHUNK, n1 = min(n, n0 + GMM_ORDER_CHUNK);
  for (int p = n0 + threadIdx.x; p < n1; p += GMM_THREADS) {
    const int k = gmm_bucket(z[p], K, B);
    if (k >= 0) atomicAdd(&h[k], 1);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < B; k += GMM_THREADS) cnt[k * GMM_ORDER_CHUNKS + blockIdx.x] = h[k];
}

// perm: the slab's points (plus `first`) in bucket order; start [B + 1], if
// given: where each bucket's begin.
__global__ void __launch_bounds__(GMM_THREADS)
gmm_place_kernel(int n, int K, int B, int first, const int* __restrict__ z, const int* __restrict__ cnt,
                 int* __restrict__ perm, int* __restrict__ start) {
  constexpr int NW = GMM_THREADS / 32, PER = GMM_ORDER_CHUNK / NW;
  __shared__ int tot[GMM_MAX_K + 1], before[GMM_MAX_K + 1], cur[NW][GMM_MAX_K + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = blockIdx.x;
  for (int k = warp; k < B; k += NW) {
    int t = 0, f = 0;
    for (int c = lane; c < (int)gridDim.x; c += 32) {
      const int v = cnt[k * GMM_ORDER_CHUNKS + c];
      t += v;
      f += c < b ? v : 0;
    }
    t = __reduce_add_sync(0xffffffffu, t);
    f = __reduce_add_sync(0xffffffffu, f);
    if (lane == 0) { tot[k] = t; before[k] = f; }
  }
  // this warp's points, and its counts by component
  const int p0 = b * GMM_ORDER_CHUNK + warp * PER;
  int kk[PER / 32];
  for (int k = lane; k < B; k += 32) cur[warp][k] = 0;
  __syncwarp();
#pragma unroll
  for (int q = 0; q < PER / 32; ++q) {
    const int p = p0 + q * 32 + lane;
    kk[q] = p < n ? gmm_bucket(z[p], K, B) : -1;
    if (kk[q] >= 0) atomicAdd(&cur[warp][kk[q]], 1);
  }
  __syncthreads();
  if (threadIdx.x < (unsigned)B) {
    int s = 0;
    for (int k = 0; k < (int)threadIdx.x; ++k) s += tot[k];
    if (b == 0 && start != nullptr) {
      start[threadIdx.x] = s;
      if ((int)threadIdx.x == B - 1) start[B] = s + tot[B - 1];
    }
    s += before[threadIdx.x];
    for (int w = 0; w < NW; ++w) {   // counts become cursors
      const int c = cur[w][threadIdx.x];
      cur[w][threadIdx.x] = s;
      s += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PER / 32; ++q) {
    const bool act = kk[q] >= 0;
    const unsigned mask = __ballot_sync(0xffffffffu, act);
    if (act) {
      const unsigned peers = __match_any_sync(mask, kk[q]);
      const int rank = __popc(peers & ((1u << lane) - 1u));
      const int base = cur[warp][kk[q]];
      perm[base + rank] = first + p0 + q * 32 + lane;
      __syncwarp(mask);
      if (rank == 0) cur[warp][kk[q]] = base + __popc(peers);
    }
    __syncwarp();
  }
}

// The segment blockIdx.x: its component and its number in it, found by the
// first warp (lane l takes components l and l + 32; start: [K + 1]); k = -1 past
// the last segment.
__device__ __forceinline__ void gmm_find_segment(const int* __restrict__ start, int K, int seg, int r, int* out) {
  const int lane = threadIdx.x & 31;
  int base = 0, k = -1, i = 0;
#pragma unroll
  for (int h = 0; h < GMM_MAX_K; h += 32) {
    const int q = h + lane;
    const int ns = q < K ? (start[q + 1] - start[q] + seg - 1) / seg : 0;
    int inc = ns;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, r >= base + inc - ns && r < base + inc);
    if (hit) {
      k = h + __ffs(hit) - 1;
      i = r - base - __shfl_sync(0xffffffffu, inc - ns, __ffs(hit) - 1);
    }
    base += __shfl_sync(0xffffffffu, inc, 31);
  }
  if (lane == 0) {
    out[0] = k;
    out[1] = i;
    out[2] = k >= 0 ? start[k] + i * seg : 0;
    out[3] = k >= 0 ? min(seg, start[k + 1] - start[k] - i * seg) : 0;
  }
}

__host__ __device__ inline int gmm_obs_tiles(int d) { const int t = (d + 3) / 4; return t * (t + 1) / 2; }
__host__ __device__ inline int gmm_obs_groups(int d) {
  const int g = GMM_THREADS / gmm_obs_tiles(d);
  return g < GMM_SEG_GROUPS ? g : GMM_SEG_GROUPS;
}
__host__ __device__ inline int gmm_seg_pitch(int d) { return (d + 3) / 4 * 4 + 2; }

// The points p_lo .. p_hi - 1 with label k, in order, into pts, and their
// number: every warp takes an equal share of the labels, counts, and places
// behind the warps before it.
__device__ __forceinline__ int gmm_gather_points(int p_lo, int p_hi, int k, const int* __restrict__ z, int* pts) {
  constexpr int NW = GMM_THREADS / 32;
  __shared__ int found[NW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int share = (p_hi - p_lo + GMM_THREADS - 1) / GMM_THREADS * 32;
  const int p0 = p_lo + warp * share, p1 = min(p_hi, p0 + share);
  int c = 0;
#pragma unroll 8
  for (int p = p0; p < p1; p += 32) c += __popc(__ballot_sync(0xffffffffu, z[min(p + lane, p_hi - 1)] == k && p + lane < p1));
  if (lane == 0) found[warp] = c;
  __syncthreads();
  int at = 0, m = 0;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    at += w < warp ? found[w] : 0;
    m += found[w];
  }
#pragma unroll 8
  for (int p = p0; p < p1; p += 32) {
    const bool in = z[min(p + lane, p_hi - 1)] == k && p + lane < p1;
    const unsigned bal = __ballot_sync(0xffffffffu, in);
    if (in) pts[at + __popc(bal & ((1u << lane) - 1u))] = p + lane;
    at += __popc(bal);
  }
  return m;
}

// One row of part per segment: sums [d] if wanted, then the scatter's lower
// triangle, row by row, if wanted.
// GATHER (small n): no order and no segments; a CTA per component and share of
// `seg` points finds the component's points in its share itself.  Its row is
// k gridDim.y + share, and cnt_part there its number of points; a component's
// only share stores the results.
// Sums: a group of pow2(d) lanes (32 lanes taking two coordinates each past
// d = 32) takes points in turn, one coordinate a lane.
// Scatter: the points are centred in binary64 once each, 64 at a time, into
// shared memory; a thread owns a 4 x 4 tile of the lower triangle (8
// values read for 16 multiply-adds), and as many groups of threads as fit
// the CTA share the points; the groups' tiles are added in group order.
// CW (16, 32 or 64, at least d): coordinates staged side by side.  All loads of
// a round are issued together, their indices clamped into the segment rather
// than guarded one by one (guarded loads waited for each other: 71 us for the
// scatter pass at K = 16, d = 32, N = 200,000).
template <int CW, bool GATHER>
__global__ void __launch_bounds__(GMM_THREADS)
gmm_segment_kernel(int n, int d, int K, int seg, int want_sum, int want_obs, const float* __restrict__ Y,
                   const int* __restrict__ z, const double* __restrict__ mu, const int* __restrict__ perm,
                   const int* __restrict__ start, double* __restrict__ part, int pts_at, int* __restrict__ cnt_part,
                   int* __restrict__ cnt, double* __restrict__ sum, double* __restrict__ obs) {
  extern __shared__ __align__(16) double sh[];
  __shared__ double mk[GMM_MAX_D];
  __shared__ int where[4];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* pts = reinterpret_cast<int*>(sh + pts_at);
  const bool whole = GATHER && gridDim.y == 1;
  const int W = (want_sum ? d : 0) + (want_obs ? d * (d + 1) / 2 : 0);
  int k, m, at;
  if (GATHER) {
    k = blockIdx.x;
    at = k * gridDim.y + blockIdx.y;
    m = gmm_gather_points(blockIdx.y * seg, min(n, (int)(blockIdx.y + 1) * seg), k, z, pts);
    if (tid == 0) *(whole ? cnt + k : cnt_part + at) = m;
    if (m == 0) {        // uniform
      for (int e = tid; e < (whole ? 0 : W); e += GMM_THREADS) part[(size_t)at * W + e] = 0.0;
      for (int e = tid; e < (whole && want_sum ? d : 0); e += GMM_THREADS) sum[(size_t)k * d + e] = 0.0;
      for (int e = tid; e < (whole && want_obs ? d * d : 0); e += GMM_THREADS) obs[(size_t)k * d * d + e] = 0.0;
      return;
    }
  } else {
    if (tid < 32) gmm_find_segment(start, K, seg, blockIdx.x, where);
    __syncthreads();
    k = where[0];
    m = where[3];
    if (k < 0) return;   // uniform
    at = blockIdx.x;
    for (int p = tid; p < m; p += GMM_THREADS) pts[p] = perm[where[2] + p];
  }
  __syncthreads();
  double* row = part + (size_t)at * W;
  if (want_sum) {
    int dp = 1;
    while (dp < d && dp < 32) dp <<= 1;
    const int c = lane & (dp - 1), per = 32 / dp;             // coordinate, points of a warp at a time
    const int step = per * (GMM_THREADS / 32);
    double s0 = 0.0, s1 = 0.0;
    const int c0 = min(c, d - 1), c1 = min(c + 32, d - 1);
    for (int p = warp * per + lane / dp; p < m; p += 8 * step) {
      float y0[8], y1[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float* y = Y + (size_t)pts[min(p + q * step, m - 1)] * d;
        y0[q] = y[c0];
        if (CW > 32) y1[q] = y[c1];
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (p + q * step < m) {
          s0 = __dadd_rn(s0, (double)y0[q]);
          if (CW > 32) s1 = __dadd_rn(s1, (double)y1[q]);
        }
    }
    for (int o = 16; o >= dp; o >>= 1) s0 = __dadd_rn(s0, __shfl_xor_sync(0xffffffffu, s0, o));   // s1: dp == 32
    if (lane < dp) {
      if (c < d) sh[warp * GMM_MAX_D + c] = s0;
      if (c + 32 < d) sh[warp * GMM_MAX_D + c + 32] = s1;
    }
    __syncthreads();
    if (tid < d) {
      double a = 0.0;
      for (int w = 0; w < GMM_THREADS / 32; ++w) a = __dadd_rn(a, sh[w * GMM_MAX_D + tid]);
      (whole ? sum + (size_t)k * d : row)[tid] = a;
    }
    __syncthreads();
    row += d;
  }
  if (!want_obs) return;
  const int pd = gmm_seg_pitch(d), dz = pd - 2;                // pitch, d rounded up to tiles
  const int nt = gmm_obs_tiles(d), G = gmm_obs_groups(d);
  const int g = tid / nt, tile = tid - g * nt;
  int ti = 0;
  while ((ti + 1) * (ti + 2) / 2 <= tile) ++ti;
  const int tj = tile - ti * (ti + 1) / 2;
  double acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
  if (tid < d) mk[tid] = mu[(size_t)k * d + tid];
  __syncthreads();
  // a thread stages one coordinate of every (256 / CW)-th point; the next
  // tile's values are loaded while this one's products are formed
  constexpr int PSTEP = GMM_THREADS / CW, NQ = GMM_SEG_TILE / PSTEP;
  const int c = tid & (CW - 1), pr = tid / CW;
  const float* yc = Y + min(c, d - 1);
  // a point's coordinates 4t, 4t + 1 of all t, then its 4t + 2, 4t + 3: the
  // tiles' 16-byte reads are then side by side
  const int cp = ((c >> 1) & 1) * (dz / 2) + 2 * (c >> 2) + (c & 1);
  float v[NQ];
  auto fetch = [&](int p0) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = yc[(size_t)pts[min(p0 + pr + q * PSTEP, m - 1)] * d];
  };
  fetch(0);
  const double mc = c < d ? mk[c] : 0.0;
  for (int p0 = 0; p0 < m; p0 += GMM_SEG_TILE) {
    const int np = min(GMM_SEG_TILE, m - p0);
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (c < dz) sh[(pr + q * PSTEP) * pd + cp] = c < d ? __dadd_rn((double)v[q], -mc) : 0.0;
    if (p0 + GMM_SEG_TILE < m) fetch(p0 + GMM_SEG_TILE);
    __syncthreads();
    if (g < G) {
      for (int p = g; p < np; p += G) {
        const double2* x = reinterpret_cast<const double2*>(sh + p * pd) + ti;
        const double2* y = reinterpret_cast<const double2*>(sh + p * pd) + tj;
        const double2 x0 = x[0], x1 = x[dz / 4], y0 = y[0], y1 = y[dz / 4];
        const double xa[4] = {x0.x, x0.y, x1.x, x1.y}, ya[4] = {y0.x, y0.y, y1.x, y1.y};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) acc[a][b] = __fma_rn(xa[a], ya[b], acc[a][b]);
      }
    }
    __syncthreads();
  }
  if (g < G) {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) sh[(g * nt + tile) * 16 + 4 * a + b] = acc[a][b];
  }
  __syncthreads();
  for (int e = tid; e < nt * 16; e += GMM_THREADS) {
    double a = 0.0;
    for (int q = 0; q < G; ++q) a = __dadd_rn(a, sh[q * nt * 16 + e]);
    int t = e >> 4, r = 0;
    while (t >= r + 1) { t -= r + 1; ++r; }
    const int ii = 4 * r + ((e >> 2) & 3), jj = 4 * t + (e & 3);
    if (ii >= d || jj > ii) continue;
    if (whole) {
      obs[(size_t)k * d * d + ii * d + jj] = a;
      obs[(size_t)k * d * d + jj * d + ii] = a;
    } else {
      row[ii * (ii + 1) / 2 + jj] = a;
    }
  }
}

// Component blockIdx.y's rows (its segments', or `shares` rows of a gathering
// pass) added: 32 entries per CTA, eight interleaved
// partial sums of each, then those in order; `add`: onto an earlier slab's.
// The counts of all but the last slab gather in scratch (so_far): `cnt` is
// stored once, with the final count, as other streams may be reading the same
// labels' counts from an earlier pass there.
__global__ void __launch_bounds__(GMM_THREADS)
gmm_stats_reduce_kernel(int d, int K, int seg, int shares, int want_sum, int want_obs,
                        const double* __restrict__ part, const int* __restrict__ start,
                        const int* __restrict__ cnt_part, int add, int last, int* __restrict__ so_far,
                        int* __restrict__ cnt, double* __restrict__ sum, double* __restrict__ obs) {
  __shared__ double red[8][33];
  const int k = blockIdx.y, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  int r0 = 0, n = 0, ns = shares;
  if (shares > 0) {
    r0 = k * shares;
    if (blockIdx.x == 0 && threadIdx.x < 32) {
      for (int r = tx; r < shares; r += 32) n += cnt_part[r0 + r];
      n = __reduce_add_sync(0xffffffffu, n);
    }
  } else {
    for (int q = 0; q < k; ++q) r0 += (start[q + 1] - start[q] + seg - 1) / seg;
    n = start[k + 1] - start[k];
    ns = (n + seg - 1) / seg;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) (last ? cnt : so_far)[k] = n + (add ? so_far[k] : 0);
  const int W = (want_sum ? d : 0) + (want_obs ? d * (d + 1) / 2 : 0);
  const int e = blockIdx.x * 32 + tx;
  double a = 0.0;
  if (e < W) {
#pragma unroll 8
    for (int r = ty; r < ns; r += 8) a = __dadd_rn(a, __ldg(part + (size_t)(r0 + r) * W + e));
  }
  red[ty][tx] = a;
  __syncthreads();
  if (ty != 0 || e >= W) return;
  a = red[0][tx];
#pragma unroll
  for (int q = 1; q < 8; ++q) a = __dadd_rn(a, red[q][tx]);
  if (want_sum && e < d) {
    double* o = sum + (size_t)k * d + e;
    *o = add ? __dadd_rn(*o, a) : a;
  } else {
    int t = e - (want_sum ? d : 0);
    int i = 0;
    while (t >= i + 1) { t -= i + 1; ++i; }
    double* o = obs + (size_t)k * d * d;
    if (add) a = __dadd_rn(o[(size_t)i * d + t], a);
    o[(size_t)i * d + t] = a;
    o[(size_t)t * d + i] = a;
  }
}

// ---- conjugate draws -----------------------------------------------------------
// Dirichlet(alpha + cnt) for the weights (augur_dist.c:526-538), element
// substream (k, iter, 7|comp<<8); sequential normaliser.
__global__ void gmm_conj_pis_kernel(int K, const double* __restrict__ alpha, const int* __restrict__ cnt,
                                    double* __restrict__ pis, uint64_t seed, uint32_t iter, uint32_t comp) {
  __shared__ double g[GMM_MAX_K];
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    Stream s = make_stream(seed, (uint32_t)k, iter, TAG_PI | (comp << 8));
    g[k] = gamma_draw(s, __dadd_rn(alpha[k], (double)cnt[k]), 1.0);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double acc = 0.0;
    for (int k = 0; k < K; ++k) acc = __dadd_rn(acc, g[k]);
    for (int k = 0; k < K; ++k) pis[k] = __ddiv_rn(g[k], acc);
  }
}

// augur_mvnormal_mvnormal_conj (augur_dist.c:633-669) for component k, one
// CTA, substream (k, iter, 8|comp<<8).  The two halves of the CTA invert the
// prior and the component covariance in step, then all of it inverts and
// factors the posterior precision.  Bound: the chain of the d columns of three
// factorisations, about 1400 cycles each (157 -> 81 us at d = 32, K = 16; one
// warp per matrix before).
template <int DT>
__global__ void __launch_bounds__(GMM_THREADS)
gmm_conj_mu_kernel(int d, int shared_cov, const double* __restrict__ mu0, const double* __restrict__ cov0,
                   const int* __restrict__ cnt, const double* __restrict__ sum, const double* __restrict__ cov,
                   double* __restrict__ mu, uint64_t seed, uint32_t iter, uint32_t comp) {
  constexpr int HALF = GMM_THREADS / 2;
  constexpr int TE = DT * (DT + 1) / 2;
  constexpr int NH = (TE + HALF - 1) / HALF, NE = (TE + GMM_THREADS - 1) / GMM_THREADS;
  extern __shared__ double sm[];
  __shared__ double piv[2][DT];
  const int k = blockIdx.x, tid = threadIdx.x;
  const int half = tid / HALF, t = tid - half * HALF;
  const int dd = d * d, dp = d * pitch(d);
  double* L0 = sm;
  double* L = L0 + dp;
  double* M0 = L + dp;
  double* M1 = M0 + dp;
  double* res = M1 + dp;
  double* w0 = res + d;
  double* mean = w0 + d;
  double* sk = mean + d;
  double* nrm = sk + d;
  double* mu0s = nrm + d;
  const double* ck = cov + (size_t)(shared_cov ? 0 : k) * dd;
  const int n = cnt[k];
  const double sc = n == 0 ? 1.0 : __ddiv_rn(1.0, (double)n);                       // augur_vec_scale
  for (int e = tid; e < dd; e += GMM_THREADS) {
    GP(L0, e / d, e % d) = cov0[e];
    GP(L, e / d, e % d) = ck[e];
  }
  for (int i = tid; i < d; i += GMM_THREADS) {
    sk[i] = __dmul_rn(sc, sum[(size_t)k * d + i]);
    mu0s[i] = mu0[i];
    Stream s = make_stream(seed, (uint32_t)k, iter, TAG_MU | (comp << 8));
    s.pos = (uint32_t)i;
    nrm[i] = s.normal();
  }
  double* A = half ? L : L0;
  double* M = half ? M1 : M0;
  {
    Tri<NH> T;
    T.deal(t, HALF, d);
    g_factor<NH, true>(T, A, M, piv[half], d);
    g_inverse(T, M, A, d);
  }
  if (half) {
    for (int e = t; e < dp; e += HALF) L[e] = __dmul_rn((double)n, L[e]);           // augur_mat_ms
  } else {
    g_mvm(res, L0, mu0s, t, HALF, d);
  }
  __syncthreads();
  if (half) g_mvm(w0, L, sk, t, HALF, d);
  __syncthreads();
  for (int i = tid; i < d; i += GMM_THREADS) res[i] = __dadd_rn(res[i], w0[i]);
  for (int e = tid; e < dp; e += GMM_THREADS) L0[e] = __dadd_rn(L0[e], L[e]);      // augur_mat_plus
  Tri<NE> T;
  T.deal(tid, GMM_THREADS, d);
  g_factor<NE, true>(T, L0, M0, piv[0], d);
  g_inverse(T, M0, L0, d);
  g_mvm(mean, L0, res, tid, GMM_THREADS, d);
  // augur_mvnormal_sample (augur_dist.c:622-630): chol(cov) nrm + mean
  for (int e = tid; e < dp; e += GMM_THREADS) L[e] = L0[e];
  g_factor<NE, false>(T, L, nullptr, piv[1], d);
  for (int i = tid; i < d; i += GMM_THREADS) {
    double s = 0.0;
#pragma unroll 8
    for (int j = 0; j <= i; ++j) s = __dadd_rn(s, __dmul_rn(GP(L, i, j), nrm[j]));
    mu[(size_t)k * d + i] = __dadd_rn(s, mean[i]);
  }
}

// Bartlett diagonal for the inverse-Wishart draw (bartlett_decomp,
// augur_dist.c:722-738): the chi-square of n - i degrees of freedom in row i
// is the sum of squares of the n - i normals at stream positions
// i*n + i + t, t < n - i (n = cnt[k] + df), substream (k, iter, 9|comp<<8).
// One CTA per (k, i): thread-strided partial sums, then the fixed-order
// block sum.  That is O(d * cnt[k]) normals per component per sweep (the
// reference's algorithm), spread over K * d CTAs.  Row i's sum of component
// k goes to chi[k * sk + i * si]: the diagonal of cov[k] (sk = d * d,
// si = d + 1), which gmm_conj_cov_kernel then reads and overwrites with the
// draw, or a [K][d] table of its own (sk = d, si = 1) when the draw runs
// beside the steps that still read cov.
__global__ void __launch_bounds__(GMM_THREADS)
gmm_bartlett_chi_kernel(int d, int df, const int* __restrict__ cnt, double* __restrict__ chi, int sk, int si,
                        uint64_t seed, uint32_t iter, uint32_t comp) {
  __shared__ double red[34];
  const int k = blockIdx.x / d, i = blockIdx.x - k * d;
  const int n = cnt[k] + df;
  const Stream s0 = make_stream(seed, (uint32_t)k, iter, TAG_COV | (comp << 8));
  double local = 0.0;
  for (int t = threadIdx.x; t < n - i; t += blockDim.x) {
    Stream s = s0;
    s.pos = (uint32_t)(i * n + i + t);
    const double zz = s.normal();
    local = __dadd_rn(local, __dmul_rn(zz, zz));
  }
  const double sum = block_sum_f64(local, red);
  if (threadIdx.x == 0) chi[(size_t)k * sk + (size_t)i * si] = sum;
}

// augur_invwishart_mvnormal_conj (augur_dist.c:751-757) and
// augur_invwishart_sample (:740-749) with bartlett_decomp (:722-738) for
// component k, one thread block, substream (k, iter, 9|comp<<8).  The
// Bartlett normals are drawn at the stream positions the reference's loop
// consumes them (row-major over the lower triangle; each diagonal
// chi-square of n - i normals follows its row's off-diagonal normals).  The
// chi-square sums of up to cnt + df squares come from
// gmm_bartlett_chi_kernel (chi[k * sk + i * si]), added in a fixed tree order
// instead of sequentially (a rounding-level difference).  Bound: the chain of
// the d columns of two factorisations and one inverse (126 -> 51 us at d = 32).
template <int DT>
__global__ void __launch_bounds__(GMM_THREADS)
gmm_conj_cov_kernel(int d, int df, const double* __restrict__ scale0, const int* __restrict__ cnt,
                    const double* __restrict__ obs, const double* chi, int sk, int si, double* cov, uint64_t seed,
                    uint32_t iter, uint32_t comp) {
  constexpr int NE = (DT * (DT + 1) / 2 + GMM_THREADS - 1) / GMM_THREADS;
  extern __shared__ double sm[];
  __shared__ double piv[DT];
  const int k = blockIdx.x, tid = threadIdx.x;
  const int dd = d * d, dp = d * pitch(d);
  double* L = sm;          // obs + scale0, then its inverse's factor
  double* M = L + dp;
  double* A = M + dp;
  double* P = A + dp;
  for (int e = tid; e < dd; e += GMM_THREADS) GP(L, e / d, e % d) = __dadd_rn(obs[(size_t)k * dd + e], scale0[e]);
  const int n = cnt[k] + df;
  // Bartlett factor: element (i, j < i) is the normal at position i*n + j;
  // the diagonal (i, i) is the square root of the row's chi-square sum.
  const Stream s0 = make_stream(seed, (uint32_t)k, iter, TAG_COV | (comp << 8));
  for (int e = tid; e < dd; e += GMM_THREADS) {
    const int i = e / d, j = e - i * d;
    if (j < i) {
      Stream s = s0;
      s.pos = (uint32_t)(i * n + j);
      GP(A, i, j) = s.normal();
    } else if (j > i) {
      GP(A, i, j) = 0.0;
    } else {
      GP(A, i, j) = __dsqrt_rn(chi[(size_t)k * sk + (size_t)i * si]);
    }
  }
  Tri<NE> T;
  T.deal(tid, GMM_THREADS, d);
  g_factor<NE, true>(T, L, M, piv, d);
  g_inverse(T, M, L, d);
  g_factor<NE, false>(T, L, nullptr, piv, d);
  // augur_mat_trtrmm (:381-392): the entries above the diagonal of L are not
  // read; A's are zeros, so the product's upper entries are sums of zeros
  for (int e = tid; e < dd; e += GMM_THREADS) {
    const int i = e / d, j = e - i * d;
    double s = 0.0;
#pragma unroll 8
    for (int q = 0; q <= i; ++q) s = __dadd_rn(s, __dmul_rn(GP(L, i, q), GP(A, q, j)));
    GP(P, i, j) = s;
  }
  g_trmi(T, P, M, piv, tid, GMM_THREADS, d);
  g_inverse(T, M, L, d);
  for (int e = tid; e < dd; e += GMM_THREADS) cov[(size_t)k * dd + e] = GP(L, e / d, e % d);
}

// ---- ESlice / MWG on the means ---------------------------------------------------
// The full conditional of mu[k] (CgLike.hs:236-265) is its prior MvNormal(mu0,
// cov0) and the points of component k.  Both moves only compare it at a
// candidate m with its value at the current mean mu: with S = sum (y_n - mu)
// over the component's n points, P = Linv and delta = P (m - mu),
//   sum_n [log N(y_n | m) - log N(y_n | mu)] = delta . (P S) - n |delta|^2 / 2,
// so one pass over the points gives S and n, and a candidate costs two d x d
// products (before, every candidate was evaluated at every point by a single
// CTA per component: 420-820 us a move at N = 6007, K = 5, d = 6).  The terms
// common to both values never enter, so the difference is at least as exact.
// A cluster of eight CTAs serves a component: seven walk the labels and add
// the component's points, in a fixed order, while the first prepares the
// tables and the proposal; it then collects the sums and makes the move.
// Sweep of that case 1020 -> 55 us.
constexpr int GMM_MOVE_CLUSTER = 8;
constexpr int GMM_MOVE_BATCH = 256;      // labels a warp reads at a time

// Sum over the component's points of y - mu (S, [d]) and their number, of
// part r of np of the labels.  sh: [warps][GMM_MAX_D] doubles, then
// [warps][GMM_MOVE_BATCH] ints.
__device__ void gmm_move_sums(int N, int d, int k, int r, int np, const float* __restrict__ Y,
                              const int* __restrict__ z, const double* __restrict__ mu, double* sh, double* S,
                              int* count) {
  constexpr int NW = GMM_THREADS / 32, NL = GMM_MOVE_BATCH / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* list = reinterpret_cast<int*>(sh + NW * GMM_MAX_D) + warp * GMM_MOVE_BATCH;
  __shared__ int counts[NW];
  int dp = 1;
  while (dp < d && dp < 32) dp <<= 1;
  const int c = lane & (dp - 1), sub = lane / dp, per = 32 / dp;   // coordinate; points of a warp at a time
  const int c0 = min(c, d - 1), c1 = min(c + 32, d - 1);
  const double m0 = mu[c0], m1 = mu[c1];
  double s0 = 0.0, s1 = 0.0;
  int total = 0;
  const int n0 = (int)((long long)N * r / np), n1 = (int)((long long)N * (r + 1) / np);
  for (int b = n0 + warp * GMM_MOVE_BATCH; b < n1; b += NW * GMM_MOVE_BATCH) {
    int lab[NL];
#pragma unroll
    for (int q = 0; q < NL; ++q) lab[q] = z[min(b + q * 32 + lane, n1 - 1)];
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < NL; ++q) {
      const bool in = lab[q] == k && b + q * 32 + lane < n1;
      const unsigned bal = __ballot_sync(0xffffffffu, in);
      if (in) list[cnt + __popc(bal & ((1u << lane) - 1u))] = b + q * 32 + lane;
      cnt += __popc(bal);
    }
    __syncwarp();
    for (int t = sub; t < cnt; t += 8 * per) {   // eight points in flight a lane group
      float y0[8], y1[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float* y = Y + (size_t)list[min(t + q * per, cnt - 1)] * d;
        y0[q] = y[c0];
        y1[q] = y[c1];
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (t + q * per < cnt) {
          s0 = __dadd_rn(s0, __dadd_rn((double)y0[q], -m0));
          s1 = __dadd_rn(s1, __dadd_rn((double)y1[q], -m1));
        }
    }
    total += cnt;
    __syncwarp();
  }
  for (int o = 16; o >= dp; o >>= 1) s0 = __dadd_rn(s0, __shfl_xor_sync(0xffffffffu, s0, o));   // s1: dp == 32
  if (lane < dp) {
    if (c < d) sh[warp * GMM_MAX_D + c] = s0;
    if (c + 32 < d) sh[warp * GMM_MAX_D + c + 32] = s1;
  }
  if (lane == 0) counts[warp] = total;
  __syncthreads();
  if (tid < d) {
    double a = 0.0;
    for (int w = 0; w < NW; ++w) a = __dadd_rn(a, sh[w * GMM_MAX_D + tid]);
    S[tid] = a;
  }
  if (tid == 0) {
    int n = 0;
    for (int w = 0; w < NW; ++w) n += counts[w];
    *count = n;
  }
}

// L x (lower triangle, row pitch as GP) for rows lane and lane + 32: the
// squared norm and, with `with`, the dot product with it, summed over the warp.
__device__ __forceinline__ void gmm_tri_norm(const double* L, const double* x, const double* with, int d, int lane,
                                             double& sq, double& dot) {
  sq = 0.0;
  dot = 0.0;
  for (int i = lane; i < d; i += 32) {
    double s = 0.0;
#pragma unroll 4
    for (int j = 0; j <= i; ++j) s = __fma_rn(GP(L, i, j), x[j], s);
    sq = __fma_rn(s, s, sq);
    if (with) dot = __fma_rn(s, with[i], dot);
  }
  sq = warp_sum_f64(sq);
  dot = warp_sum_f64(dot);
}

// SLICE: augur_mcmc_eslice (augur_mcmclib.h:439-485) on mu[k]; substream
// (k, iter, 10|comp<<8): nu (d normals), u, theta, one uniform per shrink.
// Otherwise MWG [mu] ~ MvNormal(mu[k], covp) (CgUserProp.hs:131-260 over
// augur_mcmc_mwg); compat uses the generated log-correction ll(mu; mu, covp) -
// ll(mu'; mu, covp) = |Linv_p (mu' - mu)|^2 / 2, else 0.  Substream (k, iter,
// 11|comp<<8): d normals, then the accept uniform.  `cov`: cov0 or covp;
// `tally`: the slice's shrinks, or the accepts added to.
template <int DT, bool SLICE>
__global__ void __cluster_dims__(GMM_MOVE_CLUSTER, 1, 1) __launch_bounds__(GMM_THREADS)
gmm_move_kernel(int N, int d, int shared_cov, const float* __restrict__ Y, const int* __restrict__ z,
                const double* __restrict__ mu0, const double* __restrict__ cov, const double* __restrict__ Linv,
                const double* __restrict__ hdet, int prior_slot, int prop_slot, int compat, double* __restrict__ mu,
                uint64_t seed, uint32_t iter, uint32_t comp, int* __restrict__ tally) {
  constexpr int NE = (DT * (DT + 1) / 2 + GMM_THREADS - 1) / GMM_THREADS;
  extern __shared__ __align__(16) double sm[];
  __shared__ double S[GMM_MAX_D], piv[GMM_MAX_D], cur[GMM_MAX_D], prop[GMM_MAX_D], mu0s[GMM_MAX_D], x[GMM_MAX_D],
      R[GMM_MAX_D], nrm[GMM_MAX_D];
  __shared__ int count;
  const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int rank = (int)cl.block_rank(), k = blockIdx.x / GMM_MOVE_CLUSTER, kc = shared_cov ? 0 : k;
  const int tid = threadIdx.x, lane = tid & 31, dd = d * d, dp = d * pitch(d);
  double* P = sm;            // Linv of the component
  double* P0 = P + dp;       // Linv of the prior
  double* C = P0 + dp;       // the proposal covariance's factor
  const uint32_t tag = (SLICE ? TAG_ESLICE : TAG_MWG) | (comp << 8);
  Stream s = make_stream(seed, (uint32_t)k, iter, tag);
  if (rank > 0) {
    gmm_move_sums(N, d, k, rank - 1, GMM_MOVE_CLUSTER - 1, Y, z, mu + (size_t)k * d, sm, S, &count);
  } else {
    for (int e = tid; e < dd; e += GMM_THREADS) {
      const int i = e / d, j = e - i * d;
      GP(P, i, j) = Linv[(size_t)kc * dd + e];
      GP(P0, i, j) = Linv[(size_t)prior_slot * dd + e];
      GP(C, i, j) = cov[e];
    }
    if (tid < d) {
      cur[tid] = mu[(size_t)k * d + tid];
      mu0s[tid] = mu0[tid];
      Stream si = s;
      si.pos = (uint32_t)tid;
      nrm[tid] = si.normal();
    }
    Tri<NE> T;
    T.deal(tid, GMM_THREADS, d);
    g_factor<NE, false>(T, C, nullptr, piv, d);
    // augur_mvnormal_sample (augur_dist.c:622-630) around mu0 or the current mean
    if (tid < d) {
      double a = 0.0;
      for (int j = 0; j <= tid; ++j) a = __dadd_rn(a, __dmul_rn(GP(C, tid, j), nrm[j]));
      prop[tid] = __dadd_rn(a, SLICE ? mu0s[tid] : cur[tid]);
    }
  }
  cl.sync();
  if (rank == 0 && tid < d) {
    double a = 0.0;
    for (int r = 1; r < GMM_MOVE_CLUSTER; ++r) a = __dadd_rn(a, cl.map_shared_rank(S, r)[tid]);
    x[tid] = a;
  }
  int n = 0;
  if (rank == 0)
    for (int r = 1; r < GMM_MOVE_CLUSTER; ++r) n += *cl.map_shared_rank(&count, r);
  cl.sync();                 // the other CTAs' shared memory has been read
  if (rank > 0 || tid >= 32) return;
  bool finite = true;                        // S is, unless a point or the mean is not
  for (int i = lane; i < d; i += 32) {       // R = P S
    double a = 0.0;
    for (int j = 0; j <= i; ++j) a = __fma_rn(GP(P, i, j), x[j], a);
    R[i] = a;
    finite = finite && isfinite(x[i]);
  }
  finite = __all_sync(0xffffffffu, finite);
  __syncwarp();
  double q0, unused;
  for (int i = lane; i < d; i += 32) x[i] = __dadd_rn(cur[i], -mu0s[i]);
  __syncwarp();
  gmm_tri_norm(P0, x, nullptr, d, lane, q0, unused);
  // a density that is not finite at any point rejects every candidate, as its
  // comparison would
  const double scale = (n > 0 ? hdet[kc] : 0.0) + hdet[prior_slot];
  const double bad = finite && isfinite(scale) ? 0.0 : NAN;
  // log density at `m` minus the one at the current mean
  auto gain = [&](const double* m) {
    double q1, sq, dot;
    __syncwarp();
    for (int i = lane; i < d; i += 32) x[i] = __dadd_rn(m[i], -mu0s[i]);
    __syncwarp();
    gmm_tri_norm(P0, x, nullptr, d, lane, q1, unused);
    __syncwarp();
    for (int i = lane; i < d; i += 32) x[i] = __dadd_rn(m[i], -cur[i]);
    __syncwarp();
    gmm_tri_norm(P, x, R, d, lane, sq, dot);
    const double data = n > 0 ? __dadd_rn(dot, -__dmul_rn(__dmul_rn(0.5, (double)n), sq)) : 0.0;
    return __dadd_rn(__dadd_rn(data, -__dmul_rn(0.5, __dadd_rn(q1, -q0))), bad);
  };
  s.pos = (uint32_t)d;       // every lane advances the same cursor
  const double logu = log(s.uniform());
  if (SLICE) {
    const double PI2 = 2.0 * 3.14159265358979323846264338327950288;
    double theta = __dadd_rn(0.0, __dmul_rn(s.uniform(), __dadd_rn(PI2, -0.0)));
    double tmin = __dadd_rn(theta, -PI2), tmax = theta;
    int ns = 0;
    for (int i = lane; i < d; i += 32) nrm[i] = prop[i];     // nu
    bool moved = false;
    for (int guard = 0; guard < 2000; ++guard) {
      const double diff = __dadd_rn(tmax, -tmin);
      if (diff < 1e-8) break;
      const double ct = cos(theta), st = sin(theta);
      for (int i = lane; i < d; i += 32) {
        const double mi = mu0s[i];
        const double a = __dmul_rn(__dadd_rn(cur[i], -mi), ct);
        const double b = __dmul_rn(__dadd_rn(nrm[i], -mi), st);
        prop[i] = __dadd_rn(__dadd_rn(a, b), mi);
      }
      if (gain(prop) > logu) {
        moved = true;
        break;
      }
      if (theta < 0) tmin = theta; else tmax = theta;
      theta = __dadd_rn(tmin, __dmul_rn(s.uniform(), __dadd_rn(tmax, -tmin)));
      ++ns;
    }
    if (moved)
      for (int i = lane; i < d; i += 32) mu[(size_t)k * d + i] = prop[i];
    if (lane == 0) tally[k] = ns;
  } else {
    double corr = 0.0;
    if (compat) {
      for (int i = lane; i < d; i += 32) x[i] = __dadd_rn(prop[i], -cur[i]);
      for (int e = lane; e < dd; e += 32) GP(C, e / d, e % d) = Linv[(size_t)prop_slot * dd + e];
      __syncwarp();
      double sq;
      gmm_tri_norm(C, x, nullptr, d, lane, sq, unused);
      corr = __dmul_rn(0.5, sq) + (isfinite(hdet[prop_slot]) ? 0.0 : NAN);
    }
    const bool acc = logu < __dadd_rn(gain(prop), corr);
    if (acc)
      for (int i = lane; i < d; i += 32) mu[(size_t)k * d + i] = prop[i];
    if (lane == 0) tally[k] += acc;
  }
}

#undef GP

// ---- launchers -------------------------------------------------------------------
static int gmm_check(int N, int d, int K) {
  AB_REQUIRE(N > 0 && d > 0 && d <= GMM_MAX_D && K > 0 && K <= GMM_MAX_K, AB_ERR_ARG,
             "gmm: need N > 0, 0 < d <= %d, 0 < K <= %d (N=%d d=%d K=%d)", GMM_MAX_D, GMM_MAX_K, N, d, K);
  return AB_OK;
}

template <int DT, bool U>
static void launch_z_t(int N, int d, int K, int shared, const float* Y, const double* pis, const double* mu,
                       const double* Linv, const double* hdet, int* z, uint64_t seed, uint32_t iter,
                       uint32_t comp, cudaStream_t st) {
  gmm_z_kernel<DT, U><<<ceil_div(N, GMM_THREADS), GMM_THREADS, 0, st>>>(N, d, K, shared, Y, pis, mu, Linv, hdet,
                                                                     z, seed, iter, comp);
}

int launch_gmm_z(int N, int d, int K, int shared, const float* Y, const double* pis, const double* mu,
                 const double* Linv, const double* hdet, int* z, uint64_t seed, uint32_t iter, uint32_t comp,
                 cudaStream_t st) {
  if (d <= 2) launch_z_t<2, true>(N, d, K, shared, Y, pis, mu, Linv, hdet, z, seed, iter, comp, st);
  else if (d <= 4) launch_z_t<4, true>(N, d, K, shared, Y, pis, mu, Linv, hdet, z, seed, iter, comp, st);
  else if (d <= 8) launch_z_t<8, true>(N, d, K, shared, Y, pis, mu, Linv, hdet, z, seed, iter, comp, st);
  else if (d <= 16) launch_z_t<16, true>(N, d, K, shared, Y, pis, mu, Linv, hdet, z, seed, iter, comp, st);
  else if (d <= 32) launch_z_t<32, true>(N, d, K, shared, Y, pis, mu, Linv, hdet, z, seed, iter, comp, st);
  else launch_z_t<GMM_MAX_D, false>(N, d, K, shared, Y, pis, mu, Linv, hdet, z, seed, iter, comp, st);
  AB_LAUNCH_CHECK("gmm_z_kernel");
  return AB_OK;
}

// Scratch of the screened draw: the component tables, the exact-path flag
// and queue length, the queue.
static inline size_t gmm_al256(size_t x) { return (x + 255) & ~(size_t)255; }
static inline size_t gmm_zs_smem(int d, int K) { return sizeof(float) * (size_t)K * gmm_zs_stride(d); }
// Whether the screened draw takes the points in the order of their current
// labels (two small launches, about 11 us at 200,000 points): then a warp's
// points are near one component and the others' rows are mostly left out.
// That depends on a state the host does not see, so the line lies where the
// order gains more with components apart and most labels right than it loses
// with random labels or components in one another: at N = 200,000 the draw takes,
// in order so, otherwise, and without the order,
//   d = 32: K = 30  298, 649, 597 us;  K = 16  155, 290, 235;  K = 8  107, 167, 136;
//   d = 24: K = 30  209, 390, 297 us;  K = 16  134, 227, 164;  K = 8  92, 132, 94;
// at N = 30,000, d = 32, K = 30 and 16 171, 232, 138 and 101, 137, 89.
static inline bool gmm_zs_ordered(int N, int d, int K) { return d > 24 && (double)N * K * d * d >= 1.5e9; }
static inline size_t gmm_zs_queue_bytes(int N) { return gmm_al256(sizeof(int) * (size_t)N); }
size_t gmm_zs_scratch(int N, int d, int K) {
  return gmm_al256(gmm_zs_smem(d, K)) + 256 + gmm_zs_queue_bytes(N) +
         (gmm_zs_ordered(N, d, K) ? gmm_zs_queue_bytes(N) + sizeof(int) * (size_t)(K + 1) * GMM_ORDER_CHUNKS : 0);
}
bool gmm_zs_fits(int d, int K) { return K <= GMM_ZS_MAXK && d <= 32 && gmm_zs_smem(d, K) <= 100 * 1024; }

template <int DT, int H>
static int launch_zs_t(int N, int d, int K, const float* Y, const float* tab, const int* perm, const int* flag,
                       int* queue, int* qn, int* z, uint64_t seed, uint32_t iter, uint32_t comp, cudaStream_t st) {
  const size_t smem = gmm_zs_smem(d, K);
  AB_CUDA(allow_smem((const void*)gmm_zs_kernel<DT, H>, smem));
  const int vec = d % 4 == 0 && (reinterpret_cast<uintptr_t>(Y) & 15) == 0;
  // a tile of 32 H points for each of a CTA's warps; with fewer, still a CTA per
  // SM, and where the tables that each reads are large, not more CTAs than run
  // at once (K = 30, d = 24 to 32: 1 to 3 % faster; K = 30, d = 2 at 400,000 points
  // 10 % slower)
  const unsigned tiles = ceil_div(N, 32 * H), warps = GMM_ZS_THREADS / 32;
  const unsigned resident = 148u * std::min<unsigned>(gmm_zs_ctas(DT, H), 227 * 1024 / (smem + 1024));
  const unsigned grid = std::min(std::max(ceil_div(tiles, warps), std::min(tiles, 148u)), smem > 10 * 1024 ? resident : ~0u);
  gmm_zs_kernel<DT, H><<<grid, GMM_ZS_THREADS, smem, st>>>(N, d, K, vec, Y, tab, perm, flag, queue, qn, z, seed,
                                                                 iter, comp);
  AB_LAUNCH_CHECK("gmm_zs_kernel");
  return AB_OK;
}

int launch_gmm_z_screened(int N, int d, int K, int shared, const float* Y, const double* pis, const double* mu,
                          const double* Linv, const double* hdet, int* z, uint64_t seed, uint32_t iter,
                          uint32_t comp, void* scratch, cudaStream_t st) {
  if (!gmm_zs_fits(d, K)) return launch_gmm_z(N, d, K, shared, Y, pis, mu, Linv, hdet, z, seed, iter, comp, st);
  char* base = static_cast<char*>(scratch);
  float* tab = reinterpret_cast<float*>(base);
  int* ctl = reinterpret_cast<int*>(base + gmm_al256(gmm_zs_smem(d, K)));
  int* flag = ctl;
  int* qn = ctl + 1;
  int* queue = reinterpret_cast<int*>(reinterpret_cast<char*>(ctl) + 256);
  AB_CUDA(cudaMemsetAsync(ctl, 0, 2 * sizeof(int), st));
  gmm_zs_prep_kernel<<<K, 64, 0, st>>>(d, K, shared, pis, mu, Linv, hdet, tab, flag);
  AB_LAUNCH_CHECK("gmm_zs_prep_kernel");
  int* perm = nullptr;
  if (gmm_zs_ordered(N, d, K)) {
    perm = reinterpret_cast<int*>(reinterpret_cast<char*>(queue) + gmm_zs_queue_bytes(N));
    int* chunk_cnt = reinterpret_cast<int*>(reinterpret_cast<char*>(perm) + gmm_zs_queue_bytes(N));
    for (long long at = 0; at < N; at += GMM_SLAB) {   // 64 bits: past the last slab the offset may not fit 32
      const int n0 = (int)at, n = std::min(GMM_SLAB, N - n0), chunks = (int)ceil_div(n, GMM_ORDER_CHUNK);
      gmm_count_kernel<<<chunks, GMM_THREADS, 0, st>>>(n, K, K + 1, z + n0, chunk_cnt);
      AB_LAUNCH_CHECK("gmm_count_kernel");
      gmm_place_kernel<<<chunks, GMM_THREADS, 0, st>>>(n, K, K + 1, n0, z + n0, chunk_cnt, perm + n0, nullptr);
      AB_LAUNCH_CHECK("gmm_place_kernel");
    }
  }
  int rc;
#define AB_ZS(DT, H) launch_zs_t<DT, H>(N, d, K, Y, tab, perm, flag, queue, qn, z, seed, iter, comp, st)
  rc = d <= 2   ? AB_ZS(2, 1)
       : d <= 4 ? AB_ZS(4, 1)
       : d <= 8 ? AB_ZS(8, 1)
       : d <= 16 ? AB_ZS(16, 1)
       : perm    ? AB_ZS(32, 2)
                 : AB_ZS(32, 1);
#undef AB_ZS
  if (rc) return rc;
  gmm_zx_kernel<<<592, 32 * K, 0, st>>>(d, K, shared, Y, pis, mu, Linv, hdet, queue, qn, z, seed, iter, comp);
  AB_LAUNCH_CHECK("gmm_zx_kernel");
  return AB_OK;
}

// The thread-group kernels are built for d <= 16, 32 and 64 (the entries a
// thread carries in registers).
#define AB_GMM_BY_D(d, CALL) \
  ((d) <= 16 ? CALL(16) : (d) <= 32 ? CALL(32) : CALL(GMM_MAX_D))

template <int DT>
static int launch_prep_t(int Kc, int d, const double* cov, double* Linv, double* hdet, cudaStream_t st) {
  const size_t smem = sizeof(double) * 2 * (size_t)d * pitch(d);
  AB_CUDA(allow_smem((const void*)gmm_prep_kernel<DT>, smem));
  gmm_prep_kernel<DT><<<Kc, GMM_THREADS, smem, st>>>(d, cov, Linv, hdet);
  AB_LAUNCH_CHECK("gmm_prep_kernel");
  return AB_OK;
}

int launch_gmm_prep(int Kc, int d, const double* cov, double* Linv, double* hdet, cudaStream_t st) {
#define AB_CALL(DT) launch_prep_t<DT>(Kc, d, cov, Linv, hdet, st)
  return AB_GMM_BY_D(d, AB_CALL);
#undef AB_CALL
}

// Scratch of the statistics: the component order, chunk counts, component
// starts, the earlier slabs' counts, and a row of partial sums per segment.
struct GmmStatScratch {
  size_t perm, cnt, start, so_far, part, total;
};
static GmmStatScratch gmm_stat_layout(int d, int K) {
  GmmStatScratch L;
  const size_t W = (size_t)d + (size_t)d * (d + 1) / 2;
  L.perm = 0;
  L.cnt = L.perm + sizeof(int) * (size_t)GMM_SLAB;
  L.start = L.cnt + sizeof(int) * (size_t)K * GMM_ORDER_CHUNKS;
  L.so_far = L.start + gmm_al256(sizeof(int) * ((size_t)K + 1));
  L.part = L.so_far + gmm_al256(sizeof(int) * (size_t)K);
  L.total = L.part + sizeof(double) * ((size_t)GMM_SEGMENTS + K) * W;
  return L;
}
size_t gmm_stats_scratch(int d, int K) { return gmm_stat_layout(d, K).total; }

// The points of a share of the gathering pass, 0 for the ordered one.  One or
// two launches instead of four, which is what a sweep of few points in few
// dimensions waits for (N = 2,000, K = 3, d = 2: 122 us with the ordered pass,
// 92 with this), and no ordering: per pass 5 and 9 us (sums, scatter) against
// 11 and 12 at N = 8,000, K = 2, d = 2, 6 and 15 against 13 and 22 at N = 32,000, d =
// 32.  A share bounds what a CTA does if all labels are equal (16 turns of the
// scatter's loop, 8 or 2 of the slower ones of wide d); twice that where the
// rows of partial sums would not suffice otherwise, and the ordered pass beyond.
static inline int gmm_stats_share(int N, int d, int K) {
  const int base = d <= 16 ? 1024 : d <= 32 ? 512 : 128;
  for (int share : {base, 2 * base})
    if (N <= 131072 && K * (int)ceil_div(N, share) <= GMM_SEGMENTS) return share;
  return 0;
}

int launch_gmm_stats(int N, int d, int K, const float* Y, const int* z, const double* mu, int want_sum,
                     int want_obs, int* cnt, double* sum, double* obs, void* scratch, cudaStream_t st) {
  const int W = (want_sum ? d : 0) + (want_obs ? d * (d + 1) / 2 : 0);
  AB_REQUIRE(1 + W <= GMM_STAT_W, AB_ERR_ARG, "gmm: d too large for the statistics pass");
  const GmmStatScratch L = gmm_stat_layout(d, K);
  char* base = static_cast<char*>(scratch);
  int* perm = reinterpret_cast<int*>(base + L.perm);
  int* chunk_cnt = reinterpret_cast<int*>(base + L.cnt);
  int* start = reinterpret_cast<int*>(base + L.start);
  int* so_far = reinterpret_cast<int*>(base + L.so_far);
  double* part = reinterpret_cast<double*>(base + L.part);
  size_t smem = want_sum ? sizeof(double) * (GMM_THREADS / 32) * GMM_MAX_D : 0;
  if (want_obs) {
    smem = std::max(smem, sizeof(double) * (size_t)GMM_SEG_TILE * gmm_seg_pitch(d));
    smem = std::max(smem, sizeof(double) * 16 * (size_t)gmm_obs_groups(d) * gmm_obs_tiles(d));
  }
  const int pts_at = (int)(smem / sizeof(double));   // then the segment's points
  if (const int share = gmm_stats_share(N, d, K)) {
    const int shares = (int)ceil_div(N, share);
    smem += sizeof(int) * (size_t)std::min(N, share);
    const auto gather = d <= 16   ? gmm_segment_kernel<16, true>
                        : d <= 32 ? gmm_segment_kernel<32, true>
                                  : gmm_segment_kernel<64, true>;
    AB_CUDA(allow_smem((const void*)gather, smem));
    gather<<<dim3(K, shares), GMM_THREADS, smem, st>>>(N, d, K, share, want_sum, want_obs, Y, z, mu, nullptr, nullptr, part,
                                                       pts_at, chunk_cnt, cnt, sum, obs);
    AB_LAUNCH_CHECK("gmm_segment_kernel");
    if (shares == 1) return AB_OK;
    gmm_stats_reduce_kernel<<<dim3(std::max(1u, ceil_div(W, 32)), K), GMM_THREADS, 0, st>>>(
        d, K, 0, shares, want_sum, want_obs, part, nullptr, chunk_cnt, 0, 1, so_far, cnt, sum, obs);
    AB_LAUNCH_CHECK("gmm_stats_reduce_kernel");
    return AB_OK;
  }
  smem += sizeof(int) * (size_t)std::max(32, (int)ceil_div(std::min(N, GMM_SLAB), GMM_SEGMENTS));
  const auto segments = d <= 16   ? gmm_segment_kernel<16, false>
                        : d <= 32 ? gmm_segment_kernel<32, false>
                                  : gmm_segment_kernel<64, false>;
  AB_CUDA(allow_smem((const void*)segments, smem));
  for (long long at = 0; at < N; at += GMM_SLAB) {   // 64 bits: past the last slab the offset may not fit 32
    const int n0 = (int)at;
    const int n = std::min(GMM_SLAB, N - n0);
    const int chunks = (int)ceil_div(n, GMM_ORDER_CHUNK);
    const int seg = std::max(32, (int)ceil_div(n, GMM_SEGMENTS));   // at most GMM_SEGMENTS + K segments
    gmm_count_kernel<<<chunks, GMM_THREADS, 0, st>>>(n, K, K, z + n0, chunk_cnt);
    AB_LAUNCH_CHECK("gmm_count_kernel");
    gmm_place_kernel<<<chunks, GMM_THREADS, 0, st>>>(n, K, K, 0, z + n0, chunk_cnt, perm, start);
    AB_LAUNCH_CHECK("gmm_place_kernel");
    if (W > 0) {
      segments<<<ceil_div(n, seg) + K, GMM_THREADS, smem, st>>>(n, d, K, seg, want_sum, want_obs, Y + (size_t)n0 * d,
                                                                z + n0, mu, perm, start, part, pts_at, nullptr, nullptr,
                                                                nullptr, nullptr);
      AB_LAUNCH_CHECK("gmm_segment_kernel");
    }
    gmm_stats_reduce_kernel<<<dim3(std::max(1u, ceil_div(W, 32)), K), GMM_THREADS, 0, st>>>(
        d, K, seg, 0, want_sum, want_obs, part, start, nullptr, n0 > 0, n0 + n == N, so_far, cnt, sum, obs);
    AB_LAUNCH_CHECK("gmm_stats_reduce_kernel");
  }
  return AB_OK;
}

template <int DT>
static int launch_conj_mu_t(int K, int d, int shared, const double* mu0, const double* cov0, const int* cnt,
                            const double* sum, const double* cov, double* mu, uint64_t seed, uint32_t iter,
                            uint32_t comp, cudaStream_t st) {
  const size_t smem = sizeof(double) * (4 * (size_t)d * pitch(d) + 6 * (size_t)d);
  AB_CUDA(allow_smem((const void*)gmm_conj_mu_kernel<DT>, smem));
  gmm_conj_mu_kernel<DT><<<K, GMM_THREADS, smem, st>>>(d, shared, mu0, cov0, cnt, sum, cov, mu, seed, iter, comp);
  AB_LAUNCH_CHECK("gmm_conj_mu_kernel");
  return AB_OK;
}

int launch_gmm_conj_mu(int K, int d, int shared, const double* mu0, const double* cov0, const int* cnt,
                       const double* sum, const double* cov, double* mu, uint64_t seed, uint32_t iter,
                       uint32_t comp, cudaStream_t st) {
#define AB_CALL(DT) launch_conj_mu_t<DT>(K, d, shared, mu0, cov0, cnt, sum, cov, mu, seed, iter, comp, st)
  return AB_GMM_BY_D(d, AB_CALL);
#undef AB_CALL
}

// The Bartlett chi-square sums into chi (chi == nullptr: cov's diagonal).
int launch_gmm_bartlett(int K, int d, int df, const int* cnt, double* chi, double* cov, uint64_t seed,
                        uint32_t iter, uint32_t comp, cudaStream_t st) {
  if (chi != nullptr)
    gmm_bartlett_chi_kernel<<<K * d, GMM_THREADS, 0, st>>>(d, df, cnt, chi, d, 1, seed, iter, comp);
  else
    gmm_bartlett_chi_kernel<<<K * d, GMM_THREADS, 0, st>>>(d, df, cnt, cov, d * d, d + 1, seed, iter, comp);
  AB_LAUNCH_CHECK("gmm_bartlett_chi_kernel");
  return AB_OK;
}

template <int DT>
static int launch_conj_cov_t(int K, int d, int df, const double* scale0, const int* cnt, const double* obs,
                             const double* chi, int sk, int si, double* cov, uint64_t seed, uint32_t iter,
                             uint32_t comp, cudaStream_t st) {
  const size_t smem = sizeof(double) * 4 * (size_t)d * pitch(d);
  AB_CUDA(allow_smem((const void*)gmm_conj_cov_kernel<DT>, smem));
  gmm_conj_cov_kernel<DT><<<K, GMM_THREADS, smem, st>>>(d, df, scale0, cnt, obs, chi, sk, si, cov, seed, iter, comp);
  AB_LAUNCH_CHECK("gmm_conj_cov_kernel");
  return AB_OK;
}

// The inverse-Wishart draw from the chi-square sums in chi (chi == nullptr:
// cov's diagonal).
int launch_gmm_conj_cov_from(int K, int d, int df, const double* scale0, const int* cnt, const double* obs,
                             const double* chi, double* cov, uint64_t seed, uint32_t iter, uint32_t comp,
                             cudaStream_t st) {
  const int sk = chi != nullptr ? d : d * d, si = chi != nullptr ? 1 : d + 1;
  if (chi == nullptr) chi = cov;
#define AB_CALL(DT) launch_conj_cov_t<DT>(K, d, df, scale0, cnt, obs, chi, sk, si, cov, seed, iter, comp, st)
  return AB_GMM_BY_D(d, AB_CALL);
#undef AB_CALL
}

int launch_gmm_conj_cov(int K, int d, int df, const double* scale0, const int* cnt, const double* obs,
                        double* cov, uint64_t seed, uint32_t iter, uint32_t comp, cudaStream_t st) {
  int rc = launch_gmm_bartlett(K, d, df, cnt, nullptr, cov, seed, iter, comp, st);
  if (rc) return rc;
  return launch_gmm_conj_cov_from(K, d, df, scale0, cnt, obs, nullptr, cov, seed, iter, comp, st);
}

template <int DT, bool SLICE>
static int launch_move_t(int N, int d, int K, int shared, const float* Y, const int* z, const double* mu0,
                         const double* cov, const double* Linv, const double* hdet, int prior_slot, int prop_slot,
                         int compat, double* mu, uint64_t seed, uint32_t iter, uint32_t comp, int* tally,
                         cudaStream_t st) {
  const size_t tables = sizeof(double) * 3 * (size_t)d * pitch(d);
  const size_t sums = (GMM_THREADS / 32) * (sizeof(double) * GMM_MAX_D + sizeof(int) * GMM_MOVE_BATCH);
  const size_t smem = std::max(tables, sums);
  AB_CUDA(allow_smem((const void*)gmm_move_kernel<DT, SLICE>, smem));
  gmm_move_kernel<DT, SLICE><<<K * GMM_MOVE_CLUSTER, GMM_THREADS, smem, st>>>(
      N, d, shared, Y, z, mu0, cov, Linv, hdet, prior_slot, prop_slot, compat, mu, seed, iter, comp, tally);
  AB_LAUNCH_CHECK("gmm_move_kernel");
  return AB_OK;
}

int launch_gmm_move(bool slice, int N, int d, int K, int shared, const float* Y, const int* z, const double* mu0,
                    const double* cov, const double* Linv, const double* hdet, int prior_slot, int prop_slot,
                    int compat, double* mu, uint64_t seed, uint32_t iter, uint32_t comp, int* tally, cudaStream_t st) {
#define AB_CALL(DT)                                                                                              \
  (slice ? launch_move_t<DT, true>(N, d, K, shared, Y, z, mu0, cov, Linv, hdet, prior_slot, prop_slot, compat, mu, \
                                   seed, iter, comp, tally, st)                                                  \
         : launch_move_t<DT, false>(N, d, K, shared, Y, z, mu0, cov, Linv, hdet, prior_slot, prop_slot, compat,  \
                                    mu, seed, iter, comp, tally, st))
  return AB_GMM_BY_D(d, AB_CALL);
#undef AB_CALL
}

}  // namespace ab

using namespace ab;

// ------------------------------- C ABI ----------------------------------------------

extern "C" size_t ab_gmm_table_doubles(int Kc, int d) { return (size_t)Kc * d * d + (size_t)Kc; }

extern "C" int ab_gmm_prep(int Kc, int d, const double* cov, double* Linv, double* hdet, void* stream) {
  AB_REQUIRE(Kc > 0 && d > 0 && d <= GMM_MAX_D, AB_ERR_ARG, "ab_gmm_prep: bad sizes");
  AB_REQUIRE(cov && Linv && hdet, AB_ERR_ARG, "ab_gmm_prep: null pointer");
  return launch_gmm_prep(Kc, d, cov, Linv, hdet, as_stream(stream));
}

extern "C" size_t ab_gmm_z_scratch_bytes(int N, int d, int K) {
  if (N <= 0 || d <= 0 || K <= 0) return 0;
  return gmm_zs_scratch(N, d, K);
}

extern "C" size_t ab_gmm_z_queue_offset(int d, int K) {
  if (d <= 0 || K <= 0) return 0;
  return gmm_al256(gmm_zs_smem(d, K)) + sizeof(int);
}

extern "C" int ab_gmm_disc_z_screened(int N, int d, int K, int shared_cov, const float* Y, const double* pis,
                                      const double* mu, const double* Linv, const double* hdet, int* z,
                                      uint64_t seed, uint32_t iter, uint32_t comp, void* scratch, void* stream) {
  int rc = gmm_check(N, d, K);
  if (rc) return rc;
  AB_REQUIRE(Y && pis && mu && Linv && hdet && z && scratch, AB_ERR_ARG, "ab_gmm_disc_z_screened: null pointer");
  AB_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 255) == 0, AB_ERR_ARG,
             "ab_gmm_disc_z_screened: scratch must be 256-byte aligned");
  return launch_gmm_z_screened(N, d, K, shared_cov, Y, pis, mu, Linv, hdet, z, seed, iter, comp, scratch,
                               as_stream(stream));
}

extern "C" int ab_gmm_disc_z(int N, int d, int K, int shared_cov, const float* Y, const double* pis,
                             const double* mu, const double* Linv, const double* hdet, int* z, uint64_t seed,
                             uint32_t iter, uint32_t comp, void* stream) {
  int rc = gmm_check(N, d, K);
  if (rc) return rc;
  AB_REQUIRE(Y && pis && mu && Linv && hdet && z, AB_ERR_ARG, "ab_gmm_disc_z: null pointer");
  return launch_gmm_z(N, d, K, shared_cov, Y, pis, mu, Linv, hdet, z, seed, iter, comp, as_stream(stream));
}

extern "C" size_t ab_gmm_stats_scratch_bytes(int d, int K) { return gmm_stats_scratch(d, K); }

extern "C" int ab_gmm_stats(int N, int d, int K, const float* Y, const int* z, const double* mu, int* cnt,
                            double* sum, double* obs, void* scratch, void* stream) {
  int rc = gmm_check(N, d, K);
  if (rc) return rc;
  AB_REQUIRE(Y && z && cnt && scratch, AB_ERR_ARG, "ab_gmm_stats: null pointer");
  AB_REQUIRE(!obs || mu, AB_ERR_ARG, "ab_gmm_stats: the scatter matrices need mu");
  return launch_gmm_stats(N, d, K, Y, z, mu, sum != nullptr, obs != nullptr, cnt, sum, obs,
                          scratch, as_stream(stream));
}

extern "C" int ab_gmm_conj_pis(int K, const double* alpha, const int* cnt, double* pis, uint64_t seed,
                               uint32_t iter, uint32_t comp, void* stream) {
  AB_REQUIRE(K > 0 && K <= GMM_MAX_K, AB_ERR_ARG, "ab_gmm_conj_pis: bad K");
  AB_REQUIRE(alpha && cnt && pis, AB_ERR_ARG, "ab_gmm_conj_pis: null pointer");
  gmm_conj_pis_kernel<<<1, 64, 0, as_stream(stream)>>>(K, alpha, cnt, pis, seed, iter, comp);
  AB_LAUNCH_CHECK("gmm_conj_pis_kernel");
  return AB_OK;
}

extern "C" int ab_gmm_conj_mu(int K, int d, int shared_cov, const double* mu0, const double* cov0, const int* cnt,
                              const double* sum, const double* cov, double* mu, uint64_t seed, uint32_t iter,
                              uint32_t comp, void* stream) {
  AB_REQUIRE(K > 0 && K <= GMM_MAX_K && d > 0 && d <= GMM_MAX_D, AB_ERR_ARG, "ab_gmm_conj_mu: bad sizes");
  AB_REQUIRE(mu0 && cov0 && cnt && sum && cov && mu, AB_ERR_ARG, "ab_gmm_conj_mu: null pointer");
  return launch_gmm_conj_mu(K, d, shared_cov, mu0, cov0, cnt, sum, cov, mu, seed, iter, comp, as_stream(stream));
}

extern "C" int ab_gmm_conj_cov(int K, int d, int df, const double* scale0, const int* cnt, const double* obs,
                               double* cov, uint64_t seed, uint32_t iter, uint32_t comp, void* stream) {
  AB_REQUIRE(K > 0 && K <= GMM_MAX_K && d > 0 && d <= GMM_MAX_D, AB_ERR_ARG, "ab_gmm_conj_cov: bad sizes");
  AB_REQUIRE(df > 0 && df < 100000, AB_ERR_ARG, "ab_gmm_conj_cov: bad degrees of freedom");
  AB_REQUIRE(scale0 && cnt && obs && cov, AB_ERR_ARG, "ab_gmm_conj_cov: null pointer");
  return launch_gmm_conj_cov(K, d, df, scale0, cnt, obs, cov, seed, iter, comp, as_stream(stream));
}

extern "C" int ab_gmm_bartlett(int K, int d, int df, const int* cnt, double* chi, uint64_t seed, uint32_t iter,
                               uint32_t comp, void* stream) {
  AB_REQUIRE(K > 0 && K <= GMM_MAX_K && d > 0 && d <= GMM_MAX_D, AB_ERR_ARG, "ab_gmm_bartlett: bad sizes");
  AB_REQUIRE(df > 0 && df < 100000, AB_ERR_ARG, "ab_gmm_bartlett: bad degrees of freedom");
  AB_REQUIRE(cnt && chi, AB_ERR_ARG, "ab_gmm_bartlett: null pointer");
  return launch_gmm_bartlett(K, d, df, cnt, chi, nullptr, seed, iter, comp, as_stream(stream));
}

extern "C" int ab_gmm_conj_cov_chi(int K, int d, int df, const double* scale0, const int* cnt, const double* obs,
                                   const double* chi, double* cov, uint64_t seed, uint32_t iter, uint32_t comp,
                                   void* stream) {
  AB_REQUIRE(K > 0 && K <= GMM_MAX_K && d > 0 && d <= GMM_MAX_D, AB_ERR_ARG, "ab_gmm_conj_cov_chi: bad sizes");
  AB_REQUIRE(df > 0 && df < 100000, AB_ERR_ARG, "ab_gmm_conj_cov_chi: bad degrees of freedom");
  AB_REQUIRE(scale0 && cnt && obs && chi && cov, AB_ERR_ARG, "ab_gmm_conj_cov_chi: null pointer");
  return launch_gmm_conj_cov_from(K, d, df, scale0, cnt, obs, chi, cov, seed, iter, comp, as_stream(stream));
}

extern "C" int ab_gmm_eslice(int N, int d, int K, int shared_cov, const float* Y, const int* z, const double* mu0,
                             const double* cov0, const double* Linv, const double* hdet, int prior_slot,
                             double* mu, uint64_t seed, uint32_t iter, uint32_t comp, int* shrinks,
                             void* stream) {
  int rc = gmm_check(N, d, K);
  if (rc) return rc;
  AB_REQUIRE(Y && z && mu0 && cov0 && Linv && hdet && mu && shrinks, AB_ERR_ARG, "ab_gmm_eslice: null pointer");
  return launch_gmm_move(true, N, d, K, shared_cov, Y, z, mu0, cov0, Linv, hdet, prior_slot, 0, 0, mu, seed, iter, comp,
                         shrinks, as_stream(stream));
}

extern "C" int ab_gmm_mwg(int N, int d, int K, int shared_cov, const float* Y, const int* z, const double* mu0,
                          const double* covp, const double* Linv, const double* hdet, int prior_slot,
                          int prop_slot, int compat, double* mu, uint64_t seed, uint32_t iter, uint32_t comp,
                          int* accepts, void* stream) {
  int rc = gmm_check(N, d, K);
  if (rc) return rc;
  AB_REQUIRE(Y && z && mu0 && covp && Linv && hdet && mu && accepts, AB_ERR_ARG, "ab_gmm_mwg: null pointer");
  return launch_gmm_move(false, N, d, K, shared_cov, Y, z, mu0, covp, Linv, hdet, prior_slot, prop_slot, compat, mu, seed,
                         iter, comp, accepts, as_stream(stream));
}
