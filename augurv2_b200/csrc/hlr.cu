// Hierarchical logistic regression: log-density and gradient over the data,
// and the HMC / NUTS / MWG transitions that consume them.
//
// Model (compiler/augur/test/hlr.rv, and its InvGamma-variance variant
// without the bias):
//   v ~ Exponential(lam) | InvGamma(a0, s0);  b ~ Normal(0, v)  (optional)
//   theta[k] ~ Normal(0, v);  y[n] ~ Bernoulli(sigmoid(theta . x[n] + b))
// Parameters of a chain are one binary64 vector par = [theta[0..D-1], b, v];
// a block (the unit an HMC / NUTS kernel moves) is a list of indices into par
// in the schedule's order.
//
// Data layout in HBM: X row-major [N][ldx] (f32 or bf16), y int32 [N],
// par f64 [C][D+2].
//
// Engine: one CTA per chain runs whole iterations of the schedule on chip
// (hlr_chain_kernel), with X in shared memory where it fits.  A data pass
// computes, at the chain's current theta and b, ll_data = sum_n log Bern(y_n | sigmoid(t_n)) and its gradient
//   d/dtheta_k = sum_n r_n x_nk,  d/db = sum_n r_n,  r_n = y_n - sigmoid(t_n)
// in FP32 per row (numerically stable logistic terms), with Kahan-compensated
// per-thread sums and fixed-order FP64 block reductions, so the result is
// deterministic.  Priors, momenta, energies and the accept tests are binary64
// in the reference's operation order (cbits/augur_dist.c, augur_mcmclib.h).
#include <cuda_bf16.h>
#include <math.h>

#include "common.cuh"
#include "philox.cuh"

namespace ab {

constexpr int HLR_THREADS = 256;         // threads that walk the rows: each row's place in the compensated sums
constexpr int HLR_BLOCK = HLR_THREADS + 32;   // and, in the chain kernel, a warp for the prior and, past D = 30, the
                                              // log-likelihood sums (otherwise the last of the row threads' warps)
constexpr int HLR_CHUNK = 1024;          // rows per data-pass chunk (r buffer)
constexpr int HLR_MAX_COLS = 4;          // columns per thread in the gradient pass
constexpr int HLR_MAX_D = HLR_THREADS * HLR_MAX_COLS - 1;
constexpr int HLR_STK = 16;              // NUTS stack entries (cbits/augur_blkstk.h:26)
constexpr int HLR_MAX_COMPS = 8;

enum { COMP_HMC = 0, COMP_NUTS = 1, COMP_MWG = 2, COMP_RSLICE = 3 };

struct HlrModelDev {
  int N, D, ldx, has_b, vprior, compat, x_bf16;
  double lam, a0, s0;
  const void* X;
  const int* y;
  int lik;              // AB_LIK_*
  float inv_var;        // AB_LIK_NORMAL: 1 / obs_var
  double ll_add;        // AB_LIK_NORMAL: N times the per-row normaliser, added once
  double vp_const;      // the variance prior's normaliser: log(lam), or a0 log(s0) - lgamma(a0)
  const float* yr;
};

struct HlrComp {
  int kind, P, idx_off, max_depth;
  double simlen, eps, mwg_var;
};

__device__ __forceinline__ void kahan_add(float& s, float& c, float x) {
  const float yv = x - c;
  const float t = s + yv;
  c = (t - s) - yv;
  s = t;
}

// Stable log Bern(y | sigmoid(t)) and its derivative, FP32.
__device__ __forceinline__ void bern_terms(bool want_ll, int y, float t, float& ll, float& r) {
  if (want_ll) {
    const float sp = fmaxf(t, 0.0f) + log1pf(__expf(-fabsf(t)));
    ll = y ? t - sp : -sp;
  }
  const float sg = 1.0f / (1.0f + __expf(-t));
  r = (float)y - sg;
}

// Data factor of a row at t (if wanted) and its derivative in t, FP32: the logistic terms above, Poisson(exp(t)): y t - exp(t) -
// lgamma(y + 1) and y - exp(t) (the reference's y log(rate) - rate -
// sum_{k <= y} log k and its adjoint through exp), Normal(t, obs_var):
// -(y - t)^2 / (2 var) and (y - t) / var (the normaliser is added once per
// pass, ll_add).  lab: the row's label, as the bits of y or yr.
__device__ __forceinline__ void lik_terms(const HlrModelDev& m, bool want_ll, int lab, float t, float& ll, float& r) {
  if (m.lik == AB_LIK_POISSON) {
    const float rate = expf(t);
    if (want_ll) ll = (float)lab * t - rate - lgammaf((float)lab + 1.0f);
    r = (float)lab - rate;
  } else if (m.lik == AB_LIK_NORMAL) {
    const float d = __int_as_float(lab) - t;
    if (want_ll) ll = -0.5f * d * d * m.inv_var;
    r = d * m.inv_var;
  } else {
    bern_terms(want_ll, lab, t, ll, r);
  }
}

__device__ __forceinline__ int load_label(const HlrModelDev& m, int n) {
  return m.lik == AB_LIK_NORMAL ? __float_as_int(m.yr[n]) : m.y[n];
}

// Shared-memory workspace of one chain CTA (sizes fixed by D).
struct Ws {
  double* par;     // [D+2]  current state
  double* prop;    // [D+2]  proposal state
  double* g;       // [D+1]  data gradient (theta..., b)
  double* blk_g;   // [D+2]  block gradient, block order
  double* p0;      // [D+2]  momentum at start
  double* ps;      // [D+2]  momentum working
  double* q;       // [D+2]  block position working
  double* aux1;    // [D+2]  spare (NUTS frontiers)
  double* aux2;    // [D+2]
  double* aux3;    // [D+2]
  double* aux4;    // [D+2]
  double* gpart;   // [HLR_THREADS] per-thread partials (double)
  float* th;       // [D]    theta in FP32 for the data pass
  float* r;        // [HLR_CHUNK] residuals of a chunk of rows
  float* l;        // [HLR_CHUNK] their log-likelihood terms
  double* red;     // [34]
  double* bcast;   // [8]   broadcast slots
  int* ibcast;     // [8]
  int* idx;        // [D+2]  block indices of the running component
  double* gfr;     // [3][P] NUTS: gradients at both frontiers and at the walk's position
  // the copy of X in shared memory, float or bf16 (null: it stays in global
  // memory), and of the labels
  void* xs;
  int* lab;
  int xpitch;
};

// Which parameters a block moves.
struct BlockInfo {
  bool th, b, v;
};

// Small-D pass widths: D gradient columns, the bias column, the
// log-likelihood; 16 columns for D + 2 <= 16, else 32.
constexpr int SMALL_COLS = 32;

// Sum over the warp's lanes of each of COLS per-lane values, transposed: on
// return v[0] of lane L holds the warp sum of column L % COLS (fixed
// butterfly order, so deterministic; COLS - 1 shuffles, plus one more round
// folding the two half-warps when COLS = 16).
template <int COLS>
__device__ __forceinline__ void warp_transpose_sum(double (&v)[COLS], int lane) {
#pragma unroll
  for (int sft = COLS / 2; sft >= 1; sft >>= 1) {
    const bool up = (lane & sft) != 0;
#pragma unroll
    for (int i = 0; i < sft; ++i) {
      const double send = up ? v[i] : v[i + sft];
      const double keep = up ? v[i + sft] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, sft);
    }
  }
  if (COLS == 16) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
}

// Where the rows are read: the shared copy in X's type, or global memory (the
// data passes then take X's type as a template argument too, G_F32 or G_BF16:
// a test of it at every load kept the loads of a row from being in flight
// together; with row_dot's groups, 20,000 rows of D = 20 176 -> 87 us).
enum { X_GLOBAL = 0, X_F32 = 1, X_BF16 = 2, G_F32 = 3, G_BF16 = 4 };
__host__ __device__ constexpr bool in_shared(int res) { return res == X_F32 || res == X_BF16; }
template <int RES>
__device__ __forceinline__ float row_x(const HlrModelDev& m, const Ws& ws, int i, int k) {
  if (RES == X_F32) return static_cast<const float*>(ws.xs)[i * ws.xpitch + k];
  if (RES == X_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(ws.xs)[i * ws.xpitch + k]);
  const size_t at = (size_t)i * m.ldx + k;
  if (RES == G_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(m.X)[at]);
  return __ldg(static_cast<const float*>(m.X) + at);
}
template <int RES>
__device__ __forceinline__ int row_label(const HlrModelDev& m, const Ws& ws, int i) {
  return in_shared(RES) ? ws.lab[i] : load_label(m, i);
}

// Data pass for D + 2 <= COLS: one row per thread (t, the log-likelihood term
// and the residual's contributions to all D + 1 gradient columns in
// registers, Kahan-compensated), then one transposed warp reduction and a
// fixed-order sum over the warps, all in FP64: the row-per-thread walk keeps
// every thread busy at small N.  By the row threads; leaves the sums in ws.g and
// ws.red[33].
// A row's values (zeros past D) and their dot product with th.  From global
// memory eight at a time without a test between them, so that they are issued
// together.
template <int RES, int K>
__device__ __forceinline__ float row_dot(const HlrModelDev& m, const Ws& ws, int i, const float (&th)[K], float (&x)[K]) {
  const int D = m.D;
#pragma unroll
  for (int k0 = 0; k0 < K; k0 += 8) {
    const bool whole = !in_shared(RES) && k0 + 8 <= K && k0 + 8 <= D;
    if (whole) {
#pragma unroll
      for (int k = k0; k < k0 + 8 && k < K; ++k) x[k] = row_x<RES>(m, ws, i, k);
    } else {
#pragma unroll
      for (int k = k0; k < k0 + 8 && k < K; ++k) x[k] = k < D ? row_x<RES>(m, ws, i, k) : 0.0f;
    }
  }
  float t = 0.0f;
#pragma unroll
  for (int k = 0; k < K; ++k) t += x[k] * th[k];
  return t;
}

template <int COLS, int RES>
__device__ __forceinline__ void data_rows_small(const HlrModelDev& m, bool want_ll, bool want_grad, float bias, const Ws& ws) {
  const int D = m.D;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < HLR_THREADS) {
    float th[COLS - 2];
#pragma unroll
    for (int k = 0; k < COLS - 2; ++k) th[k] = k < D ? ws.th[k] : 0.0f;
    double v[COLS];
    if (!want_grad) {
      // two rows in flight, which the gradient's sums leave no registers for
      float ls = 0.0f, lc = 0.0f;
#pragma unroll 1
      for (int i = tid; i < m.N; i += 2 * HLR_THREADS) {
        const int i1 = min(i + HLR_THREADS, m.N - 1);
        float x0[COLS - 2], x1[COLS - 2];
        const float t0 = row_dot<RES>(m, ws, i, th, x0), t1 = row_dot<RES>(m, ws, i1, th, x1);
        const int y0 = row_label<RES>(m, ws, i), y1 = row_label<RES>(m, ws, i1);
        float l0, l1, rv;
        lik_terms(m, true, y0, t0 + bias, l0, rv);
        lik_terms(m, true, y1, t1 + bias, l1, rv);
        kahan_add(ls, lc, l0);
        if (i + HLR_THREADS < m.N) kahan_add(ls, lc, l1);
      }
#pragma unroll
      for (int j = 0; j < COLS - 1; ++j) v[j] = 0.0;
      v[COLS - 1] = (double)ls - (double)lc;
    } else {
      float s[COLS], c[COLS];
#pragma unroll
      for (int j = 0; j < COLS; ++j) { s[j] = 0.0f; c[j] = 0.0f; }
#pragma unroll 1
      for (int i = tid; i < m.N; i += HLR_THREADS) {
        float x[COLS - 2];
        const float t = row_dot<RES>(m, ws, i, th, x);
        float llv, rv;
        lik_terms(m, want_ll, row_label<RES>(m, ws, i), t + bias, llv, rv);
        if (want_ll) kahan_add(s[COLS - 1], c[COLS - 1], llv);
#pragma unroll
        for (int k = 0; k < COLS - 2; ++k)
          if (k < D) kahan_add(s[k], c[k], rv * x[k]);
#pragma unroll
        for (int k = 0; k < COLS - 1; ++k)
          if (k == D) kahan_add(s[k], c[k], rv);
      }
#pragma unroll
      for (int j = 0; j < COLS; ++j) v[j] = (double)s[j] - (double)c[j];
    }
    warp_transpose_sum<COLS>(v, lane);
    if (lane < COLS) ws.gpart[warp * COLS + lane] = v[0];
  }
  __syncthreads();
  if (tid < COLS) {
    constexpr int NW = HLR_THREADS / 32;
    double a[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) a[w] = ws.gpart[w * COLS + tid];
    const double acc = ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
    if (tid == COLS - 1) ws.red[33] = acc;
    else if (tid <= D) ws.g[tid] = acc;
  }
}

// Data pass for wider D, a chunk of rows at a time: the rows' dot products (X
// in shared memory: a row per thread, its 32 interleaved partial sums in
// registers and added as the warp tree of the global-memory walk adds them;
// otherwise a warp per row) and their terms; then the row threads, owners of
// gradient columns, walk the chunk's residuals, while eight lanes of the last
// warp walk its log-likelihood terms.
template <int RES, int BLOCK>
__device__ __forceinline__ void data_rows_wide(const HlrModelDev& m, bool want_ll, bool want_grad, float bias, const Ws& ws) {
  constexpr int NW = HLR_THREADS / 32, LAST = BLOCK / 32 - 1;
  const int D = m.D, N = m.N;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // gradient accumulators: thread owns columns c = tid + i*HLR_THREADS (cols
  // D+1 including the bias column) for rows n = grp (mod ngrp)
  const int ncol = D + 1;
  const int ngrp = ncol >= HLR_THREADS ? 1 : HLR_THREADS / ncol;
  const int grp = ncol >= HLR_THREADS ? 0 : tid / ncol;
  const int col0 = ncol >= HLR_THREADS ? tid : tid % ncol;
  const bool gactive = tid < HLR_THREADS && grp < ngrp;
  float gs[HLR_MAX_COLS], gc[HLR_MAX_COLS];
#pragma unroll
  for (int i = 0; i < HLR_MAX_COLS; ++i) { gs[i] = 0.0f; gc[i] = 0.0f; }
  float lls = 0.0f, llc = 0.0f;   // log-likelihood terms of rows = lane (mod NW), lanes below NW of the last warp
  for (int n0 = 0; n0 < N; n0 += HLR_CHUNK) {
    const int nc = min(HLR_CHUNK, N - n0);
    if (in_shared(RES)) {
      for (int i = tid; i < nc; i += BLOCK) {
        float p[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) p[q] = 0.0f;
        for (int k0 = 0; k0 < D; k0 += 32) {
#pragma unroll
          for (int q = 0; q < 32; ++q)
            if (k0 + q < D) p[q] += row_x<RES>(m, ws, n0 + i, k0 + q) * ws.th[k0 + q];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int q = 0; q < o; ++q) p[q] += p[q + o];
        float llv, rv;
        lik_terms(m, want_ll, ws.lab[n0 + i], p[0] + bias, llv, rv);
        if (want_ll) ws.l[i] = llv;
        ws.r[i] = rv;
      }
    } else if (warp < NW) {
      // eight rows of a warp at a time; the transposed reduction adds each
      // row's 32 partial sums in the tree of a full one (lanes i and i ^ 16, ...)
      for (int i0 = warp * 8; i0 < nc; i0 += NW * 8) {
        float part[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) part[r] = 0.0f;
        for (int k = lane; k < D; k += 32) {
          const float tk = ws.th[k];
#pragma unroll
          for (int r = 0; r < 8; ++r) part[r] += row_x<RES>(m, ws, n0 + min(i0 + r, nc - 1), k) * tk;
        }
#pragma unroll
        for (int o = 16, h = 4; h > 0; o >>= 1, h >>= 1) {
          const bool up = (lane & o) != 0;
#pragma unroll
          for (int r = 0; r < h; ++r) {
            const float send = up ? part[r] : part[r + h], keep = up ? part[r + h] : part[r];
            part[r] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
        }
        part[0] += __shfl_xor_sync(0xffffffffu, part[0], 2);
        part[0] += __shfl_xor_sync(0xffffffffu, part[0], 1);
        const int i = i0 + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
        if ((lane & 3) == 0 && i < nc) {
          float llv, rv;
          lik_terms(m, want_ll, row_label<RES>(m, ws, n0 + i), part[0] + bias, llv, rv);
          if (want_ll) ws.l[i] = llv;
          ws.r[i] = rv;
        }
      }
    }
    __syncthreads();
    if (want_grad && gactive) {
      if (ncol < HLR_THREADS) {
        if (col0 < D) {
          // eight rows' values in flight, added in row order
          for (int i = grp; i < nc; i += 8 * ngrp) {
            float xv[8], rv[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const int ii = min(i + q * ngrp, nc - 1);
              xv[q] = row_x<RES>(m, ws, n0 + ii, col0);
              rv[q] = ws.r[ii];
            }
#pragma unroll
            for (int q = 0; q < 8; ++q)
              if (i + q * ngrp < nc) kahan_add(gs[0], gc[0], rv[q] * xv[q]);
          }
        } else {
#pragma unroll 4
          for (int i = grp; i < nc; i += ngrp) kahan_add(gs[0], gc[0], ws.r[i]);
        }
      } else {
        for (int i = 0; i < nc; ++i) {
          const float rv = ws.r[i];
#pragma unroll
          for (int j = 0; j < HLR_MAX_COLS; ++j) {
            const int c = col0 + j * HLR_THREADS;
            if (c < D) kahan_add(gs[j], gc[j], rv * row_x<RES>(m, ws, n0 + i, c));
            else if (c == D) kahan_add(gs[j], gc[j], rv);
          }
        }
      }
    }
    if (want_ll && warp == LAST && lane < NW) {
#pragma unroll 4
      for (int i = lane; i < nc; i += NW) kahan_add(lls, llc, ws.l[i]);
    }
    if (n0 + HLR_CHUNK < N) __syncthreads();
  }
  if (want_ll && warp == LAST) {
    const double v = warp_sum_f64((double)lls - (double)llc);
    if (lane == 0) ws.red[33] = v;
  }
  if (want_grad) {
    if (ncol >= HLR_THREADS) {
      for (int j = 0; j < HLR_MAX_COLS; ++j)
        if (gactive && col0 + j * HLR_THREADS < ncol) ws.g[col0 + j * HLR_THREADS] = (double)gs[j] - (double)gc[j];
    } else {
      // combine the groups column by column in a fixed order
      if (tid < HLR_THREADS) ws.gpart[tid] = gactive ? (double)gs[0] - (double)gc[0] : 0.0;
      __syncthreads();
      if (tid < ncol) {
        double acc = 0.0;
#pragma unroll 4
        for (int q = 0; q < ngrp; ++q) acc += ws.gpart[q * ncol + tid];
        ws.g[tid] = acc;
      }
    }
  }
}

template <int COLS, int RES, int BLOCK>
__device__ __forceinline__ void data_rows(const HlrModelDev& m, bool want_ll, bool want_grad, float bias, const Ws& ws) {
  if constexpr (COLS > 0) data_rows_small<COLS, RES>(m, want_ll, want_grad, bias, ws);
  else data_rows_wide<RES, BLOCK>(m, want_ll, want_grad, bias, ws);
}

// ---- priors (binary64; reference formulas when compat) ----------------------
__device__ __forceinline__ double normal_ll(const HlrModelDev& m, double pt, double mean, double var) {
  const double t = pt - mean;
  if (m.compat) return var > 0.0 ? (-log(var)) - (0.5 * t * t / var) : -1e8;
  if (!(var > 0.0)) return -INFINITY;
  return -0.5 * log(2.0 * 3.14159265358979323846 * var) - 0.5 * t * t / var;
}
// d/dvar of the former at mean 0, iv = 1 / var, whose square may be out of range.
__device__ __forceinline__ double normal_dvar(const HlrModelDev& m, double t, double var, double iv) {
  const double ti = t * iv;
  return (m.compat ? -0.5 * var : -0.5 * iv) + 0.5 * (ti * ti);
}
__device__ __forceinline__ double vprior_ll(const HlrModelDev& m, double v) {
  if (m.vprior == 0) return (m.lam > 0.0 && v > 0.0) ? m.vp_const - m.lam * v : (m.compat ? -1e8 : -INFINITY);
  if (!(v > 0.0)) return m.compat ? -1e8 : -INFINITY;
  return m.vp_const - (m.a0 + 1.0) * log(v) - m.s0 / v;
}
__device__ __forceinline__ double vprior_dot(const HlrModelDev& m, double v, double iv) {
  if (m.vprior == 0) return (m.lam > 0.0 && v > 0.0) ? -m.lam : 0.0;
  return -(m.a0 + 1.0) * iv + (m.s0 * iv) * iv;
}

__device__ __forceinline__ BlockInfo block_info(const HlrModelDev& m, const int* idx, int P) {
  BlockInfo bi{false, false, false};
  for (int j = 0; j < P; ++j) {
    const int i = idx[j];
    if (i < m.D) bi.th = true;
    else if (i == m.D) bi.b = m.has_b != 0;
    else bi.v = true;
  }
  return bi;
}

// Full conditional of the block at `par` (returned if wanted) and its
// gradient, if wanted, in block order into ws.blk_g.  Factor order as the
// generated ll_/grad_ functions (CgLike.hs:139-147, CgGrad.hs:165-376); the
// coefficients' prior terms are added in a fixed tree.  The last warp forms the
// prior - its logarithm and the shared 1 / v are the longest chains of binary64
// operations of an evaluation - while the row threads pass over the data.
// COLS: the data pass, 16 or 32 columns of the row-per-thread one, or 0 for the
// wide one.
template <int RES, int COLS, int BLOCK = HLR_BLOCK>
__device__ __forceinline__ double block_eval(const HlrModelDev& m, bool want_ll, bool want_grad, const double* par,
                                          const BlockInfo bi, int P, Ws& ws) {
  const int D = m.D, tid = threadIdx.x, lane = tid & 31;
  const bool data = bi.th || bi.b;
  const double v = par[D + 1];
  if (data)
    for (int k = tid; k < D; k += BLOCK) ws.th[k] = (float)par[k];
  const float bias = m.has_b ? (float)par[D] : 0.0f;
  const double iv = 1.0 / v;
  __syncthreads();
  if ((tid >= BLOCK - 32 || !data) && (want_ll || bi.v)) {
    // the prior: lanes take the coefficients (of all warps if none passes over
    // the data), lane 0 of the last warp the variance and the bias
    double pl = 0.0, pd = 0.0;
    if (bi.th || bi.v)
      for (int k = data ? lane : tid; k < D; k += data ? 32 : BLOCK) {
        if (want_ll) pl += normal_ll(m, par[k], 0.0, v);
        if (bi.v) pd += normal_dvar(m, par[k], v, iv);
      }
    if (want_ll) pl = warp_sum_f64(pl);
    if (bi.v) pd = warp_sum_f64(pd);
    if (!data) {
      constexpr int NW = BLOCK / 32;
      if (lane == 0) {
        ws.gpart[tid >> 5] = pl;
        ws.gpart[NW + (tid >> 5)] = pd;
      }
      __syncthreads();
      pl = pd = 0.0;
      for (int w = 0; w < NW; ++w) {
        pl += ws.gpart[w];
        pd += ws.gpart[NW + w];
      }
    }
    if (tid == BLOCK - 32) {
      double ll = 0.0, gv = 0.0;
      if (bi.v) {
        if (want_ll) ll += vprior_ll(m, v);
        gv += vprior_dot(m, v, iv);
      }
      if (m.has_b && (bi.b || bi.v)) {
        if (want_ll) ll += normal_ll(m, par[D], 0.0, v);
        if (bi.v) gv += normal_dvar(m, par[D], v, iv);
      }
      ws.bcast[0] = ll + pl;
      ws.bcast[1] = gv + pd;
    }
  }
  if (data) {
    if constexpr (RES != X_GLOBAL) data_rows<COLS, RES, BLOCK>(m, want_ll, want_grad, bias, ws);
    else if (m.x_bf16) data_rows<COLS, G_BF16, BLOCK>(m, want_ll, want_grad, bias, ws);
    else data_rows<COLS, G_F32, BLOCK>(m, want_ll, want_grad, bias, ws);
  }
  __syncthreads();
  if (want_grad) {
    for (int j = tid; j < P; j += BLOCK) {
      const int i = ws.idx[j];
      ws.blk_g[j] = i < D ? -par[i] * iv + ws.g[i] : i == D ? (m.has_b ? -par[D] * iv + ws.g[D] : 0.0) : ws.bcast[1];
    }
  }
  const double ll = want_ll ? ws.bcast[0] + (data ? ws.red[33] + m.ll_add : 0.0) : 0.0;
  __syncthreads();
  return ll;
}

__device__ __forceinline__ void set_block(double* par, const int* idx, int P, const double* q) {
  for (int j = threadIdx.x; j < P; j += blockDim.x) par[idx[j]] = q[j];
  __syncthreads();
}

// The running component's block indices, next to the other state.
__device__ __forceinline__ BlockInfo stage_block(const HlrModelDev& m, const int* idx, int P, Ws& ws) {
  __syncthreads();
  for (int j = threadIdx.x; j < P; j += blockDim.x) ws.idx[j] = idx[j];
  __syncthreads();
  return block_info(m, ws.idx, P);
}

// Binary64 dot product, by the first warp in a fixed tree, broadcast.
__device__ double block_dot(const double* a, const double* b, int P, Ws& ws) {
  if (threadIdx.x < 32) {
    double acc = 0.0;
    for (int j = threadIdx.x; j < P; j += 32) acc += a[j] * b[j];
    acc = warp_sum_f64(acc);
    if (threadIdx.x == 0) ws.bcast[2] = acc;
  }
  __syncthreads();
  const double r = ws.bcast[2];
  __syncthreads();
  return r;
}

// ---- HMC: cbits/augur_mcmclib.h:343-424 -------------------------------------
// `known`: ws.aux1 and *ll_known hold the block gradient and log density at
// the current state (left there by the previous iteration of a schedule whose
// only component this is); on return they hold the new state's.
template <int RES, int COLS>
__device__ int hmc_transition(const HlrModelDev& m, const HlrComp& cp, const BlockInfo bi, Ws& ws, uint64_t seed,
                              uint32_t iter, uint32_t chain, uint32_t ci, bool known, double* ll_known) {
  const int P = cp.P;
  const int tid = threadIdx.x;
  const int* idx = ws.idx;
  for (int j = tid; j < P; j += blockDim.x) {
    Stream s = make_stream(seed, chain * (uint32_t)P + j, iter, TAG_MOM | (ci << 8));
    ws.p0[j] = s.normal();
  }
  if (tid == HLR_THREADS) {
    Stream h = make_stream(seed, chain, iter, TAG_HMC | (ci << 8));
    const double scale_eps = 0.8 + h.uniform() * (1.2 - 0.8);
    const double stepsize = scale_eps * cp.eps;
    const double sj = 0.9 + h.uniform() * (1.1 - 0.9);
    const unsigned rl = (unsigned)round(sj * cp.simlen / stepsize);
    ws.bcast[3] = stepsize;
    ws.ibcast[0] = (int)min(rl > 1u ? rl : 1u, 1u << 20);   // host bounds simlen/eps
    ws.bcast[4] = h.uniform();   // accept uniform (position 2)
  }
  for (int i = tid; i < m.D + 2; i += blockDim.x) ws.prop[i] = ws.par[i];
  __syncthreads();
  const double step = ws.bcast[3];
  const int L = ws.ibcast[0];
  const double u = ws.bcast[4];
  for (int j = tid; j < P; j += blockDim.x) ws.q[j] = ws.par[idx[j]];
  // l = 0: gradient and log density at the current state, unless known; then
  // L positions, the log density needed at the last
  double ll_curr = *ll_known, ll_prop = 0.0;
  for (int l = known ? 1 : 0;; ++l) {
    if (l > 0) {
      // each thread moves its own coordinates
      for (int j = tid; j < P; j += blockDim.x) {
        const double* g = l == 1 ? ws.aux1 : ws.blk_g;
        const double p = __dadd_rn(l == 1 ? ws.p0[j] : ws.ps[j], __dmul_rn(l == 1 ? step / 2.0 : step, g[j]));
        const double q = __dadd_rn(ws.q[j], __dmul_rn(step, p));
        ws.ps[j] = p;
        ws.q[j] = q;
        ws.prop[idx[j]] = q;
      }
      __syncthreads();
    }
    const double v = block_eval<RES, COLS>(m, l == 0 || l == L, true, l == 0 ? ws.par : ws.prop, bi, P, ws);
    if (l == 0) {
      ll_curr = v;
      for (int j = tid; j < P; j += blockDim.x) ws.aux1[j] = ws.blk_g[j];
    } else if (l == L) {
      ll_prop = v;
      break;
    }
  }
  for (int j = tid; j < P; j += blockDim.x) ws.ps[j] = __dadd_rn(ws.ps[j], __dmul_rn(step / 2.0, ws.blk_g[j]));
  __syncthreads();
  const double k0 = block_dot(ws.p0, ws.p0, P, ws);
  const double k1 = block_dot(ws.ps, ws.ps, P, ws);
  const double auxll = k0 / 2.0 - k1 / 2.0;
  const double dlog = ll_prop - ll_curr + auxll;   // minus the energy error
  const int acc = log(u) < dlog;
  // divergent: the energy error passed the bound, or is not finite
  const int div = !(dlog > -AB_DIVERGENCE_DH);
  if (acc) {
    for (int i = tid; i < m.D + 2; i += blockDim.x) ws.par[i] = ws.prop[i];
    for (int j = tid; j < P; j += blockDim.x) ws.aux1[j] = ws.blk_g[j];
  }
  *ll_known = acc ? ll_prop : ll_curr;
  __syncthreads();
  return acc | (div << 1);
}

// ---- NUTS: cbits/augur_mcmclib.h:575-776 (iterative restatement) ------------
// Stacks live in global scratch: [3][HLR_STK][P] doubles per chain.
struct NutsFrame {
  int j, phase, ln, ls;
};

__device__ int nuts_update_s(int s, const double* tp, const double* mp, const double* tm,
                             const double* mm, int P, Ws& ws) {
  int res = 0;
  if (s == 1) {
    for (int j = threadIdx.x; j < P; j += blockDim.x) ws.blk_g[j] = __dadd_rn(tp[j], __dmul_rn(-1.0, tm[j]));
    __syncthreads();
    const double d1 = block_dot(ws.blk_g, mp, P, ws);
    const double d2 = block_dot(ws.blk_g, mm, P, ws);
    res = (d1 >= 0.0 && d2 >= 0.0) ? 1 : 0;
  }
  return res;
}

// The gradient at a leaf's start is the one found at the previous leaf's end
// (the reference evaluates it again): it is kept for the walk (ws.blk_g between
// leaves, wg) and for both frontiers (gm, gp), so a leaf is one evaluation.
template <int RES, int COLS>
__device__ int nuts_transition(const HlrModelDev& m, const HlrComp& cp, const BlockInfo bi, Ws& ws,
                               double* stk, uint64_t seed, uint32_t iter, uint32_t chain, uint32_t ci,
                               int* depth_out, int* leaves_out, int* error_out, int* div_out) {
  const int P = cp.P;
  const int tid = threadIdx.x;
  const int* idx = ws.idx;
  double* gm = ws.gfr;                           // gradient at theta_minus
  double* gp = ws.gfr + P;                       // gradient at theta_plus
  double* wg = ws.gfr + 2 * P;                   // gradient at the walk's position
  double* tp_stk = stk;                          // theta_prop stack
  double* ts_stk = stk + (size_t)HLR_STK * P;    // theta stack
  double* ms_stk = stk + (size_t)2 * HLR_STK * P;  // mom stack
  double* th0 = ws.aux1;   // theta0 (block)
  double* thm = ws.aux2;   // theta_minus
  double* thp = ws.aux3;   // theta_plus
  double* thprop = ws.q;   // working theta
  double* mm = ws.p0;      // mom_minus
  double* mp = ws.ps;      // mom_plus
  double* aux4 = ws.aux4;  // spare copy buffer
  // initialise
  for (int j = tid; j < P; j += blockDim.x) {
    th0[j] = ws.par[idx[j]];
    thm[j] = th0[j];
    thp[j] = th0[j];
    Stream s = make_stream(seed, chain * (uint32_t)P + j, iter, TAG_MOM | (ci << 8));
    mm[j] = s.normal();
    mp[j] = mm[j];
  }
  for (int i = tid; i < m.D + 2; i += blockDim.x) ws.prop[i] = ws.par[i];
  __syncthreads();
  // h substream position counter lives in ibcast[1] (read/advanced by thread 0)
  const double ll0 = block_eval<RES, COLS>(m, true, true, ws.par, bi, P, ws);
  for (int j = tid; j < P; j += blockDim.x) gm[j] = gp[j] = ws.blk_g[j];
  const double mm2 = block_dot(mm, mm, P, ws);
  if (tid == 0) {
    Stream h = make_stream(seed, chain, iter, TAG_NUTS | (ci << 8));
    const double e = -1.0 * log(h.uniform());
    ws.bcast[5] = ll0 - 0.5 * mm2 - e;   // logu
    ws.ibcast[1] = (int)h.pos;
    ws.ibcast[2] = -1; ws.ibcast[3] = -1; ws.ibcast[4] = -1;  // tp, ts, ms stack heads
    ws.ibcast[5] = 0;  // leaves
    ws.ibcast[6] = 0;  // overflow flag
    ws.ibcast[7] = 0;  // divergence flag
  }
  __syncthreads();
  const double logu = ws.bcast[5];
  auto draw_u = [&]() -> double {   // next uniform of the sequential h stream (uniform across threads)
    __syncthreads();
    if (tid == 0) {
      Stream h = make_stream(seed, chain, iter, TAG_NUTS | (ci << 8));
      h.pos = (uint32_t)ws.ibcast[1];
      ws.bcast[6] = h.uniform();
      ws.ibcast[1] = (int)h.pos;
    }
    __syncthreads();
    const double r = ws.bcast[6];
    __syncthreads();
    return r;
  };
  auto push = [&](double* base, int head_slot, const double* v) {
    __syncthreads();
    int hd = ws.ibcast[head_slot] + 1;
    if (hd >= HLR_STK) { if (tid == 0) ws.ibcast[6] = 1; hd = HLR_STK - 1; }
    for (int j = tid; j < P; j += blockDim.x) base[(size_t)hd * P + j] = v[j];
    __syncthreads();
    if (tid == 0) ws.ibcast[head_slot] = hd;
    __syncthreads();
  };
  auto head = [&](int head_slot) -> int {
    const int h = ws.ibcast[head_slot];
    return h < 0 ? 0 : h;
  };
  auto pop = [&](int head_slot) -> int {   // returns the popped slot index
    __syncthreads();
    const int h = ws.ibcast[head_slot];
    __syncthreads();
    if (tid == 0) ws.ibcast[head_slot] = h - 1;
    __syncthreads();
    return h < 0 ? 0 : h;
  };
  int n = 1, jd = 0, s = 1;
  double stepsize = cp.eps;
  NutsFrame fr[24];
  for (;;) {
    int f_cpy = 0;
    if (tid == 0) { ws.ibcast[3] = -1; ws.ibcast[4] = -1; }
    __syncthreads();
    const int dir = draw_u() < 0.5 ? 0 : 1;   // 0 = MINUS
    stepsize = dir == 0 ? -cp.eps : cp.eps;
    double* mom = dir == 0 ? mm : mp;
    for (int j = tid; j < P; j += blockDim.x) {
      thprop[j] = dir == 0 ? thm[j] : thp[j];
      wg[j] = dir == 0 ? gm[j] : gp[j];
    }
    __syncthreads();
    // ---- build_tree(thprop, mom, jd, dir) as an explicit post-order walk
    int sp = 0;
    fr[0].j = jd; fr[0].phase = 0;
    int rn = 0, rs = 0;       // return value of the last finished subtree
    while (sp >= 0) {
      NutsFrame& F = fr[sp];
      if (F.j == 0) {
        // leaf: leapfrog1 (:305-325) - half kick, drift, gradient, half kick
        for (int j = tid; j < P; j += blockDim.x) {
          mom[j] = __dadd_rn(mom[j], __dmul_rn(stepsize / 2.0, wg[j]));
          thprop[j] = __dadd_rn(thprop[j], __dmul_rn(stepsize, mom[j]));
          ws.prop[idx[j]] = thprop[j];
        }
        __syncthreads();
        const double llp = block_eval<RES, COLS>(m, true, true, ws.prop, bi, P, ws);
        for (int j = tid; j < P; j += blockDim.x) {
          wg[j] = ws.blk_g[j];
          mom[j] = __dadd_rn(mom[j], __dmul_rn(stepsize / 2.0, wg[j]));
        }
        __syncthreads();
        if (tid == 0) ws.ibcast[5] += 1;
        push(tp_stk, 2, thprop);
        const double ll = llp - 0.5 * block_dot(mom, mom, P, ws);
        rn = logu <= ll ? 1 : 0;
        rs = logu < 1000.0 + ll ? 1 : 0;
        // a leaf outside the slice by the reference's deltaMax (1000) ends
        // the tree: the iteration counts as divergent
        if (tid == 0 && !rs) ws.ibcast[7] = 1;
        --sp;
        continue;
      }
      if (F.phase == 0) {
        F.phase = 1;
        fr[sp + 1].j = F.j - 1; fr[sp + 1].phase = 0;
        ++sp;
        continue;
      }
      if (F.phase == 1) {             // left subtree finished
        F.ln = rn; F.ls = rs;
        if (F.ls == 1) {
          if (F.j == 1) { push(ts_stk, 3, thprop); push(ms_stk, 4, mom); }
          F.phase = 2;
          fr[sp + 1].j = F.j - 1; fr[sp + 1].phase = 0;
          ++sp;
        } else {
          rn = F.ln; rs = F.ls;
          --sp;
        }
        continue;
      }
      // phase 2: right subtree finished (rn, rs)
      const int p1 = pop(2);
      const int p2 = pop(2);
      const double bias = ((double)rn) / (F.ln + rn);
      const double uu = draw_u();
      // push(prop2) or push(prop1): copy through the spare buffer
      const int src = (uu < bias) ? p1 : p2;
      for (int j = tid; j < P; j += blockDim.x) aux4[j] = tp_stk[(size_t)src * P + j];
      push(tp_stk, 2, aux4);
      F.ln += rn;
      const double* tpv; const double* mpv; const double* tmv; const double* mmv;
      const int th_slot = head(3), mo_slot = head(4);
      if (dir == 0) { tpv = ts_stk + (size_t)th_slot * P; mpv = ms_stk + (size_t)mo_slot * P; tmv = thprop; mmv = mom; }
      else { tmv = ts_stk + (size_t)th_slot * P; mmv = ms_stk + (size_t)mo_slot * P; tpv = thprop; mpv = mom; }
      F.ls = nuts_update_s(rs, tpv, mpv, tmv, mmv, P, ws);
      if (F.j > 1) { pop(3); pop(4); }
      rn = F.ln; rs = F.ls;
      --sp;
    }
    // ---- outer loop body (:744-774)
    for (int j = tid; j < P; j += blockDim.x) {
      (dir == 0 ? thm : thp)[j] = thprop[j];
      (dir == 0 ? gm : gp)[j] = wg[j];
    }
    __syncthreads();
    const int pp = pop(2);
    if (rs == 1) {
      const unsigned ratio = (unsigned)(((double)rn) / n);   // augur_min is unsigned
      const double bias = (double)(ratio < 1u ? ratio : 1u);
      if (draw_u() < bias) {
        for (int j = tid; j < P; j += blockDim.x) thprop[j] = tp_stk[(size_t)pp * P + j];
        f_cpy = 1;
      }
      __syncthreads();
    }
    n += rn;
    s = nuts_update_s(rs, thp, mp, thm, mm, P, ws);
    jd += 1;
    if (s != 1 || jd >= cp.max_depth || ws.ibcast[6]) {
      if (f_cpy) for (int j = tid; j < P; j += blockDim.x) th0[j] = thprop[j];
      __syncthreads();
      break;
    }
  }
  set_block(ws.par, idx, P, th0);
  if (tid == 0) {
    *depth_out = jd;
    *leaves_out = ws.ibcast[5];
    *error_out = ws.ibcast[6];
    *div_out = ws.ibcast[7];
  }
  __syncthreads();
  return 0;
}

// ---- Reflective slice: cbits/augur_mcmclib.h:498-543 ------------------------
// Momentum from (c*P + j, iter, MOM|ci<<8); slice level z = ll(curr) - Exp(1)
// with the exponential from (c, iter, RSLICE|ci<<8); augur_max(1,
// round(simlen / eps)) steps of q += eps p0, each followed by the log density
// at the new point and, outside the slice, a reflection of p0 off the block
// gradient there (p0 += -2 (p0.g)/(g.g) g, dot products in block_dot's tree).  The
// move is kept only if the last point is inside the slice.
template <int RES, int COLS>
__device__ int rslice_transition(const HlrModelDev& m, const HlrComp& cp, const BlockInfo bi, Ws& ws,
                                 uint64_t seed, uint32_t iter, uint32_t chain, uint32_t ci, int* refl_out) {
  const int P = cp.P;
  const int tid = threadIdx.x;
  const int* idx = ws.idx;
  for (int j = tid; j < P; j += blockDim.x) {
    Stream s = make_stream(seed, chain * (uint32_t)P + j, iter, TAG_MOM | (ci << 8));
    ws.p0[j] = s.normal();
  }
  if (tid == 0) {
    Stream h = make_stream(seed, chain, iter, TAG_RSLICE | (ci << 8));
    ws.bcast[3] = -1.0 * log(h.uniform());
    const unsigned rl = (unsigned)round(cp.simlen / cp.eps);
    ws.ibcast[0] = (int)min(rl > 1u ? rl : 1u, 1u << 20);   // host bounds simlen/eps
  }
  for (int i = tid; i < m.D + 2; i += blockDim.x) ws.prop[i] = ws.par[i];
  __syncthreads();
  const double expo = ws.bcast[3];
  const int L = ws.ibcast[0];
  const double step = cp.eps;
  for (int j = tid; j < P; j += blockDim.x) ws.q[j] = ws.par[idx[j]];
  // l = 0: the log density at the current state; then at each of L points, and
  // where it is outside the slice (cond) the gradient there: one evaluation a
  // turn, so that the kernel holds its code once
  bool cond = false;
  int refl = 0;
  double z = 0.0;
  for (int l = 0;;) {
    const double ll = block_eval<RES, COLS>(m, !cond, cond, l == 0 ? ws.par : ws.prop, bi, P, ws);
    if (cond) {
      const double a1 = block_dot(ws.p0, ws.blk_g, P, ws);
      const double a2 = block_dot(ws.blk_g, ws.blk_g, P, ws);
      const double sc = __dmul_rn(-2.0, a1 / a2);
      for (int j = tid; j < P; j += blockDim.x) ws.p0[j] = __dadd_rn(ws.p0[j], __dmul_rn(sc, ws.blk_g[j]));
      __syncthreads();
      ++refl;
      if (l == L) break;
      cond = false;
    } else if (l == 0) {
      z = ll - expo;
    } else {
      cond = ll < z;                     // same value on every thread
      if (cond) continue;
      if (l == L) break;
    }
    for (int j = tid; j < P; j += blockDim.x) ws.q[j] = __dadd_rn(ws.q[j], __dmul_rn(step, ws.p0[j]));
    __syncthreads();
    set_block(ws.prop, idx, P, ws.q);
    ++l;
  }
  if (!cond)
    for (int i = tid; i < m.D + 2; i += blockDim.x) ws.par[i] = ws.prop[i];
  __syncthreads();
  *refl_out = refl;
  return !cond;
}

// ---- MWG on one scalar of par: augur_mcmclib.h:89-105,178-193 ---------------
template <int RES, int COLS>
__device__ int mwg_transition(const HlrModelDev& m, const HlrComp& cp, const BlockInfo bi, Ws& ws,
                              uint64_t seed, uint32_t iter, uint32_t chain, uint32_t ci) {
  const int which = ws.idx[0];
  if (threadIdx.x == 0) {
    Stream s = make_stream(seed, chain, iter, TAG_MWG | (ci << 8));
    const double x = ws.par[which];
    const double xp = x + sqrt(cp.mwg_var) * s.normal();
    ws.bcast[3] = xp;
    ws.bcast[4] = s.uniform();
    ws.bcast[5] = m.compat ? normal_ll(m, x, x, cp.mwg_var) - normal_ll(m, xp, x, cp.mwg_var) : 0.0;
  }
  for (int i = threadIdx.x; i < m.D + 2; i += blockDim.x) ws.prop[i] = ws.par[i];
  __syncthreads();
  if (threadIdx.x == 0) ws.prop[which] = ws.bcast[3];
  __syncthreads();
  double lc = 0.0, lp = 0.0;
#pragma unroll 1
  for (int l = 0; l < 2; ++l) {
    lc = lp;
    lp = block_eval<RES, COLS>(m, true, false, l == 0 ? ws.par : ws.prop, bi, 1, ws);
  }
  const int acc = log(ws.bcast[4]) < lp - lc + ws.bcast[5];
  if (acc && threadIdx.x == 0) ws.par[which] = ws.prop[which];
  __syncthreads();
  return acc;
}

// Shared memory of a chain CTA: the state vectors, the NUTS gradients and
// stacks, then X in its own type (rows of an odd number of 4-byte words) and
// the labels.
struct HlrLayout {
  int res;         // X_GLOBAL, X_F32 or X_BF16
  int xpitch;      // elements of a row of the copy
  int stk;         // NUTS stacks in shared memory (else the caller's scratch)
  int nuts;        // a NUTS component is present
};

static __host__ __device__ inline size_t hlr_layout_bytes(int N, int D, const HlrLayout& l) {
  const size_t V = (size_t)D + 2;
  size_t d = 11 * V + HLR_THREADS + 34 + 8 + 8 + (V + 1) / 2 + 1 + ((size_t)D + 1) / 2 + 1 + HLR_CHUNK;
  if (l.nuts) d += 3 * V;
  if (l.stk) d += 3 * (size_t)HLR_STK * V;
  return sizeof(double) * d +
         (l.res ? sizeof(int) * (size_t)N + (l.res == X_F32 ? 4 : 2) * (size_t)N * l.xpitch : 0);
}

__device__ Ws carve(void* base, int N, int D, const HlrLayout& l, double*& stk) {
  Ws w;
  double* d = reinterpret_cast<double*>(base);
  const int V = D + 2;
  w.par = d; d += V; w.prop = d; d += V; w.g = d; d += V; w.blk_g = d; d += V;
  w.p0 = d; d += V; w.ps = d; d += V; w.q = d; d += V; w.aux1 = d; d += V; w.aux2 = d; d += V;
  w.aux3 = d; d += V; w.aux4 = d; d += V;
  w.gpart = d; d += HLR_THREADS;
  w.red = d; d += 34;
  w.bcast = d; d += 8;
  w.ibcast = reinterpret_cast<int*>(d); d += 8;
  w.idx = reinterpret_cast<int*>(d); d += (V + 1) / 2 + 1;
  w.th = reinterpret_cast<float*>(d); d += (D + 1) / 2 + 1;
  w.r = reinterpret_cast<float*>(d);
  w.l = w.r + HLR_CHUNK;
  d += HLR_CHUNK;
  w.gfr = d; if (l.nuts) d += 3 * V;
  stk = d; if (l.stk) d += 3 * (size_t)HLR_STK * V;
  w.lab = reinterpret_cast<int*>(d);
  w.xs = l.res ? w.lab + N : nullptr;
  w.xpitch = l.xpitch;
  return w;
}

// X and the labels into shared memory, STAGE_DEPTH values of a thread in flight
// (a row a warp, one load after another, took 45 us for 1000 x 10 values, as
// long as ten evaluations).
constexpr int STAGE_DEPTH = 8;
template <typename T>
__device__ __forceinline__ void stage_rows(const HlrModelDev& m, const T* __restrict__ X, T* xs, int pitch) {
  const int N = m.N, D = m.D, di = HLR_BLOCK / D, dk = HLR_BLOCK % D;
  int i = threadIdx.x / D, k = threadIdx.x % D;
  while (i < N) {
    T v[STAGE_DEPTH];
    int at[STAGE_DEPTH];
#pragma unroll
    for (int u = 0; u < STAGE_DEPTH; ++u) {
      at[u] = i < N ? i * pitch + k : -1;
      if (i < N) v[u] = X[(size_t)i * m.ldx + k];
      i += di;
      k += dk;
      if (k >= D) { k -= D; ++i; }
    }
#pragma unroll
    for (int u = 0; u < STAGE_DEPTH; ++u)
      if (at[u] >= 0) xs[at[u]] = v[u];
  }
}
__device__ __forceinline__ void stage_labels(const HlrModelDev& m, int* lab) {
  for (int i0 = threadIdx.x; i0 < m.N; i0 += STAGE_DEPTH * HLR_BLOCK) {
    int v[STAGE_DEPTH];
#pragma unroll
    for (int u = 0; u < STAGE_DEPTH; ++u) v[u] = load_label(m, min(i0 + u * HLR_BLOCK, m.N - 1));
#pragma unroll
    for (int u = 0; u < STAGE_DEPTH; ++u)
      if (i0 + u * HLR_BLOCK < m.N) lab[i0 + u * HLR_BLOCK] = v[u];
  }
}

// One CTA per chain: n_iter iterations of the schedule `comps`.
// stats[c][ci][5] = {accepts, sum depth, sum leaves, errors, divergent iterations}.
// Bound: the chain of one evaluation - barriers, the compensated sums of a
// thread's rows, binary64 reductions - at 11 evaluations an HMC iteration.
// Measured, ten HMC iterations at N = 1000, D = 10: 890 -> 334 us; a NUTS
// iteration of depth 5 for 48 chains at N = 2003, D = 41 (bf16): 5.30 -> 0.40 ms,
// where every evaluation walked X a warp per row and every leaf took two.
// Issue slots 37 and 52 % busy, no pipe near its limit, stalls on fixed latencies
// and barriers.
template <int RES, int COLS>
__global__ void __launch_bounds__(HLR_BLOCK, 1)
hlr_chain_kernel(const __grid_constant__ HlrModelDev m, HlrLayout l, const HlrComp* __restrict__ comps, int n_comps,
                 const int* __restrict__ idx_all, double* __restrict__ pars, int n_iter,
                 uint32_t iter0, uint64_t seed, double* __restrict__ stats,
                 double* __restrict__ nuts_stk, int stk_P) {
  extern __shared__ __align__(16) double smem_d[];
  double* stk;
  Ws ws = carve(smem_d, m.N, m.D, l, stk);
  const int c = blockIdx.x;
  if (!l.stk) stk = nuts_stk + (size_t)c * 3 * HLR_STK * stk_P;
  if (RES == X_F32) stage_rows(m, static_cast<const float*>(m.X), static_cast<float*>(ws.xs), l.xpitch);
  if (RES == X_BF16) stage_rows(m, static_cast<const __nv_bfloat16*>(m.X), static_cast<__nv_bfloat16*>(ws.xs), l.xpitch);
  if (RES) stage_labels(m, ws.lab);
  double* par_g = pars + (size_t)c * (m.D + 2);
  for (int i = threadIdx.x; i < m.D + 2; i += blockDim.x) ws.par[i] = par_g[i];
  __syncthreads();
  const bool tell = threadIdx.x == 0;
  BlockInfo bi{false, false, false};
  double ll_known = 0.0;
  for (int it = 0; it < n_iter; ++it) {
    const uint32_t iter = iter0 + (uint32_t)it;
    for (int ci = 0; ci < n_comps; ++ci) {
      const HlrComp cp = comps[ci];
      if (n_comps > 1 || it == 0) bi = stage_block(m, idx_all + cp.idx_off, cp.P, ws);
      double* st = stats + ((size_t)c * n_comps + ci) * AB_HLR_STATS;
      if (cp.kind == COMP_HMC) {
        const int a = hmc_transition<RES, COLS>(m, cp, bi, ws, seed, iter, (uint32_t)c, (uint32_t)ci,
                                          n_comps == 1 && it > 0, &ll_known);
        if (tell) { st[0] += a & 1; st[4] += a >> 1; }
      } else if (cp.kind == COMP_NUTS) {
        __shared__ int sh_out[4];
        nuts_transition<RES, COLS>(m, cp, bi, ws, stk, seed, iter, (uint32_t)c, (uint32_t)ci, &sh_out[0], &sh_out[1],
                             &sh_out[2], &sh_out[3]);
        if (tell) { st[1] += sh_out[0]; st[2] += sh_out[1]; st[3] += sh_out[2]; st[4] += sh_out[3]; }
      } else if (cp.kind == COMP_RSLICE) {
        int refl = 0;
        const int a = rslice_transition<RES, COLS>(m, cp, bi, ws, seed, iter, (uint32_t)c, (uint32_t)ci, &refl);
        if (tell) { st[0] += a; st[2] += refl; }
      } else {
        const int a = mwg_transition<RES, COLS>(m, cp, bi, ws, seed, iter, (uint32_t)c, (uint32_t)ci);
        if (tell) st[0] += a;
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < m.D + 2; i += blockDim.x) par_g[i] = ws.par[i];
}

// Log-density and gradient of a block for C parameter vectors (one CTA per
// vector): the data pass and priors used by the transitions, exposed for
// parity checks and for callers that drive their own samplers.
// 256 threads of at most 128 registers, two CTAs per SM: with many vectors that
// counts for more than a warp for the prior (500 vectors of D = 28, 5000 rows:
// 104 us, 150 with one CTA of 288 threads per SM).
template <int COLS>
__global__ void __launch_bounds__(HLR_THREADS, 2)
hlr_ll_grad_kernel(const __grid_constant__ HlrModelDev m, HlrLayout l, const int* __restrict__ idx, int P, const double* __restrict__ pars,
                   double* __restrict__ ll, double* __restrict__ grad) {
  extern __shared__ __align__(16) double smem_d[];
  double* stk;
  Ws ws = carve(smem_d, m.N, m.D, l, stk);
  const int c = blockIdx.x;
  for (int i = threadIdx.x; i < m.D + 2; i += blockDim.x) ws.par[i] = pars[(size_t)c * (m.D + 2) + i];
  const BlockInfo bi = stage_block(m, idx, P, ws);
  const double v = block_eval<X_GLOBAL, COLS, HLR_THREADS>(m, true, grad != nullptr, ws.par, bi, P, ws);
  if (threadIdx.x == 0) ll[c] = v;
  if (grad != nullptr)
    for (int j = threadIdx.x; j < P; j += blockDim.x) grad[(size_t)c * P + j] = ws.blk_g[j];
}

static int make_model(HlrModelDev& m, const ab_hlr_model* d) {
  AB_REQUIRE(d != nullptr, AB_ERR_ARG, "hlr: null model");
  AB_REQUIRE(d->N > 0 && d->D > 0 && d->D <= HLR_MAX_D, AB_ERR_ARG,
             "hlr: need N > 0 and 0 < D <= %d (N=%d D=%d)", HLR_MAX_D, d->N, d->D);
  AB_REQUIRE(d->lik == AB_LIK_BERNOULLI || d->lik == AB_LIK_POISSON || d->lik == AB_LIK_NORMAL, AB_ERR_ARG,
             "hlr: unknown likelihood %d", d->lik);
  AB_REQUIRE(d->X && (d->lik == AB_LIK_NORMAL ? d->yr != nullptr : d->y != nullptr), AB_ERR_ARG,
             "hlr: null data pointer");
  AB_REQUIRE(d->lik != AB_LIK_NORMAL || d->obs_var > 0.0, AB_ERR_ARG, "hlr: the observation variance must be > 0");
  AB_REQUIRE(d->x_dtype == AB_F32 || d->x_dtype == AB_BF16, AB_ERR_ARG, "hlr: X must be f32 or bf16");
  AB_REQUIRE(d->ldx >= d->D, AB_ERR_ARG, "hlr: ldx < D");
  AB_REQUIRE(d->vprior == 0 || d->vprior == 1, AB_ERR_ARG, "hlr: vprior must be 0 or 1");
  m.N = d->N; m.D = d->D; m.ldx = d->ldx; m.has_b = d->has_b != 0; m.vprior = d->vprior;
  m.compat = d->compat != 0; m.x_bf16 = d->x_dtype == AB_BF16;
  m.lam = d->lam; m.a0 = d->a0; m.s0 = d->s0; m.X = d->X; m.y = d->y;
  m.lik = d->lik;
  m.yr = d->yr;
  m.inv_var = d->lik == AB_LIK_NORMAL ? (float)(1.0 / d->obs_var) : 0.0f;
  // per-row Normal normaliser: the reference's -log(var) (compat) or -log(2 pi var) / 2
  m.ll_add = d->lik != AB_LIK_NORMAL ? 0.0
             : (double)d->N * (m.compat ? -log(d->obs_var) : -0.5 * log(2.0 * M_PI * d->obs_var));
  m.vp_const = m.vprior == 0 ? log(m.lam) : m.a0 * log(m.s0) - lgamma(m.a0);
  return AB_OK;
}

// What a chain's CTA keeps in shared memory: X and the labels, if a component
// evaluates the data, and the NUTS stacks, where they fit 224 KB (an SM holds
// one CTA, whatever its shared memory: 288 threads of 153 to 168 registers).
// Every evaluation then reads X from there instead of walking it through the
// caches.
static HlrLayout choose_layout(const HlrModelDev& m, bool nuts, bool data) {
  const size_t room = 224 * 1024;
  const auto fits = [&](const HlrLayout& l) { return hlr_layout_bytes(m.N, m.D, l) <= room; };
  if (data) {
    HlrLayout x{m.x_bf16 ? X_BF16 : X_F32, m.x_bf16 ? 2 * (((m.D + 1) / 2) | 1) : (m.D | 1), nuts, nuts};
    if (fits(x)) return x;
    x.stk = 0;
    if (fits(x)) return x;
  }
  HlrLayout l{X_GLOBAL, 0, nuts, nuts};
  if (!fits(l)) l.stk = 0;
  return l;
}

template <int COLS>
static auto chain_kernel(int res) {
  return res == X_F32    ? hlr_chain_kernel<X_F32, COLS>
         : res == X_BF16 ? hlr_chain_kernel<X_BF16, COLS>
                         : hlr_chain_kernel<X_GLOBAL, COLS>;
}

static int check_idx_host(const int* idx_host, int P, int D) {
  for (int j = 0; j < P; ++j)
    AB_REQUIRE(idx_host[j] >= 0 && idx_host[j] < D + 2, AB_ERR_ARG, "hlr: block index %d out of range", idx_host[j]);
  return AB_OK;
}

}  // namespace ab

using namespace ab;

extern "C" size_t ab_hlr_chain_scratch_bytes(int C, int D) {
  return sizeof(double) * (size_t)C * 3 * HLR_STK * (size_t)(D + 2);
}

extern "C" int ab_hlr_ll_grad(const ab_hlr_model* model, const int* idx_dev, const int* idx_host, int P,
                              int C, const double* pars, double* ll, double* grad, void* stream) {
  HlrModelDev m;
  int rc = make_model(m, model);
  if (rc) return rc;
  AB_REQUIRE(C > 0 && P > 0 && P <= m.D + 2, AB_ERR_ARG, "ab_hlr_ll_grad: bad C or P");
  AB_REQUIRE(idx_dev && idx_host && pars && ll, AB_ERR_ARG, "ab_hlr_ll_grad: null pointer");
  rc = check_idx_host(idx_host, P, m.D);
  if (rc) return rc;
  const HlrLayout l{X_GLOBAL, 0, 0, 0};
  const size_t smem = hlr_layout_bytes(m.N, m.D, l);
  const auto kernel = m.D + 2 <= 16           ? hlr_ll_grad_kernel<16>
                      : m.D + 2 <= SMALL_COLS ? hlr_ll_grad_kernel<SMALL_COLS>
                                              : hlr_ll_grad_kernel<0>;
  AB_CUDA(allow_smem((const void*)kernel, smem));
  kernel<<<C, HLR_THREADS, smem, as_stream(stream)>>>(m, l, idx_dev, P, pars, ll, grad);
  AB_LAUNCH_CHECK("hlr_ll_grad_kernel");
  return AB_OK;
}

extern "C" int ab_hlr_run_chains(const ab_hlr_model* model, const ab_hlr_comp* comps_host,
                                 const void* comps_dev, int n_comps, const int* idx_dev,
                                 const int* idx_host, int C, double* pars, int n_iter, uint32_t iter0,
                                 uint64_t seed, double* stats, void* scratch, void* stream) {
  HlrModelDev m;
  int rc = make_model(m, model);
  if (rc) return rc;
  AB_REQUIRE(C > 0 && n_iter >= 0, AB_ERR_ARG, "ab_hlr_run_chains: bad C or n_iter");
  AB_REQUIRE(n_comps > 0 && n_comps <= HLR_MAX_COMPS, AB_ERR_ARG, "ab_hlr_run_chains: 1..%d components",
             HLR_MAX_COMPS);
  AB_REQUIRE(comps_host && comps_dev && idx_dev && idx_host && pars && stats, AB_ERR_ARG,
             "ab_hlr_run_chains: null pointer");
  bool has_nuts = false, data = false;
  for (int i = 0; i < n_comps; ++i) {
    const ab_hlr_comp& c = comps_host[i];
    AB_REQUIRE(c.kind >= 0 && c.kind <= 3, AB_ERR_ARG, "component %d: unknown kind", i);
    AB_REQUIRE(c.P > 0 && c.P <= m.D + 2, AB_ERR_ARG, "component %d: bad block size", i);
    AB_REQUIRE(c.kind != 2 || c.P == 1, AB_ERR_ARG, "component %d: MWG moves one scalar", i);
    AB_REQUIRE(c.kind == 2 || c.eps > 0.0, AB_ERR_ARG, "component %d: step size must be > 0", i);
    AB_REQUIRE((c.kind != 0 && c.kind != 3) || (c.simlen >= 0.0 && c.simlen / c.eps <= 1e5), AB_ERR_ARG,
               "component %d: HMC / RSlice simlen/eps must be <= 1e5 steps", i);
    AB_REQUIRE(c.kind != 2 || c.mwg_var > 0.0, AB_ERR_ARG, "component %d: MWG variance must be > 0", i);
    AB_REQUIRE(c.kind != 1 || (c.max_depth > 0 && c.max_depth <= 14), AB_ERR_ARG,
               "component %d: NUTS max_depth must be 1..14", i);
    rc = check_idx_host(idx_host + c.idx_off, c.P, m.D);
    if (rc) return rc;
    has_nuts |= c.kind == 1;
    for (int j = 0; j < c.P; ++j) data |= idx_host[c.idx_off + j] < m.D + (m.has_b ? 1 : 0);
  }
  AB_REQUIRE(!has_nuts || scratch, AB_ERR_ARG, "ab_hlr_run_chains: NUTS needs scratch");
  static_assert(sizeof(ab_hlr_comp) == sizeof(HlrComp), "component layout");
  const HlrLayout l = choose_layout(m, has_nuts, data);
  const size_t smem = hlr_layout_bytes(m.N, m.D, l);
  AB_REQUIRE(smem <= 224 * 1024, AB_ERR_ARG, "hlr: D too large for the per-chain engine");
  const auto kernel = m.D + 2 <= 16 ? chain_kernel<16>(l.res) : m.D + 2 <= SMALL_COLS ? chain_kernel<SMALL_COLS>(l.res)
                                                                                       : chain_kernel<0>(l.res);
  AB_CUDA(allow_smem((const void*)kernel, smem));
  kernel<<<C, HLR_BLOCK, smem, as_stream(stream)>>>(m, l, reinterpret_cast<const HlrComp*>(comps_dev), n_comps, idx_dev,
                                                    pars, n_iter, iter0, seed, stats,
                                                    reinterpret_cast<double*>(scratch), m.D + 2);
  AB_LAUNCH_CHECK("hlr_chain_kernel");
  return AB_OK;
}
