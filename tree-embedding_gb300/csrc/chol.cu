// Cholesky factors of Grams and what a basis is multiplied by after them.
//
//  chol_inverse_batched     : G (fp64, l <= 144) -> T = R^-1, the CholeskyQR
//    step that replaces LUfraction (Code/frpca.c:4-41) between frPCA's products.
//  chol_shift_solve_batched : K (fp32, l <= 256) -> x L^-T with a shift, the
//    cheap basis of the wide merge's subspace iteration.
//
// A factorization here is a chain of l dependent pivots, far too little work
// for its latency: a column at a time, with three CTA barriers each, it took
// 350 us at l = 133 (2.6 us a column). panel_factor takes 32 columns at a time,
// one row per thread, in groups of eight whose triangle one warp factors by
// shuffles, so a barrier covers eight pivots, and the columns before a panel
// are subtracted from all of it at once (4 x 4 register tiles).
#include <algorithm>

#include "internal.h"
#include "pairs.h"

namespace tsvd {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int CH_THREADS = 512;
constexpr int CH_NB = 32;

// L in shared memory by panels: panel J holds the rows from 32 J down of its 32
// columns, column c at c * (ldn - 32 J + 4).
__host__ __device__ __forceinline__ int panel_ld(int J, int ldn) { return ldn - CH_NB * J + 4; }
__host__ __device__ __forceinline__ int panel_off(int J, int ldn) {
  return CH_NB * (J * (ldn + 4) - 16 * J * (J - 1));
}

// The factor of an n x n matrix whose entry (i, j) is entry(i, j), i >= j, into
// L (panels); a pivot for which root(k, d) returns 0 is dropped: unit pivot,
// zero column, inv[k] = 0. inv[k] = 1 / L_kk otherwise, root the reciprocal of
// the pivot's square root. CH_THREADS threads.
template <class Entry, class Root>
__device__ __forceinline__ void panel_factor(int n, int ldn, float *L, float *inv, Entry entry,
                                             Root root) {
  const int tid = threadIdx.x, ti = tid >> 3, tj = tid & 7;
  for (int J = 0; J * CH_NB < n; ++J) {
    const int J0 = J * CH_NB, m = ldn - J0, ld = panel_ld(J, ldn);
    float *P = L + panel_off(J, ldn);
    const int i0 = 4 * ti, j0 = 4 * tj;
    if (i0 < m) {
      float s[4][4];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = J0 + i0 + p, j = J0 + j0 + q;
          s[p][q] = i < n && j <= i ? entry(i, j) : 0.f;
        }
      for (int K = 0; K < J; ++K) {
        const int lk = panel_ld(K, ldn);
        const float *Q = L + panel_off(K, ldn) + J0 - K * CH_NB;
#pragma unroll 4
        for (int k = 0; k < CH_NB; ++k) {
          const float4 a = *reinterpret_cast<const float4 *>(Q + k * lk + i0);
          const float4 b = *reinterpret_cast<const float4 *>(Q + k * lk + j0);
          const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = 0; q < 4; ++q) s[p][q] = fmaf(-av[p], bv[q], s[p][q]);
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<float4 *>(P + (j0 + q) * ld + i0) =
            make_float4(s[0][q], s[1][q], s[2][q], s[3][q]);
    }
    __syncthreads();
    for (int b = 0; b < CH_NB; b += 8) {
      const bool row = tid < m;
      float h[8];
      if (row) {
#pragma unroll
        for (int q = 0; q < 8; ++q) h[q] = P[(b + q) * ld + tid];
        for (int k = 0; k < b; ++k) {
          const float x = P[k * ld + tid];
          const float4 u = *reinterpret_cast<const float4 *>(P + k * ld + b);
          const float4 v = *reinterpret_cast<const float4 *>(P + k * ld + b + 4);
          const float l[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
          for (int q = 0; q < 8; ++q) h[q] = fmaf(-x, l[q], h[q]);
        }
      }
      if (tid < 32) {  // rows J0 .. J0 + 31: the 8 x 8 triangle by shuffles
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float d = __shfl_sync(kFull, h[q], b + q);
          const float y = J0 + b + q < n ? root(J0 + b + q, d) : 0.f;
          h[q] = y > 0.f ? h[q] * y : (tid == b + q ? 1.f : 0.f);
          if (tid == b + q) inv[J0 + b + q] = y;
#pragma unroll
          for (int t = q + 1; t < 8; ++t)
            h[t] = fmaf(-h[q], __shfl_sync(kFull, h[q], b + t), h[t]);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) P[(b + q) * ld + tid] = tid >= b + q ? h[q] : 0.f;
      }
      __syncthreads();
      if (row && tid >= 32) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          h[q] *= inv[J0 + b + q];
#pragma unroll
          for (int t = q + 1; t < 8; ++t) h[t] = fmaf(-h[q], P[(b + q) * ld + b + t], h[t]);
          P[(b + q) * ld + tid] = h[q];
        }
      }
    }
    __syncthreads();
  }
}

// 1 / sqrt(d) to working precision
__device__ __forceinline__ float inv_sqrt(float d) {
  const float y = rsqrt_approx(d);
  return fmaf(0.5f * y, fmaf(-d * y, y, 1.f), y);
}

// The inverse of panel J's diagonal block (one warp): column `lane` in x.
__device__ __forceinline__ void diag_inverse(const float *P, int ld, const float *inv, float *x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < CH_NB; ++i) x[i] = i == lane ? 1.f : 0.f;
#pragma unroll
  for (int k = 0; k < CH_NB; ++k) {
    const float r = inv[k];
    x[k] = k >= lane ? x[k] * (r > 0.f ? r : 1.f) : 0.f;
#pragma unroll
    for (int i = k + 1; i < CH_NB; ++i) x[i] = fmaf(-P[k * ld + i], x[k], x[i]);
  }
}

// ------------------------------------------------------------------ T = R^-1
// One CTA per problem. G is scaled by a power of two to a largest diagonal
// entry near 1; pivots at or below 1e-12 of it are dropped (zero column of T).
// Of a dependent column only rounding is left, about 2^-24 of its own entry:
// such a pivot is raised to 2e-7 of it, so that the column, as large in its
// off-diagonal entries, stays small after the division.
// The inverse W = L^-1 goes block row by block row: W_IJ = -W_II (sum L_IK W_KJ),
// all columns J < I of a row at once. l = 133, measured: 350 -> 72 us for one
// problem, 730 -> 158 us for 256 (two waves of one CTA per SM).
__global__ void __launch_bounds__(CH_THREADS) chol_inverse_kernel(double *const *gs,
                                                                  float *const *ts, int l) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float inv[kLp + CH_NB];
  __shared__ int sc_s;
  __shared__ float tol_s;
  __shared__ float low[kLp];  // 2e-7 of the diagonal
  const int ldn = (l + 31) & ~31, nb = ldn / CH_NB, ldw = ldn + 4, tid = threadIdx.x;
  float *L = sm, *W = L + panel_off(nb, ldn), *S = W + ldn * ldw;  // W row-major [ldn][ldw]
  const long long *G = reinterpret_cast<const long long *>(gs[blockIdx.x]);
  if (tid < 32) {
    long long mx = 0;
    for (int i = tid; i < l; i += 32) mx = max(mx, G[(int64_t)i * l + i]);
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(kFull, mx, o));
    const int raw = (int)(mx >> 52);
    if (tid == 0) {
      float hi, lo;
      sc_s = raw > 0 && raw < 0x7ff ? -(((raw - 1023) >> 1) + 1) : 0;
      pair_of(mx, 2 * sc_s, hi, lo);
      tol_s = hi * 1e-12f;
    }
  }
  for (int i = tid; i < ldn * ldw; i += CH_THREADS) W[i] = 0.f;
  __syncthreads();
  const int sc = sc_s;
  auto entry = [&](int i, int j) {
    float hi, lo;
    pair_of(G[(int64_t)i * l + j], 2 * sc, hi, lo);
    return hi + lo;
  };
  for (int i = tid; i < l; i += CH_THREADS) low[i] = 2e-7f * entry(i, i);
  __syncthreads();
  const float tol = tol_s;
  panel_factor(l, ldn, L, inv, entry,
               [&](int k, float d) { return d > tol ? inv_sqrt(fmaxf(d, low[k])) : 0.f; });
  for (int J = tid >> 5; J < nb; J += CH_THREADS / 32) {
    float x[CH_NB];
    diag_inverse(L + panel_off(J, ldn), panel_ld(J, ldn), inv + J * CH_NB, x);
#pragma unroll
    for (int i = 0; i < CH_NB; ++i) W[(J * CH_NB + i) * ldw + J * CH_NB + (tid & 31)] = x[i];
  }
  __syncthreads();
  const int ti = tid & 7, tj = tid >> 3;  // 4 x 4 tiles: rows of the block row, columns
  for (int I = 1; I < nb; ++I) {
    const bool act = 4 * tj < CH_NB * I;
    const int i0 = 4 * ti, j0 = 4 * tj;
    float s[4][4] = {};
    if (act) {
      for (int K = j0 / CH_NB; K < I; ++K) {
        const int lk = panel_ld(K, ldn);
        const float *Q = L + panel_off(K, ldn) + (I - K) * CH_NB;
#pragma unroll 4
        for (int k = 0; k < CH_NB; ++k) {
          const float4 a = *reinterpret_cast<const float4 *>(Q + k * lk + i0);
          const float4 b = *reinterpret_cast<const float4 *>(W + (K * CH_NB + k) * ldw + j0);
          const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = 0; q < 4; ++q) s[p][q] = fmaf(-av[p], bv[q], s[p][q]);
        }
      }
#pragma unroll
      for (int p = 0; p < 4; ++p)
        *reinterpret_cast<float4 *>(S + (i0 + p) * ldw + j0) =
            make_float4(s[p][0], s[p][1], s[p][2], s[p][3]);
    }
    __syncthreads();
    if (act) {
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) s[p][q] = 0.f;
#pragma unroll 4
      for (int k = 0; k < CH_NB; ++k) {
        const float4 b = *reinterpret_cast<const float4 *>(S + k * ldw + j0);
        const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const float av = W[(I * CH_NB + i0 + p) * ldw + I * CH_NB + k];
#pragma unroll
          for (int q = 0; q < 4; ++q) s[p][q] = fmaf(av, bv[q], s[p][q]);
        }
      }
#pragma unroll
      for (int p = 0; p < 4; ++p)
        *reinterpret_cast<float4 *>(W + (I * CH_NB + i0 + p) * ldw + j0) =
            make_float4(s[p][0], s[p][1], s[p][2], s[p][3]);
    }
    __syncthreads();
  }
  // T = (L^-1)^T, dropped directions zeroed
  float *T = ts[blockIdx.x];
  const float back = scalbnf(1.f, sc);
  for (int i = tid; i < l * kLp; i += CH_THREADS) {
    const int r = i / kLp, c = i % kLp;
    T[i] = c < l && c >= r && inv[c] > 0.f ? W[c * ldw + r] * back : 0.f;
  }
}

size_t chol_inverse_smem(int l) {
  const int ldn = (l + 31) & ~31;
  return (size_t)(panel_off(ldn / CH_NB, ldn) + (ldn + CH_NB) * (ldn + 4)) * sizeof(float);
}

// ------------------------------------------------------------------ x L^-T
// A factor for solve_rows_kernel, in global memory: L row-major [ldn][ldn], then
// the inverses of its diagonal blocks [nb][32][32], row-major.
__host__ __device__ __forceinline__ size_t factor_floats(int ldn) {
  return (size_t)ldn * ldn + (size_t)ldn * CH_NB;
}

// Shifted Cholesky in fp32 for the basis of a subspace iteration: K + s I =
// L L^T with s = shift * trace(K) / l, so no direction is dropped and x L^-T
// is a well-conditioned (not exactly orthonormal) basis. One CTA per problem;
// l = 256, measured: 936 us a column at a time, 84 us by panels.
__global__ void __launch_bounds__(CH_THREADS) chol_shift_kernel(const float *__restrict__ K,
                                                                float *__restrict__ out, int l,
                                                                float shift) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float inv[256 + CH_NB];
  __shared__ float tr_s;
  const int ldn = (l + 31) & ~31, nb = ldn / CH_NB, tid = threadIdx.x;
  const float *Kb = K + (int64_t)blockIdx.x * l * l;
  if (tid < 32) {
    float acc = 0.f;
    for (int i = tid; i < l; i += 32) acc += Kb[(int64_t)i * l + i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    if (tid == 0) tr_s = fmaxf(acc, 1.17549435e-38f) * shift / (float)l;
  }
  __syncthreads();
  const float tr = tr_s;
  panel_factor(
      l, ldn, sm, inv,
      [&](int i, int j) { return Kb[(int64_t)i * l + j] + (i == j ? tr : 0.f); },
      [&](int, float d) { return inv_sqrt(fmaxf(d, tr)); });
  float *F = out + blockIdx.x * factor_floats(ldn);
  for (int i = tid; i < ldn * ldn; i += CH_THREADS) {
    const int r = i / ldn, c = i % ldn, J = c / CH_NB;
    F[i] = r >= J * CH_NB ? sm[panel_off(J, ldn) + (c % CH_NB) * panel_ld(J, ldn) + r - J * CH_NB]
                          : 0.f;
  }
  F += (int64_t)ldn * ldn;
  for (int J = tid >> 5; J < nb; J += CH_THREADS / 32) {
    float x[CH_NB];
    diag_inverse(sm + panel_off(J, ldn), panel_ld(J, ldn), inv + J * CH_NB, x);
#pragma unroll
    for (int i = 0; i < CH_NB; ++i) F[(J * CH_NB + i) * CH_NB + (tid & 31)] = x[i];
  }
}

// y = x L^-T for the rows of x (rows x l, ld l, problem b at b * stride): a CTA
// takes 32 rows and goes through the 32-column blocks of the factor, y_J =
// (x_J - sum_{K<J} y_K L_JK^T) L_JJ^-T, y kept in shared memory (transposed) and
// the factor's block rows staged from L2. Threads: 4 x 4 output tiles (64) times
// four slices of K, added up in a fixed order. 1500 rows, l = 256, 8 problems,
// measured: 61 us; a warp per row, a column at a time, took 309 us.
constexpr int SR_ROWS = 32, SR_THREADS = 256;
constexpr int SR_LD = SR_ROWS + 4;
__global__ void __launch_bounds__(SR_THREADS) solve_rows_kernel(const float *__restrict__ x,
                                                                float *__restrict__ y,
                                                                const float *__restrict__ factor,
                                                                int rows, int l, int64_t stride) {
  extern __shared__ __align__(16) float sm[];
  const int ldn = (l + 31) & ~31, tid = threadIdx.x, r0 = blockIdx.x * SR_ROWS;
  float *Y = sm;                          // [ldn][SR_LD]: column k of y
  float *B = Y + ldn * SR_LD;             // [ldn][SR_LD]: L_JK^T, k-major
  float *R = B + ldn * SR_LD;             // [4][32][SR_LD]: partial tiles
  const float *F = factor + blockIdx.y * factor_floats(ldn);
  const float *D = F + (int64_t)ldn * ldn;
  const float *xb = x + blockIdx.y * stride;
  float *yb = y + blockIdx.y * stride;
  const int slice = tid >> 6, t = tid & 63, i0 = 4 * (t & 7), j0 = 4 * (t >> 3);
  for (int J0 = 0; J0 < l; J0 += CH_NB) {
    // L rows J0 .. J0 + 31, columns 0 .. J0 - 1, transposed; then L_JJ^-1
    for (int i = tid; i < CH_NB * J0; i += SR_THREADS) {
      const int j = i / J0, k = i % J0;
      B[k * SR_LD + j] = F[(int64_t)(J0 + j) * ldn + k];
    }
    __syncthreads();
    float s[4][4] = {};
    for (int k = slice; k < J0; k += 4) {
      const float4 a = *reinterpret_cast<const float4 *>(Y + k * SR_LD + i0);
      const float4 b = *reinterpret_cast<const float4 *>(B + k * SR_LD + j0);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) s[p][q] = fmaf(-av[p], bv[q], s[p][q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<float4 *>(R + (slice * CH_NB + j0 + q) * SR_LD + i0) =
          make_float4(s[0][q], s[1][q], s[2][q], s[3][q]);
    __syncthreads();
    // residual of the block into R[0], the diagonal inverse (k-major) into B
    for (int i = tid; i < SR_ROWS * CH_NB; i += SR_THREADS) {
      const int j = i % CH_NB, r = i / CH_NB;
      float v = r0 + r < rows && J0 + j < l ? xb[(int64_t)(r0 + r) * l + J0 + j] : 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q) v += R[(q * CH_NB + j) * SR_LD + r];
      R[j * SR_LD + r] = v;
      B[j * SR_LD + r] = D[(J0 + r) * CH_NB + j];  // B[k][j] = (L_JJ^-1)[j][k]
    }
    __syncthreads();
    // 32 x 32 outputs, 2 x 2 per thread: y[r][j] = sum_k R[k][r] Linv[j][k]
    {
      const int a0 = 2 * (tid & 15), b0 = 2 * (tid >> 4);
      float o[2][2] = {};
#pragma unroll 8
      for (int k = 0; k < CH_NB; ++k) {
        const float2 u = *reinterpret_cast<const float2 *>(R + k * SR_LD + a0);
        const float2 v = *reinterpret_cast<const float2 *>(B + k * SR_LD + b0);
        o[0][0] = fmaf(u.x, v.x, o[0][0]);
        o[0][1] = fmaf(u.x, v.y, o[0][1]);
        o[1][0] = fmaf(u.y, v.x, o[1][0]);
        o[1][1] = fmaf(u.y, v.y, o[1][1]);
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        Y[(J0 + b0 + q) * SR_LD + a0] = o[0][q];
        Y[(J0 + b0 + q) * SR_LD + a0 + 1] = o[1][q];
      }
    }
    __syncthreads();
  }
  for (int i = tid; i < SR_ROWS * l; i += SR_THREADS) {
    const int r = i / l, k = i % l;
    if (r0 + r < rows) yb[(int64_t)(r0 + r) * l + k] = Y[k * SR_LD + r];
  }
}

size_t solve_rows_smem(int l) {
  const size_t ldn = (l + 31) & ~31;
  return (2 * ldn + 4 * CH_NB) * SR_LD * sizeof(float);
}

}  // namespace

tsvd_status chol_inverse_batched(double *const *g, float *const *t, int l, int nprob,
                                 cudaStream_t st) {
  if (nprob == 0) return TSVD_OK;
  if (l > kLp) return fail(TSVD_ERR_INVALID, "chol: l=%d > %d", l, kLp);
  const size_t smem = chol_inverse_smem(l);
  TSVD_TRY(raise_smem_ceiling((const void *)chol_inverse_kernel, smem));
  chol_inverse_kernel<<<nprob, CH_THREADS, smem, st>>>(g, t, l);
  TSVD_LAUNCH_CHECK();
  return TSVD_OK;
}

size_t chol_factor_floats(int l) { return factor_floats((l + 31) & ~31); }

tsvd_status chol_shift_solve_batched(const float *K, float *factor, const float *x, float *y,
                                     int rows, int l, int64_t stride, float shift, int nprob,
                                     cudaStream_t st) {
  if (nprob == 0) return TSVD_OK;
  if (l > 256 || l < 1) return fail(TSVD_ERR_INVALID, "chol shift: l=%d", l);
  const int ldn = (l + 31) & ~31;
  const size_t csm = (size_t)panel_off(ldn / CH_NB, ldn) * sizeof(float);
  const size_t rsm = solve_rows_smem(l);
  TSVD_TRY(raise_smem_ceiling((const void *)chol_shift_kernel, csm));
  TSVD_TRY(raise_smem_ceiling((const void *)solve_rows_kernel, rsm));
  chol_shift_kernel<<<nprob, CH_THREADS, csm, st>>>(K, factor, l, shift);
  TSVD_LAUNCH_CHECK();
  solve_rows_kernel<<<dim3((unsigned)ceil_div(rows, SR_ROWS), nprob), SR_THREADS, rsm, st>>>(
      x, y, factor, rows, l, stride);
  TSVD_LAUNCH_CHECK();
  return TSVD_OK;
}

}  // namespace tsvd
