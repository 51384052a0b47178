// Batched FP32 GEMM for the wide merge: C = op(A) B with op(A) = A or A^T,
// row-major operands, problem z at offset z * stride of each operand.
//
// The merges wider than 256 columns (the reference's run.sh arity 8,
// Code/Tree_u_NC.cpp:723-850) run a subspace iteration whose products are
// plain fp32 GEMMs of at most |S| x 2048 by 2048 x 256. They are bound by the
// issue of the FMAs, so a thread's 8 x 8 outputs take four 16-byte shared-memory
// reads a step for 64 of them, and the next slice of K is on its way from L2
// while one is multiplied. A root merge has 48 tiles of 128 x 64 for 152 SMs: K
// is then split over CTAs, and a second kernel adds their sums in order, so every
// output is a fixed-order fp32 sum (deterministic). 1500 x 1024 by 1024 x 256
// takes 22 us and 5 for the sums, eight such 169 and 20; the 118 products of a tree
// of arity 8 over 64 blocks, measured: 14.7 -> 9.8 ms (4 x 4 outputs a thread,
// slices fetched between barriers, no split, before).
#include <algorithm>

#include "internal.h"

namespace tsvd {

namespace {

constexpr int TM = 128, TN = 64, TK = 16, SG_THREADS = 128;
constexpr int SG_MAX_SPLIT = 16;

struct SgemmArgs {
  int M, N, K;
  const float *A;
  int lda;
  int64_t sa;
  const float *B;
  int ldb;
  int64_t sb;
  float *C;      // the result, or with kc < K the partial sums [split][problem][M][N]
  int ldc;
  int64_t sc;
  int kc;        // K values a CTA takes
  int nprob;
  int lower;     // tiles above the diagonal are left out
};

// Four consecutive floats of a row of len, zeros past it (VEC: len and the
// address are multiples of four floats).
template <bool VEC>
__device__ __forceinline__ float4 load4(const float *row, int at, int len) {
  if (VEC) return at < len ? *reinterpret_cast<const float4 *>(row + at) : make_float4(0, 0, 0, 0);
  return make_float4(at < len ? row[at] : 0.f, at + 1 < len ? row[at + 1] : 0.f,
                     at + 2 < len ? row[at + 2] : 0.f, at + 3 < len ? row[at + 3] : 0.f);
}

template <bool TRANS_A, bool VEC>
__global__ void __launch_bounds__(SG_THREADS) sgemm_kernel(SgemmArgs a) {
  __shared__ __align__(16) float As[2][TK][TM + 4];
  __shared__ __align__(16) float Bs[2][TK][TN + 4];
  const int z = blockIdx.z % a.nprob, split = blockIdx.z / a.nprob;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  if (a.lower && n0 > m0 + TM - 1) return;
  const float *A = a.A + z * a.sa, *B = a.B + z * a.sb;
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  const int kb = split * a.kc, ke = min(a.K, kb + a.kc);
  float4 ra[4], rb[2];
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = tid + q * SG_THREADS;
      if (TRANS_A) {  // A is K x M: 32 float4 of m per k
        const int k = k0 + (e >> 5), m = m0 + 4 * (e & 31);
        ra[q] = k < ke ? load4<VEC>(A + (int64_t)k * a.lda, m, a.M) : none;
      } else {        // A is M x K: 4 float4 of k per m
        const int m = m0 + (e >> 2), k = k0 + 4 * (e & 3);
        ra[q] = m < a.M ? load4<VEC>(A + (int64_t)m * a.lda, k, ke) : none;
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = tid + q * SG_THREADS, k = k0 + (e >> 4), n = n0 + 4 * (e & 15);
      rb[q] = k < ke ? load4<VEC>(B + (int64_t)k * a.ldb, n, a.N) : none;
    }
  };
  auto stage = [&](int s) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = tid + q * SG_THREADS;
      if (TRANS_A) {
        *reinterpret_cast<float4 *>(&As[s][e >> 5][4 * (e & 31)]) = ra[q];
      } else {
        const int m = e >> 2, k = 4 * (e & 3);
        As[s][k][m] = ra[q].x;
        As[s][k + 1][m] = ra[q].y;
        As[s][k + 2][m] = ra[q].z;
        As[s][k + 3][m] = ra[q].w;
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = tid + q * SG_THREADS;
      *reinterpret_cast<float4 *>(&Bs[s][e >> 4][4 * (e & 15)]) = rb[q];
    }
  };
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  fetch(kb);
  stage(0);
  __syncthreads();
  int s = 0;
  for (int k0 = kb; k0 < ke; k0 += TK, s ^= 1) {
    const bool more = k0 + TK < ke;
    if (more) fetch(k0 + TK);
#pragma unroll
    for (int k = 0; k < TK; ++k) {
      float av[8], bv[8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        *reinterpret_cast<float4 *>(av + 4 * h) =
            *reinterpret_cast<const float4 *>(&As[s][k][64 * h + 4 * ty]);
        *reinterpret_cast<float4 *>(bv + 4 * h) =
            *reinterpret_cast<const float4 *>(&Bs[s][k][32 * h + 4 * tx]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    if (more) stage(s ^ 1);  // its readers passed the barrier of the slice before
    __syncthreads();
  }
  const bool whole = a.kc >= a.K;
  float *C = whole ? a.C + z * a.sc : a.C + ((int64_t)split * a.nprob + z) * a.M * a.N;
  const int ldc = whole ? a.ldc : a.N;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + 64 * (i >> 2) + 4 * ty + (i & 3);
    if (m >= a.M) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = n0 + 32 * h + 4 * tx;
      float *c = C + (int64_t)m * ldc + n;
      if (VEC) {
        if (n < a.N)
          *reinterpret_cast<float4 *>(c) = make_float4(acc[i][4 * h], acc[i][4 * h + 1],
                                                       acc[i][4 * h + 2], acc[i][4 * h + 3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < a.N) c[j] = acc[i][4 * h + j];
      }
    }
  }
}

// C[z] = the sum of its splits' partial sums, in order (lower: of tiles not left out).
__global__ void __launch_bounds__(256) sgemm_sum_kernel(SgemmArgs a, const float *part, int splits,
                                                        float *out) {
  const int64_t mn = (int64_t)a.M * a.N, all = mn * a.nprob;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < all;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int z = (int)(i / mn), m = (int)(i % mn / a.N), n = (int)(i % a.N);
    if (a.lower && n / TN * TN > m / TM * TM + TM - 1) continue;
    float sum = 0.f;
    for (int s = 0; s < splits; ++s) sum += __ldcg(part + s * all + i);
    out[z * a.sc + (int64_t)m * a.ldc + n] = sum;
  }
}

}  // namespace

tsvd_status sgemm_batched(bool trans_a, int M, int N, int K, const float *A, int lda, int64_t sa,
                          const float *B, int ldb, int64_t sb, float *C, int ldc, int64_t sc,
                          int nprob, void *work, size_t work_bytes, cudaStream_t st, bool lower) {
  if (M <= 0 || N <= 0 || nprob <= 0) return TSVD_OK;
  const int tm = (int)ceil_div(M, TM), tn = (int)ceil_div(N, TN);
  // split K until every SM has three CTAs, with 64 values of K or more each
  const int64_t tiles = (int64_t)tm * tn * nprob;
  int64_t splits = std::min<int64_t>({ceil_div(3 * sm_count(), tiles), (int64_t)K / 64,
                                      (int64_t)SG_MAX_SPLIT, 65535 / nprob,
                                      (int64_t)(work_bytes / sizeof(float)) /
                                          ((int64_t)M * N * nprob)});
  int kc = K;
  if (splits > 1) {
    kc = (int)round_up(ceil_div(K, splits), TK);
    splits = ceil_div(K, kc);
  }
  if (splits <= 1) {
    splits = 1;
    kc = std::max(K, 1);
  }
  if (nprob > 65535) return fail(TSVD_ERR_INVALID, "sgemm: %d problems", nprob);
  float *part = static_cast<float *>(work);
  SgemmArgs a{M, N, K, A, lda, sa, B, ldb, sb, splits > 1 ? part : C, ldc, sc, kc, nprob,
              lower ? 1 : 0};
  auto four = [](const void *p, int64_t x, int64_t y, int64_t z) {
    return ((uintptr_t)p % 16 == 0) && x % 4 == 0 && y % 4 == 0 && z % 4 == 0;
  };
  const bool vec = four(A, lda, sa, trans_a ? M : K) && four(B, ldb, sb, N) &&
                   (splits > 1 ? four(part, 0, 0, 0) : four(C, ldc, sc, 0));
  auto *fn = trans_a ? (vec ? sgemm_kernel<true, true> : sgemm_kernel<true, false>)
                     : (vec ? sgemm_kernel<false, true> : sgemm_kernel<false, false>);
  fn<<<dim3((unsigned)tn, (unsigned)tm, (unsigned)(nprob * splits)), SG_THREADS, 0, st>>>(a);
  TSVD_LAUNCH_CHECK();
  if (splits > 1) {
    sgemm_sum_kernel<<<grid_for((int64_t)M * N * nprob, 256), 256, 0, st>>>(a, part, (int)splits,
                                                                            C);
    TSVD_LAUNCH_CHECK();
  }
  return TSVD_OK;
}

}  // namespace tsvd
