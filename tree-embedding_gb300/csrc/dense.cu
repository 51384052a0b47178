// Dense kernels of the blockwise randomized SVD and the tree merge.
//
//  gemm_fwd / gemm_bwd : the two products of every frPCA pass,
//      Y = A X   and   Z = A^T Y   (Code/frpca.c:259,280,282,294 via
//      csr_matrix_{,transpose_}matrix_mult, ..._ext.c:364-398),
//    with A stored once per block as A^T in half precision (vertex-major, the
//    layout the PPR state has) and the skinny operand split into hi + lo
//    halves so that it keeps ~22 significant bits. 5th-generation tensor
//    cores: tcgen05.mma kind::f16 into a tensor-memory accumulator (fp32),
//    operands brought into shared memory by TMA (cp.async.bulk.tensor) in a
//    5-stage pipeline of full / empty mbarriers.
//  gram_batched : X^T X with compensated sums per row chunk, chunks summed in
//    fp64 (Code/frpca.c:101, cblas_dgemm TN).
//  apply_right_batched : X W, with chol_inverse_batched (chol.cu) the
//    CholeskyQR2 normalization replacing LUfraction (Code/frpca.c:4-41); the
//    span of the basis, which is all the power iteration keeps, is the same.
#include <algorithm>
#include <map>
#include <mutex>
#include <cstring>

#include "internal.h"

namespace tsvd {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// ------------------------------------------------------------------ GEMM tiles
// The two frPCA products run on the 5th-generation tensor cores: one CTA
// computes three 128 x 144 fp32 tiles in tensor memory (TMEM) with tcgen05.mma
// kind::f16, issued by one thread. The operand tiles are brought into shared
// memory by the Tensor Memory Accelerator: one producer thread issues
// cp.async.bulk.tensor copies whose completion is counted (in bytes) on the
// stage's "full" mbarrier; the MMA thread waits on it, issues the stage's
// MMAs and commits them to the stage's "empty" mbarrier, which the producer
// waits on before refilling the stage. Four stages of 32 K values are in
// flight.
//
// Shared-memory layouts are the swizzled canonical ones of the tensor cores,
// written by the TMA with the matching swizzle, so that every copy moves
// whole 64- or 128-byte rows:
//  * skinny operand (hi and lo halves, [k][144] in global memory, MN-major):
//    three 64-column atoms of 32 K rows x 128 bytes, 128-byte swizzle
//    (columns 144-191 of the third atom are outside the tensor: zeros, never
//    read by an N = 144 MMA). Descriptor: LBO = 4 KB between atoms along N,
//    SBO = 1 KB between 8-row groups along K;
//  * A of the forward product (A^T [n_c][Sp]: M = Sp contiguous, MN-major):
//    six 64-row atoms of 32 K rows x 128 bytes, 128-byte swizzle; row tile h
//    is atoms 2h, 2h + 1 (LBO 4 KB, SBO 1 KB);
//  * A of the backward product (A^T rows are M, K = Sp contiguous, K-major):
//    one 128-row x 64-byte box per row tile, 64-byte swizzle (SBO = 512
//    bytes between 8-row groups); the second 16-deep K step starts 32 bytes
//    into the rows.
// Rows past a block's n_c and K past its end lie outside the tensors, and the
// TMA fills them with zeros. Every copy starts at an innermost coordinate
// that is a multiple of 8 values (16 bytes).
constexpr int BM = 128, MH = 3, BN = kLp, BK = 32, STAGES = 4, GEMM_THREADS = 128;
constexpr int kAtom = 64;                              // values per 128-byte swizzle row
constexpr int kAtomBytes = BK * 128;                   // one 32-row x 128-byte atom: 4 KB
constexpr int kBAtoms = (BN + kAtom - 1) / kAtom;      // 3
constexpr int SA_BYTES = BM * BK * 2;                  // 8 KB per row tile (two atoms)
constexpr int SB_BYTES = kBAtoms * kAtomBytes;         // 12 KB per skinny half
constexpr int STAGE_BYTES = MH * SA_BYTES + 2 * SB_BYTES;
constexpr size_t kGemmSmem = (size_t)STAGES * STAGE_BYTES + 2048;  // + alignment slack, barriers
constexpr int kLayoutSw128 = 2, kLayoutSw64 = 4;       // descriptor swizzle modes
constexpr int kTmemCols = 512;                         // MH accumulators, kAccStride apart
constexpr int kAccStride = 160;
static_assert(MH * kAccStride <= kTmemCols && kAccStride >= BN, "accumulators fit in TMEM");
static_assert(BN % 16 == 0 && BN <= 256, "tcgen05.mma with M = 128 needs N % 16 == 0, N <= 256");
static_assert(STAGE_BYTES % 1024 == 0 && SA_BYTES % 1024 == 0 && kAtomBytes % 1024 == 0,
              "swizzle atoms stay 1024-byte aligned");
static_assert(BM % kAtom == 0 && SA_BYTES == 2 * kAtomBytes, "a row tile is two atoms");

// Counts waits that ran out (a kernel that gives up skips its tile and
// frees its tensor memory; the host turns a non-zero count into an error).
__device__ int g_umma_timeouts = 0;

// tcgen05 shared-memory descriptor: start, leading / stride byte offsets (16-
// byte units), version 1, base offset 0, swizzle mode.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t saddr, int lbo, int sbo, int layout) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)(layout & 7) << 61;
  return d;
}

// kind::f16 instruction descriptor: fp32 accumulator, fp16 A and B, A K-major
// (0) or MN-major (1), B MN-major, N = BN, M = BM.
__host__ __device__ constexpr uint32_t umma_idesc(int a_mn) {
  return (1u << 4) | ((uint32_t)a_mn << 15) | (1u << 16) | ((uint32_t)(BN >> 3) << 17) |
         ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (int it = 0; it < (1 << 24); ++it)
    if (mbar_try(bar, parity)) return true;
  return false;
}

// The same wait, also ending (false) once the CTA's failure flag is set.
__device__ __forceinline__ bool mbar_wait_or_fail(uint32_t bar, uint32_t parity,
                                                  volatile int *failed) {
  for (int it = 0; it < (1 << 24); ++it) {
    if (mbar_try(bar, parity)) return true;
    if (*failed) return false;
  }
  return false;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

struct GemmArgs {
  const CUtensorMap *maps;  // 3 per problem: A, skinny hi, skinny lo
  const int32_t *ncols;
  int lda;  // Sp
  int has_lo;
  float *const *out;
  float scale;
  int splits;  // fwd split-K
};

// FWD: Y (Sp x BN) [+]= A (Sp x nc) * X (nc x BN), A given as A^T [nc][lda].
// BWD: Z (nc x BN) = A^T (nc x Sp) * Y (Sp x BN).
// The skinny operand is hi (+ lo), both accumulated into the same tile.
template <bool FWD>
__global__ void __launch_bounds__(GEMM_THREADS, 1) umma_gemm_kernel(GemmArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // swizzle atoms must sit on 1024-byte boundaries of the shared window
  unsigned char *stage_base =
      smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint64_t *full = reinterpret_cast<uint64_t *>(stage_base + (size_t)STAGES * STAGE_BYTES);
  uint64_t *empty = full + STAGES;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(empty + STAGES);
  volatile int *failed = reinterpret_cast<volatile int *>(tslot + 1);
  const int prob = blockIdx.z;
  const int nc = a.ncols[prob];
  const int m0 = blockIdx.x * (BM * MH);
  const int mrows = FWD ? a.lda : nc;  // rows of the output
  if (m0 >= mrows) return;
  const int nk_total = FWD ? (nc + BK - 1) / BK : a.lda / BK;
  const int per = (nk_total + a.splits - 1) / a.splits;
  const int kt0 = blockIdx.y * per, kt1 = min(nk_total, kt0 + per);
  if (kt0 >= kt1) return;
  const int nk = kt1 - kt0;
  const CUtensorMap *map_a = a.maps + 3 * (int64_t)prob;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t tx_bytes = MH * SA_BYTES + (a.has_lo ? 2 : 1) * SB_BYTES;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(full + s), 1);
      mbar_init(smem_u32(empty + s), 1);
    }
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(tslot)),
                 "n"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *tslot;

  if (warp == 0 && lane == 0) {
    // producer: fill stage i % STAGES with K tile kt0 + i once the MMAs that
    // read its previous contents (tile i - STAGES) have completed
    for (int j = 0; j < 3; ++j)
      asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(map_a + j))
                   : "memory");
    int filled = 0;
    for (int i = 0; i < nk; ++i) {
      const int st = i % STAGES;
      if (i >= STAGES &&
          !mbar_wait_or_fail(smem_u32(empty + st), (uint32_t)((i / STAGES - 1) & 1), failed)) {
        *failed = 1;
        break;
      }
      const uint32_t fb = smem_u32(full + st);
      const uint32_t sa = smem_u32(stage_base + (size_t)st * STAGE_BYTES);
      const int k0 = (kt0 + i) * BK;
      mbar_expect_tx(fb, tx_bytes);
      if (FWD) {  // six 64-row atoms of M at K rows k0 .. k0 + 31
#pragma unroll
        for (int t = 0; t < MH * BM / kAtom; ++t)
          tma_load_2d(sa + t * kAtomBytes, map_a, m0 + t * kAtom, k0, fb);
      } else {  // per row tile: 128 rows of M, K values k0 .. k0 + 31
#pragma unroll
        for (int h = 0; h < MH; ++h) tma_load_2d(sa + h * SA_BYTES, map_a, k0, m0 + h * BM, fb);
      }
#pragma unroll
      for (int t = 0; t < kBAtoms; ++t) {
        tma_load_2d(sa + MH * SA_BYTES + t * kAtomBytes, map_a + 1, t * kAtom, k0, fb);
        if (a.has_lo)
          tma_load_2d(sa + MH * SA_BYTES + SB_BYTES + t * kAtomBytes, map_a + 2, t * kAtom, k0, fb);
      }
      filled = i + 1;
    }
    // no copy may still be writing shared memory when the CTA exits: wait for
    // the last fill of every stage (those the MMA thread consumed are done)
    for (int i = max(0, filled - STAGES); i < filled; ++i)
      if (!mbar_wait(smem_u32(full + i % STAGES), (uint32_t)((i / STAGES) & 1))) *failed = 1;
  } else if (warp == 1 && lane == 0) {
    // MMA issuer
    constexpr uint32_t idesc = umma_idesc(FWD ? 1 : 0);
    // per 16-deep K step: MN-major tiles advance two 8-row groups (2 KB),
    // the K-major A 32 bytes along its rows
    constexpr int a_lbo = FWD ? kAtomBytes : 16, a_sbo = FWD ? 1024 : 512;
    constexpr int a_layout = FWD ? kLayoutSw128 : kLayoutSw64, a_kstep = FWD ? 2048 : 32;
    int issued = 0;
    for (int i = 0; i < nk; ++i) {
      const int st = i % STAGES;
      if (!mbar_wait_or_fail(smem_u32(full + st), (uint32_t)((i / STAGES) & 1), failed)) {
        *failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t sa = smem_u32(stage_base + (size_t)st * STAGE_BYTES);
      const uint32_t sbh = sa + MH * SA_BYTES, sbl = sbh + SB_BYTES;
#pragma unroll
      for (int ks = 0; ks < BK / 16; ++ks) {
        const uint64_t bdh = umma_smem_desc(sbh + ks * 2048, kAtomBytes, 1024, kLayoutSw128);
        const uint64_t bdl = umma_smem_desc(sbl + ks * 2048, kAtomBytes, 1024, kLayoutSw128);
        const uint32_t acc0 = (i > 0 || ks > 0) ? 1u : 0u;
#pragma unroll
        for (int h = 0; h < MH; ++h) {
          const uint64_t ad =
              umma_smem_desc(sa + h * SA_BYTES + ks * a_kstep, a_lbo, a_sbo, a_layout);
          const uint32_t td = tmem + (uint32_t)(h * kAccStride);
          asm volatile(
              "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(td),
              "l"(ad), "l"(bdh), "r"(idesc), "r"(acc0));
          if (a.has_lo)
            asm volatile(
                "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(td),
                "l"(ad), "l"(bdl), "r"(idesc), "r"(1u));
        }
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
              smem_u32(empty + st))
          : "memory");
      issued = i + 1;
    }
    // the last commit covers every MMA issued before it; wait for it even
    // after a failure, so no MMA still writes the tensor memory freed below
    if (issued > 0) {
      const int li = issued - 1;
      if (!mbar_wait(smem_u32(empty + li % STAGES), (uint32_t)((li / STAGES) & 1))) *failed = 1;
    }
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const bool ok = *failed == 0;
  if (!ok) {
    if (lane == 0) atomicAdd(&g_umma_timeouts, 1);
  } else {
    // epilogue: warp w reads TMEM lanes 32w..32w+31 of accumulator h = output
    // rows m0 + 128 h + 32 w + lane
    float *out = a.out[prob];
    const bool atomic = FWD && a.splits > 1;
#pragma unroll 1
    for (int h = 0; h < MH; ++h) {
      const int row = m0 + h * BM + warp * 32 + lane;
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 16) {
        uint32_t v[16];
        const uint32_t ta =
            tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(h * kAccStride + c0);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
            "%14,%15}, [%16];\n"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
              "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(ta));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        if (row < mrows) {
          float *o = out + (int64_t)row * BN + c0;
          if (atomic) {  // split-K partial tiles: float4 reductions (rows are 576-byte aligned)
#pragma unroll
            for (int j = 0; j < 16; j += 4)
              atomicAdd(reinterpret_cast<float4 *>(o + j),
                        make_float4(__uint_as_float(v[j]) * a.scale,
                                    __uint_as_float(v[j + 1]) * a.scale,
                                    __uint_as_float(v[j + 2]) * a.scale,
                                    __uint_as_float(v[j + 3]) * a.scale));
          } else {
#pragma unroll
            for (int j = 0; j < 16; j += 4)
              *reinterpret_cast<float4 *>(o + j) = make_float4(
                  __uint_as_float(v[j]) * a.scale, __uint_as_float(v[j + 1]) * a.scale,
                  __uint_as_float(v[j + 2]) * a.scale, __uint_as_float(v[j + 3]) * a.scale);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                 "n"(kTmemCols));
}

// ------------------------------------------------------------------ Gram
// Compensated sums of error-free products (Ogita, Rump, Oishi, "Accurate sum and dot
// product", SISC 2005): S + C carries a chunk's sum to 2^-45 of the sum of its
// terms' magnitudes, and the chunks are added in fp64. Of TwoSum's error of u = S + p,
// (S - S') + (p - z) with z = u - S and S' = u - z, the second difference is taken of the
// exact product instead of p, by one fused multiply-add: eight operations a term, where
// p's own error and TwoSum take ten. (u itself from the exact product would take seven,
// but u - z then rounds where S and the product cancel: 2^-28. Four are enough with S held
// near an anchor above the column norms, but entries then carry 2^-45 of the norms'
// product, and those of nearly orthogonal columns 2^-30 of their terms.) The kernel is
// bound by the issue of these operations; with the sum of the chunks, measured, 32
// problems of 1500 x 256: ten 996 us, these 652, anchored 583; 64 of 3125 x 133: 1084,
// 732, 643.
constexpr int GRAM_MIN_ROWS = 128;    // rows per CTA (one fp64 partial per chunk); fewer
                                      // where CTAs are few (gram_batched)
constexpr int GRAM_MAX_CHUNKS = 2048;  // chunks over all problems (bounds the work buffer)
constexpr int GRAM_HALVED = 64;   // chunks of a problem that halving may make
constexpr int GRAM_SUB = 32;      // rows staged in smem at a time
constexpr int GRAM_THREADS = 256;
constexpr int GRAM_LMAX = 256;

struct GramArgs {
  const float *const *x;
  const int32_t *rows;
  int ld;
  int l;
  int tiles;      // ceil(l/4)
  int nchunks;    // per problem
  int chunk_rows;
  double *work;   // [prob][chunk][l*l]
};

// (S, C) += a b
__device__ __forceinline__ void comp_add(float &S, float &C, float a, float b) {
  const float u = __fadd_rn(S, __fmul_rn(a, b)), z = __fsub_rn(u, S);
  C = __fadd_rn(C, __fadd_rn(__fsub_rn(S, __fsub_rn(u, z)), __fmaf_rn(a, b, -z)));
  S = u;
}

// grid: (row chunk, tile group, problem). A thread owns one upper-triangle 4 x 4
// tile of the l x l output and accumulates it over the chunk's rows.
__global__ void __launch_bounds__(GRAM_THREADS) gram_partial_kernel(GramArgs a) {
  extern __shared__ __align__(16) float sx[];  // [GRAM_SUB][4 tiles]
  const int prob = blockIdx.z, chunk = blockIdx.x;
  const int rows = a.rows[prob];
  const int r0 = chunk * a.chunk_rows;
  double *out = a.work + ((int64_t)prob * a.nchunks + chunk) * a.l * a.l;
  const int T = a.tiles, sld = 4 * T;  // staged row stride covers every 4 x 4 tile column
  const float *x = a.x[prob];
  const int r1 = min(rows, r0 + a.chunk_rows);
  const int t = blockIdx.y * GRAM_THREADS + threadIdx.x;
  const bool mine = t < T * (T + 1) / 2;
  int ti = 0, tj = 0;
  if (mine) {
    int J = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
    while ((J + 1) * (J + 2) / 2 <= t) ++J;
    while (J * (J + 1) / 2 > t) --J;
    ti = 4 * (t - J * (J + 1) / 2);
    tj = 4 * J;
  }
  float S[16], C[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) S[e] = C[e] = 0.f;
  for (int rb = r0; rb < r1; rb += GRAM_SUB) {
    const int nr = min(GRAM_SUB, r1 - rb);
    __syncthreads();
    for (int i = threadIdx.x; i < GRAM_SUB * sld; i += GRAM_THREADS) {
      int rr = i / sld, cc = i % sld;
      sx[i] = (rr < nr && cc < a.l) ? x[(int64_t)(rb + rr) * a.ld + cc] : 0.f;
    }
    __syncthreads();
    if (!mine) continue;
#pragma unroll 2
    for (int rr = 0; rr < nr; ++rr) {
      float xi[4], xj[4];
      *reinterpret_cast<float4 *>(xi) = *reinterpret_cast<const float4 *>(sx + rr * sld + ti);
      *reinterpret_cast<float4 *>(xj) = *reinterpret_cast<const float4 *>(sx + rr * sld + tj);
#pragma unroll
      for (int e = 0; e < 16; ++e) comp_add(S[e], C[e], xi[e >> 2], xj[e & 3]);
    }
  }
  if (!mine) return;
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int i = ti + (e >> 2), j = tj + (e & 3);
    if (i < a.l && j < a.l) out[i * a.l + j] = (double)S[e] + (double)C[e];
  }
}

// Sums the chunks' upper 4 x 4 tiles and mirrors them.
__global__ void gram_reduce_kernel(const double *__restrict__ work, int nchunks, int l,
                                   double *const *g, int nprob) {
  const int prob = blockIdx.y;
  const int64_t ll = (int64_t)l * l;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ll;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / l), c = (int)(i % l);
    if (r / 4 > c / 4) continue;
    double s = 0.0;
    const double *w = work + (int64_t)prob * nchunks * ll + i;
#pragma unroll 8
    for (int k = 0; k < nchunks; ++k) s += w[k * ll];
    g[prob][i] = s;
    g[prob][(int64_t)c * l + r] = s;
  }
}

// ------------------------------------------------------------------ X * W
// Y = X W diag(colscale) (rows x n_out, written up to ldy <= 144 columns,
// zero past n_out), optionally split into fp16 hi/lo. A CTA takes a tile of 32 R
// rows: warp w owns columns 16 w .. 16 w + 15, lane l rows l, l + 32, ..; K goes
// APPLY_KS at a time through two stages of shared memory, the next slab of X and W
// on its way (cp.async) while one is multiplied. Per four k a warp reads its X as
// R float4 a lane and its 64 W values by broadcast, 32 shared-memory wavefronts for
// 256 FMAs at R = 4, whose issue (three operands each from the register file, about
// 75 lanes a clock) bounds large batches; small ones wait for their slabs, and take
// R = 1. The tile goes out through shared memory, in whole rows of 16-byte stores.
// upper: W is upper triangular, and a warp stops at its last column's row. Every
// sum runs over k in ascending order, whatever R. X may alias Y (in-place
// CholeskyQR): a tile is read whole before it is written. Measured, slabs fetched
// between barriers and 4-byte stores before: 64 problems of 3125 x 133 (triangular,
// with the split) 406 -> 205 us, 32 of 1500 x 256 208 -> 112, one of 1500 x 133 28
// -> 13, of 1500 x 256 47 -> 20.
constexpr int APPLY_THREADS = 288;
constexpr int APPLY_KS = 32;
constexpr int APPLY_WLD = kLp;            // staged W row
constexpr int APPLY_OLD = kLp + 4;        // output tile row
struct ApplyArgs {
  const float *const *x;
  const int32_t *rows;
  int ldx;
  const float *const *w;
  int ldw;
  int n_in, n_out;
  const float *const *colscale;
  float *const *y;
  int ldy;
  __half *const *yhi;
  __half *const *ylo;
  float split_scale;
  int upper;
  int vec;  // ldx and ldw are multiples of four
};

constexpr int APPLY_XLD = APPLY_KS + 4;   // staged X row
template <int R>
constexpr size_t apply_smem() {
  return sizeof(float) * std::max((size_t)2 * (32 * R * APPLY_XLD + APPLY_KS * APPLY_WLD),
                                  (size_t)32 * R * APPLY_OLD);
}

// BYTES (16 or 4) to shared memory, of which the first `in` come from src.
template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(float *dst, const float *src, int in) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(in));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(in));
}

// One slab (APPLY_KS deep, from k0) of X and W to shared memory, asynchronously; what
// lies outside is zero. VEC: by 16 bytes (rows that begin on 16 bytes), else by 4.
template <int R, bool VEC>
__device__ __forceinline__ void apply_fetch(const ApplyArgs &a, const float *X, const float *W,
                                            int r0, int rows, int k0, float *sx, float *sw) {
  constexpr int V = VEC ? 4 : 1;
  const int ks = min(APPLY_KS, a.n_in - k0);
  for (int i = threadIdx.x; i < 32 * R * (APPLY_KS / V); i += APPLY_THREADS) {
    const int k = V * (i % (APPLY_KS / V)), rr = i / (APPLY_KS / V);
    const int in = r0 + rr < rows ? max(0, min(V, ks - k)) : 0;
    cp_async_zfill<4 * V>(sx + rr * APPLY_XLD + k,
                          in ? X + (int64_t)(r0 + rr) * a.ldx + k0 + k : X, 4 * in);
  }
  for (int i = threadIdx.x; i < APPLY_KS * (APPLY_WLD / V); i += APPLY_THREADS) {
    const int c = V * (i % (APPLY_WLD / V)), k = i / (APPLY_WLD / V);
    const int in = k < ks ? max(0, min(V, a.n_out - c)) : 0;
    cp_async_zfill<4 * V>(sw + k * APPLY_WLD + c, in ? W + (int64_t)(k0 + k) * a.ldw + c : W,
                          4 * in);
  }
}

template <int R>
__global__ void __launch_bounds__(APPLY_THREADS, 2) apply_right_kernel(ApplyArgs a) {
  extern __shared__ __align__(16) float sm[];
  constexpr int RT = 32 * R, STAGE = RT * APPLY_XLD + APPLY_KS * APPLY_WLD;
  const int prob = blockIdx.y, r0 = blockIdx.x * RT;
  const int rows = a.rows[prob];
  if (r0 >= rows) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c0 = 16 * warp;
  const float *X = a.x[prob], *W = a.w[prob];
  const bool act = c0 < a.n_out;
  float acc[R][16];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[r][j] = 0.f;
  const bool vec = a.vec && (((uintptr_t)X | (uintptr_t)W) & 15) == 0;
  auto fetch = [&](int k0, float *to) {
    if (vec) apply_fetch<R, true>(a, X, W, r0, rows, k0, to, to + RT * APPLY_XLD);
    else apply_fetch<R, false>(a, X, W, r0, rows, k0, to, to + RT * APPLY_XLD);
    asm volatile("cp.async.commit_group;\n" ::);
  };
  fetch(0, sm);
  for (int k0 = 0, s = 0; k0 < a.n_in; k0 += APPLY_KS, s ^= 1) {
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();  // the slab is there, and every warp is done with the one before
    if (k0 + APPLY_KS < a.n_in) fetch(k0 + APPLY_KS, sm + (s ^ 1) * STAGE);
    if (!act || (a.upper && k0 > c0 + 15)) continue;
    const float *sx = sm + s * STAGE + lane * APPLY_XLD, *sw = sm + s * STAGE + RT * APPLY_XLD + c0;
    const int ks = min(APPLY_KS, a.n_in - k0);  // (what lies past it is zero)
    for (int k = 0; k < ks; k += 4) {
      float xv[R][4];
#pragma unroll
      for (int r = 0; r < R; ++r)
        *reinterpret_cast<float4 *>(xv[r]) =
            *reinterpret_cast<const float4 *>(sx + 32 * r * APPLY_XLD + k);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float wv[16];
#pragma unroll
        for (int j = 0; j < 16; j += 4)
          *reinterpret_cast<float4 *>(wv + j) =
              *reinterpret_cast<const float4 *>(sw + (k + q) * APPLY_WLD + j);
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[r][j] = fmaf(xv[r][q], wv[j], acc[r][j]);
      }
    }
  }
  __syncthreads();  // every warp is done with the staged slabs
  float *so = sm;   // [RT][APPLY_OLD]
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int j = 0; j < 16; j += 4)
      *reinterpret_cast<float4 *>(so + (lane + 32 * r) * APPLY_OLD + c0 + j) =
          make_float4(acc[r][j], acc[r][j + 1], acc[r][j + 2], acc[r][j + 3]);
  __syncthreads();
  const float *cs = a.colscale ? a.colscale[prob] : nullptr;
  float *Y = a.y[prob];
  __half *Yh = a.yhi ? a.yhi[prob] : nullptr;
  __half *Yl = a.ylo ? a.ylo[prob] : nullptr;
  auto split = [&](float v, __half &h, __half &l) {
    const float sv = v * a.split_scale;
    h = __float2half_rn(sv);
    l = __float2half_rn(sv - __half2float(h));
  };
  // (columns past n_out are zero, as W was staged as zero there)
  if (a.ldy % 4 == 0 && (((uintptr_t)Y | (uintptr_t)Yh | (uintptr_t)Yl) & 15) == 0) {
    const int v4 = a.ldy / 4;
    for (int i = tid; i < RT * v4; i += APPLY_THREADS) {
      const int rr = i / v4, c = 4 * (i % v4);
      if (r0 + rr >= rows) break;
      float4 v = *reinterpret_cast<const float4 *>(so + rr * APPLY_OLD + c);
      if (cs && c < a.n_out) {
        v.x *= cs[c];
        v.y *= c + 1 < a.n_out ? cs[c + 1] : 0.f;
        v.z *= c + 2 < a.n_out ? cs[c + 2] : 0.f;
        v.w *= c + 3 < a.n_out ? cs[c + 3] : 0.f;
      }
      const int64_t at = (int64_t)(r0 + rr) * a.ldy + c;
      *reinterpret_cast<float4 *>(Y + at) = v;
      if (Yh) {
        __align__(8) __half h[4], l[4];
        split(v.x, h[0], l[0]);
        split(v.y, h[1], l[1]);
        split(v.z, h[2], l[2]);
        split(v.w, h[3], l[3]);
        *reinterpret_cast<uint2 *>(Yh + at) = *reinterpret_cast<const uint2 *>(h);
        *reinterpret_cast<uint2 *>(Yl + at) = *reinterpret_cast<const uint2 *>(l);
      }
    }
    return;
  }
  for (int i = tid; i < RT * a.ldy; i += APPLY_THREADS) {
    const int rr = i / a.ldy, c = i % a.ldy;
    if (r0 + rr >= rows) break;
    const float v = so[rr * APPLY_OLD + c] * (cs && c < a.n_out ? cs[c] : 1.f);
    const int64_t at = (int64_t)(r0 + rr) * a.ldy + c;
    Y[at] = v;
    if (Yh) split(v, Yh[at], Yl[at]);
  }
}

}  // namespace

// ------------------------------------------------------------------ host side
int sm_count() {
  // initialized once, thread-safely (a pipelined run calls this from two threads)
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 1;
  }();
  return n;
}

int grid_for(int64_t work_items, int threads_per_block, int blocks_per_sm) {
  int64_t need = ceil_div(std::max<int64_t>(work_items, 1), threads_per_block);
  int64_t cap = (int64_t)sm_count() * blocks_per_sm;
  return (int)std::max<int64_t>(1, std::min(need, cap));
}

// A kernel's dynamic shared-memory ceiling is a process-wide attribute, and
// sessions on other threads launch the same kernels with other sizes: it is
// only ever raised (under a lock), so no thread's launch can find it lowered
// below what that launch asks for.
tsvd_status raise_smem_ceiling(const void *fn, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, size_t> ceiling;
  int dev = 0;
  TSVD_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(mu);
  size_t &cur = ceiling[std::make_pair(fn, dev)];
  if (bytes <= cur) return TSVD_OK;
  TSVD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  cur = bytes;
  return TSVD_OK;
}

// cuTensorMapEncodeTiled, resolved from the driver at run time (the library
// links only the runtime).
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn tensor_map_encoder() {
  static const EncodeTiledFn fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    cudaError_t e =
        cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return (EncodeTiledFn) nullptr;
    }
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// A row-major fp16 matrix [rows][pitch] (the first `cols` values of each row
// in use) as a 2-D tensor for the TMA: {cols, rows}, a {box_cols, box_rows}
// box, the given shared-memory swizzle.
static tsvd_status encode_2d(CUtensorMap *m, const __half *base, int64_t cols, int64_t rows,
                             int pitch, int box_cols, int box_rows, CUtensorMapSwizzle swz) {
  const EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return fail(TSVD_ERR_DEVICE, "cuTensorMapEncodeTiled is not available from the driver");
  if (!base || (reinterpret_cast<uintptr_t>(base) & 15) != 0 || pitch % 8 != 0)
    return fail(TSVD_ERR_INVALID, "tensor map: operand %p / pitch %d not 16-byte aligned",
                (const void *)base, pitch);
  const cuuint64_t dims[2] = {(cuuint64_t)std::max<int64_t>(cols, 1),
                              (cuuint64_t)std::max<int64_t>(rows, 1)};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch * 2};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  const cuuint32_t estride[2] = {1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void *)base, dims, strides, box,
                        estride, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(TSVD_ERR_DEVICE,
                "cuTensorMapEncodeTiled: error %d (%lld x %lld, pitch %d, box %d x %d)", (int)r,
                (long long)rows, (long long)cols, pitch, box_rows, box_cols);
  return TSVD_OK;
}

tsvd_status gemm_encode_maps(int fwd, int nprob, const __half *const *at, const int32_t *nc,
                             int lda, const __half *const *hi, const __half *const *lo,
                             CUtensorMap *out) {
  for (int i = 0; i < nprob; ++i) {
    CUtensorMap *m = out + 3 * (int64_t)i;
    if (fwd)  // M = Sp along the rows of A^T, K = its n_c rows: 64 x 32 boxes
      TSVD_TRY(encode_2d(m, at[i], lda, nc[i], lda, kAtom, BK, CU_TENSOR_MAP_SWIZZLE_128B));
    else      // K = Sp along the rows, M = the n_c rows: 32 x 128 boxes
      TSVD_TRY(encode_2d(m, at[i], lda, nc[i], lda, BK, BM, CU_TENSOR_MAP_SWIZZLE_64B));
    const int64_t brows = fwd ? nc[i] : lda;
    TSVD_TRY(encode_2d(m + 1, hi[i], BN, brows, BN, kAtom, BK, CU_TENSOR_MAP_SWIZZLE_128B));
    if (lo && lo[i])
      TSVD_TRY(encode_2d(m + 2, lo[i], BN, brows, BN, kAtom, BK, CU_TENSOR_MAP_SWIZZLE_128B));
    else
      memset(m + 2, 0, sizeof(CUtensorMap));
  }
  return TSVD_OK;
}

tsvd_status gemm_fwd(const GemmBatch &gb, bool has_lo, float *const *y, float *y_base,
                     size_t y_bytes, int sp, int max_nc, float inv_xscale, cudaStream_t st) {
  if (gb.nprob == 0) return TSVD_OK;
  if (sp % BM != 0) return fail(TSVD_ERR_INVALID, "gemm_fwd: Sp = %d not a multiple of %d", sp, BM);
  if (!gb.maps) return fail(TSVD_ERR_INVALID, "gemm_fwd: no tensor maps");
  TSVD_TRY(raise_smem_ceiling((const void *)umma_gemm_kernel<true>, kGemmSmem));
  const int mtiles = (int)ceil_div(sp, BM * MH);
  int splits = 1;
  int64_t base_ctas = (int64_t)mtiles * gb.nprob;
  int64_t target = sm_count();  // one CTA per SM (shared memory)
  if (base_ctas < target)
    splits = (int)std::min<int64_t>(ceil_div(target, base_ctas),
                                    std::max<int64_t>(1, ceil_div(max_nc, 1024)));
  // split-K partial tiles are accumulated with atomics into zeroed outputs
  if (splits > 1) TSVD_CUDA(cudaMemsetAsync(y_base, 0, y_bytes, st));
  GemmArgs a{gb.maps, gb.ncols, gb.lda, has_lo ? 1 : 0, y, inv_xscale, splits};
  dim3 grid(mtiles, splits, gb.nprob);
  umma_gemm_kernel<true><<<grid, GEMM_THREADS, kGemmSmem, st>>>(a);
  TSVD_LAUNCH_CHECK();
  return TSVD_OK;
}

tsvd_status gemm_bwd(const GemmBatch &gb, bool has_lo, float *const *z, int sp, int max_nc,
                     float inv_yscale, cudaStream_t st) {
  if (gb.nprob == 0 || max_nc == 0) return TSVD_OK;
  if (sp % BK != 0) return fail(TSVD_ERR_INVALID, "gemm_bwd: Sp = %d not a multiple of %d", sp, BK);
  if (!gb.maps) return fail(TSVD_ERR_INVALID, "gemm_bwd: no tensor maps");
  TSVD_TRY(raise_smem_ceiling((const void *)umma_gemm_kernel<false>, kGemmSmem));
  GemmArgs a{gb.maps, gb.ncols, sp, has_lo ? 1 : 0, z, inv_yscale, 1};
  dim3 grid((unsigned)ceil_div(max_nc, BM * MH), 1, gb.nprob);
  umma_gemm_kernel<false><<<grid, GEMM_THREADS, kGemmSmem, st>>>(a);
  TSVD_LAUNCH_CHECK();
  return TSVD_OK;
}

tsvd_status gemm_check(cudaStream_t st) {
  int h = 0;
  TSVD_CUDA(cudaMemcpyFromSymbolAsync(&h, g_umma_timeouts, sizeof(int), 0, cudaMemcpyDeviceToHost, st));
  TSVD_CUDA(cudaStreamSynchronize(st));
  if (h != 0) {
    const int zero = 0;
    TSVD_CUDA(cudaMemcpyToSymbolAsync(g_umma_timeouts, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, st));
    TSVD_CUDA(cudaStreamSynchronize(st));
    return fail(TSVD_ERR_TIMEOUT, "tensor-core GEMM: %d warps gave up waiting for their MMAs", h);
  }
  return TSVD_OK;
}

static void gram_chunks(int max_rows, int nprob, int *nchunks, int *chunk_rows) {
  int64_t want = ceil_div(std::max(max_rows, 1), GRAM_MIN_ROWS);
  int64_t cap = std::max<int64_t>(1, GRAM_MAX_CHUNKS / std::max(nprob, 1));
  int64_t nc = std::max<int64_t>(1, std::min(want, cap));
  int64_t cr = round_up(ceil_div(std::max(max_rows, 1), nc), 32);
  *chunk_rows = (int)cr;
  *nchunks = (int)ceil_div(std::max(max_rows, 1), cr);
}

size_t gram_work_bytes(int max_rows, int l, int nprob) {
  int nchunks, cr;
  gram_chunks(max_rows, nprob, &nchunks, &cr);
  return (size_t)nprob * nchunks * l * l * sizeof(double);
}

tsvd_status gram_batched(const float *const *x, const int32_t *rows, int max_rows, int l, int ld,
                         double *const *g, double *work, size_t work_bytes, int nprob,
                         cudaStream_t st) {
  if (nprob == 0) return TSVD_OK;
  if (l > GRAM_LMAX) return fail(TSVD_ERR_INVALID, "gram: l=%d > %d", l, GRAM_LMAX);
  int nchunks, chunk_rows;
  gram_chunks(max_rows, nprob, &nchunks, &chunk_rows);
  if (gram_work_bytes(max_rows, l, nprob) > work_bytes)
    return fail(TSVD_ERR_INVALID, "gram: work buffer too small");
  int tiles = (l + 3) / 4;
  int groups = (int)ceil_div(tiles * (tiles + 1) / 2, GRAM_THREADS);
  // A slab of 32 rows is 3 us of a CTA's issue: halve the chunks until every SM has
  // two, as far as the buffer goes and to GRAM_HALVED of a problem at most, as their sum
  // is a chain. With it, chunks of 128 rows / halved / halved without that limit: 1000 x
  // 69, 4 problems 35 / 20 / 20 us; one of 1500 x 256 47 / 42 / 42, 3000 x 133 43 / 33 /
  // 39, 6000 x 133 47 / 47 / 60, 3000 x 69 37 / 31 / 29; two of 6000 x 37 31 / 31 / 39.
  while (chunk_rows > GRAM_SUB && (int64_t)nchunks * groups * nprob < 2 * sm_count()) {
    const int cr = (int)round_up(chunk_rows / 2, GRAM_SUB);
    const int64_t nc = ceil_div(max_rows, cr);
    if (cr == chunk_rows || nc > GRAM_HALVED || nc * nprob > GRAM_MAX_CHUNKS ||
        (size_t)(nc * nprob) * l * l * sizeof(double) > work_bytes)
      break;
    chunk_rows = cr;
    nchunks = (int)nc;
  }
  size_t smem = (size_t)GRAM_SUB * (4 * tiles) * sizeof(float);
  TSVD_TRY(raise_smem_ceiling((const void *)gram_partial_kernel, smem));
  // (a chunk past a problem's row count writes zeros)
  GramArgs a{x, rows, ld, l, tiles, nchunks, chunk_rows, work};
  gram_partial_kernel<<<dim3(nchunks, groups, nprob), GRAM_THREADS, smem, st>>>(a);
  TSVD_LAUNCH_CHECK();
  gram_reduce_kernel<<<dim3((unsigned)ceil_div((int64_t)l * l, 256), nprob), 256, 0, st>>>(
      work, nchunks, l, g, nprob);
  TSVD_LAUNCH_CHECK();
  return TSVD_OK;
}

tsvd_status apply_right_batched(const float *const *x, const int32_t *rows, int max_rows, int ldx,
                                const float *const *w, int ldw, int n_in, int n_out,
                                const float *const *colscale, float *const *y, int ldy,
                                __half *const *yhi, __half *const *ylo, float split_scale,
                                int nprob, cudaStream_t st, bool upper) {
  if (nprob == 0 || max_rows == 0) return TSVD_OK;
  if (n_out > kLp || ldy > kLp || n_in > 256 || n_in < 1)
    return fail(TSVD_ERR_INVALID, "apply_right: sizes %d %d %d", n_in, n_out, ldy);
  ApplyArgs a{x, rows, ldx, w, ldw, n_in, n_out, colscale, y, ldy, yhi, ylo, split_scale,
              upper ? 1 : 0, ldx % 4 == 0 && ldw % 4 == 0 ? 1 : 0};
  // 128-row tiles where they fill the SMs, 32-row tiles where they do not
  if (ceil_div(max_rows, 128) * nprob >= sm_count()) {
    TSVD_TRY(raise_smem_ceiling((const void *)apply_right_kernel<4>, apply_smem<4>()));
    apply_right_kernel<4><<<dim3((unsigned)ceil_div(max_rows, 128), nprob), APPLY_THREADS,
                            apply_smem<4>(), st>>>(a);
  } else {
    TSVD_TRY(raise_smem_ceiling((const void *)apply_right_kernel<1>, apply_smem<1>()));
    apply_right_kernel<1><<<dim3((unsigned)ceil_div(max_rows, 32), nprob), APPLY_THREADS,
                            apply_smem<1>(), st>>>(a);
  }
  TSVD_LAUNCH_CHECK();
  return TSVD_OK;
}

}  // namespace tsvd
