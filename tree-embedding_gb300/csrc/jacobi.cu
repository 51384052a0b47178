// Two-sided cyclic Jacobi on a Gram, its rows spread over the shared memory of
// a thread-block cluster, replacing LAPACKE_dsyevd (Code/frpca.c:102) and the
// Gram route to LAPACKE_dgesvd (..._mkl.c:1278).
//
// The solver of the entry points that hand singular vectors of a matrix of up to 256
// columns to the caller (tsvd_frpca*, tsvd_merge_svd); the sessions' eigen-solves, and
// the end of a wider merge, take the one-sided solver of eig.cu. The two differ in what
// they are good at. Its rotations shorten the vectors here, by 1e-6 (16 columns) to 4.4e-5
// (256), where the one-sided solver's stay within 1e-6; but a vector's small entries
// keep their relative accuracy here, and only an absolute one of 1e-7 there. Left
// vectors are M V / s: of 300 x 16 with columns of norms 1 to 1e-6 they are orthogonal to
// 3.5e-6 this way and to 3.2e-4 the other, which is what a caller of these entry points
// sees. The tree works on its factors' products, and the root's is off by 0.9e-6 (d = 16)
// to 1.8e-5 (128) by this solver and by 2.0e-6 to 6.4e-6 by the other.
#include <algorithm>

#include <cooperative_groups.h>

#include "internal.h"
#include "jacobi_sched.h"

namespace tsvd {

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ uint32_t remote_addr(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Stores to a CTA of the cluster that count towards its barrier mbar.
__device__ __forceinline__ void send_b32(uint32_t addr, float v, uint32_t mbar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
      "r"(__float_as_uint(v)), "r"(mbar)
      : "memory");
}
__device__ __forceinline__ void send_b64(uint32_t addr, uint64_t v, uint32_t mbar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
      "l"(v), "r"(mbar)
      : "memory");
}
__device__ __forceinline__ bool try_wait(uint32_t mbar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(mbar), "r"(phase)
      : "memory");
  return ok != 0;
}

// ------------------------------------------------------------------ Jacobi
constexpr int JAC_THREADS = 1024;
constexpr int kJacWaits = 1 << 22;  // polls of a barrier before a cluster gives up
constexpr int JAC_MAX_SWEEPS = 30;
constexpr int kJacMaxCluster = 8;  // CTAs per eigenproblem (portable cluster size)
constexpr int kJacRotBase = 512;   // first thread computing rotations (P <= 128 of them)
constexpr int kJacSendBase = 768;  // first thread broadcasting (2 L <= 256 rows)

struct JacobiArgs {
  double *const *g;
  int n;
  float *const *lambda;
  float2 *log;        // [prob][JAC_MAX_SWEEPS][np-1][np/2]
  int32_t *sweeps;    // [prob]
  int32_t *rank;      // [prob][n]
  int32_t *most_sweeps;  // maximum over the batch
  int refine;         // 1: the diagonal is carried in fp64 (see jacobi_kernel)
  const float *const *vinit;  // replay starts from these rows (null: identity)
};

// Shared-memory layout of one CTA of jacobi_kernel (C CTAs per problem).
struct JacobiSmem {
  int n, np, P, L, nbuf;
  size_t off_dbase, off_lam, off_rows, off_cs, off_pt, off_diag, off_coup, off_top,
      off_bot, off_slot, off_flag, off_mbar, bytes;
  __host__ __device__ JacobiSmem(int n_, int C) {
    n = n_;
    np = n + (n & 1);
    P = np / 2;
    L = (P + C - 1) / C;
    nbuf = 2 * L + 4;  // the rows of the owned slots' players, mailboxes [2 parities][L, R]
    size_t o = 0;
    off_dbase = o; o += (size_t)np * sizeof(double);
    off_lam = o; o += (size_t)np * sizeof(double);
    off_rows = o; o += (size_t)nbuf * np * sizeof(float);
    off_cs = o; o += (size_t)P * sizeof(float2);
    off_pt = o; o += (size_t)P * sizeof(float);
    off_diag = o; o += (size_t)2 * np * sizeof(float);  // [parity][player]
    off_coup = o; o += (size_t)2 * P * sizeof(float);   // [parity][slot]
    off_top = o; o += (size_t)2 * L * sizeof(int);      // two map pairs (renamed each round)
    off_bot = o; o += (size_t)2 * L * sizeof(int);
    o = (o + 7) & ~(size_t)7;
    off_slot = o; o += (size_t)2 * L * sizeof(int2);    // [parity][slot]
    off_flag = o; o += (size_t)(JAC_MAX_SWEEPS + 2) * sizeof(int);
    o = (o + 7) & ~(size_t)7;
    off_mbar = o; o += 2 * sizeof(uint64_t);  // [parity]
    bytes = (o + 15) & ~(size_t)15;
  }
};

// One symmetric eigenproblem per thread-block cluster of C CTAs: cyclic
// two-sided Jacobi in the round-robin order of circle_player (np/2 disjoint
// pairs per round, np - 1 rounds per sweep). CTA c owns the pair slots
// [c L, c L + L) and holds the full rows (indexed by player, so a warp's
// lanes touch consecutive words) of the two players of each owned slot.
// A round: every CTA applies all of the round's rotations to its rows, 2 x 2
// block by block (G <- J_k1^T G J_k2, each entry summed in an order that is
// the same for its transposed twin, so the two copies of an entry that
// different CTAs hold stay equal); then the schedule advances: each CTA
// passes one row to each neighbour (into the neighbour's mailbox, in
// distributed shared memory) and broadcasts, for every row it holds, the
// diagonal entry and the coupling to the row's next partner. These are stores that
// count their bytes on a barrier in the receiver (st.async, mbarrier): a CTA goes on
// when its round's bytes have come, one trip, where stores and a cluster barrier
// after them take two. Meanwhile it renames its rows (circle_arrivals, circle_next);
// then it computes all rotations of the next round itself, from the same values in
// the same order, so every CTA has the same rotations without a second exchange.
// Mailboxes, broadcast values and barriers alternate between two by round parity:
// nobody sends for round g + 2 before it has what all others send in g + 1, and so
// nothing is overwritten that is yet to be read. A wait that runs out (kJacWaits)
// makes the CTA leave at the sweep's end, and the solve an error.
//
// Rotate when the pair is coupled: relative to the pair (Demmel-Veselic) and
// above an absolute floor. The first pass only resolves the couplings above
// 1e-5 of max|a_ii| (a few sweeps: the Grams of merges and of frPCA's Z are
// nearly diagonal at that scale); it settles in fp32 the strong couplings
// whose small eigenvalues come from cancellation, which H = V^T G V then
// recomputes in fp64. Refinement mode (a.refine): g = H, the diagonal is kept
// as an fp64 base (dbase, fixed) plus an fp32 correction in the rows, so the
// small eigenvalues keep their relative accuracy: the rotation angle uses
// (dbase_q - dbase_p) rounded once, and the updates only move the
// corrections. The eigenvalues span 1e-7 of the largest, so below 1e-4 of it
// most pairs are still coupled; the refinement's floor (1e-11 of max|a_ii|)
// sits above the fp32 rounding its own rotations leave, so the tiny
// eigenvalues' pairs cannot cycle.
//
// A round is a chain (clocks at n = 256, one problem: update 1800, which 32 warps'
// issue bounds, sends and the wait for the others 1800, rotations 800), so what can
// be known before the loop or while the data travel is taken off it: the divisions by
// P and C, the row names and where each slot's rows begin, the players (one step on
// the circle a round), the angle beside its test; the first pass does no fp64
// arithmetic. The rotations and their order are those of the plain loop. First
// pass, refinement and replay together, measured: n = 256 8.55 -> 5.2 ms, 133 3.89 ->
// 2.24, 69 1.41 -> 0.79 (16 CTAs at n = 256: 5.5).
__global__ void __launch_bounds__(JAC_THREADS) jacobi_kernel(JacobiArgs a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char jsm[];
  const int C = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
  const JacobiSmem lay(a.n, C);
  const int n = lay.n, np = lay.np, P = lay.P, L = lay.L;
  double *dbase = reinterpret_cast<double *>(jsm + lay.off_dbase);
  double *lam_all = reinterpret_cast<double *>(jsm + lay.off_lam);
  float *rows = reinterpret_cast<float *>(jsm + lay.off_rows);
  float2 *rot = reinterpret_cast<float2 *>(jsm + lay.off_cs);  // cosine, sine of each slot
  float *pt = reinterpret_cast<float *>(jsm + lay.off_pt);
  float *diag = reinterpret_cast<float *>(jsm + lay.off_diag);  // [2][np]
  float *coup = reinterpret_cast<float *>(jsm + lay.off_coup);  // [2][P]
  int *const top_m = reinterpret_cast<int *>(jsm + lay.off_top);  // [2][L]
  int *const bot_m = reinterpret_cast<int *>(jsm + lay.off_bot);
  int *flag = reinterpret_cast<int *>(jsm + lay.off_flag);  // [sweep]: some pair rotated
  int *top = top_m, *bot = bot_m;  // the current maps: slot s0+i -> row buffers
  // where the rows of the slot's lower- and higher-numbered player begin
  int2 *const slot_m = reinterpret_cast<int2 *>(jsm + lay.off_slot);
  const bool refine = a.refine != 0;
  const int prob = blockIdx.x / C;
  const int s0 = crank * L, nloc = min(P, s0 + L) - s0;  // >= 1 (host)
  const int cgroups = (int)blockDim.x / P;  // >= 8 (P <= 128)
  const double *Gin = a.g[prob];
  // G times a power of two, its largest diagonal entry in [1, 2): the products of two
  // entries in the rotations' tests stay in range, and nothing else changes
  double down, up;
  {
    long long big = 0;
    for (int i = threadIdx.x & 31; i < n; i += 32)
      big = max(big, __double_as_longlong(fabs(Gin[(int64_t)i * n + i])));
    for (int o = 16; o > 0; o >>= 1) big = max(big, __shfl_xor_sync(0xffffffffu, big, o));
    const int raw = (int)(big >> 52);  // 0: zero or denormal, 0x7ff: not finite
    const int e = raw > 0 && raw < 0x7ff ? raw - 1023 : 0;
    down = scalbn(1.0, -e);
    up = scalbn(1.0, e);
  }
  float2 *log = a.log + (int64_t)prob * JAC_MAX_SWEEPS * (np - 1) * P;
  // at every sweep start slot k holds players k (top) and np-1-k (bottom)
  auto player_of = [&](int i) { return (i & 1) ? np - 1 - (s0 + i / 2) : s0 + i / 2; };
  auto row_of = [&](int i) { return rows + (size_t)((i & 1) ? bot[i / 2] : top[i / 2]) * np; };
  for (int i = threadIdx.x; i < nloc; i += blockDim.x) {
    top[i] = 2 * i;
    bot[i] = 2 * i + 1;
    slot_m[i] = slot_m[L + i] = make_int2(2 * i * np, (2 * i + 1) * np);
  }
  for (int i = threadIdx.x; i < np; i += blockDim.x) {
    dbase[i] = (refine && i < n) ? Gin[(int64_t)i * n + i] * down : 0.0;
    diag[i] = (!refine && i < n) ? (float)(Gin[(int64_t)i * n + i] * down) : 0.f;
  }
  for (int k = threadIdx.x; k < P; k += blockDim.x) {  // round 0 pairs (k, np-1-k)
    const int q = np - 1 - k;
    coup[k] = q < n ? (float)(Gin[(int64_t)k * n + q] * down) : 0.f;
  }
  for (int i = threadIdx.x; i <= JAC_MAX_SWEEPS + 1; i += blockDim.x) flag[i] = 0;
  volatile int *dead = flag + JAC_MAX_SWEEPS + 1;  // a wait ran out
  const uint32_t sbase = smem_u32(jsm), mbar = sbase + (uint32_t)lay.off_mbar;
  if (C > 1 && threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar + 8 * i) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int idx = threadIdx.x; idx < 2 * nloc * np; idx += blockDim.x) {
    const int b = idx / np, col = idx % np, x = player_of(b);
    float v = 0.f;
    if (x < n && col < n && !(refine && x == col)) v = (float)(Gin[(int64_t)x * n + col] * down);
    rows[(size_t)b * np + col] = v;
  }
  if (C > 1) cluster.sync(); else __syncthreads();
  // The rotation of slot k, players x and y (sweep `sw`, global round g), from the
  // broadcast values of parity `par`.
  float dmax = 0.f;  // max|a_ii| at the start of the sweep (rotation warps)
  auto sweep_dmax = [&](int par) {
    float m = 0.f;
    for (int x = threadIdx.x & 31; x < n; x += 32)
      m = fmaxf(m, fabsf(refine ? (float)(dbase[x] + (double)diag[par * np + x])
                               : diag[par * np + x]));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    return m;
  };
  auto rotations = [&](int k, int x, int y, int sw, int g, int par) {
    const int p = min(x, y), q = max(x, y);
    float c = 1.f, s = 0.f, tt = 0.f;
    if (q < n) {
      const float cp = diag[par * np + p], cq = diag[par * np + q], apq = coup[par * P + k];
      // (the first pass has no fp64 base: no arithmetic in fp64, 2 lanes a clock)
      const float app = refine ? (float)(dbase[p] + (double)cp) : cp,
                  aqq = refine ? (float)(dbase[q] + (double)cq) : cq;
      const float floor_abs = (refine ? 1e-11f : 1e-5f) * dmax;
      const float rel_tol = refine ? 1e-7f : 1e-6f;
      // the angle does not wait for the test's square root
      const float diff = refine ? (float)(dbase[q] - dbase[p]) + (cq - cp) : aqq - app;
      const float tau = diff / (2.f * apq);
      const float sg = tau >= 0.f ? 1.f : -1.f;
      const float tan = sg / (fabsf(tau) + sqrtf(1.f + tau * tau));
      const float cosine = rsqrtf(1.f + tan * tan);
      if (fabsf(apq) > floor_abs && fabsf(apq) > rel_tol * sqrtf(fabsf(app) * fabsf(aqq))) {
        tt = tan;
        c = cosine;
        s = tt * c;
        flag[sw] = 1;
      }
    }
    rot[k] = make_float2(c, s);
    pt[k] = tt;
    if (k >= s0 && k < s0 + nloc) log[(int64_t)g * P + k] = make_float2(c, s);
  };
  // the rotations are computed by warps 16-19 and the broadcast sent by warps
  // 24-31, while warps 0-7 move rows, so the phases of a round overlap
  const int rt = (int)threadIdx.x - kJacRotBase, bt = (int)threadIdx.x - kJacSendBase;
  if (rt >= 0 && rt < ((P + 31) & ~31)) dmax = sweep_dmax(0);
  if (rt >= 0 && rt < P) rotations(rt, rt, np - 1 - rt, 0, 0, 0);
  __syncthreads();
  int sweeps_done = JAC_MAX_SWEEPS;
  // what a thread does every round, found once
  const int k2 = (int)threadIdx.x % P, kl0 = (int)threadIdx.x / P;
  // broadcast: a thread per held row and CTA
  const int bt_n = (JAC_THREADS - kJacSendBase) / C;
  const int bt_r = bt >= 0 ? bt % C : 0, bt_i = bt >= 0 ? bt / C : 2 * L;
  const bool updates = (int)threadIdx.x < cgroups * P;
  // the players of column slot k2, or (rotation threads) of slot rt: one step on
  // the circle a round
  const int my = rt >= 0 && rt < P ? rt : k2;
  int px = k2, py = np - 1 - k2, rx = my, ry = np - 1 - my;
  auto step = [&](int x) { return x == 0 ? 0 : x == np - 1 ? 1 : x + 1; };
  // shared memory of the CTAs this thread sends to: threads 0-127 the left
  // neighbour's, 128-255 the right one's, from kJacSendBase on bt_r's
  const int to = bt >= 0 ? bt_r : threadIdx.x < 128 ? max(crank - 1, 0) : min(crank + 1, C - 1);
  const uint32_t rbase = remote_addr(sbase, to);
  const uint32_t round_bytes =
      4 * (np + P) + 4 * np * ((crank > 0 ? 1 : 0) + (crank < C - 1 ? 1 : 0));
  int t = 0, sw = 0;  // round of the sweep, sweep
  for (int g = 0;; ++g) {
    // every rotation applied to the owned rows, 2 x 2 block (owned slot k1,
    // slot k2) by block: a thread keeps one column slot k2 for the round and
    // walks the owned slots (groups of P threads; the column pair's players
    // and rotation are loaded once)
    if (updates) {
      const int p2 = min(px, py), q2 = max(px, py);
      const float2 r2 = rot[k2];
      const float c2 = r2.x, s2v = r2.y;
      const int2 *slot = slot_m + (g & 1) * L;
      for (int kl = kl0; kl < nloc; kl += cgroups) {
        const float2 r1 = rot[s0 + kl];
        const float c1 = r1.x, s1v = r1.y;
        if (s1v == 0.f && s2v == 0.f) continue;
        const int2 at = slot[kl];
        float *rp = rows + at.x, *rq = rows + at.y;
        if (k2 == s0 + kl) {  // the rotation's own 2 x 2 block
          const float t1 = pt[k2];
          if (q2 < n && t1 != 0.f) {
            const float apq = rp[q2];
            rp[p2] -= t1 * apq;
            rq[q2] += t1 * apq;
            rp[q2] = 0.f;
            rq[p2] = 0.f;
          }
          continue;
        }
        const float cc = __fmul_rn(c1, c2), cs = __fmul_rn(c1, s2v), sc = __fmul_rn(s1v, c2),
                    ss = __fmul_rn(s1v, s2v);
        const float b00 = rp[p2], b01 = rp[q2], b10 = rq[p2], b11 = rq[q2];
        // J1^T B J2 with J = [[c, s], [-s, c]]; the twin block (k2, k1) sums
        // the same four products in the same pairs
        rp[p2] = __fsub_rn(__fadd_rn(__fmul_rn(cc, b00), __fmul_rn(ss, b11)),
                           __fadd_rn(__fmul_rn(cs, b01), __fmul_rn(sc, b10)));
        rp[q2] = __fsub_rn(__fadd_rn(__fmul_rn(cs, b00), __fmul_rn(cc, b01)),
                           __fadd_rn(__fmul_rn(ss, b10), __fmul_rn(sc, b11)));
        rq[p2] = __fsub_rn(__fadd_rn(__fmul_rn(sc, b00), __fmul_rn(cc, b10)),
                           __fadd_rn(__fmul_rn(ss, b01), __fmul_rn(cs, b11)));
        rq[q2] = __fadd_rn(__fadd_rn(__fmul_rn(ss, b00), __fmul_rn(cc, b11)),
                           __fadd_rn(__fmul_rn(sc, b01), __fmul_rn(cs, b10)));
      }
    }
    __syncthreads();
    // the next round: position j -> j - 1 (j >= 2), 1 -> np - 1, 0 stays
    const int g1 = g + 1, t1 = t + 1 == np - 1 ? 0 : t + 1, sw1 = t1 ? sw : sw + 1, par = g1 & 1;
    const uint32_t bar = rbase + (uint32_t)lay.off_mbar + 8 * par;
    if (C > 1) {
      if (threadIdx.x == kJacRotBase - 32)  // the round's data, from every CTA
        asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(
                         mbar + 8 * par),
                     "r"(round_bytes)
                     : "memory");
      // hand-over: first owned top row left, last owned bottom row right
      if (threadIdx.x < 256) {
        const int j = threadIdx.x & 127, left = threadIdx.x < 128;
        const uint64_t *src =
            reinterpret_cast<const uint64_t *>(rows + (size_t)(left ? top[0] : bot[nloc - 1]) * np);
        const uint32_t dst = rbase + (uint32_t)lay.off_rows +
                             4 * (uint32_t)((2 * L + 2 * par + left) * np) + 8 * j;
        if (left ? crank > 0 : crank < C - 1)
          if (j < np / 2) send_b64(dst, src[j], bar);
      }
    }
    // each held row's diagonal, and its coupling to its next partner (sent by
    // the lower-numbered of the two), to every CTA
    for (int i = bt_i; i < 2 * nloc; i += bt_n) {
      const int k = s0 + i / 2, pos = (i & 1) ? np - 1 - k : k;
      const int x = circle_player(pos, t, np);
      const float *row = rows + (size_t)((i & 1) ? bot[i / 2] : top[i / 2]) * np;
      const int pos1 = pos == 0 ? 0 : (pos == 1 ? np - 1 : pos - 1);
      const int k1 = min(pos1, np - 1 - pos1), y = circle_player(np - 1 - pos1, t1, np);
      const float dx = row[x], cx = x < y && y < n ? row[y] : 0.f;
      if (C > 1) {
        send_b32(rbase + (uint32_t)lay.off_diag + 4 * (par * np + x), dx, bar);
        if (x < y) send_b32(rbase + (uint32_t)lay.off_coup + 4 * (par * P + k1), cx, bar);
      } else {
        diag[par * np + x] = dx;
        if (x < y) coup[par * P + k1] = cx;
      }
    }
    // the row names of the next round, while the data travel (only this CTA's maps
    // are involved)
    int dl = -1, dr = -1;
    int *ntop = top == top_m ? top_m + L : top_m, *nbot = bot == bot_m ? bot_m + L : bot_m;
    if (P >= 2 && (int)threadIdx.x < 256) {
      circle_arrivals(top, bot, s0, nloc, P, &dl, &dr);
      for (int i = threadIdx.x; i < nloc; i += 256)
      {
        int nt, nb;
        circle_next(top, bot, s0, nloc, P, i, dl, dr, &nt, &nb);
        ntop[i] = nt;
        nbot[i] = nb;
        const bool up = circle_player(s0 + i, t1, np) < circle_player(np - 1 - s0 - i, t1, np);
        slot_m[par * L + i] = up ? make_int2(nt * np, nb * np) : make_int2(nb * np, nt * np);
      }
    }
    px = step(px);
    py = step(py);
    rx = step(rx);
    ry = step(ry);
    if (C > 1) {
      if (threadIdx.x < 256 || (rt >= 0 && rt < ((P + 31) & ~31))) {
        const uint32_t phase = ((uint32_t)(g1 - 1) >> 1) & 1;
        int polls = 0;
        while (!try_wait(mbar + 8 * par, phase))
          if (*dead || ++polls > kJacWaits) {
            *dead = 1;
            break;
          }
      }
      // the rows sent are overwritten next: their readers, warps 0-7 and 24-31, are done
      if (threadIdx.x < 256)
        asm volatile("bar.sync 1, 512;" ::: "memory");
      else if (bt >= 0)
        asm volatile("bar.arrive 1, 512;" ::: "memory");
      if (P >= 2 && (int)threadIdx.x < np) {  // arrived rows take the freed buffers
        const float *mbox = rows + (size_t)(2 * L + 2 * par) * np;  // [from left, from right]
        const int i = threadIdx.x;
        if (dl >= 0) rows[(size_t)dl * np + i] = mbox[i];
        if (dr >= 0) rows[(size_t)dr * np + i] = mbox[np + i];
      }
    } else {
      __syncthreads();
    }
    if (P >= 2) {
      top = ntop;
      bot = nbot;
    }
    if (t1 == 0) {  // sweep boundary: stop after a sweep without rotations
      __syncthreads();
      // (the same in every CTA, but for a wait that ran out)
      if (!flag[sw1 - 1] || sw1 == JAC_MAX_SWEEPS || *dead) {
        sweeps_done = sw1;
        break;
      }
      if (rt >= 0 && rt < ((P + 31) & ~31)) dmax = sweep_dmax(par);
    }
    if (rt >= 0 && rt < P) rotations(rt, rx, ry, sw1, g1, par);
    __syncthreads();
    t = t1;
    sw = sw1;
  }
  if (threadIdx.x == 0) {
    if (crank == 0) a.sweeps[prob] = sweeps_done;
    const int32_t report = jacobi_report(crank, *dead != 0, sweeps_done);
    if (report) atomicMax(a.most_sweeps, report);
  }
  // eigenvalues to every CTA of the cluster, then each ranks its own players
  for (int i = threadIdx.x; i < 2 * nloc; i += blockDim.x) {
    const int x = player_of(i);
    const double lx = dbase[x] + (double)row_of(i)[x];
    for (int r = 0; r < C; ++r) cluster.map_shared_rank(lam_all, r)[x] = lx;
  }
  if (C > 1) cluster.sync(); else __syncthreads();  // the last remote access is above
  float *lam = a.lambda[prob];
  for (int i = threadIdx.x; i < 2 * nloc; i += blockDim.x) {
    const int x = player_of(i);
    if (x >= n) continue;
    const double li = lam_all[x];
    int r = 0;
    for (int j = 0; j < n; ++j) {
      const double lj = lam_all[j];
      r += (lj > li) || (lj == li && j < x);
    }
    a.rank[prob * n + x] = r;
    lam[r] = (float)(li * up);
  }
}

// V = product of the logged rotations, rows processed independently;
// column c of the product lands in column rank[c] of the output. The log is
// streamed into shared memory REPLAY_CHUNK rounds at a time with cp.async,
// double buffered, so a round waits on its barrier only, not on L2.
constexpr int REPLAY_ROWS = 16;  // at most; 2 where that still leaves the batch few blocks
constexpr int REPLAY_CHUNK = 16;

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_u32(smem)), "l"(gmem));
}

__global__ void __launch_bounds__(256) jacobi_replay_kernel(JacobiArgs a, float *const *vout,
                                                            int rows) {
  extern __shared__ __align__(16) float sv[];  // [rows][n], then [2][REPLAY_CHUNK][P] float2
  const int n = a.n, np = n + (n & 1), P = np / 2;
  const int prob = blockIdx.y;
  const int r0 = blockIdx.x * rows;
  const int nr = min(rows, n - r0);
  if (nr <= 0) return;
  float2 *lb = reinterpret_cast<float2 *>(sv + ((rows * n + 1) & ~1));
  const float *vin = a.vinit ? a.vinit[prob] : nullptr;
  for (int i = threadIdx.x; i < rows * n; i += blockDim.x) {
    int rr = i / n, cc = i % n;
    sv[i] = rr >= nr ? 0.f : vin ? vin[(int64_t)(r0 + rr) * n + cc] : (r0 + rr == cc ? 1.f : 0.f);
  }
  const float2 *log = a.log + (int64_t)prob * JAC_MAX_SWEEPS * (np - 1) * P;
  const int rounds = a.sweeps[prob] * (np - 1);
  const int nchunks = (rounds + REPLAY_CHUNK - 1) / REPLAY_CHUNK;
  const int G = max(1, (int)blockDim.x / P);                // row groups (P <= 128)
  const int g = (int)threadIdx.x / P, k = (int)threadIdx.x % P;
  auto issue = [&](int c) {
    const int first = c * REPLAY_CHUNK, cnt = min(REPLAY_CHUNK, rounds - first);
    const float2 *src = log + (int64_t)first * P;
    float2 *dst = lb + (c & 1) * REPLAY_CHUNK * P;
    for (int i = threadIdx.x; i < cnt * P; i += blockDim.x) cp_async8(dst + i, src + i);
    cp_async_commit();
  };
  if (nchunks > 0) issue(0);
  for (int c = 0; c < nchunks; ++c) {
    if (c + 1 < nchunks) {
      issue(c + 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();  // chunk c visible to every thread; sv initialized
    const float2 *buf = lb + (c & 1) * REPLAY_CHUNK * P;
    const int first = c * REPLAY_CHUNK, cnt = min(REPLAY_CHUNK, rounds - first);
    for (int q = 0; q < cnt; ++q) {
      const int t = (first + q) % (np - 1);
      // thread (group g, pair k): one rotation, applied to rows g, g+G, ...
      if (g < G) {
        const float2 cs = buf[q * P + k];
        const int x = circle_player(k, t, np), y = circle_player(np - 1 - k, t, np);
        const int p = min(x, y), qq = max(x, y);
        if (cs.y != 0.f && qq < n)
          for (int rr = g; rr < nr; rr += G) {
            const float vp = sv[rr * n + p], vq = sv[rr * n + qq];
            sv[rr * n + p] = cs.x * vp - cs.y * vq;
            sv[rr * n + qq] = cs.y * vp + cs.x * vq;
          }
      }
      __syncthreads();
    }
  }
  float *V = vout[prob];
  const int32_t *rank = a.rank + prob * n;
  for (int i = threadIdx.x; i < nr * n; i += blockDim.x) {
    int rr = i / n, cc = i % n;
    V[(int64_t)(r0 + rr) * n + rank[cc]] = sv[rr * n + cc];
  }
}

}  // namespace

size_t jacobi_work_bytes(int n, int nprob) {
  int np = n + (n & 1);
  size_t logb = (size_t)nprob * JAC_MAX_SWEEPS * (np - 1) * (np / 2) * sizeof(float2);
  return round_up(logb, 256) + round_up((size_t)nprob * sizeof(int32_t), 256) +
         round_up((size_t)nprob * n * sizeof(int32_t), 256);
}

tsvd_status jacobi_eig_batched(double *const *g, int n, float *const *lambda, float *const *v,
                               int nprob, void *work, size_t work_bytes, cudaStream_t st,
                               int32_t *sweeps, int refine, const float *const *vinit) {
  if (nprob == 0) return TSVD_OK;
  if (n > 256 || n < 2) return fail(TSVD_ERR_INVALID, "jacobi: n=%d", n);
  if (jacobi_work_bytes(n, nprob) > work_bytes) return fail(TSVD_ERR_INVALID, "jacobi: work");
  int np = n + (n & 1);
  char *w = (char *)work;
  JacobiArgs a;
  a.g = g;
  a.n = n;
  a.lambda = lambda;
  a.log = (float2 *)w;
  w += round_up((size_t)nprob * JAC_MAX_SWEEPS * (np - 1) * (np / 2) * sizeof(float2), 256);
  a.sweeps = (int32_t *)w;
  w += round_up((size_t)nprob * sizeof(int32_t), 256);
  a.rank = (int32_t *)w;
  a.refine = refine;
  a.most_sweeps = sweeps;
  a.vinit = vinit;
  const int P = np / 2;
  // CTAs per problem: as many as keep the whole batch within one wave of
  // clusters (up to 8), at least as many as the rows need for shared memory,
  // and no CTA without a slot
  const size_t smem_cap = 200 * 1024;
  int C = 1;
  while (C < kJacMaxCluster && (int64_t)nprob * 2 * C <= sm_count()) C *= 2;
  while (C < kJacMaxCluster && JacobiSmem(n, C).bytes > smem_cap) C *= 2;
  while (C > 1 && (C - 1) * JacobiSmem(n, C).L >= P) C /= 2;
  int cmin = 1;
  while (cmin < kJacMaxCluster && JacobiSmem(n, cmin).bytes > smem_cap) cmin *= 2;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(JAC_THREADS);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto configure = [&](int c) -> tsvd_status {
    cfg.gridDim = dim3((unsigned)(nprob * c));
    cfg.dynamicSmemBytes = JacobiSmem(n, c).bytes;
    attr[0].val.clusterDim.x = (unsigned)c;
    return raise_smem_ceiling((const void *)jacobi_kernel, cfg.dynamicSmemBytes);
  };
  // a cluster must fit in one GPC: fewer CTAs per problem when the batch's
  // clusters would not all be resident at once (a second wave doubles the
  // time, as 16 clusters of 8 did)
  while (C > cmin) {
    TSVD_TRY(configure(C));
    int active = 0;
    if (cudaOccupancyMaxActiveClusters(&active, (const void *)jacobi_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      break;
    }
    if (active >= nprob) break;
    C /= 2;
  }
  TSVD_TRY(configure(C));
  if (cfg.dynamicSmemBytes > smem_cap)
    return fail(TSVD_ERR_INVALID, "jacobi: n=%d needs %zu B per CTA", n, cfg.dynamicSmemBytes);
  TSVD_CUDA(cudaLaunchKernelEx(&cfg, jacobi_kernel, a));
  // rows a block: a round costs a block its rows, one after the other (n = 256,
  // one problem: 16 rows 1.2 ms, 2 rows 0.5 ms)
  const int rrows = ceil_div(n, 2) * nprob <= 4 * sm_count() ? 2 : REPLAY_ROWS;
  const size_t rsmem = (size_t)((rrows * n + 1) & ~1) * sizeof(float) +
                       (size_t)2 * REPLAY_CHUNK * P * sizeof(float2);
  if (rsmem > 48 * 1024) TSVD_TRY(raise_smem_ceiling((const void *)jacobi_replay_kernel, rsmem));
  jacobi_replay_kernel<<<dim3((unsigned)ceil_div(n, rrows), nprob), 256, rsmem, st>>>(a, v, rrows);
  TSVD_LAUNCH_CHECK();
  return TSVD_OK;
}

}  // namespace tsvd
