// frPCA over a caller's CSR matrix: the drop-in for Code/frpca.c:239-326
// (frPCA(mat_csr*, mat**, mat**, mat**, k, q)) and a status-returning form.
//
// The matrix goes to the device as the caller has it; there it is checked, its
// empty columns are compacted away and it becomes the half-precision A^T of the
// mixed form (tsvd_frpca; values scaled by a power of two into half range,
// products on the tensor cores) or an FP32 CSR / CSC pair (tsvd_frpca_fp32 and
// the legacy frPCA symbol; both products as SpMM, the plain form's products).
// Built on one host thread instead, with some 40 allocations a call, this and
// the results' transposition were most of a call. 1500 x 6000 with 900k entries,
// k = 128, measured with the kernels of then: 12.7 -> 6.3 ms (5.6 now); 600 x 3001 with
// 90k entries, k = 32: 3.9 -> 1.8 ms (1.8 now).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>

#include "factor.h"
#include "internal.h"
#include "plain.h"

using namespace tsvd;

namespace {

uint64_t g_frpca_seed = 20231;

// One call's stream and device memory, given back when the call returns.
struct CallMemory {
  cudaStream_t st = nullptr;
  std::vector<void *> held;
  ~CallMemory() {
    if (st) cudaStreamDestroy(st);
    for (void *p : held) cudaFree(p);
    cudaGetLastError();  // the launch checks read this slot: leave nothing from teardown in it
  }
  tsvd_status open() {
    TSVD_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    return TSVD_OK;
  }
  // Runs take(arena) twice: to add up what it takes, then to carve it.
  template <typename F>
  tsvd_status carve(F take) {
    DeviceArena A;
    A.count = true;
    TSVD_TRY(take(A));
    A.cap = A.used;
    A.used = 0;
    A.count = false;
    TSVD_CUDA(cudaMalloc(&A.base, std::max<size_t>(A.cap, 256)));
    held.push_back(A.base);
    return take(A);
  }
};

// What the checks of a matrix found.
enum : uint32_t { kBadEntry = 1, kHasZeros = 2, kUnsorted = 4 };
struct MatrixInfo {
  unsigned long long vmax_bits;  // largest magnitude, as the bits of a double
  int64_t nnz;                   // entries that are not zero (sparse form)
  uint32_t found;
  int32_t nc;                    // columns that are not empty
};

// The caller's entries [0, nnz) on the device, indices still based at `base`.
struct RawMatrix {
  const int64_t *rp;  // nrows + 1, offset by org
  const int32_t *col;
  const double *val;
  int64_t nnz, org;
  int32_t nrows, ncols, base;
  __device__ int32_t row_of(int64_t t) const {  // the last row that begins at or before t
    int32_t lo = 0, hi = nrows;
    while (hi - lo > 1) {
      const int32_t mid = lo + (hi - lo) / 2;
      if (rp[mid] - org <= t) lo = mid; else hi = mid;
    }
    return lo;
  }
};

__device__ __forceinline__ float scaled(double v, double scale) {
  return (float)((double)(float)v * scale);
}

// flag[c] = 1 for columns with a nonzero, cnt[c] their number (cnt may be null).
__global__ void check_kernel(RawMatrix m, int32_t *flag, int32_t *cnt, MatrixInfo *info) {
  unsigned long long vmax = 0;
  uint32_t found = 0;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < m.nnz;
       t += (int64_t)gridDim.x * blockDim.x) {
    const double v = m.val[t];
    const int32_t c = m.col[t] - m.base;
    if (c < 0 || c >= m.ncols || !(fabs(v) <= (double)FLT_MAX)) {
      found |= kBadEntry;
      continue;
    }
    if (t > 0 && m.col[t - 1] - m.base > c && m.rp[m.row_of(t)] - m.org != t) found |= kUnsorted;
    if (v == 0.0) {
      found |= kHasZeros;
      continue;
    }
    flag[c] = 1;
    if (cnt) atomicAdd(&cnt[c], 1);
    const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(v));
    if (b > vmax) vmax = b;
  }
  // non-negative doubles order as their bits do
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, vmax, o);
    if (w > vmax) vmax = w;
  }
  found = __reduce_or_sync(0xffffffffu, found);
  if ((threadIdx.x & 31) == 0) {
    if (vmax) atomicMax(&info->vmax_bits, vmax);
    if (found) atomicOr(&info->found, found);
  }
}

// cinv[c] = compacted column or -1 (in place of flag), cmap its inverse. cpos: where
// each column's nonzeros begin (may be null).
__global__ void compact_kernel(int32_t *cinv, const int64_t *pos, const int64_t *cpos,
                               int32_t ncols, int32_t *cmap, MatrixInfo *info) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < ncols;
       c += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i = (int32_t)pos[c];
    if (cinv[c]) {
      cmap[i] = (int32_t)c;
      cinv[c] = i;
    } else {
      cinv[c] = -1;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    info->nc = (int32_t)pos[ncols];
    if (cpos) info->nnz = cpos[ncols];
  }
}

__global__ void densify_kernel(RawMatrix m, const int32_t *cinv, double scale, int sp,
                               __half *at) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < m.nnz;
       t += (int64_t)gridDim.x * blockDim.x) {
    const double v = m.val[t];
    if (v == 0.0) continue;
    at[(int64_t)cinv[m.col[t] - m.base] * sp + m.row_of(t)] = __float2half_rn(scaled(v, scale));
  }
}

// (column, entry) pairs for the sort that gives the CSC, zeros past the last column;
// column pointers of the compacted columns; and, of a matrix whose rows ascend and hold
// no zeros, the CSR.
__global__ void csr_kernel(RawMatrix m, const int32_t *cinv, const int64_t *cpos, double scale,
                           bool ready, SparseBlock b, uint32_t *keys, uint32_t *vals) {
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = i0; t < m.nnz; t += step) {
    const double v = m.val[t];
    const int32_t c = v == 0.0 ? b.cols : cinv[m.col[t] - m.base];
    keys[t] = (uint32_t)c;
    vals[t] = (uint32_t)t;
    if (ready) {
      b.colidx[t] = c;
      b.rval[t] = scaled(v, scale);
    }
  }
  if (ready)
    for (int64_t i = i0; i <= b.rows; i += step)
      b.rowptr[i] = i < m.nrows ? m.rp[i] - m.org : m.nnz;
  for (int64_t c = i0; c <= m.ncols; c += step) {
    if (c == m.ncols) b.colptr[b.cols] = b.nnz;
    else if (cinv[c] >= 0) b.colptr[cinv[c]] = cpos[c];
  }
}

// rows receives each entry's row, the key of the sort back to rows; null if the CSR is
// there already.
__global__ void csc_gather_kernel(RawMatrix m, const uint32_t *order, double scale, SparseBlock b,
                                  uint32_t *rows) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < b.nnz;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = order[i];
    const int32_t r = m.row_of(t);
    b.rowidx[i] = r;
    b.cval[i] = rows ? scaled(m.val[t], scale) : b.rval[t];
    if (rows) rows[i] = (uint32_t)r;
  }
}

// The CSR of entries sorted by row, in each row by column.
__global__ void csr_gather_kernel(RawMatrix m, const int32_t *cinv, const uint32_t *order,
                                  const uint32_t *row, double scale, SparseBlock b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= b.nnz;
       i += (int64_t)gridDim.x * blockDim.x) {
    // the rows that begin here: those past the entry before's, up to this one's
    const int64_t last = i < b.nnz ? (int64_t)row[i] : b.rows;
    for (int64_t r = i > 0 ? (int64_t)row[i - 1] + 1 : 0; r <= last; ++r) b.rowptr[r] = i;
    if (i == b.nnz) break;
    const int64_t t = order[i];
    b.colidx[i] = cinv[m.col[t] - m.base];
    b.rval[i] = scaled(m.val[t], scale);
  }
}

// Elements [f0, f0 + n) of the column-major double matrix whose row r is row
// cinv[r] (r without cinv; zeros for -1) of the row-major x (pitch k).
__global__ void widen_columns_kernel(const float *x, int k, const int32_t *cinv, int64_t rows,
                                     int64_t f0, int64_t n, double *out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = (f0 + i) / rows, r = (f0 + i) % rows, s = cinv ? cinv[r] : r;
    out[i] = s >= 0 ? (double)x[s * k + j] : 0.0;
  }
}

// Elements [f0, f0 + n) of the column-major in to the row-major fp32 m.
__global__ void narrow_rows_kernel(const double *in, int64_t rows, int cols, int64_t f0, int64_t n,
                                   float *m) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    m[(f0 + i) % rows * cols + (f0 + i) / rows] = (float)in[i];
}

// Results and dense inputs pass through at most this many doubles at a time.
constexpr int64_t kStage = 1 << 23;

tsvd_status fetch_columns(const float *x, int k, const int32_t *cinv, int64_t rows, double *stage,
                          double *out, cudaStream_t st) {
  for (int64_t f0 = 0; f0 < rows * k; f0 += kStage) {
    const int64_t n = std::min(kStage, rows * k - f0);
    widen_columns_kernel<<<grid_for(n, 256), 256, 0, st>>>(x, k, cinv, rows, f0, n, stage);
    TSVD_LAUNCH_CHECK();
    // fresh pages are mapped here, while the kernel runs: a fault of the copy
    // costs more (600 x 128 results: 0.69 -> 0.01 ms of copies)
    for (int64_t i = f0; i < f0 + n; i += 512) out[i] = 0.0;
    TSVD_CUDA(cudaMemcpyAsync(out + f0, stage, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
  }
  TSVD_CUDA(cudaStreamSynchronize(st));
  return TSVD_OK;
}

}  // namespace

extern "C" void tsvd_set_frpca_seed(uint64_t seed) { g_frpca_seed = seed; }

namespace {

// A caller's CSR with its empty columns compacted away: triplets in row
// order (explicit zeros dropped), the compacted -> original column map and
// the largest magnitude.
struct HostBlock {
  std::vector<int32_t> trow, tcol, cmap, cinv;
  std::vector<double> tval;
  double vmax = 0.0;
};

tsvd_status host_block(int32_t nrows, int32_t ncols, int64_t nnz, const int64_t *row_ptr,
                       const int32_t *col_idx, const double *values, int32_t index_base,
                       HostBlock &H) {
  if (nrows < 1 || ncols < 1 || nnz < 0 || !row_ptr || (nnz > 0 && (!col_idx || !values)))
    return fail(TSVD_ERR_INVALID, "frpca: bad matrix arguments");
  if (index_base != 0 && index_base != 1) return fail(TSVD_ERR_INVALID, "frpca: index_base");
  H.cinv.assign(ncols, -1);
  H.trow.reserve(nnz);
  H.tcol.reserve(nnz);
  H.tval.reserve(nnz);
  for (int32_t i = 0; i < nrows; ++i) {
    int64_t b = row_ptr[i] - index_base, e = row_ptr[i + 1] - index_base;
    if (b < 0 || e < b || e > nnz) return fail(TSVD_ERR_INVALID, "frpca: bad row pointers");
    for (int64_t t = b; t < e; ++t) {
      int32_t c = col_idx[t] - index_base;
      if (c < 0 || c >= ncols) return fail(TSVD_ERR_INVALID, "frpca: column out of range");
      if (values[t] == 0.0) continue;
      if (!std::isfinite(values[t])) return fail(TSVD_ERR_NUMERIC, "frpca: non-finite value");
      if (std::fabs(values[t]) > (double)FLT_MAX)
        return fail(TSVD_ERR_INVALID, "frpca: |value| above the float range");
      H.cinv[c] = 1;
      H.trow.push_back(i);
      H.tcol.push_back(c);
      H.tval.push_back(values[t]);
      H.vmax = std::max(H.vmax, std::fabs(values[t]));
    }
  }
  for (int32_t c = 0; c < ncols; ++c)
    if (H.cinv[c] > 0) {
      H.cinv[c] = (int32_t)H.cmap.size();
      H.cmap.push_back(c);
    }
  for (auto &c : H.tcol) c = H.cinv[c];
  return TSVD_OK;
}

// A compacted matrix on the device, ready for the products.
struct DirectBlock {
  int32_t nc = 0;
  double scale = 1.0;
  const int32_t *cmap = nullptr, *cinv = nullptr;
  const __half *at = nullptr;
  SparseBlock sb;
  bool sparse = false;
};

// The power of two that takes the largest magnitude to 2^14 (undone on sigma).
double scale_for(double vmax) {
  int e2 = 0;
  if (vmax > 0) std::frexp(vmax, &e2);
  return std::ldexp(1.0, 14 - e2);
}

tsvd_status take_sparse(DeviceArena &A, SparseBlock &sb, int rows, int cols, int64_t nnz) {
  sb.rows = rows;
  sb.cols = cols;
  sb.nnz = nnz;
  TSVD_TRY(device_take(&A, &sb.rowptr, (size_t)rows + 1));
  TSVD_TRY(device_take(&A, &sb.colidx, (size_t)nnz));
  TSVD_TRY(device_take(&A, &sb.rval, (size_t)nnz));
  TSVD_TRY(device_take(&A, &sb.colptr, (size_t)cols + 1));
  TSVD_TRY(device_take(&A, &sb.rowidx, (size_t)nnz));
  return device_take(&A, &sb.cval, (size_t)nnz);
}

// The block from the caller's arrays, on the device. *ready stays false where the
// matrix is left to the host: an entry is not valid (the host's walk says which
// comes first) or, for the sparse form, the entries do not fit the sort's 32-bit
// positions. Of a sparse matrix whose rows do not ascend or hold zeros, the sort by
// column drops the zeros and a second one by row gives the CSR: both are stable, so the
// entries come in the order of the host's build. The whole call, k = 128, 1500 x 6000
// with 900k entries, 10 % of them zeros, rows mixed, measured: 47 ms with the host's
// build, 5.3 so (rows in order without zeros: 5.3); 600 x 3001 with 90k, k = 32: 4.6 and
// 1.3 ms.
tsvd_status block_on_device(CallMemory &M, int32_t nrows, int32_t ncols, int64_t nnz_arg,
                            const int64_t *row_ptr, const int32_t *col_idx, const double *values,
                            int32_t base, bool sparse, DirectBlock &D, bool *ready) {
  *ready = false;
  const int64_t org = row_ptr[0], nnz = row_ptr[nrows] - org;
  if (org < base || row_ptr[nrows] - base > nnz_arg || (sparse && nnz >= (1ll << 31)))
    return TSVD_OK;
  for (int32_t i = 0; i < nrows; ++i)
    if (row_ptr[i + 1] < row_ptr[i]) return TSVD_OK;
  cudaStream_t st = M.st;
  RawMatrix m{nullptr, nullptr, nullptr, nnz, org, nrows, ncols, base};
  int64_t *rp;
  int32_t *col, *cinv, *cmap, *cnt = nullptr;
  double *val;
  int64_t *pos, *cpos = nullptr;
  void *tmp;
  MatrixInfo *info, h;
  TSVD_TRY(M.carve([&](DeviceArena &A) -> tsvd_status {
    TSVD_TRY(device_take(&A, &rp, (size_t)nrows + 1));
    TSVD_TRY(device_take(&A, &col, (size_t)nnz));
    TSVD_TRY(device_take(&A, &val, (size_t)nnz));
    TSVD_TRY(device_take(&A, &cmap, (size_t)ncols));
    TSVD_TRY(device_take(&A, &pos, (size_t)ncols + 1));
    if (sparse) TSVD_TRY(device_take(&A, &cpos, (size_t)ncols + 1));
    TSVD_TRY(device_take(&A, (char **)&tmp, scan_tmp_bytes(ncols)));
    // cleared together
    TSVD_TRY(device_take(&A, &info, 1));
    TSVD_TRY(device_take(&A, &cinv, (size_t)ncols));
    return sparse ? device_take(&A, &cnt, (size_t)ncols) : TSVD_OK;
  }));
  TSVD_CUDA(cudaMemsetAsync(
      info, 0, (char *)(sparse ? cnt + ncols : cinv + ncols) - (char *)info, st));
  TSVD_CUDA(cudaMemcpyAsync(rp, row_ptr, sizeof(int64_t) * (nrows + 1), cudaMemcpyHostToDevice, st));
  m.rp = rp;
  m.col = col;
  m.val = val;
  if (nnz > 0) {
    TSVD_CUDA(cudaMemcpyAsync(col, col_idx + (org - base), sizeof(int32_t) * nnz,
                              cudaMemcpyHostToDevice, st));
    TSVD_CUDA(cudaMemcpyAsync(val, values + (org - base), sizeof(double) * nnz,
                              cudaMemcpyHostToDevice, st));
    check_kernel<<<grid_for(nnz, 256), 256, 0, st>>>(m, cinv, cnt, info);
    TSVD_LAUNCH_CHECK();
  }
  TSVD_TRY(scan_i32_to_i64(cinv, pos, ncols, tmp, st));
  if (sparse) TSVD_TRY(scan_i32_to_i64(cnt, cpos, ncols, tmp, st));
  compact_kernel<<<grid_for(ncols, 256), 256, 0, st>>>(cinv, pos, cpos, ncols, cmap, info);
  TSVD_LAUNCH_CHECK();
  TSVD_CUDA(cudaMemcpyAsync(&h, info, sizeof h, cudaMemcpyDeviceToHost, st));
  TSVD_CUDA(cudaStreamSynchronize(st));
  if (h.found & kBadEntry) return TSVD_OK;
  D.nc = h.nc;
  D.cmap = cmap;
  D.cinv = cinv;
  D.sparse = sparse;
  double vmax;
  std::memcpy(&vmax, &h.vmax_bits, sizeof vmax);
  D.scale = scale_for(vmax);
  *ready = true;
  if (D.nc == 0) return TSVD_OK;
  const int sp = (int)round_up(nrows, kRowPad);
  if (!sparse) {
    __half *at;
    const size_t n = (size_t)D.nc * sp;
    TSVD_TRY(M.carve([&](DeviceArena &A) { return device_take(&A, &at, n); }));
    TSVD_CUDA(cudaMemsetAsync(at, 0, sizeof(__half) * n, st));
    densify_kernel<<<grid_for(nnz, 256), 256, 0, st>>>(m, cinv, D.scale, sp, at);
    TSVD_LAUNCH_CHECK();
    D.at = at;
    return TSVD_OK;
  }
  const bool in_order = h.found == 0;
  uint32_t *keys, *vals, *keys2, *vals2;
  void *stmp;
  TSVD_TRY(M.carve([&](DeviceArena &A) -> tsvd_status {
    TSVD_TRY(take_sparse(A, D.sb, sp, D.nc, h.nnz));
    for (uint32_t **p : {&keys, &vals, &keys2, &vals2}) TSVD_TRY(device_take(&A, p, (size_t)nnz));
    return device_take(&A, (char **)&stmp, sort_tmp_bytes(nnz));
  }));
  csr_kernel<<<grid_for(std::max<int64_t>(nnz, ncols), 256), 256, 0, st>>>(
      m, cinv, cpos, D.scale, in_order, D.sb, keys, vals);
  TSVD_LAUNCH_CHECK();
  // zeros have the key nc
  auto bits_for = [](int64_t keys_up_to) {
    int bits = 1;
    while ((1ll << bits) <= keys_up_to) ++bits;
    return bits;
  };
  bool in_alt = false;
  TSVD_TRY(stable_sort_pairs(keys, vals, keys2, vals2, nnz,
                             bits_for(in_order ? D.nc - 1 : D.nc), stmp, st, &in_alt));
  if (in_alt) {
    std::swap(keys, keys2);
    std::swap(vals, vals2);
  }
  csc_gather_kernel<<<grid_for(h.nnz, 256), 256, 0, st>>>(m, vals, D.scale, D.sb,
                                                         in_order ? nullptr : keys);
  TSVD_LAUNCH_CHECK();
  if (in_order) return TSVD_OK;
  TSVD_TRY(stable_sort_pairs(keys, vals, keys2, vals2, h.nnz, bits_for(nrows - 1), stmp, st,
                             &in_alt));
  csr_gather_kernel<<<grid_for(h.nnz + 1, 256), 256, 0, st>>>(
      m, cinv, in_alt ? vals2 : vals, in_alt ? keys2 : keys, D.scale, D.sb);
  TSVD_LAUNCH_CHECK();
  return TSVD_OK;
}

// The sparse block of any valid matrix, built on the host: CSR over the padded
// rows and CSC over the compacted columns, both with ascending minor indices
// (counting sorts of the row-ordered triplets).
tsvd_status sparse_from_host(CallMemory &M, int32_t nrows, int32_t ncols, const HostBlock &H,
                             DirectBlock &D) {
  const int32_t nc = (int32_t)H.cmap.size();
  const int64_t nnz = (int64_t)H.tval.size();
  const int sp = (int)round_up(nrows, kRowPad);
  D.nc = nc;
  D.scale = scale_for(H.vmax);
  D.sparse = true;
  if (nc == 0) return TSVD_OK;
  std::vector<float> tval(nnz);
  for (int64_t t = 0; t < nnz; ++t) tval[t] = (float)((float)H.tval[t] * D.scale);
  std::vector<int64_t> rp(sp + 1, 0), cp(nc + 1, 0);
  for (int64_t t = 0; t < nnz; ++t) {
    rp[H.trow[t] + 1]++;
    cp[H.tcol[t] + 1]++;
  }
  for (int i = 0; i < sp; ++i) rp[i + 1] += rp[i];
  for (int c = 0; c < nc; ++c) cp[c + 1] += cp[c];
  std::vector<int32_t> ci(nnz), ri(nnz);
  std::vector<float> rv(nnz), cv(nnz);
  std::vector<int64_t> rpos(rp.begin(), rp.end() - 1), cpos(cp.begin(), cp.end() - 1);
  std::vector<int64_t> order(nnz);
  for (int64_t t = 0; t < nnz; ++t) order[t] = t;
  std::stable_sort(order.begin(), order.end(), [&](int64_t a, int64_t b) {
    return H.trow[a] != H.trow[b] ? H.trow[a] < H.trow[b] : H.tcol[a] < H.tcol[b];
  });
  for (int64_t t : order) {
    const int64_t a = rpos[H.trow[t]]++;
    ci[a] = H.tcol[t];
    rv[a] = tval[t];
    const int64_t b = cpos[H.tcol[t]]++;
    ri[b] = H.trow[t];
    cv[b] = tval[t];
  }
  cudaStream_t st = M.st;
  int32_t *cmap, *cinv;
  TSVD_TRY(M.carve([&](DeviceArena &A) -> tsvd_status {
    TSVD_TRY(take_sparse(A, D.sb, sp, nc, nnz));
    TSVD_TRY(device_take(&A, &cmap, (size_t)nc));
    return device_take(&A, &cinv, (size_t)ncols);
  }));
  const SparseBlock &sb = D.sb;
  auto up = [&](void *d, const void *src, size_t bytes) {
    return cudaMemcpyAsync(d, src, bytes, cudaMemcpyHostToDevice, st);
  };
  TSVD_CUDA(up(sb.rowptr, rp.data(), sizeof(int64_t) * rp.size()));
  TSVD_CUDA(up(sb.colptr, cp.data(), sizeof(int64_t) * cp.size()));
  TSVD_CUDA(up(sb.colidx, ci.data(), sizeof(int32_t) * nnz));
  TSVD_CUDA(up(sb.rowidx, ri.data(), sizeof(int32_t) * nnz));
  TSVD_CUDA(up(sb.rval, rv.data(), sizeof(float) * nnz));
  TSVD_CUDA(up(sb.cval, cv.data(), sizeof(float) * nnz));
  TSVD_CUDA(up(cmap, H.cmap.data(), sizeof(int32_t) * nc));
  TSVD_CUDA(up(cinv, H.cinv.data(), sizeof(int32_t) * ncols));
  TSVD_CUDA(cudaStreamSynchronize(st));  // the host vectors go out of scope
  D.cmap = cmap;
  D.cinv = cinv;
  return TSVD_OK;
}

tsvd_status frpca_direct(int32_t nrows, int32_t ncols, int64_t nnz, const int64_t *row_ptr,
                         const int32_t *col_idx, const double *values, int32_t index_base,
                         int32_t k, int32_t q, uint64_t seed, bool sparse, double *U, double *S,
                         double *V) {
  if (nrows < 1 || ncols < 1 || nnz < 0 || !row_ptr || (nnz > 0 && (!col_idx || !values)))
    return fail(TSVD_ERR_INVALID, "frpca: bad matrix arguments");
  if (index_base != 0 && index_base != 1) return fail(TSVD_ERR_INVALID, "frpca: index_base");
  const bool args_ok = k >= 1 && k + 5 <= kLp && q >= 1;
  DirectBlock D;
  CallMemory M;
  bool ready = false;
  tsvd_status s1 = TSVD_OK;
  if (args_ok) {
    s1 = M.open();
    if (s1 == TSVD_OK)
      s1 = block_on_device(M, nrows, ncols, nnz, row_ptr, col_idx, values, index_base, sparse, D,
                           &ready);
  }
  HostBlock H;
  bool walked = false;
  // The host's walk and, for the sparse form, its build in place of the device's: 16
  // bytes an entry on the device, where the device's own build takes up to 44.
  auto from_host = [&]() -> tsvd_status {
    cudaGetLastError();
    if (!walked)
      TSVD_TRY(host_block(nrows, ncols, nnz, row_ptr, col_idx, values, index_base, H));
    walked = true;
    if (!args_ok) return fail(TSVD_ERR_INVALID, "frpca: k=%d q=%d", k, q);
    D = DirectBlock();
    if (H.cmap.empty()) return TSVD_OK;
    if (!M.st || !sparse) return s1 != TSVD_OK ? s1 : fail(TSVD_ERR_STATE, "frpca: matrix");
    for (void *p : M.held) cudaFree(p);
    M.held.clear();
    return sparse_from_host(M, nrows, ncols, H, D);
  };
  // its errors come before those of the device and of k and q
  if (s1 != TSVD_OK || !ready) TSVD_TRY(from_host());
  if (D.nc == 0) {
    if (S) std::fill(S, S + k, 0.0);
    if (U) std::fill(U, U + (size_t)nrows * k, 0.0);
    if (V) std::fill(V, V + (size_t)ncols * k, 0.0);
    return TSVD_OK;
  }
  const int sp = (int)round_up(nrows, kRowPad);
  const int64_t stage_n = std::min<int64_t>(kStage, (int64_t)std::max(nrows, ncols) * k);
  float *du, *dv, *ds;
  double *stage;
  FrpcaWork W;
  auto take_work = [&]() {
    return M.carve([&](DeviceArena &A) -> tsvd_status {
      TSVD_TRY(device_take(&A, &du, (size_t)sp * k));
      TSVD_TRY(device_take(&A, &dv, (size_t)D.nc * k));
      TSVD_TRY(device_take(&A, &ds, (size_t)k));
      TSVD_TRY(device_take(&A, &stage, (size_t)stage_n));
      return frpca_work_alloc(W, 1, D.nc, sp, k + 5, k, true, &A, M.st);
    });
  };
  s1 = take_work();
  if (s1 == TSVD_ERR_OOM && sparse && !walked) {
    // the call fits beside the 16 bytes an entry, but not beside what the build has left
    frpca_work_free(W);
    s1 = from_host();
    if (s1 == TSVD_OK) s1 = take_work();
  }
  if (s1 == TSVD_OK) {
    FrpcaProblem P;
    P.block = 0;
    P.at = D.at;
    P.ncols = D.nc;
    P.colmap = D.cmap;
    P.col_base = 0;
    P.b_out = nullptr;
    P.sigma_out = ds;
    P.u_out = du;
    P.v_out = dv;
    P.sparse = D.sparse ? &D.sb : nullptr;
    double ssum = 0;
    s1 = frpca_batch(W, &P, 1, q, seed, nrows, M.st, &ssum);
  }
  // descending sigma; U nrows x k, V ncols x k, column-major
  std::vector<float> hs(k);
  auto results = [&]() -> tsvd_status {
    TSVD_CUDA(cudaMemcpyAsync(hs.data(), ds, sizeof(float) * k, cudaMemcpyDeviceToHost, M.st));
    TSVD_CUDA(cudaStreamSynchronize(M.st));
    if (U) TSVD_TRY(fetch_columns(du, k, nullptr, nrows, stage, U, M.st));
    if (V) TSVD_TRY(fetch_columns(dv, k, D.cinv, ncols, stage, V, M.st));
    for (int j = 0; S && j < k; ++j) S[j] = hs[j] / D.scale;
    return TSVD_OK;
  };
  if (s1 == TSVD_OK) s1 = results();
  frpca_work_free(W);
  return s1;
}

}  // namespace

extern "C" tsvd_status tsvd_frpca(int32_t nrows, int32_t ncols, int64_t nnz, const int64_t *row_ptr,
                                  const int32_t *col_idx, const double *values, int32_t index_base,
                                  int32_t k, int32_t q, uint64_t seed, double *U, double *S,
                                  double *V) {
  return frpca_direct(nrows, ncols, nnz, row_ptr, col_idx, values, index_base, k, q, seed, false, U,
                      S, V);
}

extern "C" tsvd_status tsvd_frpca_fp32(int32_t nrows, int32_t ncols, int64_t nnz,
                                       const int64_t *row_ptr, const int32_t *col_idx,
                                       const double *values, int32_t index_base, int32_t k,
                                       int32_t q, uint64_t seed, double *U, double *S,
                                       double *V) {
  return frpca_direct(nrows, ncols, nnz, row_ptr, col_idx, values, index_base, k, q, seed, true, U,
                      S, V);
}

extern "C" void frPCA(mat_csr *A, mat **U, mat **S, mat **V, int k, int q) {
  if (!A || !U || !S || !V || !*U || !*S || !*V) {
    fail(TSVD_ERR_INVALID, "frPCA: null argument");
    return;
  }
  const int m = A->nrows, n = A->ncols;
  std::vector<int64_t> rp(m + 1, 0);
  std::vector<int32_t> ci;
  std::vector<double> va;
  ci.reserve(A->nnz > 0 ? A->nnz : 0);
  va.reserve(A->nnz > 0 ? A->nnz : 0);
  for (int i = 0; i < m; ++i) {
    for (int t = A->pointerB[i] - 1; t < A->pointerE[i] - 1; ++t) {
      ci.push_back(A->cols[t] - 1);
      va.push_back(A->values[t]);
    }
    rp[i + 1] = (int64_t)ci.size();
  }
  std::vector<double> u((size_t)m * k), s(k), v((size_t)n * k);
  // the caller's doubles enter as FP32 (SpMM products), the precision the
  // reference's path keeps most closely on this hardware
  tsvd_status st = tsvd_frpca_fp32(m, n, (int64_t)ci.size(), rp.data(), ci.data(), va.data(), 0,
                                   k, q, g_frpca_seed, u.data(), s.data(), v.data());
  mat *Um = *U, *Sm = *S, *Vm = *V;
  if (st != TSVD_OK) {
    std::memset(Um->d, 0, sizeof(double) * (size_t)Um->nrows * Um->ncols);
    std::memset(Sm->d, 0, sizeof(double) * (size_t)Sm->nrows * Sm->ncols);
    std::memset(Vm->d, 0, sizeof(double) * (size_t)Vm->nrows * Vm->ncols);
    return;
  }
  // ascending order, as dsyevd hands them to the reference (frpca.c:298-310)
  for (int j = 0; j < k; ++j) {
    int src = k - 1 - j;
    Sm->d[j] = s[src];
    std::memcpy(Um->d + (size_t)j * Um->nrows, u.data() + (size_t)src * m, sizeof(double) * m);
    std::memcpy(Vm->d + (size_t)j * Vm->nrows, v.data() + (size_t)src * n, sizeof(double) * n);
  }
}

// dense_sub_svd_function (Code/Tree_u_NC.cpp:238-262) over
// truncated_singular_value_decomposition (matrix_vector_functions_intel_mkl.c
// :1259-1300): US = U_d diag(s_d) of the dense rows x cols matrix M
// (column-major, as the reference's mat), sigma = s_d descending. The tree
// merge's own path: compensated Gram, eigen-solve, and for more
// than 256 columns the subspace iteration of the wide merge.
extern "C" tsvd_status tsvd_merge_svd(int32_t rows, int32_t cols, const double *M, int32_t d,
                                      double *US, double *sigma) {
  if (rows < 1 || cols < 1 || !M || !US || !sigma) return fail(TSVD_ERR_INVALID, "merge_svd: bad arguments");
  if (d < 1 || d > std::min(rows, cols) || d > kLp || cols > 2048 || (cols > 256 && std::min(rows, 256) < d))
    return fail(TSVD_ERR_INVALID, "merge_svd: d = %d for %d x %d (d <= %d, cols <= 2048)", d, rows,
                cols, kLp);
  const int sp = (int)round_up(rows, kRowPad);
  CallMemory M1;
  TSVD_TRY(M1.open());
  cudaStream_t st = M1.st;
  float *m, *dout, *dsig;  // m row-major fp32, as the merge keeps factors
  double *stage;
  const int64_t total = (int64_t)rows * cols;
  FrpcaWork W;
  auto run = [&]() -> tsvd_status {
    TSVD_TRY(M1.carve([&](DeviceArena &A) -> tsvd_status {
      TSVD_TRY(device_take(&A, &m, (size_t)total));
      TSVD_TRY(device_take(&A, &dout, (size_t)rows * d));
      TSVD_TRY(device_take(&A, &dsig, (size_t)d));
      TSVD_TRY(device_take(&A, &stage, (size_t)std::min(kStage, total)));
      return frpca_work_alloc(W, 1, rows, sp, std::min(kLp, d + 5), d, true, &A, st);
    }));
    for (int64_t f0 = 0; f0 < total; f0 += kStage) {
      const int64_t n = std::min(kStage, total - f0);
      TSVD_CUDA(cudaMemcpyAsync(stage, M + f0, sizeof(double) * n, cudaMemcpyHostToDevice, st));
      narrow_rows_kernel<<<grid_for(n, 256), 256, 0, st>>>(stage, rows, cols, f0, n, m);
      TSVD_LAUNCH_CHECK();
    }
    TSVD_TRY(merge_matrix(W, m, rows, cols, dout, dsig, st));
    std::vector<float> hs(d);
    TSVD_CUDA(cudaMemcpyAsync(hs.data(), dsig, sizeof(float) * d, cudaMemcpyDeviceToHost, st));
    TSVD_TRY(eig_sweeps_fetch(W, st));
    TSVD_CUDA(cudaStreamSynchronize(st));
    TSVD_TRY(eig_check(W));
    for (int32_t j = 0; j < d; ++j) sigma[j] = hs[j];
    return fetch_columns(dout, d, nullptr, rows, stage, US, st);
  };
  const tsvd_status s1 = run();
  frpca_work_free(W);
  return s1;
}
