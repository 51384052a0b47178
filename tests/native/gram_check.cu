// Largest error of the Gram kernel's off-diagonal entries against long double, relative
// to the sum of the entry's terms' magnitudes, as a power of two; one line per matrix.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "internal.h"

using namespace tsvd;

static double worst(int kind, int rows, int l) {
  std::mt19937_64 gen(kind + rows + l);
  std::normal_distribution<double> normal;
  std::vector<float> x((size_t)rows * l);
  for (int r = 0; r < rows; ++r)
    for (int c = 0; c < l; ++c) {
      double v = normal(gen);
      if (kind == 1 && r % l != c) v *= 1e-5;                   // nearly orthogonal columns
      if (kind == 2) v *= std::pow(10.0, -5.0 * c / l);         // very different norms
      if (kind == 3) v = (c % 2 && r % 2 ? -1 : 1) * (1 + 1e-3 * v);  // sums that cancel
      x[(size_t)r * l + c] = (float)v;
    }
  float *dx;
  double *dg, *work;
  const float **px;
  double **pg;
  int32_t *dr;
  const size_t bytes = 4 * gram_work_bytes(rows, l, 1);
  cudaMalloc(&dx, x.size() * sizeof(float));
  cudaMalloc(&dg, sizeof(double) * l * l);
  cudaMalloc(&work, bytes);
  cudaMalloc(&px, sizeof *px);
  cudaMalloc(&pg, sizeof *pg);
  cudaMalloc(&dr, sizeof *dr);
  cudaMemcpy(dx, x.data(), x.size() * sizeof(float), cudaMemcpyHostToDevice);
  cudaMemcpy(px, &dx, sizeof dx, cudaMemcpyHostToDevice);
  cudaMemcpy(pg, &dg, sizeof dg, cudaMemcpyHostToDevice);
  cudaMemcpy(dr, &rows, sizeof rows, cudaMemcpyHostToDevice);
  const tsvd_status st = gram_batched(px, dr, rows, l, l, pg, work, bytes, 1, nullptr);
  std::vector<double> g((size_t)l * l);
  const cudaError_t e =
      cudaMemcpy(g.data(), dg, sizeof(double) * l * l, cudaMemcpyDeviceToHost);
  for (void *p : {(void *)dx, (void *)dg, (void *)work, (void *)px, (void *)pg, (void *)dr})
    cudaFree(p);
  if (st != TSVD_OK || e != cudaSuccess) return 1.0;
  double most = 0;
  for (int i = 0; i < l; ++i)
    for (int j = 0; j < i; ++j) {
      long double sum = 0, abs = 0;
      for (int r = 0; r < rows; ++r) {
        const long double p = (long double)x[(size_t)r * l + i] * x[(size_t)r * l + j];
        sum += p;
        abs += fabsl(p);
      }
      for (double v : {g[(size_t)i * l + j], g[(size_t)j * l + i]})
        most = std::max(most, (double)(fabsl(v - sum) / abs));
    }
  return most;
}

int main() {
  for (int kind = 0; kind < 4; ++kind)
    for (int rows : {1, 31, 33, 300, 1500})
      for (int l : {2, 37, 133})
        std::printf("%d %d %d %.2f\n", kind, rows, l, std::log2(worst(kind, rows, l) + 1e-30));
  return 0;
}
