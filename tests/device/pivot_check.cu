// GPU driver for tests/test_pivot_math.py: the pivots' reciprocal and root
// (csrc/gbba_pivot.cuh) beside CUDA's division and square root.
//
// Input:  doubles d[n].  Output: double rcp[n], root[n], inverse root[n],
//         1 / d [n], sqrt(d) [n].
#include <cstdio>
#include <vector>

#include "gbba_pivot.cuh"

__global__ void k_check(const double* d, long n, double* out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s, r;
  gbba::sqrt_newton(d[i], s, r);
  out[i] = gbba::rcp_series(d[i]);
  out[n + i] = s;
  out[2 * n + i] = r;
  out[3 * n + i] = 1.0 / d[i];
  out[4 * n + i] = sqrt(d[i]);
}

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  FILE* in = fopen(argv[1], "rb");
  FILE* out = fopen(argv[2], "wb");
  if (!in || !out) return 2;
  fseek(in, 0, SEEK_END);
  const long n = ftell(in) / 8;
  rewind(in);
  std::vector<double> d(n), o(5 * n);
  if (n == 0 || (long)fread(d.data(), 8, n, in) != n) return 2;
  double *dd = nullptr, *od = nullptr;
  if (cudaMalloc(&dd, 8 * n) || cudaMalloc(&od, 40 * n)) return 3;
  if (cudaMemcpy(dd, d.data(), 8 * n, cudaMemcpyHostToDevice)) return 3;
  k_check<<<(unsigned)((n + 255) / 256), 256>>>(dd, n, od);
  if (cudaGetLastError() || cudaMemcpy(o.data(), od, 40 * n, cudaMemcpyDeviceToHost)) return 3;
  const bool ok = (long)fwrite(o.data(), 8, 5 * n, out) == 5 * n;
  fclose(out);
  return ok ? 0 : 2;
}
