// Device functions of the library on arrays, for tests/test_gpu_device_functions.py.
#include "../examinimd_gb300/csrc/f32_pairs.cuh"

using namespace emd;

namespace {
__global__ void k_recip(const double* d, double* y, double* ref, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  y[i] = recip_rn(d[i]);
  ref[i] = 1.0 / d[i];
}
__global__ void k_sincos(const double* x, double* sn, double* cs, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  F2 s, c;
  f2_sincos(f2_split(x[i]), s, c);
  sn[i] = double(s.h) + double(s.l);
  cs[i] = double(c.h) + double(c.l);
}
__global__ void k_rsqrt(const double* x, double* y, double* split, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const F2 v = f2_split(x[i]), r = f2_rsqrt(v);
  y[i] = double(r.h) + double(r.l);
  split[i] = double(v.h) + double(v.l);
}

template <typename K>
int run(K k, const double* a, double* b, double* c, int n) {
  double *da = nullptr, *db = nullptr, *dc = nullptr;
  const size_t bytes = sizeof(double) * size_t(n);
  if (n <= 0 || cudaMalloc(&da, bytes) || cudaMalloc(&db, bytes) || cudaMalloc(&dc, bytes)) return 1;
  if (cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice)) return 2;
  k<<<(n + 255) / 256, 256>>>(da, db, dc, n);
  if (cudaGetLastError() || cudaDeviceSynchronize()) return 3;
  if (cudaMemcpy(b, db, bytes, cudaMemcpyDeviceToHost) || cudaMemcpy(c, dc, bytes, cudaMemcpyDeviceToHost)) return 4;
  cudaFree(da);
  cudaFree(db);
  cudaFree(dc);
  return 0;
}
}  // namespace

extern "C" int probe_recip(const double* d, double* y, double* ref, int n) { return run(k_recip, d, y, ref, n); }
extern "C" int probe_sincos(const double* x, double* s, double* c, int n) { return run(k_sincos, x, s, c, n); }
extern "C" int probe_rsqrt(const double* x, double* y, double* split, int n) { return run(k_rsqrt, x, y, split, n); }
