// Evaluates the quotients, reciprocals and roots of rod_fast.cuh on arrays
// (for test_gpu_rod_fast.py).
#include "rod_fast.cuh"

namespace {

__global__ void probe(int op, int n, const double* a, const double* b, double* o, double* o2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], y = b[i];
  double r = 0.0, r2 = 0.0;
  switch (op) {
    case 0: r = eb::rcp_from(x, eb::rcp_near(x)); break;
    case 1: r = eb::rcp_from(x, y); break;
    case 2: r = eb::rcp_from_rough(x, y); break;
    case 3: r = eb::div_from(x, y, eb::rcp_from(y, eb::rcp_near(y))); break;
    case 4: {
      const eb::Length l = eb::length_of(x);
      r = l.l;
      r2 = l.il;
      break;
    }
  }
  o[i] = r;
  o2[i] = r2;
}

}  // namespace

extern "C" int rod_fast_probe(int op, int n, const double* a, const double* b, double* o, double* o2) {
  double* d[4] = {nullptr, nullptr, nullptr, nullptr};
  const size_t bytes = static_cast<size_t>(n) * sizeof(double);
  cudaError_t e = cudaSuccess;
  for (auto& p : d)
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&p), bytes);
  if (e == cudaSuccess) e = cudaMemcpy(d[0], a, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d[1], b, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    probe<<<(n + 255) / 256, 256>>>(op, n, d[0], d[1], d[2], d[3]);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(o, d[2], bytes, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(o2, d[3], bytes, cudaMemcpyDeviceToHost);
  for (double* p : d) cudaFree(p);
  return static_cast<int>(e);
}
