// The primitives of seeded.cuh over arrays, beside CUDA's own operators (test
// of test_gpu_seeded.py).
#include "../proteuscfd_gb300/csrc/seeded.cuh"

__global__ void k_apply(int op, long long n, const double* a, const double* b, double* out, double* ref) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], y = b[i];
  double inv;
  switch (op) {
    case 0: out[i] = pcfd::recip(x); ref[i] = 1.0 / x; break;
    case 1: out[i] = pcfd::quot(x, y); ref[i] = x / y; break;
    case 2: out[i] = pcfd::Quot64(y).of(x); ref[i] = x / y; break;
    case 3: out[i] = pcfd::root(x); ref[i] = sqrt(x); break;
    case 4: out[i] = pcfd::sqrt_inv(x, &inv); ref[i] = sqrt(x); break;
    case 5: pcfd::sqrt_inv(x, &inv); out[i] = inv; ref[i] = 1.0 / sqrt(x); break;
    case 6: out[i] = pcfd::widen((float)x); ref[i] = (double)(float)x; break;
    case 7: out[i] = (double)pcfd::est_f32(x); ref[i] = (double)(float)x; break;
    case 8: out[i] = pcfd::key_gt(x, y) ? 1.0 : 0.0; ref[i] = x > y ? 1.0 : 0.0; break;
  }
}

// a, b, out, ref: host arrays of n; returns a cudaError_t
extern "C" int seeded_apply(int op, long long n, const double* a, const double* b, double* out, double* ref) {
  double* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 4 * n * sizeof(double));
  if (e != cudaSuccess) return e;
  if (e == cudaSuccess) e = cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_apply<<<(unsigned)((n + 127) / 128), 128>>>(op, n, d, d + n, d + 2 * n, d + 3 * n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, n * sizeof(double), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(ref, d + 3 * n, n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e;
}
