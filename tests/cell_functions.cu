// Entry points of tests/test_gpu_cell_functions.py: functions of mp_cell.cuh over
// arrays, one element per thread.
#include "mp_cell.cuh"

using namespace mpb;

template <typename T>
__global__ void plasma_coef_kernel(double denom, double chi, const T *sig, double *out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  EParams<T> p;
  p.denom_d = denom;
  p.denom_t = T(denom);
  p.chi_raw = chi;
  CellCoef<T, 0> c = {};
  plasma_coef<T, 0>(p, sig[i], c);
  out[i] = c.chi_over_denom;
}

template <typename T>
static int plasma_coef_run(double denom, double chi, const T *sig, double *out, int n) {
  T *ds = nullptr;
  double *dout = nullptr;
  cudaError_t e = cudaMalloc(&ds, n * sizeof(T));
  if (e == cudaSuccess) e = cudaMalloc(&dout, n * sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(ds, sig, n * sizeof(T), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    plasma_coef_kernel<T><<<(n + 127) / 128, 128>>>(denom, chi, ds, dout, n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dout, n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(ds);
  cudaFree(dout);
  return int(e);
}

extern "C" int plasma_coef_f32(double denom, double chi, const float *sig, double *out, int n) {
  return plasma_coef_run(denom, chi, sig, out, n);
}
extern "C" int plasma_coef_f64(double denom, double chi, const double *sig, double *out, int n) {
  return plasma_coef_run(denom, chi, sig, out, n);
}

// The start of the Kerr solve, FP64 form (f32 = 0) or FP32 form.
__global__ void kerr_start_kernel(const double *A, const double *C, const double *E2, double *out, int n, int f32) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double C2 = C[i] * C[i];
  out[i] = f32 ? kerr_start(A[i], C[i], (float)C2, (float)E2[i]) : kerr_start(A[i], C[i], C2, E2[i]);
}

extern "C" int kerr_starts(const double *A, const double *C, const double *E2, double *out, int n, int f32) {
  const double *in[3] = {A, C, E2};
  double *d[4] = {nullptr, nullptr, nullptr, nullptr};
  cudaError_t e = cudaSuccess;
  for (int q = 0; q < 4 && e == cudaSuccess; ++q) {
    e = cudaMalloc(&d[q], n * sizeof(double));
    if (e == cudaSuccess && q < 3) e = cudaMemcpy(d[q], in[q], n * sizeof(double), cudaMemcpyHostToDevice);
  }
  if (e == cudaSuccess) {
    kerr_start_kernel<<<(n + 127) / 128, 128>>>(d[0], d[1], d[2], d[3], n, f32);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d[3], n * sizeof(double), cudaMemcpyDeviceToHost);
  for (double *p : d) cudaFree(p);
  return int(e);
}
