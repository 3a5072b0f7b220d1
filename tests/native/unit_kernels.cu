// Device functions of the library that no entry point returns by themselves,
// one element per thread, for tests/test_gpu_unit_kernels.py.
#include <cuda_runtime.h>

#include "swc_recon_vjp.cuh"

namespace {

// v[5][n], rb[n], lb[n] -> vb[5][n]; two cells per thread in the lanes of
// Two<T>, as the stage adjoint pairs its variables (n even).
template <typename T>
__global__ void weno5_vjp_kernel(int n, const T* v, const T* rb, const T* lb,
                                 T* vb) {
  using O = swc::Two<T>;
  const int i = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (i + 1 >= n) return;
  typename O::V c[5], b[5];
  for (int k = 0; k < 5; ++k) {
    c[k] = O::mk(v[k * n + i], v[k * n + i + 1]);
    b[k] = O::splat(T(0));
  }
  swc::weno5_cell_vjp_v<O>(c, O::mk(rb[i], rb[i + 1]), O::mk(lb[i], lb[i + 1]),
                           b);
  for (int k = 0; k < 5; ++k) {
    vb[k * n + i] = b[k].x;
    vb[k * n + i + 1] = b[k].y;
  }
}

__global__ void rcp_normal_kernel(int n, const double* a, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = swc::rcp_normal(a[i]);
}

}  // namespace

extern "C" int unit_rcp_normal(int n, const void* a, void* out) {
  rcp_normal_kernel<<<(n + 127) / 128, 128>>>(
      n, static_cast<const double*>(a), static_cast<double*>(out));
  return cudaGetLastError() != cudaSuccess;
}

extern "C" int unit_weno5_vjp(int n, int f64, const void* v, const void* rb,
                              const void* lb, void* vb) {
  const int blocks = (n / 2 + 127) / 128;
  if (f64)
    weno5_vjp_kernel<double><<<blocks, 128>>>(
        n, static_cast<const double*>(v), static_cast<const double*>(rb),
        static_cast<const double*>(lb), static_cast<double*>(vb));
  else
    weno5_vjp_kernel<float><<<blocks, 128>>>(
        n, static_cast<const float*>(v), static_cast<const float*>(rb),
        static_cast<const float*>(lb), static_cast<float*>(vb));
  return cudaGetLastError() != cudaSuccess;
}
