// Device functions of rkdg_physics.cuh and rkdg_generic.cuh beside CUDA's own, for
// test_gpu_device_math.py.
#include "rkdg_generic.cuh"
#include "rkdg_physics.cuh"

using namespace rkdg;

// out[0] rcp_f64, [1] 1/x, [2] sqrt_f64, [3] sqrt(x)
__global__ void k_roots(int n, const double* x, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = rcp_f64(x[i]);
  out[n + i] = 1.0 / x[i];
  out[2 * n + i] = sqrt_f64(x[i]);
  out[3 * n + i] = sqrt(x[i]);
}
__global__ void k_root_n(int n, int m, double invm, const double* x, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = root_n(x[i], m, invm);
}
// bits of cut_f32 and of the conversion towards zero
__global__ void k_cut(int n, const double* x, unsigned* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = __float_as_uint(cut_f32(x[i]));
  out[n + i] = __float_as_uint(__double2float_rz(x[i]));
}
// bits of the float pair by split_value and by conversions
__global__ void k_splits(int n, const double* x, unsigned* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float h, l;
  split_value(x[i], h, l);
  out[i] = __float_as_uint(h);
  out[n + i] = __float_as_uint(l);
  h = (float)x[i];
  out[2 * n + i] = __float_as_uint(h);
  out[3 * n + i] = __float_as_uint((float)(x[i] - (double)h));
}
__global__ void k_widen(int n, const float* x, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = widen(x[i]);
}
// the FP32 flux and speed of hexahedra, quads and hanging faces
template <int DIM>
__global__ void k_plain(int n, const double* u1, const double* u2, const double* nor, double* flux, double* speed,
                        float gamma, float cov, int rs, int avg) {
  constexpr int NEQ = DIM + 2;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s1[NEQ], s2[NEQ], nn[DIM], F[NEQ];
  for (int k = 0; k < NEQ; ++k) {
    s1[k] = (float)u1[i * NEQ + k];
    s2[k] = (float)u2[i * NEQ + k];
    F[k] = 0.0f;
  }
  for (int d = 0; d < DIM; ++d) nn[d] = (float)nor[i * DIM + d];
  speed[i] = (double)riemann<DIM, float, true>(s1, s2, nn, F, gamma, cov, rs, avg);
  for (int k = 0; k < NEQ; ++k) flux[i * NEQ + k] = (double)F[k];
}

extern "C" {
int check_roots(int n, const double* x, double* out) {
  k_roots<<<(n + 255) / 256, 256>>>(n, x, out);
  return (int)cudaDeviceSynchronize();
}
int check_root_n(int n, int m, double invm, const double* x, double* out) {
  k_root_n<<<(n + 255) / 256, 256>>>(n, m, invm, x, out);
  return (int)cudaDeviceSynchronize();
}
int check_cut(int n, const double* x, unsigned* out) {
  k_cut<<<(n + 255) / 256, 256>>>(n, x, out);
  return (int)cudaDeviceSynchronize();
}
int check_split(int n, const double* x, unsigned* out) {
  k_splits<<<(n + 255) / 256, 256>>>(n, x, out);
  return (int)cudaDeviceSynchronize();
}
int check_widen(int n, const float* x, double* out) {
  k_widen<<<(n + 255) / 256, 256>>>(n, x, out);
  return (int)cudaDeviceSynchronize();
}
int check_plain(int dim, int n, const double* u1, const double* u2, const double* nor, double* flux, double* speed,
                float gamma, float cov, int rs, int avg) {
  if (dim == 2)
    k_plain<2><<<(n + 127) / 128, 128>>>(n, u1, u2, nor, flux, speed, gamma, cov, rs, avg);
  else
    k_plain<3><<<(n + 127) / 128, 128>>>(n, u1, u2, nor, flux, speed, gamma, cov, rs, avg);
  return (int)cudaDeviceSynchronize();
}
}
