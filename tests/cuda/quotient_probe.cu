// Element-wise launches of the kernels' own quotient, root and reconstruction
// functions for tests/test_gpu_quotients.py: `n` elements, one thread each, on
// host arrays.  Built with the flags of the form under test.
#include "cb_stage.cuh"

using namespace cb;

namespace {
enum { QUOT, ROOT, THIRD, BY27 };

__global__ void fp64_kernel(int op, const double *a, const double *b, double *out, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  if (op == QUOT) out[t] = Den<double>(b[t])(a[t]);
  else if (op == ROOT) out[t] = root(a[t]);
  else if (op == THIRD) out[t] = third<double, false>(a[t]);
  else out[t] = by27<false>(a[t]);
}

// v: six stencil values per element and lane (two lanes); out: left and right
// values of both lanes, packed, then scalar
__global__ void recon_kernel(int op, const float *v, float *out, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  float2 s[6], l, r;
#pragma unroll
  for (int x = 0; x < 6; x++) s[x] = make_float2(v[t * 12 + x], v[t * 12 + 6 + x]);
  float sl[2], sr[2];
  if (op == 0) muscl_2(s[1], s[2], s[3], s[4], l, r);
  else if (op == 1) weno3_2(s[1], s[2], s[3], s[4], l, r);
  else { l = weno5_2(s[0], s[1], s[2], s[3], s[4]); r = weno5_2(s[5], s[4], s[3], s[2], s[1]); }
  for (int y = 0; y < 2; y++) {
    const float *p = v + t * 12 + 6 * y;
    if (op == 0) {
      sl[y] = muscl_l<float>(p[1], p[2], p[3]);
      sr[y] = muscl_r<float>(p[2], p[3], p[4]);
    } else if (op == 1) {
      sl[y] = weno3_l<float>(p[1], p[2], p[3]);
      sr[y] = weno3_r<float>(p[2], p[3], p[4]);
    } else {
      sl[y] = weno5<float>(p[0], p[1], p[2], p[3], p[4]);
      sr[y] = weno5<float>(p[5], p[4], p[3], p[2], p[1]);
    }
  }
  const float o[8] = {l.x, l.y, r.x, r.y, sl[0], sl[1], sr[0], sr[1]};
  for (int x = 0; x < 8; x++) out[t * 8 + x] = o[x];
}

// quotient, reciprocal and root as the mixed form's functions and as its
// compiler's operators (-prec-div=false, -prec-sqrt=false)
__global__ void fp32_kernel(const float *a, const float *b, float *out, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const float o[6] = {Den<float>(b[t])(a[t]), a[t] / b[t], rcp_approx(b[t]), 1.f / b[t], root(b[t]), sqrtf(b[t])};
  for (int x = 0; x < 6; x++) out[t * 6 + x] = o[x];
}

template <class T, class L>
int run(const T *x, size_t nx, const T *y, size_t ny, T *out, size_t no, L launch) {
  T *dx = nullptr, *dy = nullptr, *dout = nullptr;
  cudaError_t e = cudaMalloc(&dx, sizeof(T) * nx);
  if (e == cudaSuccess) e = cudaMalloc(&dy, sizeof(T) * (ny ? ny : 1));
  if (e == cudaSuccess) e = cudaMalloc(&dout, sizeof(T) * no);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, sizeof(T) * nx, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && ny) e = cudaMemcpy(dy, y, sizeof(T) * ny, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    launch(dx, dy, dout);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dout, sizeof(T) * no, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dy);
  cudaFree(dout);
  return (int)e;
}
int blocks(int n) { return (n + 255) / 256; }
}  // namespace

extern "C" {
int probe_fp64(int op, const double *a, const double *b, double *out, int n) {
  return run(a, n, b, n, out, n, [&](double *x, double *y, double *o) { fp64_kernel<<<blocks(n), 256>>>(op, x, y, o, n); });
}
int probe_recon(int op, const float *v, float *out, int n) {
  return run(v, 12 * (size_t)n, (const float *)nullptr, 0, out, 8 * (size_t)n,
             [&](float *x, float *, float *o) { recon_kernel<<<blocks(n), 256>>>(op, x, o, n); });
}
int probe_fp32(const float *a, const float *b, float *out, int n) {
  return run(a, n, b, n, out, 6 * (size_t)n, [&](float *x, float *y, float *o) { fp32_kernel<<<blocks(n), 256>>>(x, y, o, n); });
}
}
