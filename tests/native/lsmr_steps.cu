// The scalar recurrences of fe_lsmr.cuh on given alpha_k, beta_k, compiled like
// the one-kernel solves: out[k] = {normr, normA, condA, normAr, c1, c2, c3}
// after step k.
#include "fe_lsmr.cuh"

__global__ void k_steps(const double* alpha, const double* beta, int n, double* out) {
  fe::Inst s;
  memset(&s, 0, sizeof(s));
  s.maxiter = 1000;
  s.ctol = 1e-8;
  s.alpha = alpha[0];
  s.beta = beta[0];
  s.s_v = 1.0 / s.alpha;
  s.u_scale = 1.0 / s.beta;
  fe::lsmr_init(s, 1);
  for (int k = 1; k <= n; ++k) {
    s.iter = k;
    s.alpha = alpha[k];
    s.beta = beta[k];
    fe::lsmr_rotate(s);
    s.normx = 1.5;
    fe::lsmr_test(s);
    const double o[7] = {s.normr, s.normA, s.condA, s.normAr, s.c1, s.c2, s.c3};
    for (int i = 0; i < 7; ++i) out[(k - 1) * 7 + i] = o[i];
  }
}

extern "C" int lsmr_steps(const double* alpha, const double* beta, int n, double* out) {
  double *a = nullptr, *b = nullptr, *o = nullptr;
  cudaError_t e = cudaMalloc(&a, (n + 1) * 8);
  if (e == cudaSuccess) e = cudaMalloc(&b, (n + 1) * 8);
  if (e == cudaSuccess) e = cudaMalloc(&o, n * 56);
  if (e == cudaSuccess) e = cudaMemcpy(a, alpha, (n + 1) * 8, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b, beta, (n + 1) * 8, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_steps<<<1, 1>>>(a, b, n, o);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, o, n * 56, cudaMemcpyDeviceToHost);
  cudaFree(a);
  cudaFree(b);
  cudaFree(o);
  return (int)e;
}
