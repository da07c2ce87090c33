// Kernels and launches of the library called one by one, for tests.
#include <cuda_runtime.h>

#include <vector>

#include "launch.h"
#include "weno.cuh"

namespace {

struct Buffers {
  std::vector<void*> p;
  cudaError_t e = cudaSuccess;
  template <typename T>
  T* up(const T* host, long long n) {
    T* d = nullptr;
    if (e == cudaSuccess) e = cudaMalloc(&d, sizeof(T) * n);
    if (e == cudaSuccess && d) p.push_back(d);
    if (e == cudaSuccess)
      e = host ? cudaMemcpy(d, host, sizeof(T) * n, cudaMemcpyHostToDevice)
               : cudaMemset(d, 0, sizeof(T) * n);
    return d;
  }
  template <typename T>
  void down(T* host, const T* d, long long n) {
    if (e == cudaSuccess) e = cudaMemcpy(host, d, sizeof(T) * n, cudaMemcpyDeviceToHost);
  }
  ~Buffers() {
    for (void* d : p) cudaFree(d);
  }
};

}  // namespace

// SSP2's plain implicit stage 2 of `count` queued cells, or with count < 0 of
// every interior cell, into out (14 planes, zero elsewhere).
extern "C" int run_stage2(const void* cfg, int count, const int* cells, const double* cons,
                          const double* aux, const double* u1, const double* flux1,
                          const double* source1, double dt, double* out) {
  mth::Grid g;
  if (!mth::grid_from_config(cfg, &g)) return -1;
  for (int q = 0; q < count; ++q)
    if (cells[q] < 0 || cells[q] >= g.Ntot) return -1;
  const long long n = 14 * g.Ntot;
  Buffers b;
  const double *c = b.up(cons, n), *a = b.up(aux, 17 * g.Ntot), *u = b.up(u1, n);
  const double *f = b.up(flux1, n), *s = b.up(source1, n);
  double* o = b.up<double>(nullptr, n);
  mth::C2PWork w;
  w.fail_list = b.up<int>(nullptr, g.Ntot);
  w.fail_count = b.up<int>(nullptr, 1);
  w.counters = b.up<long long>(nullptr, 16);
  if (b.e != cudaSuccess) return b.e;
  if (count > 0) {
    b.e = cudaMemcpy(w.fail_list, cells, sizeof(int) * count, cudaMemcpyHostToDevice);
    if (b.e == cudaSuccess)
      b.e = cudaMemcpy(w.fail_count, &count, sizeof count, cudaMemcpyHostToDevice);
    if (b.e != cudaSuccess) return b.e;
  }
  b.e = count < 0 ? mth::launch_imex_stage(g, 2, c, a, u, f, s, o, dt, w, nullptr)
                  : mth::launch_imex_stage_queued(g, 2, c, a, u, f, s, o, dt, w, nullptr);
  if (b.e == cudaSuccess) b.e = cudaDeviceSynchronize();
  b.down(out, o, n);
  return b.e;
}

// SSP2's separate closing combination (cons updated in place).
extern "C" int run_ssp2_combine(const void* cfg, double* cons, const double* flux1,
                                const double* flux2, const double* source1,
                                const double* source2, double dt) {
  mth::Grid g;
  if (!mth::grid_from_config(cfg, &g)) return -1;
  const long long n = 14 * g.Ntot;
  Buffers b;
  double* c = b.up(cons, n);
  const double *f1 = b.up(flux1, n), *f2 = b.up(flux2, n);
  const double *s1 = b.up(source1, n), *s2 = b.up(source2, n);
  if (b.e != cudaSuccess) return b.e;
  b.e = mth::launch_ssp2_combine(g, 14, c, f1, f2, s1, s2, dt, nullptr);
  if (b.e == cudaSuccess) b.e = cudaDeviceSynchronize();
  b.down(cons, c, n);
  return b.e;
}

namespace {

// out[k n + i]: 0 div_by (y = div_rcp(b)), 1 Divisor(b)(a), 2 IEEE a / b, 3 rcp64(b),
// 4 rsqrt64(b), 5 and 6 the residuals 1 - b y0 and 1 - b y0^2 of the hardware's
// approximations of 1/b and 1/sqrt(b).
__global__ void k_quotients(int n, const double* a, const double* b, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], d = b[i];
  out[i] = mth::div_by(x, d, mth::div_rcp(d));
  out[n + i] = mth::Divisor(d)(x);
  out[2 * n + i] = x / d;
  out[3 * n + i] = mth::rcp64(d);
  out[4 * n + i] = mth::rsqrt64(d);
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  out[5 * n + i] = __fma_rn(-d, y, 1.0);
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  out[6 * n + i] = __fma_rn(-(d * y), y, 1.0);
}

// out[k n + i]: the face of stencils v[2 ORDER * i ...] (ORDER cells upwind, ORDER
// downwind, in the order the points take them) by weno_face_exact with one
// operand test (0) and with two (1), and with IEEE divisions (2).
template <int ORDER>
__global__ void k_faces(int n, const double* v, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* p = v + 2 * ORDER * i;
  const double* m = p + 2 * ORDER - 1;  // read downwards
  out[i] = mth::weno_face_exact<ORDER, true>(p, m, 1);
  out[n + i] = mth::weno_face_exact<ORDER, false>(p, m, 1);
  out[2 * n + i] = mth::weno_face_ieee<ORDER>(p, m, 1);
}

}  // namespace

extern "C" int run_quotients(int n, const double* a, const double* b, double* out) {
  Buffers m;
  const double *x = m.up(a, n), *d = m.up(b, n);
  double* o = m.up<double>(nullptr, 7LL * n);
  if (m.e != cudaSuccess) return m.e;
  k_quotients<<<(n + 127) / 128, 128>>>(n, x, d, o);
  m.e = cudaDeviceSynchronize();
  m.down(out, o, 7LL * n);
  return m.e;
}

extern "C" int run_faces(int order, int n, const double* v, double* out) {
  Buffers m;
  const double* x = m.up(v, 2LL * order * n);
  double* o = m.up<double>(nullptr, 3LL * n);
  if (m.e != cudaSuccess) return m.e;
  if (order == 3)
    k_faces<3><<<(n + 127) / 128, 128>>>(n, x, o);
  else
    k_faces<5><<<(n + 127) / 128, 128>>>(n, x, o);
  m.e = cudaDeviceSynchronize();
  m.down(out, o, 3LL * n);
  return m.e;
}
