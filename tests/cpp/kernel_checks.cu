// Kernels and launches of the library called one by one, for tests.
#include <cuda_runtime.h>

#include <vector>

#include "launch.h"

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
