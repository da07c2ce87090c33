// Plain FP64 implicit stages of the IMEX integrators (SSP2, SSP3, SSP2322):
// MINPACK's hybrid method on 14 unknowns per cell.  A unit of its own because
// each instantiation of the unrolled solver takes most of a minute to compile.
// Compiled with -fmad=false like kernels_fp64.cu: every expression rounds like
// the reference's x86-64 build.
#include <cuda_runtime.h>

#include "common.cuh"
#include "ensemble.h"
#include "launch.h"
#include "minpack.cuh"
#include "srrmhd.cuh"

namespace mth {

namespace {

inline int blocks_for(long long n, int t) { return (int)((n + t - 1) / t); }

// One implicit SSP2(222) stage per interior cell: a 14-unknown Powell-hybrid
// solve whose residual runs the secant C2P and the source (SSP2.cc:72-148).
constexpr double kImexTol = 0.000000149011612;
// The reference's SSP2 assigns IMEX2Arguments(data) to its member, but
// IMEX2Arguments::operator= (IMEX2Args.cc:34-63) does not copy gam / om2gam,
// so the constants in effect are those of the default constructor
// (IMEX2Args.h:35-37): om2gam = 0.4142135623730950, one ulp above the
// parameterised constructor's 0.4142135623730949.
constexpr double kImexGam = 0.2928932188134525;
constexpr double kImexOm2Gam = 0.4142135623730950;

// One cell of the implicit stage; returns the residual evaluations and sets
// the error flag when hybrd1 did not converge.
template <int STAGE>
__device__ __forceinline__ long long imex_cell(const Grid& g, long long cell,
                                               const double* __restrict__ cons,
                                               const double* __restrict__ aux_guess,
                                               const double* __restrict__ u1,
                                               const double* __restrict__ flux1,
                                               const double* __restrict__ source1,
                                               double* __restrict__ out, double dt, C2PWork w) {
  const long long N = g.Ntot;
  double u[14], f1[14], s1[14], x[14], fv[14];
#pragma unroll
  for (int v = 0; v < 14; ++v) u[v] = cons[v * N + cell];
  if (STAGE == 1) {
#pragma unroll
    for (int v = 0; v < 14; ++v) x[v] = u[v];
  } else {
#pragma unroll
    for (int v = 0; v < 14; ++v) {
      f1[v] = flux1[v * N + cell];
      // the mixed stage 2 fills only the planes that have a source
      s1[v] = SRRMHD::sourced(v) ? source1[v * N + cell] : 0.0;
      x[v] = 0.5 * (u[v] + u1[v * N + cell] - dt * f1[v]);
    }
  }
  srrmhd::ImexResidual R;
  R.u = u;
  R.flux1 = f1;
  R.source1 = s1;
  R.flux2 = nullptr;
  R.source2 = nullptr;
  R.hmgam = 0.0;
  R.dt = dt;
  R.gam = kImexGam;
  R.om2gam = kImexOm2Gam;
  R.g = g.gamma;
  R.sigma = g.sigma;
  R.sigma_exp = g.sigma_exp;
  R.functional = g.functional_sigma;
  R.cp = g.cp;
  R.Z = aux_guess[10 * N + cell];
  R.stage = STAGE;
  R.evals = 0;
  HybrdResult res = Hybrd<14>::solve(R, x, fv, kImexTol);
#pragma unroll
  for (int v = 0; v < 14; ++v) out[v * N + cell] = x[v];
  if (res.info != 1) {
    atomicAdd((unsigned long long*)&w.counters[2], 1ull);
    atomicOr((unsigned long long*)&w.counters[3], (unsigned long long)ERR_IMPLICIT);
  }
  return res.nfev;
}

template <int STAGE>
__global__ void __launch_bounds__(64)
    k_imex_stage(Grid g, const double* __restrict__ cons, const double* __restrict__ aux_guess,
                 const double* __restrict__ u1, const double* __restrict__ flux1,
                 const double* __restrict__ source1, double* __restrict__ out, double dt,
                 C2PWork w) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long evals = 0;
  if (t < n_interior(g)) {
    int i, j, k;
    interior_ijk(g, t, i, j, k);
    evals = imex_cell<STAGE>(g, cell_id(g, i, j, k), cons, aux_guess, u1, flux1, source1, out,
                             dt, w);
  }
  unsigned mask = __ballot_sync(0xffffffffu, t < n_interior(g));
  for (int o = 16; o > 0; o >>= 1) evals += __shfl_down_sync(0xffffffffu, evals, o);
  if ((threadIdx.x & 31) == 0 && mask) {
    atomicAdd((unsigned long long*)&w.counters[0], (unsigned long long)__popc(mask));
    atomicAdd((unsigned long long*)&w.counters[1], (unsigned long long)evals);
  }
}

// The same solve for the cells of a queue (mixed-form fallback).  One block
// of 64 threads strides over the queue; the count is reset at the end by the
// block after all threads finished reading it.
template <int STAGE>
__global__ void __launch_bounds__(64)
    k_imex_stage_queued(Grid g, const double* __restrict__ cons,
                        const double* __restrict__ aux_guess, const double* __restrict__ u1,
                        const double* __restrict__ flux1, const double* __restrict__ source1,
                        double* __restrict__ out, double dt, C2PWork w) {
  const int n = *w.fail_count;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    imex_cell<STAGE>(g, w.fail_list[q], cons, aux_guess, u1, flux1, source1, out, dt, w);
    atomicAdd((unsigned long long*)&w.counters[3 + 5], 1ull);  // fallbacks (counters[8])
  }
}

__global__ void k_reset_count(int* c) { *c = 0; }

// SSP3(332) / SSP2(322) implicit stages.  FORM is the residual form of
// srrmhd::ImexResidual (1, 2, 3: SSP3 stages; 4, 5, 6: SSP2322 stages);
// XFORM the initial guess: 0 U^n, 1 U1 (SSP3.cc:114), 2 U2 + dt (F1 + F2) / 4
// (SSP3.cc:149-150), 3 (U^n + U2 - dt F2) / 2 (SSP2322.cc:169-171).  The Z
// guess comes from zaux[10]; as the reference copies args.aux back into
// tempaux after each cell's solve, the last evaluation's Z goes to zout[10],
// which then seeds that stage's recovery.
constexpr double kSsp3Tol = 0.0000000149011612;
constexpr double kSsp2322Tol = 1.48e-8;
constexpr double kImexHmGam = 0.2071067811865475;

template <int FORM, int XFORM>
__device__ __forceinline__ long long imex_sweep_cell(
    const Grid& g, long long cell, const double* __restrict__ cons, const double* zaux,
    const double* __restrict__ u1, const double* __restrict__ u2,
    const double* __restrict__ flux1, const double* __restrict__ flux2,
    const double* __restrict__ source1, const double* __restrict__ source2,
    double* __restrict__ out, double* zout, double dt, C2PWork w) {
  const long long N = g.Ntot;
  double u[14], f1[14], f2[14], s1[14], s2[14], x[14], fv[14];
#pragma unroll
  for (int v = 0; v < 14; ++v) {
    const long long o = v * N + cell;
    u[v] = cons[o];
    f1[v] = (FORM == 2 || FORM == 3) ? flux1[o] : 0.0;
    s1[v] = (FORM == 2 || FORM == 3 || FORM == 5) ? source1[o] : 0.0;
    f2[v] = (FORM == 3 || FORM == 6) ? flux2[o] : 0.0;
    s2[v] = (FORM == 6) ? source2[o] : 0.0;
    if (XFORM == 0) x[v] = u[v];
    else if (XFORM == 1) x[v] = u1[o];
    else if (XFORM == 2) x[v] = u2[o] + dt * (f1[v] + f2[v]) / 4.0;
    else x[v] = 0.5 * (u[v] + u2[o] - dt * f2[v]);
  }
  srrmhd::ImexResidual R;
  R.u = u;
  R.flux1 = f1;
  R.source1 = s1;
  R.flux2 = f2;
  R.source2 = s2;
  R.dt = dt;
  R.gam = kImexGam;
  R.om2gam = kImexOm2Gam;
  R.hmgam = kImexHmGam;
  R.g = g.gamma;
  R.sigma = g.sigma;
  R.sigma_exp = g.sigma_exp;
  R.functional = g.functional_sigma;
  R.cp = g.cp;
  R.Z = zaux[10 * N + cell];
  R.stage = FORM;
  R.evals = 0;
  HybrdResult res = Hybrd<14>::solve(R, x, fv, FORM <= 3 ? kSsp3Tol : kSsp2322Tol);
#pragma unroll
  for (int v = 0; v < 14; ++v) out[v * N + cell] = x[v];
  zout[10 * N + cell] = R.Z;
  if (res.info != 1) {
    atomicAdd((unsigned long long*)&w.counters[2], 1ull);
    atomicOr((unsigned long long*)&w.counters[3], (unsigned long long)ERR_IMPLICIT);
  }
  return res.nfev;
}

template <int FORM, int XFORM>
__global__ void __launch_bounds__(64)
    k_imex_sweep(Grid g, const double* __restrict__ cons, const double* zaux,
                 const double* __restrict__ u1, const double* __restrict__ u2,
                 const double* __restrict__ flux1, const double* __restrict__ flux2,
                 const double* __restrict__ source1, const double* __restrict__ source2,
                 double* __restrict__ out, double* zout, double dt, C2PWork w) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long evals = 0;
  if (t < n_interior(g)) {
    int i, j, k;
    interior_ijk(g, t, i, j, k);
    evals = imex_sweep_cell<FORM, XFORM>(g, cell_id(g, i, j, k), cons, zaux, u1, u2, flux1,
                                         flux2, source1, source2, out, zout, dt, w);
  }
  const unsigned mask = __ballot_sync(0xffffffffu, t < n_interior(g));
  for (int o = 16; o > 0; o >>= 1) evals += __shfl_down_sync(0xffffffffu, evals, o);
  if ((threadIdx.x & 31) == 0 && mask) {
    atomicAdd((unsigned long long*)&w.counters[0], (unsigned long long)__popc(mask));
    atomicAdd((unsigned long long*)&w.counters[1], (unsigned long long)evals);
  }
}

// The same solve for the cells the mixed-form stage queued (grid stride over
// the queue; the count is cleared afterwards by k_reset_count).
template <int FORM, int XFORM>
__global__ void __launch_bounds__(64)
    k_imex_sweep_queued(Grid g, const double* __restrict__ cons, const double* zaux,
                        const double* __restrict__ u1, const double* __restrict__ u2,
                        const double* __restrict__ flux1, const double* __restrict__ flux2,
                        const double* __restrict__ source1, const double* __restrict__ source2,
                        double* __restrict__ out, double* zout, double dt, C2PWork w) {
  const int n = *w.fail_count;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    imex_sweep_cell<FORM, XFORM>(g, w.fail_list[q], cons, zaux, u1, u2, flux1, flux2, source1,
                                 source2, out, zout, dt, w);
    atomicAdd((unsigned long long*)&w.counters[8], 1ull);  // fallbacks
  }
}

// One CTA per SRRMHD member: the cells of the member's queue that the
// mixed-form implicit solve left unconverged, solved as the reference does
// (the ensemble counterpart of k_imex_stage_queued).
template <int STAGE>
__global__ void __launch_bounds__(64) k_ens_imex_queued(const Member* __restrict__ mem) {
  const Member& d = mem[blockIdx.x];
  if (d.model != MODEL_SRRMHD) return;
  const Grid g = d.g;
  const C2PWork w{d.fail_list, d.fail_count, d.counters + 4};
  const int n = *d.fail_count;
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    imex_cell<STAGE>(g, d.fail_list[q], d.a[EA_CONS], d.a[EA_AUX], d.a[EA_U1], d.a[EA_F1],
                     d.a[EA_S1], d.a[STAGE == 1 ? EA_U1 : EA_U2], d.dt, w);
    atomicAdd((unsigned long long*)&w.counters[8], 1ull);  // implicit fallbacks
  }
  __syncthreads();
  if (threadIdx.x == 0) *d.fail_count = 0;
}

}  // namespace

cudaError_t launch_imex_stage(const Grid& g, int stage, const double* cons,
                              const double* aux_guess, const double* u1, const double* flux1,
                              const double* source1, double* out, double dt, C2PWork w,
                              cudaStream_t st) {
  const long long nI = (long long)(g.ie - g.is) * (g.je - g.js) * (g.ke - g.ks);
  if (stage == 1)
    k_imex_stage<1><<<blocks_for(nI, 64), 64, 0, st>>>(g, cons, aux_guess, u1, flux1, source1,
                                                        out, dt, w);
  else
    k_imex_stage<2><<<blocks_for(nI, 64), 64, 0, st>>>(g, cons, aux_guess, u1, flux1, source1,
                                                        out, dt, w);
  return cudaGetLastError();
}

cudaError_t launch_imex_stage_queued(const Grid& g, int stage, const double* cons,
                                     const double* aux_guess, const double* u1,
                                     const double* flux1, const double* source1, double* out,
                                     double dt, C2PWork w, cudaStream_t st) {
  if (stage == 1)
    k_imex_stage_queued<1><<<148, 64, 0, st>>>(g, cons, aux_guess, u1, flux1, source1, out, dt, w);
  else
    k_imex_stage_queued<2><<<148, 64, 0, st>>>(g, cons, aux_guess, u1, flux1, source1, out, dt, w);
  k_reset_count<<<1, 1, 0, st>>>(w.fail_count);
  return cudaGetLastError();
}

cudaError_t launch_imex_sweep(const Grid& g, int form, const double* cons, const double* zaux,
                              const double* u1, const double* u2, const double* flux1,
                              const double* flux2, const double* source1, const double* source2,
                              double* out, double* zout, double dt, C2PWork w, cudaStream_t st) {
  const long long nI = n_interior_host(g);
  const int b = blocks_for(nI, 64);
#define SWEEP(F, X)                                                                        \
  k_imex_sweep<F, X><<<b, 64, 0, st>>>(g, cons, zaux, u1, u2, flux1, flux2, source1, source2, \
                                       out, zout, dt, w)
  switch (form) {
    case 1: SWEEP(1, 0); break;  // SSP3 stage 1
    case 2: SWEEP(2, 1); break;  // SSP3 stage 2
    case 3: SWEEP(3, 2); break;  // SSP3 stage 3
    case 4: SWEEP(4, 0); break;  // SSP2322 stage 1
    case 5: SWEEP(5, 0); break;  // SSP2322 stage 2
    case 6: SWEEP(6, 3); break;  // SSP2322 stage 3
    default: return cudaErrorInvalidValue;
  }
#undef SWEEP
  return cudaGetLastError();
}

cudaError_t launch_imex_sweep_queued(const Grid& g, int form, const double* cons,
                                     const double* zaux, const double* u1, const double* u2,
                                     const double* flux1, const double* flux2,
                                     const double* source1, const double* source2, double* out,
                                     double* zout, double dt, C2PWork w, cudaStream_t st) {
#define QSWEEP(F, X)                                                                     \
  k_imex_sweep_queued<F, X><<<148, 64, 0, st>>>(g, cons, zaux, u1, u2, flux1, flux2, source1, \
                                                source2, out, zout, dt, w)
  switch (form) {
    case 1: QSWEEP(1, 0); break;
    case 2: QSWEEP(2, 1); break;
    case 3: QSWEEP(3, 2); break;
    case 4: QSWEEP(4, 0); break;
    case 5: QSWEEP(5, 0); break;
    case 6: QSWEEP(6, 3); break;
    default: return cudaErrorInvalidValue;
  }
#undef QSWEEP
  k_reset_count<<<1, 1, 0, st>>>(w.fail_count);
  return cudaGetLastError();
}

cudaError_t ens_imex_queued(const Member* mem, int n_members, int stage, cudaStream_t st) {
  if (stage == 1)
    k_ens_imex_queued<1><<<n_members, 64, 0, st>>>(mem);
  else
    k_ens_imex_queued<2><<<n_members, 64, 0, st>>>(mem);
  return cudaGetLastError();
}

}  // namespace mth
