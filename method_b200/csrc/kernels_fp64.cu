// Plain FP64 kernels.  This translation unit is compiled with -fmad=false
// (and IEEE division / square root, the nvcc defaults) so that every
// expression rounds exactly like the reference's x86-64 build, which has no
// FMA contraction at the default -march.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "ensemble.h"
#include "fvs2d.cuh"
#include "fvs2d_group.cuh"
#include "hybrid.cuh"
#include "launch.h"
#include "minpack.cuh"
#include "srmhd.cuh"
#include "srrmhd.cuh"

namespace mth {

namespace {

constexpr int kThreads = 256;

inline int blocks_for(long long n, int t = kThreads) { return (int)((n + t - 1) / t); }

// ---------------------------------------------------------------------------
// primsToAll over every cell (srmhd.cc:573-673, srrmhd.cc:358-510).
__global__ void k_prims_to_all_srmhd(Grid g, const double* __restrict__ prims,
                                     double* __restrict__ cons, double* __restrict__ aux) {
  long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (cell >= g.Ntot) return;
  const long long N = g.Ntot;
  double p[8], c[9], a[13];
#pragma unroll
  for (int v = 0; v < 8; ++v) p[v] = prims[v * N + cell];
  srmhd::prims_to_all(p, g.gamma, c, a);
#pragma unroll
  for (int v = 0; v < 9; ++v) cons[v * N + cell] = c[v];
#pragma unroll
  for (int v = 0; v < 13; ++v) aux[v * N + cell] = a[v];
}

// ---------------------------------------------------------------------------
// Boundary conditions: every ghost cell receives the interior value it maps
// to.  Sources are always interior cells, so one pass is race free.  Threads
// are ghost cells (first the x slabs, then the y slabs of the interior rows,
// then the z slabs of the interior columns) times groups of four variables,
// whose loads are in flight together.  A thread per cell of the array with a
// loop over its variables spent its time on cells that are no ghosts and on
// one load's latency per variable: the 30 variables of 1024^2, three launches,
// 31 -> 15 us, of 64^3 32 -> 19 us.  T: a type that holds the ghosts' number.
constexpr int kBcsVars = 4;
inline long long n_ghosts(const Grid& g) { return g.Ntot - n_interior_host(g); }

template <typename T>
__global__ void k_apply_bcs(Grid g, double* __restrict__ arr, int nvars, T n) {
  T t = blockIdx.x * (T)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const T Ny = g.Ny, Nz = g.Nz, mx = g.ie - g.is, my = g.je - g.js, mz = g.ke - g.ks;
  const T gy = Ny - my, gz = Nz - mz, nx = (g.Nx - mx) * Ny * Nz, ny = mx * gy * Nz;
  T i, j, k;
  if (t < nx) {
    k = t % Nz;
    t /= Nz;
    j = t % Ny;
    i = t / Ny;
    if (i >= (T)g.is) i += mx;
  } else if (t < nx + ny) {
    t -= nx;
    k = t % Nz;
    t /= Nz;
    j = t % gy;
    i = g.is + t / gy;
    if (j >= (T)g.js) j += my;
  } else {
    t -= nx + ny;
    k = t % gz;
    t /= gz;
    j = g.js + t % my;
    i = g.is + t / my;
    if (k >= (T)g.ks) k += mz;
  }
  const int v0 = blockIdx.y * kBcsVars;
  const double* src = arr + v0 * g.Ntot + mapped_cell(g, (int)i, (int)j, (int)k);
  double* dst = arr + v0 * g.Ntot + cell_id(g, (int)i, (int)j, (int)k);
  double x[kBcsVars];
#pragma unroll
  for (int v = 0; v < kBcsVars; ++v)
    if (v0 + v < nvars) x[v] = src[v * g.Ntot];
#pragma unroll
  for (int v = 0; v < kBcsVars; ++v)
    if (v0 + v < nvars) dst[v * g.Ntot] = x[v];
}

// ---------------------------------------------------------------------------
// Generic flux path, one direction at a time, on materialised ghosts.  Mirrors
// FVS::fluxReconstruction and FVS::F (fluxVectorSplitting.cc:4-131).
// Only the rows through the interior are split and reconstructed (a cell whose
// other two indices are ghosts reaches no interior cell's flux difference): at
// 64^3 79% of the cells and 71% of the faces.  With the boundary conditions
// above, an RK2 WENO5 step and its ghost fill at 64^3 0.98 -> 0.87 ms, 16^3 199 -> 138 us.
__device__ __forceinline__ bool row_interior(const Grid& g, int dir, int i, int j, int k) {
  return (dir == 0 || (i >= g.is && i < g.ie)) && (dir == 1 || (j >= g.js && j < g.je)) &&
         (dir == 2 || (k >= g.ks && k < g.ke));
}

// Flux vector and Lax-Friedrichs split of one direction over those cells.
template <class M>
__global__ void k_split_dir_full(Grid g, const double* __restrict__ cons,
                                 const double* __restrict__ prims,
                                 const double* __restrict__ aux, int dir,
                                 double* __restrict__ fplus, double* __restrict__ fminus) {
  long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (cell >= g.Ntot) return;
  const long long ij = cell / g.Nz;
  if (!row_interior(g, dir, (int)(ij / g.Ny), (int)(ij % g.Ny), (int)(cell % g.Nz))) return;
  double c[M::NC], p[M::NP], a[M::NA], f[M::NC];
  M::template load_flux_inputs<double>(cons, prims, aux, g.Ntot, cell, c, p, a);
  M::template flux<double>(c, p, a, dir, f);
#pragma unroll
  for (int v = 0; v < M::NC; ++v) {
    fplus[v * g.Ntot + cell] = 0.5 * (f[v] + 1.0 * c[v]);
    fminus[v * g.Ntot + cell] = 0.5 * (f[v] - 1.0 * c[v]);
  }
}

// ALL: every cell, zero outside [shift, N - shift), as the reference's arrays
// hold; else the faces of the interior cells alone.  blockIdx.y takes its share
// of the variables.
template <int ORDER, bool ALL>
__global__ void k_weno_dir(Grid g, int nc, int dir, const double* __restrict__ fplus,
                           const double* __restrict__ fminus, double* __restrict__ frecon) {
  long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (cell >= g.Ntot) return;
  int k = (int)(cell % g.Nz);
  long long t = cell / g.Nz;
  int j = (int)(t % g.Ny);
  int i = (int)(t / g.Ny);
  constexpr int shift = (ORDER + 1) / 2;
  int idx = dir == 0 ? i : (dir == 1 ? j : k);
  int n = dir == 0 ? g.Nx : (dir == 1 ? g.Ny : g.Nz);
  long long stride = dir == 0 ? (long long)g.Ny * g.Nz : (dir == 1 ? g.Nz : 1);
  const bool inside = idx >= shift && idx < n - shift;
  if (!ALL) {
    const int lo = dir == 0 ? g.is : (dir == 1 ? g.js : g.ks);
    const int hi = dir == 0 ? g.ie : (dir == 1 ? g.je : g.ke);
    if (idx < lo || idx > hi || !row_interior(g, dir, i, j, k)) return;
  }
  const int per = (nc + gridDim.y - 1) / gridDim.y;
  for (int v = blockIdx.y * per; v < min(nc, (int)(blockIdx.y + 1) * per); ++v) {
    double r = 0.0;  // the reference zero-initialises its reconstruction arrays
    if (inside) {
      const double* P = fplus + v * g.Ntot + cell;
      const double* Mm = fminus + v * g.Ntot + cell;
      if constexpr (ORDER <= 5) {
        r = weno_face_exact<ORDER, true>(P - shift * stride, Mm + (shift - 1) * stride, stride);
      } else {
        // upwind i-shift .. i-shift+order-1, downwind i+shift-1 .. i+shift-order
        const int s = (int)stride;
        const double up = weno_point<ORDER, double>(P - shift * stride, s);
        const double dn = weno_point<ORDER, double>(Mm + (shift - 1) * stride, -s);
        r = up + dn;
      }
    } else {
      r = 0.0 + 0.0;
    }
    frecon[v * g.Ntot + cell] = r;
  }
}

// k_weno_dir for a runtime order.  Grids of fewer than two blocks per SM split
// the variables over blocks, too: their threads wait for one reconstruction
// after the other otherwise.
template <bool ALL>
void weno_dir_launch(const Grid& g, int nc, int order, int dir, const double* fplus,
                     const double* fminus, double* frecon, cudaStream_t st) {
  const int b = blocks_for(g.Ntot);
  const dim3 n(b, b < 2 * device_sm_count() ? nc : 1);
  switch (order) {
    case 3: k_weno_dir<3, ALL><<<n, kThreads, 0, st>>>(g, nc, dir, fplus, fminus, frecon); break;
    case 5: k_weno_dir<5, ALL><<<n, kThreads, 0, st>>>(g, nc, dir, fplus, fminus, frecon); break;
    case 7: k_weno_dir<7, ALL><<<n, kThreads, 0, st>>>(g, nc, dir, fplus, fminus, frecon); break;
    case 9: k_weno_dir<9, ALL><<<n, kThreads, 0, st>>>(g, nc, dir, fplus, fminus, frecon); break;
    default: k_weno_dir<11, ALL><<<n, kThreads, 0, st>>>(g, nc, dir, fplus, fminus, frecon); break;
  }
}

__global__ void k_fnet_dir(Grid g, int nc, int dir, int first, const double* __restrict__ frecon,
                           double* __restrict__ fnet) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n_interior(g)) return;
  int i, j, k;
  interior_ijk(g, t, i, j, k);
  const long long cell = cell_id(g, i, j, k);
  const long long nb = dir == 0 ? cell_id(g, i + 1, j, k)
                                : (dir == 1 ? cell_id(g, i, j + 1, k) : cell_id(g, i, j, k + 1));
  const double d = dir == 0 ? g.dx : (dir == 1 ? g.dy : g.dz);
  for (int v = 0; v < nc; ++v) {
    const double* F = frecon + v * g.Ntot;
    double val = F[nb] / d - F[cell] / d;
    fnet[v * g.Ntot + cell] = first ? val : fnet[v * g.Ntot + cell] + val;
  }
}

__global__ void k_stage_update(Grid g, int nc, int mode, const double* u0,
                               const double* in, const double* __restrict__ fnet, double dt,
                               double* out) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n_interior(g)) return;
  int i, j, k;
  interior_ijk(g, t, i, j, k);
  const long long cell = cell_id(g, i, j, k);
  for (int v = 0; v < nc; ++v) {
    const long long o = v * g.Ntot + cell;
    if (mode == STAGE_EULER) out[o] = in[o] - dt * fnet[o];
    else if (mode == STAGE_RK2_CORR) out[o] = 0.5 * (u0[o] + in[o] - dt * fnet[o]);
    else out[o] = fnet[o];
  }
}

// ---------------------------------------------------------------------------
// SRMHD primitive recovery (srmhd.cc:390-562): one Powell-hybrid solve per
// interior cell from the previous state's guess; cells that fail are queued
// for the neighbour-average retry.
constexpr double kSrmhdTol = 1.49011612e-7;

// One interior cell: returns the residual evaluations; a failure is queued.
__device__ __forceinline__ long long c2p_srmhd_hybrd_cell(const Grid& g, long long cell,
                                                          const double* __restrict__ cons,
                                                          const double* prims_guess,
                                                          const double* aux_guess,
                                                          double* prims, double* aux,
                                                          double* __restrict__ solution,
                                                          int* fail_list, int* fail_count) {
  const long long N = g.Ntot;
  double c[9];
#pragma unroll
  for (int v = 0; v < 9; ++v) c[v] = cons[v * N + cell];
  double pg[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) pg[v] = prims_guess[v * N + cell];
  double hg = aux_guess[cell];
  srmhd::Residual R = srmhd::residual_args(c, g.gamma);
  double x[2], fv[2];
  srmhd::guess_from_prims(pg, hg, x);
  HybrdResult res = Hybrd<2>::solve(R, x, fv, kSrmhdTol);
  if (res.info == 1) {
    solution[cell] = x[0];
    solution[N + cell] = x[1];
    double p[8], a[13];
    srmhd::from_solution(c, x, g.gamma, R.BS, R.Bsq, R.Ssq, p, a);
#pragma unroll
    for (int v = 0; v < 8; ++v) prims[v * N + cell] = p[v];
#pragma unroll
    for (int v = 0; v < 13; ++v) aux[v * N + cell] = a[v];
  } else {
    prims[5 * N + cell] = c[5];
    prims[6 * N + cell] = c[6];
    prims[7 * N + cell] = c[7];
    aux[10 * N + cell] = R.BS;
    aux[11 * N + cell] = R.Bsq;
    aux[12 * N + cell] = R.Ssq;
    int slot = atomicAdd(fail_count, 1);
    fail_list[slot] = (int)cell;
  }
  return res.nfev;
}

// Registers capped at 96 (5 resident CTAs of 128 threads).  Large grids do not
// care (OT 1024^2 RK2 step 1.514 ms at 64, 1.512 at 96, 1.520 at 128
// registers: more warps against fewer spills); small ones, whose few warps
// wait on their own spills, do (KH 64 x 128 step 77.3, 75.2, 73.7 us; 64^3
// step 0.997, 0.983, 0.988 ms).  Register allocation changes no result.
__global__ void __launch_bounds__(128, 5)
    k_c2p_srmhd(Grid g, const double* __restrict__ cons, const double* prims_guess,
                const double* aux_guess, double* prims, double* aux,
                double* __restrict__ solution, C2PWork w) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long nfev = 0;
  if (t < n_interior(g)) {
    int i, j, k;
    interior_ijk(g, t, i, j, k);
    nfev = c2p_srmhd_hybrd_cell(g, cell_id(g, i, j, k), cons, prims_guess, aux_guess, prims, aux,
                                solution, w.fail_list, w.fail_count);
  }
  // one atomic per warp for the statistics
  unsigned mask = __ballot_sync(0xffffffffu, t < n_interior(g));
  for (int o = 16; o > 0; o >>= 1) nfev += __shfl_down_sync(0xffffffffu, nfev, o);
  if ((threadIdx.x & 31) == 0 && mask) {
    atomicAdd((unsigned long long*)&w.counters[0], (unsigned long long)__popc(mask));
    atomicAdd((unsigned long long*)&w.counters[1], (unsigned long long)nfev);
  }
}

// Neighbour-average retry of failed cells (srmhd.cc:458-507), processed one
// at a time in (i, j, k) order as the reference does.  The reference solves
// the retry with the residual arguments left over from the last interior cell
// of the first pass; that behaviour is kept so that results stay identical.
__device__ void c2p_retry_body(const Grid& g, const double* __restrict__ cons, double* prims,
                               double* aux, double* solution, int* fail_list, int* fail_count,
                               long long* counters) {
  const int n = *fail_count;
  if (n == 0) return;
  int* L = fail_list;
  // heap sort of the failed cell ids (ascending = the reference's loop order)
  for (int s = n / 2 - 1; s >= 0; --s) {
    for (int r = s;;) {
      int ch = 2 * r + 1;
      if (ch >= n) break;
      if (ch + 1 < n && L[ch + 1] > L[ch]) ++ch;
      if (L[r] >= L[ch]) break;
      int tmp = L[r]; L[r] = L[ch]; L[ch] = tmp;
      r = ch;
    }
  }
  for (int end = n - 1; end > 0; --end) {
    int tmp = L[0]; L[0] = L[end]; L[end] = tmp;
    for (int r = 0;;) {
      int ch = 2 * r + 1;
      if (ch >= end) break;
      if (ch + 1 < end && L[ch + 1] > L[ch]) ++ch;
      if (L[r] >= L[ch]) break;
      int t2 = L[r]; L[r] = L[ch]; L[ch] = t2;
      r = ch;
    }
  }
  const long long N = g.Ntot;
  double cl[9];
  const long long last = cell_id(g, g.ie - 1, g.je - 1, g.ke - 1);
  for (int v = 0; v < 9; ++v) cl[v] = cons[v * N + last];
  srmhd::Residual R = srmhd::residual_args(cl, g.gamma);
  long long still = 0, nfev = 0;
  for (int f = 0; f < n; ++f) {
    const long long cell = L[f];
    const int z = (int)(cell % g.Nz);
    const int y = (int)((cell / g.Nz) % g.Ny);
    const int x = (int)(cell / ((long long)g.Nz * g.Ny));
    long long nb[6];
    int cnt = 0;
    if (x > 0) nb[cnt++] = cell_id(g, x - 1, y, z);
    if (y > 0) nb[cnt++] = cell_id(g, x, y - 1, z);
    if (z > 0) nb[cnt++] = cell_id(g, x, y, z - 1);
    if (x < g.Nx - 1) nb[cnt++] = cell_id(g, x + 1, y, z);
    if (y < g.Ny - 1) nb[cnt++] = cell_id(g, x, y + 1, z);
    if (z < g.Nz - 1) nb[cnt++] = cell_id(g, x, y, z + 1);
    double s[2] = {0, 0};
    for (int q = 0; q < cnt; ++q) {
      s[0] += solution[nb[q]];
      s[1] += solution[N + nb[q]];
    }
    s[0] /= (double)cnt;
    s[1] /= (double)cnt;
    double fv[2];
    HybrdResult res = Hybrd<2>::solve(R, s, fv, kSrmhdTol);
    nfev += res.nfev;
    if (res.info != 1) ++still;
    solution[cell] = s[0];
    solution[N + cell] = s[1];
    double c[9];
    for (int v = 0; v < 9; ++v) c[v] = cons[v * N + cell];
    double p[8], a[13];
    srmhd::from_solution(c, s, g.gamma, aux[10 * N + cell], aux[11 * N + cell],
                         aux[12 * N + cell], p, a);
    for (int v = 0; v < 8; ++v) prims[v * N + cell] = p[v];
    for (int v = 0; v < 13; ++v) aux[v * N + cell] = a[v];
  }
  counters[1] += nfev;
  counters[2] += still;
  *fail_count = 0;
}

__global__ void k_c2p_retry_srmhd(Grid g, const double* __restrict__ cons, double* prims,
                                  double* aux, double* solution, C2PWork w) {
  if (threadIdx.x != 0) return;
  c2p_retry_body(g, cons, prims, aux, solution, w.fail_list, w.fail_count, w.counters);
}

// RKSplit source step: target += dt * S(cons) on the interior (rkSplit.cc:31-53).
template <int MODEL>
__global__ void k_source_add(Grid g, const double* __restrict__ cons,
                             const double* __restrict__ prims, const double* __restrict__ aux,
                             double* target, double dt) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n_interior(g)) return;
  int i, j, k;
  interior_ijk(g, t, i, j, k);
  const long long N = g.Ntot, cell = cell_id(g, i, j, k);
  if (MODEL == MODEL_SRMHD) {
    double c[9], s[9];
#pragma unroll
    for (int v = 0; v < 9; ++v) c[v] = cons[v * N + cell];
    srmhd::source(c, g.cp, s);
#pragma unroll
    for (int v = 0; v < 9; ++v) target[v * N + cell] = target[v * N + cell] + dt * s[v];
  } else {
    double c[14], a[17], s[14];
#pragma unroll
    for (int v = 0; v < 14; ++v) c[v] = cons[v * N + cell];
#pragma unroll
    for (int v = 0; v < 17; ++v) a[v] = aux[v * N + cell];
    srrmhd::source(c, a, g.cp, s);
#pragma unroll
    for (int v = 0; v < 14; ++v) target[v * N + cell] = target[v * N + cell] + dt * s[v];
  }
}

// ---------------------------------------------------------------------------
// SRRMHD primsToAll with the 4th-order central-difference charge density
// (srrmhd.cc:358-510); the stencil reads the input primitives of neighbours.
__global__ void k_prims_to_all_srrmhd(Grid g, const double* __restrict__ prims,
                                      double* __restrict__ cons, double* __restrict__ aux) {
  long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (cell >= g.Ntot) return;
  const long long N = g.Ntot;
  const int k = (int)(cell % g.Nz);
  const int j = (int)((cell / g.Nz) % g.Ny);
  const int i = (int)(cell / ((long long)g.Nz * g.Ny));
  double p[11], c[14], a[17];
#pragma unroll
  for (int v = 0; v < 11; ++v) p[v] = prims[v * N + cell];
  auto P = [&](int v, int ii, int jj, int kk) { return prims[v * N + cell_id(g, ii, jj, kk)]; };
  bool qfd = true;
  double divE = 0.0;
  if (i > 1 && j > 1 && k > 1 && i < g.Nx - 2 && j < g.Ny - 2 && k < g.Nz - 2) {
    divE = (-P(8, i + 2, j, k) + 8 * P(8, i + 1, j, k) - 8 * P(8, i - 1, j, k) + P(8, i - 2, j, k)) /
               (12 * g.dx) +
           (-P(9, i, j + 2, k) + 8 * P(9, i, j + 1, k) - 8 * P(9, i, j - 1, k) + P(9, i, j - 2, k)) /
               (12 * g.dy) +
           (-P(10, i, j, k + 2) + 8 * P(10, i, j, k + 1) - 8 * P(10, i, j, k - 1) +
            P(10, i, j, k - 2)) /
               (12 * g.dz);
  } else if (i > 1 && j > 1 && i < g.Nx - 2 && j < g.Ny - 2 && g.nz == 0) {
    divE = (-P(8, i + 2, j, k) + 8 * P(8, i + 1, j, k) - 8 * P(8, i - 1, j, k) + P(8, i - 2, j, k)) /
               (12 * g.dx) +
           (-P(9, i, j + 2, k) + 8 * P(9, i, j + 1, k) - 8 * P(9, i, j - 1, k) + P(9, i, j - 2, k)) /
               (12 * g.dy);
  } else if (i > 1 && i < g.Nx - 2 && g.ny == 0) {
    divE = (-P(8, i + 2, j, k) + 8 * P(8, i + 1, j, k) - 8 * P(8, i - 1, j, k) + P(8, i - 2, j, k)) /
           (12 * g.dx);
  } else {
    qfd = false;
  }
  srrmhd::prims_to_all(p, g.gamma, g.sigma, g.sigma_exp, g.functional_sigma, qfd, divE, c, a);
#pragma unroll
  for (int v = 0; v < 14; ++v) cons[v * N + cell] = c[v];
#pragma unroll
  for (int v = 0; v < 17; ++v) aux[v * N + cell] = a[v];
}

// SRRMHD grid primitive recovery (srrmhd.cc:314-356): secant on Z per
// interior cell, seeded from the guess array's aux[10].
__global__ void __launch_bounds__(128)
    k_c2p_srrmhd(Grid g, const double* __restrict__ cons, const double* aux_guess, double* prims,
                 double* aux, C2PWork w) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long evals = 0;
  if (t < n_interior(g)) {
    int i, j, k;
    interior_ijk(g, t, i, j, k);
    const long long N = g.Ntot, cell = cell_id(g, i, j, k);
    double c[14], p[11], a[17];
#pragma unroll
    for (int v = 0; v < 14; ++v) c[v] = cons[v * N + cell];
    a[10] = aux_guess[10 * N + cell];
    int ev = 0;
    bool ok = srrmhd::c2p_cell(c, g.gamma, sigma_of(g, c[0]), p, a, ev);
    evals = ev;
    if (ok) {
#pragma unroll
      for (int v = 0; v < 11; ++v) prims[v * N + cell] = p[v];
#pragma unroll
      for (int v = 0; v < 17; ++v) aux[v * N + cell] = a[v];
    } else {
      atomicAdd((unsigned long long*)&w.counters[2], 1ull);
      atomicOr((unsigned long long*)&w.counters[3], (unsigned long long)ERR_C2P);
    }
  }
  unsigned mask = __ballot_sync(0xffffffffu, t < n_interior(g));
  for (int o = 16; o > 0; o >>= 1) evals += __shfl_down_sync(0xffffffffu, evals, o);
  if ((threadIdx.x & 31) == 0 && mask) {
    atomicAdd((unsigned long long*)&w.counters[0], (unsigned long long)__popc(mask));
    atomicAdd((unsigned long long*)&w.counters[1], (unsigned long long)evals);
  }
}

// Model::sourceTerm into an array, over the interior (ALL = false) or every
// cell (ALL = true, the reference's sourceTerm loops, srmhd.cc:226-250).
template <int MODEL, bool ALL>
__global__ void k_source(Grid g, const double* __restrict__ cons, const double* __restrict__ aux,
                         double* __restrict__ out) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long cell;
  if (ALL) {
    if (t >= g.Ntot) return;
    cell = t;
  } else {
    if (t >= n_interior(g)) return;
    int i, j, k;
    interior_ijk(g, t, i, j, k);
    cell = cell_id(g, i, j, k);
  }
  const long long N = g.Ntot;
  if (MODEL == MODEL_SRMHD) {
    double c[9], s[9];
#pragma unroll
    for (int v = 0; v < 9; ++v) c[v] = cons[v * N + cell];
    srmhd::source(c, g.cp, s);
#pragma unroll
    for (int v = 0; v < 9; ++v) out[v * N + cell] = s[v];
  } else {
    double c[14], a[17], s[14];
#pragma unroll
    for (int v = 0; v < 14; ++v) c[v] = cons[v * N + cell];
#pragma unroll
    for (int v = 0; v < 17; ++v) a[v] = aux[v * N + cell];
    srrmhd::source(c, a, g.cp, s);
#pragma unroll
    for (int v = 0; v < 14; ++v) out[v * N + cell] = s[v];
  }
}

// SSP3(332) combination (SSP3.cc:204-214).
__global__ void k_ssp3_combine(Grid g, double* cons, const double* __restrict__ f1,
                               const double* __restrict__ f2, const double* __restrict__ f3,
                               const double* __restrict__ s1, const double* __restrict__ s2,
                               const double* __restrict__ s3, double dt) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n_interior(g)) return;
  int i, j, k;
  interior_ijk(g, t, i, j, k);
  const long long cell = cell_id(g, i, j, k);
  for (int v = 0; v < 14; ++v) {
    const long long o = v * g.Ntot + cell;
    cons[o] = cons[o] - dt * (f1[o] + f2[o] + 4 * f3[o]) / 6.0 +
              dt * (s1[o] + s2[o] + 4 * s3[o]) / 6.0;
  }
}

// SSP2(322) combination (SSP2322.cc:224-234).
__global__ void k_ssp2322_combine(Grid g, double* cons, const double* __restrict__ f2,
                                  const double* __restrict__ f3, const double* __restrict__ s2,
                                  const double* __restrict__ s3, double dt) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n_interior(g)) return;
  int i, j, k;
  interior_ijk(g, t, i, j, k);
  const long long cell = cell_id(g, i, j, k);
  for (int v = 0; v < 14; ++v) {
    const long long o = v * g.Ntot + cell;
    cons[o] = cons[o] - dt * 0.5 * (f2[o] + f3[o] - s2[o] - s3[o]);
  }
}

// SSP2 combination U += -0.5 dt (flux1 + flux2 - source1 - source2)
// (SSP2.cc:155-166).
__global__ void k_ssp2_combine(Grid g, int nc, double* cons, const double* __restrict__ flux1,
                               const double* __restrict__ flux2,
                               const double* __restrict__ source1,
                               const double* __restrict__ source2, double dt) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n_interior(g)) return;
  int i, j, k;
  interior_ijk(g, t, i, j, k);
  const long long cell = cell_id(g, i, j, k);
  for (int v = 0; v < nc; ++v) {
    const long long o = v * g.Ntot + cell;
    // as in imex_cell, of stage 1's source only these planes count
    const double s1 = SRRMHD::sourced(v) ? source1[o] : 0.0;
    cons[o] += -0.5 * dt * (flux1[o] + flux2[o] - s1 - source2[o]);
  }
}

// Model::fluxVector over every cell (srmhd.cc:72-206, srrmhd.cc:65-192).
template <class M>
__global__ void k_flux_vector(Grid g, const double* __restrict__ cons,
                              const double* __restrict__ prims, const double* __restrict__ aux,
                              int dir, double* __restrict__ f) {
  long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (cell >= g.Ntot) return;
  double c[M::NC], p[M::NP], a[M::NA], fv[M::NC];
  M::template load_flux_inputs<double>(cons, prims, aux, g.Ntot, cell, c, p, a);
  M::template flux<double>(c, p, a, dir, fv);
#pragma unroll
  for (int v = 0; v < M::NC; ++v) f[v * g.Ntot + cell] = fv[v];
}

// SRMHD::getPrimitiveVarsSingleCell (srmhd.cc:297-377) on n independent
// cells, variable-major with stride n.
__global__ void __launch_bounds__(128)
    k_c2p_cells_srmhd(long long n, double gamma, double tol, const double* __restrict__ cons,
                      double* prims, double* aux, int* flag) {
  long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= n) return;
  double c[9], pg[4];
#pragma unroll
  for (int v = 0; v < 9; ++v) c[v] = cons[v * n + q];
#pragma unroll
  for (int v = 0; v < 4; ++v) pg[v] = prims[v * n + q];
  srmhd::Residual R = srmhd::residual_args(c, gamma);
  double x[2], fv[2];
  srmhd::guess_from_prims(pg, aux[q], x);
  HybrdResult res = Hybrd<2>::solve(R, x, fv, tol);
  if (res.info != 1) {
    atomicOr(flag, 1);
    return;
  }
  double p[8], a[13];
  srmhd::from_solution(c, x, gamma, R.BS, R.Bsq, R.Ssq, p, a);
#pragma unroll
  for (int v = 0; v < 8; ++v) prims[v * n + q] = p[v];
#pragma unroll
  for (int v = 0; v < 13; ++v) aux[v * n + q] = a[v];
}

// SRRMHD::getPrimitiveVarsSingleCell (srrmhd.cc:256-312) on n cells.
__global__ void __launch_bounds__(128)
    k_c2p_cells_srrmhd(long long n, double gamma, double sigma, const double* __restrict__ cons,
                       double* prims, double* aux, int* flag) {
  long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= n) return;
  double c[14], p[11], a[17];
#pragma unroll
  for (int v = 0; v < 14; ++v) c[v] = cons[v * n + q];
  a[10] = aux[10 * n + q];
  int ev = 0;
  if (!srrmhd::c2p_cell(c, gamma, sigma, p, a, ev)) {
    aux[10 * n + q] = a[10];
    atomicOr(flag, 1);
    return;
  }
#pragma unroll
  for (int v = 0; v < 11; ++v) prims[v * n + q] = p[v];
#pragma unroll
  for (int v = 0; v < 17; ++v) aux[v * n + q] = a[v];
}

// The plain tile runs in passes of kFp64Group variables (fvs2d_group.cuh)
// with registers sized for kFp64Blocks CTAs per SM: WENO3/5 4 CTAs (64
// registers, a few spilled), WENO7 3, WENO9/11 2.  OT 1024^2 WENO5 RK2 step: two
// passes of 5 + 4 variables 1.51 ms (1.53 at 3 CTAs per SM), three of 3 1.55, all
// in one pass 1.67.
// Grids of fewer than two tiles per SM run one CTA per tile and group of
// variables: of one variable while that makes at most four CTAs per SM, else of
// three (five for the Hybrid model, whose flux costs more to evaluate again
// per group; all of SRMHD's with WENO9/11 towards two tiles per SM).  Plain RK2
// steps of Orszag-Tang grids one after another, us, with one variable per CTA,
// three, five, all in one CTA, and in passes:
//   SRMHD WENO5   64 x 128 (32 tiles) 59 63 69 82 91, 200 x 256 (200) 110 107 107 118 124,
//                 256 x 288 (288) 134 122 124 122 127, 512 x 512 (1024) 403 349 359 345 347
//   SRRMHD WENO5  128 x 128 (64) 57 50 54 77 92, 200 x 256 115 89 97 134 129,
//                 256 x 288 153 119 118 141 133
//   Hybrid WENO5  128 x 128 115 108 105 128 155, 200 x 256 193 167 163 193 197,
//                 512 x 512 825 636 581 624 561
//   SRMHD WENO7   128 x 128 97 93 103 137 145, 200 x 256 164 158 146 178 185
//   SRMHD WENO9   240 x 256 (240) 270 218 244 242 249, 280 x 256 (280): three 250, all 245
//   SRMHD WENO11  232 x 256 (232): three 291, all 315; 264 x 256 (264) 340, 320
//   SRRMHD WENO11 128 x 128 199 167 155 263 311, 256 x 288 592 468 458 521 465
// All forms give the same bits.
template <class M>
constexpr int kFp64Group = 5;
template <class M>
constexpr int kFp64SmallGroup = std::is_same<M, HYBRID>::value ? 5 : 3;
// Tiles per SM above which (and below two) SRMHD's WENO9/11, whose wide halo each
// group loads and splits again, run one CTA per tile with all variables.
template <class M, int ORDER>
constexpr double kFp64WholeTile =
    !std::is_same<M, SRMHD>::value ? 0.0 : ORDER == 9 ? 1.75 : ORDER == 11 ? 1.67 : 0.0;
// SRRMHD's WENO7 in groups of three fits 64 registers, 4 CTAs per SM (32 bytes
// spilled): the compiler's choice of 70, 3 CTAs, makes a 200 x 256 step 161 us, not 149.
template <class M, int ORDER, int G>
constexpr int kFp64CtasBlocks =
    std::is_same<M, SRRMHD>::value && G == 3 && ORDER == 7 ? 4 : 0;
template <int ORDER>
constexpr int kFp64Blocks = ORDER <= 5 ? 4 : ORDER <= 7 ? 3 : 2;

template <class M, int ORDER, int TI, int G>
cudaError_t fvs2d_group_ctas(const Grid& g, const double* cons, const double* prims,
                             const double* aux, const double* u0, double* out, double dt, int mode,
                             StageTail tail, dim3 grid, cudaStream_t st) {
  using S = Fvs2dGroupSmem<M, ORDER, TI, G>;
  auto kern = k_fvs2d_group_ctas<M, ORDER, TI, G, kFp64CtasBlocks<M, ORDER, G>>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bytes);
  if (e != cudaSuccess) return e;
  grid.z = S::NG;
  kern<<<grid, dim3(32, TI), S::bytes, st>>>(g, cons, prims, aux, u0, out, dt, mode, tail);
  return cudaGetLastError();
}

template <class M, int ORDER, int TI>
cudaError_t fvs2d_instance(const Grid& g, const double* cons, const double* prims,
                           const double* aux, const double* u0, double* out, double dt, int mode,
                           StageTail tail, cudaStream_t st) {
  dim3 grid((g.je - g.js + 31) / 32, (g.ie - g.is + TI - 1) / TI);
  dim3 block(32, TI);
  const long long tiles = (long long)grid.x * grid.y, sms = device_sm_count();
  if (tiles >= 2 * sms) {
    using S = Fvs2dGroupSmem<M, ORDER, TI, kFp64Group<M>>;
    auto kern = k_fvs2d_group<M, ORDER, TI, kFp64Group<M>, kFp64Blocks<ORDER>>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)S::bytes);
    if (e != cudaSuccess) return e;
    kern<<<grid, block, S::bytes, st>>>(g, cons, prims, aux, u0, out, dt, mode, tail);
    return cudaGetLastError();
  }
  if (tiles * M::NC <= 4LL * sms)
    return fvs2d_group_ctas<M, ORDER, TI, 1>(g, cons, prims, aux, u0, out, dt, mode, tail, grid, st);
  if constexpr (kFp64WholeTile<M, ORDER> > 0) {
    if (tiles > kFp64WholeTile<M, ORDER> * sms)
      return fvs2d_group_ctas<M, ORDER, TI, M::NC>(g, cons, prims, aux, u0, out, dt, mode, tail,
                                                   grid, st);
  }
  return fvs2d_group_ctas<M, ORDER, TI, kFp64SmallGroup<M>>(g, cons, prims, aux, u0, out, dt, mode,
                                                            tail, grid, st);
}

// ---------------------------------------------------------------------------
// Ensemble kernels: CTAs stride over a work list covering every member.
template <class M, int ORDER, int TI>
__global__ void __launch_bounds__(32 * TI)
    k_ens_fvs_fp64(const Member* __restrict__ mem, const Item* __restrict__ items, int n_items,
                   int ic, int ip, int ia, int iu0, int iout, int mode) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const Item w = items[it];
    const Member& d = mem[w.m];
    const Grid g = d.g;
    fvs2d_tile<M, double, ORDER, TI>(g, d.a[ic], d.a[ip], d.a[ia], iu0 >= 0 ? d.a[iu0] : nullptr,
                                     d.a[iout], d.dt, mode, w.a, w.b, smem_raw,
                                     StageTail{d.a[EA_F1], d.a[EA_S1], g.cp});
    __syncthreads();
  }
}

__global__ void __launch_bounds__(128, 8)
    k_ens_c2p_srmhd_hybrd(const Member* __restrict__ mem, const Item* __restrict__ items,
                          int n_items, int ic, int ipg, int iag, int ip, int ia) {
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const Item w = items[it];
    const Member& d = mem[w.m];
    const Grid g = d.g;
    const long long t = w.a + threadIdx.x;
    long long nfev = 0;
    if (t < n_interior(g)) {
      int i, j, k;
      interior_ijk(g, t, i, j, k);
      nfev = c2p_srmhd_hybrd_cell(g, cell_id(g, i, j, k), d.a[ic], d.a[ipg], d.a[iag], d.a[ip],
                                  d.a[ia], d.a[EA_SOL], d.fail_list, d.fail_count);
    }
    const unsigned mask = __ballot_sync(0xffffffffu, t < n_interior(g));
    for (int o = 16; o > 0; o >>= 1) nfev += __shfl_down_sync(0xffffffffu, nfev, o);
    if ((threadIdx.x & 31) == 0 && mask) {
      atomicAdd((unsigned long long*)&d.counters[0], (unsigned long long)__popc(mask));
      atomicAdd((unsigned long long*)&d.counters[1], (unsigned long long)nfev);
    }
  }
}

// One CTA per member: the member's neighbour-average retry.
__global__ void k_ens_c2p_retry(const Member* __restrict__ mem, int ic, int ip, int ia) {
  if (threadIdx.x != 0) return;
  const Member& d = mem[blockIdx.x];
  if (d.model != MODEL_SRMHD) return;
  const Grid g = d.g;
  c2p_retry_body(g, d.a[ic], d.a[ip], d.a[ia], d.a[EA_SOL], d.fail_list, d.fail_count,
                 d.counters);
}

// SRRMHD source of the interior cells of every SRRMHD member (srrmhd.cc:194-206);
// here, without contraction, so that members match k_source bit for bit.
__global__ void __launch_bounds__(128)
    k_ens_source(const Member* __restrict__ mem, const Item* __restrict__ items, int n_items,
                 int ic, int ia, int iout) {
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const Item w = items[it];
    const Member& d = mem[w.m];
    const Grid g = d.g;
    const long long t = w.a + threadIdx.x;
    if (t >= n_interior(g)) continue;
    int i, j, k;
    interior_ijk(g, t, i, j, k);
    const long long N = g.Ntot, cell = cell_id(g, i, j, k);
    double c[14], a[17], s[14];
#pragma unroll
    for (int v = 0; v < 14; ++v) c[v] = d.a[ic][v * N + cell];
#pragma unroll
    for (int v = 0; v < 17; ++v) a[v] = d.a[ia][v * N + cell];
    srrmhd::source(c, a, g.cp, s);
#pragma unroll
    for (int v = 0; v < 14; ++v) d.a[iout][v * N + cell] = s[v];
  }
}

// Simulation::updateTime's dt for every member (simulation.cc:113-124); the
// expression is the host's, compiled without contraction.
__global__ void k_ens_dt(Member* mem, int n) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  Member& d = mem[m];
  const Grid& g = d.g;
  double dtX(d.cfl * g.dx / (1.0 * sqrt((double)g.dims)));
  double dtY(d.cfl * g.dy / (1.0 * sqrt((double)g.dims)));
  double dtZ(d.cfl * g.dz / (1.0 * sqrt((double)g.dims)));
  double dt = (dtX <= dtY && dtX <= dtZ) ? dtX : ((dtY < dtZ) ? dtY : dtZ);
  if (d.iters < 15) dt *= 0.1;
  if (d.iters >= 15 && d.iters < 30) dt *= 0.25;
  if (d.t + dt > d.endTime) dt = d.endTime - d.t;
  d.dt = dt;
}

__global__ void k_ens_advance(Member* mem, int n) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  mem[m].t += mem[m].dt;
  mem[m].iters++;
}

template <class M, int ORDER, int TI>
cudaError_t ens_fvs_fp64_instance(const Member* mem, const Item* items, int n, int ic, int ip,
                                  int ia, int iu0, int iout, int mode, int grid,
                                  cudaStream_t st) {
  using S = Fvs2dSmem<M, double, ORDER, TI>;
  auto kern = k_ens_fvs_fp64<M, ORDER, TI>;
  static int cap = 0;  // resident CTAs of this instance on the device
  if (!cap) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)S::bytes);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0, occ = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 32 * TI, S::bytes);
    cap = std::max(1, occ) * std::max(1, sms);
  }
  grid = std::min(grid, cap);
  kern<<<grid, dim3(32, TI), S::bytes, st>>>(mem, items, n, ic, ip, ia, iu0, iout, mode);
  return cudaGetLastError();
}

}  // namespace

// ---------------------------------------------------------------------------
cudaError_t launch_prims_to_all(const Grid& g, int model, const double* prims, double* cons,
                                double* aux, cudaStream_t st) {
  if (model == MODEL_SRMHD) {
    k_prims_to_all_srmhd<<<blocks_for(g.Ntot), kThreads, 0, st>>>(g, prims, cons, aux);
    return cudaGetLastError();
  }
  return launch_prims_to_all_srrmhd(g, prims, cons, aux, st);
}

cudaError_t launch_apply_bcs(const Grid& g, double* arr, int nvars, cudaStream_t st) {
  const long long n = n_ghosts(g);
  if (n <= 0 || nvars <= 0) return cudaSuccess;
  const dim3 grid(blocks_for(n), (nvars + kBcsVars - 1) / kBcsVars);
  if (n < (1LL << 31))
    k_apply_bcs<unsigned><<<grid, kThreads, 0, st>>>(g, arr, nvars, (unsigned)n);
  else
    k_apply_bcs<long long><<<grid, kThreads, 0, st>>>(g, arr, nvars, n);
  return cudaGetLastError();
}

// The ghost cells of x-rows [r0, r1) only (k_apply_bcs on a row range).
__global__ void k_apply_bcs_rows(Grid g, double* __restrict__ arr, int nvars, int r0, int r1) {
  const long long plane = (long long)g.Ny * g.Nz;
  const long long cell = r0 * plane + blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (cell >= r1 * plane) return;
  const int k = (int)(cell % g.Nz);
  const long long t = cell / g.Nz;
  const int j = (int)(t % g.Ny);
  const int i = (int)(t / g.Ny);
  const bool ghost = (i < g.is || i >= g.ie) || (g.dims > 1 && (j < g.js || j >= g.je)) ||
                     (g.dims > 2 && (k < g.ks || k >= g.ke));
  if (!ghost) return;
  const long long src = mapped_cell(g, i, j, k);
  for (int v = 0; v < nvars; ++v) arr[v * g.Ntot + cell] = arr[v * g.Ntot + src];
}

cudaError_t launch_apply_bcs_rows(const Grid& g, double* arr, int nvars, int r0, int r1,
                                  cudaStream_t st) {
  const long long n = (long long)(r1 - r0) * g.Ny * g.Nz;
  if (n <= 0) return cudaSuccess;
  k_apply_bcs_rows<<<blocks_for(n), kThreads, 0, st>>>(g, arr, nvars, r0, r1);
  return cudaGetLastError();
}

cudaError_t launch_fvs2d_fp64(const Grid& g, int model, int order, const double* cons,
                              const double* prims, const double* aux, const double* u0,
                              double* out, double dt, int mode, cudaStream_t st,
                              StageTail tail) {
#define FVS64(MM, O) return fvs2d_instance<MM, O, 8>(g, cons, prims, aux, u0, out, dt, mode, tail, st)
  if (model == MODEL_SRMHD) {
    switch (order) {
      case 3: FVS64(SRMHD, 3);
      case 5: FVS64(SRMHD, 5);
      case 7: FVS64(SRMHD, 7);
      case 9: FVS64(SRMHD, 9);
      default: FVS64(SRMHD, 11);
    }
  }
  if (model == MODEL_HYBRID) {  // WENO3 / WENO5; higher orders take the generic path
    if (order == 3) FVS64(HYBRID, 3);
    if (order == 5) FVS64(HYBRID, 5);
    return cudaErrorInvalidValue;
  }
  switch (order) {
    case 3: FVS64(SRRMHD, 3);
    case 5: FVS64(SRRMHD, 5);
    case 7: FVS64(SRRMHD, 7);
    case 9: FVS64(SRRMHD, 9);
    default: FVS64(SRRMHD, 11);
  }
#undef FVS64
}

cudaError_t launch_weno_dir(const Grid& g, int nc, int order, int dir, const double* fplus,
                            const double* fminus, double* frecon, cudaStream_t st) {
  weno_dir_launch<true>(g, nc, order, dir, fplus, fminus, frecon, st);
  return cudaGetLastError();
}

cudaError_t launch_fvs_generic(const Grid& g, int model, int order, double* cons, double* prims,
                               double* aux, double* fplus, double* fminus, double* frecon,
                               double* fnet, cudaStream_t st) {
  const int nc = model == MODEL_SRMHD ? 9 : 14;
  const int np = model == MODEL_SRMHD ? 8 : 11;
  const int na = model == MODEL_SRMHD ? 13 : 17;
  cudaError_t e;
  if ((e = launch_apply_bcs(g, cons, nc, st)) != cudaSuccess) return e;
  if ((e = launch_apply_bcs(g, prims, np, st)) != cudaSuccess) return e;
  if ((e = launch_apply_bcs(g, aux, na, st)) != cudaSuccess) return e;
  return launch_fvs_generic_raw(g, model, order, cons, prims, aux, fplus, fminus, frecon, fnet,
                                st);
}

cudaError_t launch_fvs_generic_raw(const Grid& g, int model, int order, const double* cons,
                                   const double* prims, const double* aux, double* fplus,
                                   double* fminus, double* frecon, double* fnet,
                                   cudaStream_t st) {
  const int nc = model == MODEL_SRMHD ? 9 : 14;
  const long long nI = (long long)(g.ie - g.is) * (g.je - g.js) * (g.ke - g.ks);
  for (int dir = 0; dir < g.dims; ++dir) {
    if (model == MODEL_SRMHD) {
      k_split_dir_full<SRMHD><<<blocks_for(g.Ntot), kThreads, 0, st>>>(g, cons, prims, aux, dir,
                                                                        fplus, fminus);
    } else if (model == MODEL_HYBRID) {
      cudaError_t e = launch_hybrid_split(g, cons, prims, aux, dir, fplus, fminus, st);
      if (e != cudaSuccess) return e;
    } else {
      k_split_dir_full<SRRMHD><<<blocks_for(g.Ntot), kThreads, 0, st>>>(g, cons, prims, aux,
                                                                         dir, fplus, fminus);
    }
    weno_dir_launch<false>(g, nc, order, dir, fplus, fminus, frecon, st);
    k_fnet_dir<<<blocks_for(nI), kThreads, 0, st>>>(g, nc, dir, dir == 0, frecon, fnet);
  }
  return cudaGetLastError();
}

cudaError_t launch_stage_update(const Grid& g, int nc, int mode, const double* u0,
                                const double* in, const double* fnet, double dt, double* out,
                                cudaStream_t st) {
  const long long nI = (long long)(g.ie - g.is) * (g.je - g.js) * (g.ke - g.ks);
  k_stage_update<<<blocks_for(nI), kThreads, 0, st>>>(g, nc, mode, u0, in, fnet, dt, out);
  return cudaGetLastError();
}

cudaError_t launch_c2p_srmhd(const Grid& g, const double* cons, const double* prims_guess,
                             const double* aux_guess, double* prims, double* aux,
                             double* solution, C2PWork w, cudaStream_t st) {
  const long long nI = (long long)(g.ie - g.is) * (g.je - g.js) * (g.ke - g.ks);
  k_c2p_srmhd<<<blocks_for(nI, 128), 128, 0, st>>>(g, cons, prims_guess, aux_guess, prims, aux,
                                                    solution, w);
  k_c2p_retry_srmhd<<<1, 32, 0, st>>>(g, cons, prims, aux, solution, w);
  return cudaGetLastError();
}

cudaError_t launch_prims_to_all_srrmhd(const Grid& g, const double* prims, double* cons,
                                       double* aux, cudaStream_t st) {
  k_prims_to_all_srrmhd<<<blocks_for(g.Ntot), kThreads, 0, st>>>(g, prims, cons, aux);
  return cudaGetLastError();
}

cudaError_t launch_c2p_srrmhd(const Grid& g, const double* cons, const double* aux_guess,
                              double* prims, double* aux, C2PWork w, cudaStream_t st) {
  const long long nI = (long long)(g.ie - g.is) * (g.je - g.js) * (g.ke - g.ks);
  k_c2p_srrmhd<<<blocks_for(nI, 128), 128, 0, st>>>(g, cons, aux_guess, prims, aux, w);
  return cudaGetLastError();
}

cudaError_t launch_source(const Grid& g, int model, const double* cons, const double* aux,
                          double* out, cudaStream_t st, bool all_cells) {
  const long long nI = (long long)(g.ie - g.is) * (g.je - g.js) * (g.ke - g.ks);
  if (all_cells) {
    if (model == MODEL_SRMHD)
      k_source<MODEL_SRMHD, true><<<blocks_for(g.Ntot), kThreads, 0, st>>>(g, cons, aux, out);
    else
      k_source<MODEL_SRRMHD, true><<<blocks_for(g.Ntot), kThreads, 0, st>>>(g, cons, aux, out);
  } else if (model == MODEL_SRMHD) {
    k_source<MODEL_SRMHD, false><<<blocks_for(nI), kThreads, 0, st>>>(g, cons, aux, out);
  } else {
    k_source<MODEL_SRRMHD, false><<<blocks_for(nI), kThreads, 0, st>>>(g, cons, aux, out);
  }
  return cudaGetLastError();
}

cudaError_t launch_flux_vector(const Grid& g, int model, const double* cons, const double* prims,
                               const double* aux, int dir, double* f, cudaStream_t st) {
  if (model == MODEL_SRMHD)
    k_flux_vector<SRMHD><<<blocks_for(g.Ntot), kThreads, 0, st>>>(g, cons, prims, aux, dir, f);
  else
    k_flux_vector<SRRMHD><<<blocks_for(g.Ntot), kThreads, 0, st>>>(g, cons, prims, aux, dir, f);
  return cudaGetLastError();
}

cudaError_t launch_c2p_cells(int model, double gamma, double sigma, long long n,
                             const double* cons, double* prims, double* aux, double tol,
                             int* flag, cudaStream_t st) {
  if (model == MODEL_SRMHD)
    k_c2p_cells_srmhd<<<blocks_for(n, 128), 128, 0, st>>>(n, gamma, tol, cons, prims, aux, flag);
  else
    k_c2p_cells_srrmhd<<<blocks_for(n, 128), 128, 0, st>>>(n, gamma, sigma, cons, prims, aux,
                                                            flag);
  return cudaGetLastError();
}

cudaError_t launch_ssp3_combine(const Grid& g, double* cons, const double* f1, const double* f2,
                                const double* f3, const double* s1, const double* s2,
                                const double* s3, double dt, cudaStream_t st) {
  k_ssp3_combine<<<blocks_for(n_interior_host(g)), kThreads, 0, st>>>(g, cons, f1, f2, f3, s1, s2,
                                                                      s3, dt);
  return cudaGetLastError();
}

cudaError_t launch_ssp2322_combine(const Grid& g, double* cons, const double* f2,
                                   const double* f3, const double* s2, const double* s3,
                                   double dt, cudaStream_t st) {
  k_ssp2322_combine<<<blocks_for(n_interior_host(g)), kThreads, 0, st>>>(g, cons, f2, f3, s2, s3,
                                                                         dt);
  return cudaGetLastError();
}

cudaError_t launch_ssp2_combine(const Grid& g, int nc, double* cons, const double* flux1,
                                const double* flux2, const double* source1,
                                const double* source2, double dt, cudaStream_t st) {
  const long long nI = (long long)(g.ie - g.is) * (g.je - g.js) * (g.ke - g.ks);
  k_ssp2_combine<<<blocks_for(nI), kThreads, 0, st>>>(g, nc, cons, flux1, flux2, source1, source2,
                                                      dt);
  return cudaGetLastError();
}

cudaError_t ens_fvs_fp64(const Member* mem, const Item* items, int n, int model, int order,
                         int TI, int ic, int ip, int ia, int iu0, int iout, int mode, int grid,
                         cudaStream_t st) {
#define ENS_FVS(MM, O, T) \
  return ens_fvs_fp64_instance<MM, O, T>(mem, items, n, ic, ip, ia, iu0, iout, mode, grid, st)
  if (model == MODEL_SRMHD) {
    if (order == 3) {
      if (TI == 4) ENS_FVS(SRMHD, 3, 4);
      if (TI == 16) ENS_FVS(SRMHD, 3, 16);
      ENS_FVS(SRMHD, 3, 8);
    }
    if (TI == 4) ENS_FVS(SRMHD, 5, 4);
    if (TI == 16) ENS_FVS(SRMHD, 5, 16);
    ENS_FVS(SRMHD, 5, 8);
  }
  return cudaErrorInvalidValue;  // plain-form ensembles are SRMHD
#undef ENS_FVS
}

cudaError_t ens_c2p_srmhd_hybrd(const Member* mem, const Item* items, int n, int ic, int ipg,
                                int iag, int ip, int ia, int grid, cudaStream_t st) {
  k_ens_c2p_srmhd_hybrd<<<grid, 128, 0, st>>>(mem, items, n, ic, ipg, iag, ip, ia);
  return cudaGetLastError();
}

cudaError_t ens_c2p_retry(const Member* mem, int n_members, int ic, int ip, int ia,
                          cudaStream_t st) {
  k_ens_c2p_retry<<<n_members, 32, 0, st>>>(mem, ic, ip, ia);
  return cudaGetLastError();
}

cudaError_t ens_source(const Member* mem, const Item* items, int n, int ic, int ia, int iout,
                       int grid, cudaStream_t st) {
  k_ens_source<<<grid, 128, 0, st>>>(mem, items, n, ic, ia, iout);
  return cudaGetLastError();
}


cudaError_t ens_dt(Member* mem, int n, cudaStream_t st) {
  k_ens_dt<<<(n + 127) / 128, 128, 0, st>>>(mem, n);
  return cudaGetLastError();
}

cudaError_t ens_advance(Member* mem, int n, cudaStream_t st) {
  k_ens_advance<<<(n + 127) / 128, 128, 0, st>>>(mem, n);
  return cudaGetLastError();
}

cudaError_t launch_source_add(const Grid& g, int model, const double* cons, const double* prims,
                              const double* aux, double* target, double dt, cudaStream_t st) {
  const long long nI = (long long)(g.ie - g.is) * (g.je - g.js) * (g.ke - g.ks);
  if (model == MODEL_SRMHD)
    k_source_add<MODEL_SRMHD><<<blocks_for(nI), kThreads, 0, st>>>(g, cons, prims, aux, target, dt);
  else
    k_source_add<MODEL_SRRMHD><<<blocks_for(nI), kThreads, 0, st>>>(g, cons, prims, aux, target,
                                                                     dt);
  return cudaGetLastError();
}

}  // namespace mth
