// D1Q5 pull step for small grids: a warp per node.
//
// The arithmetic of pull_point_kernel<D1Q5, N> and pull_1d_scheme_kernel (TVD
// steps.cu:447, WENO5 :774-825, Lagrange :986-1036), split over the lanes so
// that an iteration takes about the latency of one transfer row: six lanes
// serve population k (lane 6k + e, 30 lanes), each transfers one window node
// of its population into the iterate's gauge; the lanes of a population
// gather the window by shuffle and every lane forms the moments and the test.
//
// What bounds it: the dependent chain of an iteration (square root, window,
// transfer, limiter, moments, reciprocal; float64 throughout for TVD and
// WENO5's nonlinear part), about 1 us, and the first loads and reductions of a
// step, about 4 us.  1000 nodes, TVD, float64, 3.6 iterations: 9.1 us per step
// against 32.4 us with a thread per node, whose iteration
// transfers six nodes by five populations and selects 80 weights in one chain.
#pragma once
#include "pond_step_1d.cuh"

namespace pond {
namespace w1d {

constexpr int WARPS = 8;
constexpr int THREADS = 32 * WARPS;
constexpr int LANES = 6;  // per population

// population k of grid node p (boundaries resolved) in the gauge (Uc, 1/invC):
// row k of the 5-point basis of the node's speeds, non-finite terms dropped.
// Plain loads: the kernel is resident while the step before still writes its
// inputs, and the read-only path (__ldg) is for data that nothing writes as
// long as the kernel lives.
template <typename R>
__device__ __forceinline__ R transfer_row(const StepArgs<R>& a, int p, int k, R Uc, R invC) {
  using L = Lattice<POND_D1Q5>;
  bool rv;
  const long long n = resolve_axis(p, a.nx, a.bc[0], rv);
  const R T = a.g_in[3 * a.N + n], u = a.g_in[n];
  R f[5];
#pragma unroll
  for (int b = 0; b < 5; b++) f[b] = finite_or_zero_f(a.f_in[b * a.N + n]);
  const R c = copysign(sqrt(fabs(T) * R(1.0 / L::TLat)), T);
  const R s = ((rv ? -u : u) - Uc) * invC, r = (rv ? -c : c) * invC;
  constexpr double e1s = EC1 * EC1, e2s = EC2 * EC2;
  const R D = k == 0 ? R(1.0 / (e1s * e2s))
                     : (k <= 2 ? R(1.0 / (2.0 * e1s * (e1s - e2s))) : R(1.0 / (2.0 * e2s * (e2s - e1s))));
  const R P = (k == 1 || k == 2) ? R(e2s) : R(e1s);
  const R S = k == 1 ? R(EC1) : k == 2 ? -R(EC1) : k == 3 ? R(EC2) : k == 4 ? -R(EC2) : R(0);
  const R Q = k == 0 ? R(e2s) : R(0);
  R g = R(0);
#pragma unroll
  for (int b = 0; b < 5; b++) {
    const R y = fma(r, R(L::xi1(b)), s), y2 = y * y;
    g = fma(finite_or_zero_f(D * (y2 - P) * (fma(S, y, y2) - Q)), f[b], g);
  }
  return g;
}

// positions in the union of the warp's windows [org, org + N), as
// window_positions counts them for the thread-per-node kernels
template <int N> __device__ __forceinline__ int union_positions(int org) {
  const int lo = __reduce_min_sync(0xffffffffu, org);
  if (__reduce_max_sync(0xffffffffu, org) - lo <= 32 - N)
    return __popc(__reduce_or_sync(0xffffffffu, ((1u << N) - 1u) << (org - lo)));
  int start[5];
#pragma unroll
  for (int k = 0; k < 5; k++) start[k] = __shfl_sync(0xffffffffu, org, LANES * k);
  return window_positions<N, 5>(start);
}

template <int SCHEME, typename R> __global__ void __launch_bounds__(THREADS) pull_1d_warp_kernel(StepArgs<R> a) {
  using L = Lattice<POND_D1Q5>;
  constexpr int N = SCHEME == POND_TVD ? 4 : SCHEME == POND_WENO5 ? 5 : SCHEME;  // window nodes
  __shared__ double pd[WARPS][6];
  __shared__ unsigned long long pu[WARPS][3];
  __shared__ int pm[WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = min(lane / LANES, 4), e = lane < 30 ? lane % LANES : lane - 30;  // lanes 30, 31 repeat population 4
  const int x = blockIdx.x * WARPS + warp;
  NodeSums ns = {0, 0, 0, 0, 0, 0, 0ull, 0ull, 0ull, 0};
  // launched while the step before still runs (launch_1d_warp): let the next
  // one come, then wait for the step before to be complete and visible
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  if (x < a.nx) {  // warp-uniform
    R f0[5];
    double rho0, U[3], T;
    load_center<POND_D1Q5, R>(a, x, f0, rho0, U, T);
    int niter = 0;
    bool conv = false;
    const double xik = k == 0 ? 0.0 : k == 1 ? EC1 : k == 2 ? -EC1 : k == 3 ? EC2 : -EC2;
    while (niter < a.max_iter) {
      niter++;
      const double C = sqrt(T / L::TLat);
      const double v = C * xik + U[0];
      const R Uc = R(U[0]), invC = R(1.0 / C);
      R fk;
      if constexpr (SCHEME == POND_TVD) {
        // lane m = 0..3 of the population: the cubic value at x-2v, x-v, x, x+v
        const int m = min(e, 3);
        const double mult = m == 0 ? -2.0 : m == 1 ? -1.0 : m == 2 ? 0.0 : 1.0;
        const double crd = double(x) + v * mult;
        const int org = window_origin<4>(crd, 0);
        ns.work += (unsigned long long)(__reduce_max_sync(0xffffffffu, org) + 4 - __reduce_min_sync(0xffffffffu, org));
        R w[4];
        lagr_weights<4, R>(crd - double(org), w);
        // the union of the four windows: consecutive nodes while |v| < 1
        int lo = org, hi = org;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int o = __shfl_sync(0xffffffffu, org, LANES * k + j);
          lo = min(lo, o);
          hi = max(hi, o);
        }
        R F = R(0);
        if (__all_sync(0xffffffffu, hi - lo <= LANES - 4)) {
          const R g = transfer_row<R>(a, lo + e, k, Uc, invC);
#pragma unroll
          for (int j = 0; j < 4; j++) F += w[j] * __shfl_sync(0xffffffffu, g, LANES * k + org + j - lo);
        } else {
#pragma unroll 1
          for (int j = 0; j < 4; j++)
            F += (j == 0 ? w[0] : j == 1 ? w[1] : j == 2 ? w[2] : w[3]) * transfer_row<R>(a, org + j, k, Uc, invC);
        }
        double Fm[4];
#pragma unroll
        for (int j = 0; j < 4; j++) Fm[j] = __shfl_sync(0xffffffffu, F, LANES * k + j);
        fk = R(tvd_combine(Fm[0], Fm[1], Fm[2], Fm[3], v));
      } else if constexpr (SCHEME == POND_WENO5) {
        const int base = (int)(floor(held_coordinate(double(x) - v) + 0.5) - 2);
        ns.work += (unsigned long long)(__reduce_max_sync(0xffffffffu, base) + 5 - __reduce_min_sync(0xffffffffu, base));
        const R g = transfer_row<R>(a, base + min(e, 4), k, Uc, invC);
        double u[5];
#pragma unroll
        for (int j = 0; j < 5; j++) u[j] = __shfl_sync(0xffffffffu, g, LANES * k + j);
        fk = R(weno5_combine(u, double(x) - v));
      } else {
        const double crd = double(x) - v;
        const int org = window_origin<N>(crd, 0);
        ns.work += union_positions<N>(org);
        const double sh = crd - double(org);
        R w[N];
        if (N == 2) {  // LinPol
          w[0] = R(1 - sh);
          w[N - 1] = R(sh);
        } else {
          lagr_weights<N, R>(sh, w);
        }
        const R g = transfer_row<R>(a, org + min(e, N - 1), k, Uc, invC);
        fk = R(0);
#pragma unroll
        for (int j = 0; j < N; j++) fk += w[j] * __shfl_sync(0xffffffffu, g, LANES * k + j);
      }
      R fn[5];
#pragma unroll
      for (int q = 0; q < 5; q++) fn[q] = __shfl_sync(0xffffffffu, fk, LANES * q);
      if (moments_and_test<POND_D1Q5, R>(a, fn, f0, C, rho0, U, T)) { conv = true; break; }
    }
    if (lane == 0) finish_node<POND_D1Q5, R>(a, x, f0, rho0, U, T, niter, conv, ns);
  }
  if (lane == 0) {
    const double v[6] = {ns.mass, ns.m0, ns.m1, ns.m2, ns.enrg, ns.k};
#pragma unroll
    for (int q = 0; q < 6; q++) pd[warp][q] = v[q];
    pu[warp][0] = ns.niter; pu[warp][1] = ns.nonconv; pu[warp][2] = ns.work;
    pm[warp] = ns.nmax;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double s = 0;
#pragma unroll
    for (int w = 0; w < WARPS; w++) s += pd[w][threadIdx.x];
    double* o = threadIdx.x == 0 ? &a.sums->mass : threadIdx.x < 4 ? &a.sums->mom[threadIdx.x - 1]
                : threadIdx.x == 4 ? &a.sums->enrg : &a.sums->k;
    atomicAdd(o, s);
  } else if (threadIdx.x < 9) {
    const int q = threadIdx.x - 6;
    unsigned long long s = 0;
#pragma unroll
    for (int w = 0; w < WARPS; w++) s += pu[w][q];
    if (s) atomicAdd(q == 0 ? &a.sums->niter_sum : q == 1 ? &a.sums->nonconv : &a.sums->work, s);
  } else if (threadIdx.x == 9) {
    int m = 0;
#pragma unroll
    for (int w = 0; w < WARPS; w++) m = max(m, pm[w]);
    atomicMax(&a.sums->niter_max, m);
  }
}

}  // namespace w1d
}  // namespace pond
