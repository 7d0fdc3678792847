// D3Q27 PonD pull step, float64, Lagrange order N = 2..4: three lanes per node,
// ten nodes of an x row per warp.
//
// The arithmetic of pull_point_kernel (steps.cu:356-588 LBMpull with
// propagate<N>) through a reference gauge, as in the float32 tile kernel
// (pond_step_d3q27.cuh): every staged node is transferred once per step into
// the gauge of the tile's centre node, and an iteration contracts the
// interpolation weights and the transfer R -> target against the R-gauge
// populations one axis at a time (81 multiply-adds per stencil node, column
// and row) instead of transforming every stencil node into the target gauge
// (243).  While the gauges lie within a factor 2 of the tile's (near_ref) the
// two agree to 7e-15 of the largest population; other tiles are left out.
//
//  * a CTA owns a 10 x 4 x 2 tile, staged with its +-2 halo (14 x 8 x 6 nodes,
//    161 KB); per node three slices k1 of nine populations, 10 doubles apart, so
//    consecutive (node, k1) pairs are 20 words apart and the eight lanes of a
//    16-byte load phase fall in distinct banks;
//  * lane 3n + j serves node n of its warp's row: x-class k1 = j along z and y
//    (27 accumulators would not fit a lane in float64: nine do), then, after
//    the row's exchange through shared memory, target z-class i3 = j for the x
//    contraction, the moments and the test;
//  * a warp with a node whose windows leave the halo, or whose iterate
//    moves far from the tile's gauge, runs that iteration from
//    global memory: lane 3n + j transforms each stencil node into the target's
//    z-class j directly, as the one-thread-per-node kernel does for all three.
//    That takes 2.5-3.5 times the time of the one-thread-per-node kernel (32^3
//    at c = 1.2: 10.6 against 4.1 ms, 10 nodes per warp instead of 32 and three
//    loads of each), so it serves nodes that get there while iterating; a tile
//    with a node that starts near the edge of the halo (|u| + c >= 0.98 on an
//    axis for N = 4), or with gauges far from its centre's, is flagged and left to
//    that kernel, which follows every
//    launch and returns at once where nothing is flagged (32^3 at c = 0.95 and
//    |u| up to 0.06: 4.0 ms with a quarter of the rows as the line, against 2.2).
//
// What bounds it: the float64 pipe (64 multiply-adds per clock and SM: 4,185 per
// lane and iteration at N = 4 are 2,090 cycles of the SM) and shared-memory
// bandwidth (17 wavefronts per stencil node, as much), at two warps per
// scheduler.  48^3 half-uniform blast, cubic, 1e-12 + 1e-10 |v|, 4.8 iterations
// per node: 1.75 ms per step against 7.02 ms for the one-thread-per-node kernel
// (three-pass transform of every stencil node, read from L1/L2 per iteration).
#pragma once
#include "pond_step_d3q27.cuh"

namespace pond {
namespace d27d {

constexpr int TX = F64_TX, TY = F64_TY, TZ = F64_TZ, H = 2;
constexpr int SX = TX + 2 * H, SY = TY + 2 * H, SZ = TZ + 2 * H;
constexpr int SN = SX * SY * SZ;  // 672 staged nodes
constexpr int NS = 30;            // doubles per staged node: slices k1 of nine, 10 apart
constexpr int WARPS = TY * TZ;    // a row each
constexpr int THREADS = 32 * WARPS;

struct NodeTables {   // y [0] and x [1] of the node's iterate
  double w[2][3][5];  // interpolation weights [class][offset + 2]
  double g[2][9];     // R -> target transfer [3 i + k]
};
struct Smem {
  double f[SN * NS];           // staged populations, then their transfer into R
  NodeTables nt[WARPS][TX];
  double ex[WARPS][32 * 9];    // a row's results [3 i2 + i3] of lane (n, k1)
};
static_assert(sizeof(Smem) + 4096 <= 232448, "the tile must fit one CTA");

// Whether a gauge (u, c) lies near enough to R that the way through R keeps
// float64's digits.  A transfer source -> R -> target cancels terms of
// (|u - u_ref| / c + c ratio)^2 per axis and way; for one node against the
// direct transfer, both in float64 (random states, relative to the largest
// population): c within a factor 2 of c_ref and |u - u_ref| up to 1.0 of the
// smaller c 7e-15 at most (direct: 1e-15); factor 5: 7e-13; factor 10 (a
// temperature ratio of 100): 2e-11; factor 100: 1e-5.  Looking at
// every iterate costs 3.5 % of a step (48^3: 1.75 ms, 1.69 without).
constexpr double FAR_C = 2.0, FAR_U = 1.0;
__device__ __forceinline__ bool near_ref(const double u[3], double c, const double uref[3], double cref, double slack) {
  const double least = slack * FAR_U * fmin(c, cref);
  return c <= slack * FAR_C * cref && cref <= slack * FAR_C * c && fabs(u[0] - uref[0]) <= least &&
         fabs(u[1] - uref[1]) <= least && fabs(u[2] - uref[2]) <= least;
}

// One stencil node into a column: Z[k2][i3] += sum_k3 c[i3][k3] F[k2][k3] for the
// z-classes i3 = 0, + (kPlus) and - (kMinus) of this lane's k1
template <bool kPlus, bool kMinus>
__device__ __forceinline__ void column_node(const double* slice, const double c[3][3], double Z[3][3]) {
  double v[10];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const double2 t = reinterpret_cast<const double2*>(slice)[q];
    v[2 * q] = t.x;
    v[2 * q + 1] = t.y;
  }
  v[8] = slice[8];
#pragma unroll
  for (int k2 = 0; k2 < 3; k2++)
#pragma unroll
    for (int i = 0; i < 3; i++) {
      if ((i == 1 && !kPlus) || (i == 2 && !kMinus)) continue;
      Z[k2][i] = fma(c[i][2], v[3 * k2 + 2], fma(c[i][1], v[3 * k2 + 1], fma(c[i][0], v[3 * k2], Z[k2][i])));
    }
}

template <int N> __global__ void __launch_bounds__(THREADS, 1) pull_d3q27_f64_kernel(StepArgs<double> a) {
  using L = Lattice<POND_D3Q27>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, z0 = blockIdx.z * TZ;
  constexpr double kMax = 1.7976931348623157e308;

  // ---- reference gauge of the CTA: the gauge of the tile's centre node
  //      ((0, 1) if it is not finite or its c is 0)
  double uref[3], cref;
  {
    bool rv[3];
    const int gx = resolve_axis(x0 + TX / 2, a.nx, a.bc[0], rv[0]);
    const int gy = resolve_axis(y0 + TY / 2, a.ny, a.bc[1], rv[1]);
    const int gz = resolve_axis(z0 + TZ / 2, a.nz, a.bc[2], rv[2]);
    const long long g = gx + (long long)a.nx * (gy + (long long)a.ny * gz);
    const double T = a.g_in[3 * a.N + g];
    cref = copysign(sqrt(fabs(T) * (1.0 / L::TLat)), T);
    bool ok = fabs(cref) <= kMax && fabs(cref) > 1.0e-150;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double v = a.g_in[(long long)k * a.N + g];
      uref[k] = rv[k] ? -v : v;
      ok = ok && fabs(v) <= kMax;
    }
#pragma unroll
    for (int k = 0; k < 3; k++) uref[k] = ok ? uref[k] : 0.0;
    cref = ok ? cref : 1.0;
  }
  const double icref = 1.0 / cref;

  // ---- stage: each thread copies whole nodes, then transfers its own into R
#pragma unroll 1
  for (int i = tid; i < SN; i += THREADS) {
    const int hx = i % SX, hy = (i / SX) % SY, hz = i / (SX * SY);
    bool rv[3];
    const int gx = resolve_axis(x0 - H + hx, a.nx, a.bc[0], rv[0]);
    const int gy = resolve_axis(y0 - H + hy, a.ny, a.bc[1], rv[1]);
    const int gz = resolve_axis(z0 - H + hz, a.nz, a.bc[2], rv[2]);
    const double* src = a.f_in + (gx + (long long)a.nx * (gy + (long long)a.ny * gz));
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(sm.f + i * NS));
#pragma unroll
    for (int t = 0; t < 27; t++) {
      int cx = t / 9, cy = (t / 3) % 3, cz = t % 3;
      if (rv[0]) cx = d27::rev3(cx);
      if (rv[1]) cy = d27::rev3(cy);
      if (rv[2]) cz = d27::rev3(cz);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d + 8 * (10 * (t / 9) + t % 9)),
                   "l"(src + (long long)d27::c_ref27[cx * 9 + cy * 3 + cz] * a.N)
                   : "memory");
    }
  }
  // ---- a tile with a node that starts at the edge of the halo or beyond, or whose
  //      gauges (halo included) lie further from R than FAR_C and FAR_U, is left to
  //      the one-thread-per-node kernel launched after this one (looked at while
  //      the copies are in flight)
  {
    const int n = lane % TX, x = x0 + n, y = y0 + warp % TY, z = z0 + warp / TY;
    const bool here = x < a.nx && y < a.ny && z < a.nz;
    bool far = false;
    if (here && lane < TX) {
      const long long g = x + (long long)a.nx * (y + (long long)a.ny * z);
      const double c = a.guess ? sqrt(double(a.guess[3 * a.N + g]) * (1.0 / L::TLat))
                               : sqrt(a.g_in[3 * a.N + g] * (1.0 / L::TLat));
#pragma unroll
      for (int ax = 0; ax < 3; ax++) {
        const double u = fabs(a.guess ? double(a.guess[ax * a.N + g]) : a.g_in[ax * a.N + g]);
        // the largest |v| whose window stays within two nodes, less what an iterate may add
        far = far || u + c >= 0.98 * (N == 4 ? 1.0 : N == 2 ? 2.0 : ax == 0 ? 1.5 : 1.0);
      }
    }
    for (int i = tid; i < SN; i += THREADS) {
      const int hx = i % SX, hy = (i / SX) % SY, hz = i / (SX * SY);
      bool rv[3];
      const int gx = resolve_axis(x0 - H + hx, a.nx, a.bc[0], rv[0]);
      const int gy = resolve_axis(y0 - H + hy, a.ny, a.bc[1], rv[1]);
      const int gz = resolve_axis(z0 - H + hz, a.nz, a.bc[2], rv[2]);
      const long long g = gx + (long long)a.nx * (gy + (long long)a.ny * gz);
      double u[3];
      bool ok = true;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const double v = a.g_in[(long long)k * a.N + g];
        u[k] = rv[k] ? -v : v;
        ok = ok && fabs(v) <= kMax;
      }
      const double c = sqrt(fabs(a.g_in[3 * a.N + g]) * (1.0 / L::TLat));
      // nodes without a finite gauge contribute nothing
      far = far || (ok && c <= kMax && !near_ref(u, c, uref, cref, 1.0));
    }
    const bool leave = __syncthreads_or(far);
    if (tid == 0)
      a.tile_flags[blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z)] = leave;
    if (leave) {
      d27::cp_async_wait_all();
      return;
    }
  }
  d27::cp_async_wait_all();
#pragma unroll 1
  for (int i = tid; i < SN; i += THREADS) {
    const int hx = i % SX, hy = (i / SX) % SY, hz = i / (SX * SY);
    bool rv[3];
    const int gx = resolve_axis(x0 - H + hx, a.nx, a.bc[0], rv[0]);
    const int gy = resolve_axis(y0 - H + hy, a.ny, a.bc[1], rv[1]);
    const int gz = resolve_axis(z0 - H + hz, a.nz, a.bc[2], rv[2]);
    const long long g = gx + (long long)a.nx * (gy + (long long)a.ny * gz);
    double u[3];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double v = __ldg(&a.g_in[(long long)k * a.N + g]);
      u[k] = rv[k] ? -v : v;
      ok = ok && fabs(v) <= kMax;
    }
    const double T = __ldg(&a.g_in[3 * a.N + g]);
    const double c = copysign(sqrt(fabs(T) * (1.0 / L::TLat)), T);
    ok = ok && fabs(c) <= kMax;
    double* fi = sm.f + i * NS;
    double v[27], sq[3], rq[3];
#pragma unroll
    for (int t = 0; t < 27; t++) {
      const double w = fi[10 * (t / 9) + t % 9];
      v[t] = ok ? finite_or_zero_f(w) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      sq[k] = ok ? (u[k] - uref[k]) * icref : 0.0;
      rq[k] = ok ? c * icref : 0.0;
    }
    d27::node_to_ref(v, sq, rq);
#pragma unroll
    for (int t = 0; t < 27; t++) fi[10 * (t / 9) + t % 9] = v[t];
  }
  __syncthreads();

  // ---- lane 3n + j; idle lanes 30, 31 repeat node 9 and write nothing
  const bool worker = lane < 30;
  const int n = worker ? lane / 3 : 9, j = worker ? lane % 3 : lane - 30;
  const int ly = warp % TY, lz = warp / TY;
  const int x = x0 + n, y = y0 + ly, z = z0 + lz;
  const bool active = x < a.nx && y < a.ny && z < a.nz;
  const long long idx = active ? x + (long long)a.nx * (y + (long long)a.ny * z) : 0;
  NodeSums ns = {0, 0, 0, 0, 0, 0, 0ull, 0ull, 0ull, 0};
  // c0.load (steps.cu:360-363): this lane's populations (i1, i2, j), with set_base(1, TLat) of an empty record
  double f0[3][3];
#pragma unroll
  for (int i = 0; i < 9; i++) f0[i / 3][i % 3] = a.f_in[(long long)d27::c_ref27[3 * i + j] * a.N + idx];
  double rho0 = a.rho_in[idx];
  double U[3] = {a.g_in[idx], a.g_in[a.N + idx], a.g_in[2 * a.N + idx]}, T = a.g_in[3 * a.N + idx];
  // weights of the classes (0, +-1 per axis): by the number of moving axes
  constexpr double W[4] = {lattice_weight_t<POND_D3Q27>(0), lattice_weight_t<POND_D3Q27>(1),
                           lattice_weight_t<POND_D3Q27>(4), lattice_weight_t<POND_D3Q27>(13)};
  if (rho0 == 0 && U[0] == 0 && U[1] == 0 && U[2] == 0 && T == 0) {
    rho0 = 1; T = L::TLat;
#pragma unroll
    for (int i = 0; i < 9; i++) {
      const int m = (i / 3 != 0) + (i % 3 != 0);
      f0[i / 3][i % 3] = j ? W[m + 1] : W[m];
    }
  }
  if (a.guess) { U[0] = a.guess[idx]; U[1] = a.guess[a.N + idx]; U[2] = a.guess[2 * a.N + idx]; T = a.guess[3 * a.N + idx]; }
  const double xij = j == 0 ? 0.0 : j == 1 ? 1.0 : -1.0;
  const double* centre = sm.f + (((lz + H) * SY + (ly + H)) * SX + (n + H)) * NS + 10 * j;
  NodeTables& nt = sm.nt[warp][n];
  double* ex = sm.ex[warp];
  bool done = !active, conv = false;
  int niter = 0;
  unsigned long long work = 0;
  while (__any_sync(0xffffffffu, !done)) {
    if (!done) niter++;
    const double C = sqrt(T * (1.0 / L::TLat));
    // windows: every lane the z axis, and lane j = 0 of the node y, the others x
    const int other = j == 0 ? 1 : 0;
    const double Uo = other ? U[1] : U[0];
    const int po = other ? y : x;
    int rz[3], ro[3];
    double wz[3][N], wo[3][N];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double vz = C * L::xi1(c) + U[2], vo = C * L::xi1(c) + Uo;
      const double cz = double(z) - vz, co = double(po) - vo;
      const int oz = window_origin<N>(cz, 2), oo = other ? window_origin<N>(co, 1) : window_origin<N>(co, 0);
      rz[c] = oz - z;
      ro[c] = oo - po;
      if (N == 2) {
        wz[c][0] = 1 - (cz - oz); wz[c][N - 1] = cz - oz;
        wo[c][0] = 1 - (co - oo); wo[c][N - 1] = co - oo;
      } else {
        lagr_weights<N, double>(cz - double(oz), wz[c]);
        lagr_weights<N, double>(co - double(oo), wo[c]);
      }
    }
    const int zlo = min(rz[0], min(rz[1], rz[2])), zhi = max(rz[0], max(rz[1], rz[2])) + N - 1;
    const int olo = min(ro[0], min(ro[1], ro[2])), ohi = max(ro[0], max(ro[1], ro[2])) + N - 1;
    const bool inside = zlo >= -H && zhi <= H && olo >= -H && ohi <= H && near_ref(U, C, uref, cref, 1.25);
    double acc[3][3];  // [i1][i2] of i3 = j
#pragma unroll
    for (int i = 0; i < 9; i++) acc[i / 3][i % 3] = 0.0;
    if (__all_sync(0xffffffffu, inside || done)) {
      // transfer R -> target per axis: G[i][k] = L_i(b + a xi_k), a = c_ref / C, b = (u_ref - U) / C
      const double iC = 1.0 / C, ainv = cref * iC;
      double Gz[3][3];
      d27::basis_rows((uref[2] - U[2]) * iC, ainv, Gz);
      __syncwarp();  // the previous iteration's readers are done
      {
        double G[3][3];
        d27::basis_rows(((other ? uref[1] : uref[0]) - Uo) * iC, ainv, G);
        if (worker && j < 2) {
          const int s = 1 - other;  // 0: y, 1: x
#pragma unroll
          for (int c = 0; c < 3; c++) {
#pragma unroll
            for (int o = -H; o <= H; o++) nt.w[s][c][o + H] = d27::wpick<N>(wo[c], ro[c], o);
#pragma unroll
            for (int k = 0; k < 3; k++) nt.g[s][3 * c + k] = G[c][k];
          }
        }
      }
      __syncwarp();
      const int wzl = __reduce_min_sync(0xffffffffu, done ? H : zlo), wzh = __reduce_max_sync(0xffffffffu, done ? -H : zhi);
      const int wyl = __reduce_min_sync(0xffffffffu, done || !other ? H : olo),
                wyh = __reduce_max_sync(0xffffffffu, done || !other ? -H : ohi);
      const int wxl = __reduce_min_sync(0xffffffffu, done || other ? H : olo),
                wxh = __reduce_max_sync(0xffffffffu, done || other ? -H : ohi);
      // the stencil nodes of the node's own windows (x in lane 3n + 1, y in lane 3n)
      unsigned oz = 0, oo = 0;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        oz |= ((1u << N) - 1u) << ((rz[c] + H) & 31);
        oo |= ((1u << N) - 1u) << ((ro[c] + H) & 31);
      }
      const int positions = __popc(__shfl_sync(0xffffffffu, oo, 3 * n)) * __popc(__shfl_sync(0xffffffffu, oo, 3 * n + 1)) * __popc(oz);
      if (!done) work += (unsigned long long)positions;
      // the usual z windows: every lane's + class starts at wzl, its - class one later, wzh = wzl + N;
      // the first offset then has no - class and the last one no + class
      const bool staggered = __all_sync(0xffffffffu, done || (rz[1] == wzl && rz[2] == wzl + 1 && rz[0] >= wzl &&
                                                              rz[0] <= wzl + 1)) && wzh == wzl + N;
      double cz[N + 1][3][3];  // z weight x transfer by offset from wzl
#pragma unroll
      for (int o = 0; o <= N; o++)
#pragma unroll
        for (int i = 0; i < 3; i++) {
          const double w = d27::wpick<N>(wz[i], rz[i], wzl + o);
#pragma unroll
          for (int k = 0; k < 3; k++) cz[o][i][k] = w * Gz[i][k];
        }
#pragma unroll 1
      for (int ox = wxl; ox <= wxh; ox++) {
        double Y[3][3];  // [i2][i3] of k1 = j
#pragma unroll
        for (int i = 0; i < 9; i++) Y[i / 3][i % 3] = 0.0;
#pragma unroll 1
        for (int oy = wyl; oy <= wyh; oy++) {
          double Z[3][3];  // [k2][i3]
#pragma unroll
          for (int i = 0; i < 9; i++) Z[i / 3][i % 3] = 0.0;
          const double* col = centre + (wzl * SX * SY + oy * SX + ox) * NS;
          if (staggered) {
            column_node<true, false>(col, cz[0], Z);
#pragma unroll
            for (int o = 1; o < N; o++) column_node<true, true>(col + o * SX * SY * NS, cz[o], Z);
            column_node<false, true>(col + N * SX * SY * NS, cz[N], Z);
          } else {
#pragma unroll 1
            for (int oz = wzl; oz <= wzh; oz++) {
              double c[3][3];
#pragma unroll
              for (int i = 0; i < 3; i++) {
                const double w = d27::wpick<N>(wz[i], rz[i], oz);
#pragma unroll
                for (int k = 0; k < 3; k++) c[i][k] = w * Gz[i][k];
              }
              column_node<true, true>(col + (oz - wzl) * SX * SY * NS, c, Z);
            }
          }
#pragma unroll
          for (int i2 = 0; i2 < 3; i2++) {
            const double w = nt.w[0][i2][oy + H];
            const double g0 = w * nt.g[0][3 * i2], g1 = w * nt.g[0][3 * i2 + 1], g2 = w * nt.g[0][3 * i2 + 2];
#pragma unroll
            for (int i3 = 0; i3 < 3; i3++)
              Y[i2][i3] = fma(g2, Z[2][i3], fma(g1, Z[1][i3], fma(g0, Z[0][i3], Y[i2][i3])));
          }
        }
#pragma unroll
        for (int i = 0; i < 9; i++) ex[lane * 9 + i] = Y[i / 3][i % 3];
        __syncwarp();
        double X[3][3];  // [k1][i2] of i3 = j
#pragma unroll
        for (int i = 0; i < 9; i++) X[i / 3][i % 3] = ex[(3 * n + i / 3) * 9 + 3 * (i % 3) + j];
        __syncwarp();
#pragma unroll
        for (int i1 = 0; i1 < 3; i1++) {
          const double w = nt.w[1][i1][ox + H];
          const double g0 = w * nt.g[1][3 * i1], g1 = w * nt.g[1][3 * i1 + 1], g2 = w * nt.g[1][3 * i1 + 2];
#pragma unroll
          for (int i2 = 0; i2 < 3; i2++)
            acc[i1][i2] = fma(g2, X[2][i2], fma(g1, X[1][i2], fma(g0, X[0][i2], acc[i1][i2])));
        }
      }
    } else {
      // departure points beyond the staged halo.  The node's windows of all axes:
      // z is in every lane, y in lane 3n, x in lane 3n + 1
      int ry[3], rx[3];
      double wy[3][N], wx[3][N];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        ry[c] = __shfl_sync(0xffffffffu, ro[c], 3 * n);
        rx[c] = __shfl_sync(0xffffffffu, ro[c], 3 * n + 1);
#pragma unroll
        for (int k = 0; k < N; k++) {
          wy[c][k] = __shfl_sync(0xffffffffu, wo[c][k], 3 * n);
          wx[c][k] = __shfl_sync(0xffffffffu, wo[c][k], 3 * n + 1);
        }
      }
      if (!done) {
        work += (unsigned long long)window_positions<N, 3>(rx) * window_positions<N, 3>(ry) * window_positions<N, 3>(rz);
        const double iC = 1.0 / C;
        double wzj[N];
#pragma unroll
        for (int k = 0; k < N; k++) wzj[k] = j == 0 ? wz[0][k] : j == 1 ? wz[1][k] : wz[2][k];
        const int rzj = j == 0 ? rz[0] : j == 1 ? rz[1] : rz[2];
        const int xhi = max(rx[0], max(rx[1], rx[2])) + N - 1, yhi = max(ry[0], max(ry[1], ry[2])) + N - 1;
        for (int ox = min(rx[0], min(rx[1], rx[2])); ox <= xhi; ox = window_next<N, 3>(rx, ox)) {
          bool rv[3];
          const int gx = resolve_axis(x + ox, a.nx, a.bc[0], rv[0]);
          for (int oy = min(ry[0], min(ry[1], ry[2])); oy <= yhi; oy = window_next<N, 3>(ry, oy)) {
            const int gy = resolve_axis(y + oy, a.ny, a.bc[1], rv[1]);
#pragma unroll 1
            for (int k = 0; k < N; k++) {  // this lane's z-class only
              const int gz = resolve_axis(z + rzj + k, a.nz, a.bc[2], rv[2]);
              const double wzk = k == 0 ? wzj[0] : k == 1 ? wzj[1] : k == 2 ? wzj[N > 2 ? 2 : 0] : wzj[N - 1];
              const double Uc[3] = {U[0], U[1], U[2]};
              double fn[27], s[3], r[3];
              load_node<POND_D3Q27, double>(a, gx + (long long)a.nx * (gy + (long long)a.ny * gz), rv, Uc, iC, fn, s, r);
              double B[3][3], t1[3][3], t2[3][3];
              d27::basis_rows(s[2], r[2], B);
#pragma unroll
              for (int i = 0; i < 9; i++) {
                double t = 0;
#pragma unroll
                for (int b = 0; b < 3; b++) {
                  const double m = finite_or_zero_f(j == 0 ? B[0][b] : j == 1 ? B[1][b] : B[2][b]);
                  t = fma(wzk * m, fn[3 * i + b], t);
                }
                t1[i / 3][i % 3] = t;
              }
              d27::basis_rows(s[1], r[1], B);
#pragma unroll
              for (int i2 = 0; i2 < 3; i2++) {
                const double w = d27::wpick<N>(wy[i2], ry[i2], oy);
#pragma unroll
                for (int b1 = 0; b1 < 3; b1++) {
                  double t = 0;
#pragma unroll
                  for (int b = 0; b < 3; b++) t = fma(w * finite_or_zero_f(B[i2][b]), t1[b1][b], t);
                  t2[b1][i2] = t;
                }
              }
              d27::basis_rows(s[0], r[0], B);
#pragma unroll
              for (int i1 = 0; i1 < 3; i1++) {
                const double w = d27::wpick<N>(wx[i1], rx[i1], ox);
#pragma unroll
                for (int i2 = 0; i2 < 3; i2++)
#pragma unroll
                  for (int b = 0; b < 3; b++)
                    acc[i1][i2] = fma(w * finite_or_zero_f(B[i1][b]), t2[b][i2], acc[i1][i2]);
              }
            }
          }
        }
      }
      __syncwarp();
    }
    if (!(C >= 1.0e-300)) {  // C <= 0, NaN, or 1/C beyond 1e300
      // target T = 0: every transfer term is non-finite and dropped (structs.cuh:542)
#pragma unroll
      for (int i = 0; i < 9; i++) acc[i / 3][i % 3] = 0.0;
    }
    // calcMoments (structs.cuh:315-342): the lane's sums over i1 and i2, then the
    // three lanes of the node in a fixed order
    double mv[5] = {0, 0, 0, 0, 0};
    bool ok = true;
    {
      double s1[3] = {0, 0, 0}, s2[3] = {0, 0, 0};
#pragma unroll
      for (int i1 = 0; i1 < 3; i1++)
#pragma unroll
        for (int i2 = 0; i2 < 3; i2++) {
          const double nv = acc[i1][i2];
          s1[i1] += nv;
          s2[i2] += nv;
          ok = ok && !(fabs(nv - f0[i1][i2]) >= a.tol_abs + a.tol_rel * fabs(nv));
        }
      const double vz = C * xij + U[2];
      mv[0] = s1[0] + s1[1] + s1[2];
      mv[3] = mv[0] * vz;
      mv[4] = mv[3] * vz;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double vx = C * L::xi1(c) + U[0], vy = C * L::xi1(c) + U[1];
        const double px = s1[c] * vx, py = s2[c] * vy;
        mv[1] += px;
        mv[2] += py;
        mv[4] += px * vx + py * vy;
      }
    }
    double m[5];
#pragma unroll
    for (int q = 0; q < 5; q++)
      m[q] = __shfl_sync(0xffffffffu, mv[q], 3 * n) + __shfl_sync(0xffffffffu, mv[q], 3 * n + 1) +
             __shfl_sync(0xffffffffu, mv[q], 3 * n + 2);
    if (m[0] != 0) {
      const double ir = 1.0 / m[0];
#pragma unroll
      for (int q = 1; q < 5; q++) m[q] *= ir;
    }
    double Tn = (m[4] - m[1] * m[1] - m[2] * m[2] - m[3] * m[3]) * (1.0 / L::Dim);
    if (Tn < 0) Tn = T;  // steps.cu:475
    // isConv (steps.cu:58-75)
#pragma unroll
    for (int k = 0; k < 3; k++) ok = ok && !(fabs(m[1 + k] - U[k]) >= a.tolg_abs + a.tolg_rel * fabs(m[1 + k]));
    ok = ok && !(fabs(Tn - T) >= a.tolg_abs + a.tolg_rel * fabs(Tn));
    const unsigned votes = __ballot_sync(0xffffffffu, ok);
    if (!done) {
#pragma unroll
      for (int i = 0; i < 9; i++) f0[i / 3][i % 3] = acc[i / 3][i % 3];
      rho0 = m[0]; U[0] = m[1]; U[1] = m[2]; U[2] = m[3]; T = Tn;
      conv = ((votes >> (3 * n)) & 7u) == 7u;
      done = conv || niter >= a.max_iter;
    }
  }
  // BGK toward rho*w_i (steps.cu:557-564), store, the node's share of the sums
  if (worker && active) {
#pragma unroll
    for (int i = 0; i < 9; i++) {
      const int mo = (i / 3 != 0) + (i % 3 != 0);
      const double w = j ? W[mo + 1] : W[mo], f = f0[i / 3][i % 3];
      a.f_out[(long long)d27::c_ref27[3 * i + j] * a.N + idx] = f + a.dtau * (rho0 * w - f);
    }
    if (j == 0) {
      a.rho_out[idx] = rho0;
      a.g_out[idx] = U[0]; a.g_out[a.N + idx] = U[1]; a.g_out[2 * a.N + idx] = U[2]; a.g_out[3 * a.N + idx] = T;
      if (a.niter_out) a.niter_out[idx] = niter;
      const double u2s = U[0] * U[0] + U[1] * U[1] + U[2] * U[2];
      ns.mass = rho0; ns.m0 = rho0 * U[0]; ns.m1 = rho0 * U[1]; ns.m2 = rho0 * U[2];
      ns.enrg = rho0 * (u2s + L::Dim * T);
      ns.k = a.kdx * u2s;
      ns.niter = niter; ns.nonconv = conv ? 0 : 1; ns.nmax = niter; ns.work = work;
    }
  }
  reduce_and_commit(ns, a.sums);
}

}  // namespace d27d
}  // namespace pond
