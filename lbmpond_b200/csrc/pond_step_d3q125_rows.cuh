// D3Q125 PonD pull step, float32, fixed-origin quadratic: five lanes per node,
// six nodes of an x row per warp.
//
// The arithmetic of steps.cu:151-250 PonDstepD3Q125 through a reference gauge,
// as in pull_d3q125_tile_kernel (which keeps float64 and the energy
// populations).  Organised for register reuse:
//
//  * a CTA owns a 6 x 4 x 4 tile and stages it with its +-1 halo (8 x 6 x 6
//    nodes) once per step, node-major: a staged node holds, per x-class k1,
//    five quads (k3 = 1..4 of each k2) and five singles (k3 = 0), 132 floats in
//    all, so a lane reads its 25 populations with five 16-byte and five 4-byte
//    loads, and consecutive (node, k1) pairs are 20 words apart: the eight
//    lanes of a load phase fall in distinct banks;
//  * lane 5n + j serves node n of the row.  Along z and y it holds x-class
//    k1 = j of its node, one y-class k2 at a time: the 15 products of z weight
//    and z transfer (in registers for the whole iteration) against the 15
//    populations of a column, as two-wide multiply-adds on pairs of both, then
//    the y weights and transfers of all five target classes on pairs of
//    z-classes.  Per row the five lanes of a node exchange their results
//    through shared memory and continue with target y-class i2 = j for the x
//    contraction, the moments and the test;
//  * the stencil is the same for every class and gauge, so there is no other
//    path: a node's six neighbours in the warp only share the iteration count.
//
// What bounds it: staging (copies, gauge transfer and the first loads, 35 % of
// a three-iteration step, not overlapped at one CTA per SM) and, per iteration,
// latency at two warps per scheduler (the 24,375 multiply-adds per node take
// half of an iteration's time).  96^3 shock and vortex, 2.75 iterations per
// node: 5.2 ms per step, 1.15 ms per iteration; the warp-per-node form it
// replaces (25 lanes of one node, one scalar shared load per multiply-add)
// took 14.7 ms.
#pragma once
#include "pond_step_d3q125_tile.cuh"

namespace pond {
namespace d125r {

constexpr int TX = 6, TY = 4, TZ = 4;
constexpr int SX = TX + 2, SY = TY + 2, SZ = TZ + 2;
constexpr int SN = SX * SY * SZ;  // 288 staged nodes
constexpr int ROWS = SY * SZ;     // staged x rows of 8 nodes
constexpr int NS = 132;           // floats per staged node; 4 mod 32, as 5 x 20 is
constexpr int WARPS = 8;
constexpr int THREADS = 32 * WARPS;


struct Smem {
  float f[SN * NS];           // staged populations, then their transfer into R
  float gy[WARPS][TX][3][28]; // per node and iteration: y weight x transfer [n_y][4 k2 + i2 - 1], i2 = 0 at [20 + k2]
  float gx[WARPS][TX][3][28]; // the same along x: [n_x][4 k1 + i1 - 1], i1 = 0 at [20 + k1]
  float ex[WARPS][32 * 28];   // per lane [4 i2 + i3 - 1], i3 = 0 at [20 + i2]: from the x- to the y-class split
  float u[3][SN];             // staged velocities (sign-flipped on mirrored axes)
  float c[SN];                // sqrts(T / TLat)
  int g[SN];                  // global node (-1: the inflow ghost)
  unsigned char flags[SN];    // mirrored axes (bits 0-2)
};
static_assert(sizeof(Smem) + 4096 <= 232448, "the tile must fit one CTA");

__device__ __forceinline__ float2 fma2(float g, float2 v, float2 o) { return __ffma2_rn(make_float2(g, g), v, o); }

// B[i][b] = L_i(s + r xi_b) of the 5-point basis, non-finite entries dropped
// (below 1e8 every |y| is under 4e8 and every entry finite)
__device__ __forceinline__ void basis5(float s, float r, float B[5][5]) {
#pragma unroll
  for (int b = 0; b < 5; b++) {
    float l[5];
    Basis<5, float>::eval(fmaf(r, d125t::xi5r<float>(b), s), l);
#pragma unroll
    for (int i = 0; i < 5; i++) B[i][b] = l[i];
  }
  if (!(fabsf(s) < 1e8f && fabsf(r) < 1e8f))
#pragma unroll
    for (int i = 0; i < 5; i++)
#pragma unroll
      for (int b = 0; b < 5; b++) B[i][b] = finite_or_zero_f(B[i][b]);
}

// Five values as the pairs 1, 2 and 3, 4 and the single 0.
struct Five {
  float2 a, b;
  float s;
  __device__ __forceinline__ float get(int i) const {
    return i == 0 ? s : i == 1 ? a.x : i == 2 ? a.y : i == 3 ? b.x : b.y;
  }
  __device__ __forceinline__ void clear() { a = b = make_float2(0.f, 0.f); s = 0.f; }
  __device__ __forceinline__ void add(float g, const Five& v) {  // this += g v
    a = fma2(g, v.a, a);
    b = fma2(g, v.b, b);
    s = fmaf(g, v.s, s);
  }
  __device__ __forceinline__ void scale(float g, const Five& v) {  // this = g v
    a = __fmul2_rn(make_float2(g, g), v.a);
    b = __fmul2_rn(make_float2(g, g), v.b);
    s = g * v.s;
  }
  __device__ __forceinline__ void load(const float* quad, const float* single) {
    const float4 q = *reinterpret_cast<const float4*>(quad);
    a = make_float2(q.x, q.y);
    b = make_float2(q.z, q.w);
    s = *single;
  }
  __device__ __forceinline__ void store(float* quad, float* single) const {
    *reinterpret_cast<float4*>(quad) = make_float4(a.x, a.y, b.x, b.y);
    *single = s;
  }
};
// sum over the five of c[i] v[i]
__device__ __forceinline__ float dot5(const Five& c, const Five& v) {
  const float2 p = __ffma2_rn(c.b, v.b, __fmul2_rn(c.a, v.a));
  return fmaf(c.s, v.s, p.x) + p.y;
}

__global__ void __launch_bounds__(THREADS, 1) pull_d3q125_rows_kernel(StepArgs<float> a) {
  using L = Lattice<POND_D3Q125>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, z0 = blockIdx.z * TZ;

  // ---- the gauge and the global index of every staged node
  for (int i = tid; i < SN; i += THREADS) {
    const int hx = i % SX, hy = (i / SX) % SY, hz = i / (SX * SY);
    bool rv[3], ghost = false;
    const int gx = d125t::staged_axis(x0 - 1 + hx, a.nx, a.bc[0], rv[0], ghost);
    const int gy = d125t::staged_axis(y0 - 1 + hy, a.ny, a.bc[1], rv[1], ghost);
    const int gz = d125t::staged_axis(z0 - 1 + hz, a.nz, a.bc[2], rv[2], ghost);
    if (ghost) rv[0] = rv[1] = rv[2] = false;
    const int g = ghost ? -1 : gx + a.nx * (gy + a.ny * gz);
    sm.g[i] = g;
    sm.flags[i] = (unsigned char)((rv[0] ? 1 : 0) | (rv[1] ? 2 : 0) | (rv[2] ? 4 : 0));
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float v = g < 0 ? float(a.inflow[1 + k]) : a.g_in[(long long)k * a.N + g];
      sm.u[k][i] = rv[k] ? -v : v;
    }
    const float Tn = g < 0 ? float(a.inflow[4]) : a.g_in[3 * a.N + g];
    sm.c[i] = copysignf(sqrtf(fabsf(Tn) * float(1.0 / L::TLat)), Tn);
  }
  __syncthreads();
  // ---- the populations: a warp copies eight nodes of a row times four planes
  //      whose slots are neighbours (a quad, or four of the singles), row after row
  {
    const int n = lane & 7, j = lane >> 3;
#pragma unroll 1
    for (int pk = warp; pk < 32; pk += WARPS) {
      // pk < 25: quad (k1, k2) = (pk / 5, pk % 5), else singles 4 (pk - 25) + j = 5 k1 + k2
      const int s = 4 * (pk - 25) + j;
      if (pk >= 25 && s >= 25) continue;
      const int p = pk < 25 ? 5 * pk + j + 1 : 5 * s;
      float* dst = sm.f + n * NS + (pk < 25 ? 4 * pk + j : 100 + s);
      const float* src = a.f_in + (long long)p * a.N;
      const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
#pragma unroll 12
      for (int row = 0; row < ROWS; row++) {
        const int g = sm.g[row * SX + n];
        if (g >= 0)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d + row * (SX * NS * 4)), "l"(src + g)
                       : "memory");
        else  // the inflow ghost: set_base of the inflow state
          dst[row * SX * NS] = float(a.inflow[0] * lattice_weight_t<POND_D3Q125>(p));
      }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  }
  __syncthreads();

  // ---- reference gauge R: the staged node at tile position (TX/2, TY/2, TZ/2)
  //      ((0, 1) if that node's gauge is not finite or its c is 0)
  float uref[3], cref;
  {
    constexpr int ci = ((TZ / 2 + 1) * SY + (TY / 2 + 1)) * SX + TX / 2 + 1;
    const float cc = sm.c[ci];
    bool ok = fabsf(cc) <= 3.402823466e38f && fabsf(cc) > 1.0e-20f;
#pragma unroll
    for (int ax = 0; ax < 3; ax++) {
      uref[ax] = sm.u[ax][ci];
      ok = ok && fabsf(uref[ax]) <= 3.402823466e38f;
    }
#pragma unroll
    for (int ax = 0; ax < 3; ax++) uref[ax] = ok ? uref[ax] : 0.f;
    cref = ok ? cc : 1.f;
  }

  const bool worker = lane < 30;
  const int n = worker ? lane / 5 : 5, j = worker ? lane % 5 : lane - 30;
  float* ex = sm.ex[warp];
  // ---- every staged node into R: lane 5n + j takes x-class j of a node through the
  //      z and y passes of the 5x5 basis, then y-class j through the x pass; a
  //      node with a non-finite gauge contributes nothing, non-finite populations count as 0
  {
    const float icref = 1.f / cref;
#pragma unroll 1
    for (int t = warp; t < SN / 6; t += WARPS) {
      const int i = 6 * t + n;
      const unsigned fl = sm.flags[i];
      const float cn = sm.c[i];
      bool ok = fabsf(cn) <= 3.402823466e38f;
      float sq[3], rq[3];
#pragma unroll
      for (int ax = 0; ax < 3; ax++) {
        const float un = sm.u[ax][i];
        ok = ok && fabsf(un) <= 3.402823466e38f;
        sq[ax] = (un - uref[ax]) * icref;
        rq[ax] = ((fl >> ax) & 1 ? -cn : cn) * icref;
      }
      float* fi = sm.f + i * NS;
      float B[5][5];
      Five w[5];  // [k2]: z-classes
      basis5(sq[2], rq[2], B);
#pragma unroll
      for (int k2 = 0; k2 < 5; k2++) {
        Five v;
        v.load(fi + 20 * j + 4 * k2, fi + 100 + 5 * j + k2);
        v.a.x = ok ? finite_or_zero_f(v.a.x) : 0.f; v.a.y = ok ? finite_or_zero_f(v.a.y) : 0.f;
        v.b.x = ok ? finite_or_zero_f(v.b.x) : 0.f; v.b.y = ok ? finite_or_zero_f(v.b.y) : 0.f;
        v.s = ok ? finite_or_zero_f(v.s) : 0.f;
        float z[5];
#pragma unroll
        for (int i3 = 0; i3 < 5; i3++) {
          Five c;
          c.a = make_float2(B[i3][1], B[i3][2]); c.b = make_float2(B[i3][3], B[i3][4]); c.s = B[i3][0];
          z[i3] = dot5(c, v);
        }
        w[k2].a = make_float2(z[1], z[2]); w[k2].b = make_float2(z[3], z[4]); w[k2].s = z[0];
      }
      basis5(sq[1], rq[1], B);
#pragma unroll
      for (int i2 = 0; i2 < 5; i2++) {
        Five t;
        t.scale(B[i2][0], w[0]);
#pragma unroll
        for (int k2 = 1; k2 < 5; k2++) t.add(B[i2][k2], w[k2]);
        t.store(ex + lane * 28 + 4 * i2, ex + lane * 28 + 20 + i2);
      }
      __syncwarp();
#pragma unroll
      for (int k1 = 0; k1 < 5; k1++) w[k1].load(ex + (5 * n + k1) * 28 + 4 * j, ex + (5 * n + k1) * 28 + 20 + j);
      __syncwarp();
      basis5(sq[0], rq[0], B);
#pragma unroll
      for (int i1 = 0; i1 < 5; i1++) {
        Five t;
        t.scale(B[i1][0], w[0]);
#pragma unroll
        for (int k1 = 1; k1 < 5; k1++) t.add(B[i1][k1], w[k1]);
        if (!ok) t.clear();
        if (worker) t.store(fi + 20 * i1 + 4 * j, fi + 100 + 5 * i1 + j);
      }
    }
  }
  __syncthreads();

  NodeSums ns = {0, 0, 0, 0, 0, 0, 0ull, 0ull, 0ull, 0};
#pragma unroll 1
  for (int r = warp; r < TY * TZ; r += WARPS) {
    const int ly = r % TY, lz = r / TY;
    const int x = x0 + n, y = y0 + ly, z = z0 + lz;
    if (y >= a.ny || z >= a.nz) continue;  // warp-uniform
    const bool active = x < a.nx;
    const long long idx = (active ? x : x0) + (long long)a.nx * (y + (long long)a.ny * z);
    // c0.load: this lane's populations (i1, j, i3)
    float f0[5][5];
#pragma unroll
    for (int i1 = 0; i1 < 5; i1++)
#pragma unroll
      for (int i3 = 0; i3 < 5; i3++) f0[i1][i3] = a.f_in[(long long)(25 * i1 + 5 * j + i3) * a.N + idx];
    double rho0 = a.rho_in[idx];
    double U[3] = {(double)a.g_in[idx], (double)a.g_in[a.N + idx], (double)a.g_in[2 * a.N + idx]};
    double Tc = a.g_in[3 * a.N + idx];
    if (rho0 == 0 && U[0] == 0 && U[1] == 0 && U[2] == 0 && Tc == 0) {  // set_base(1, TLat)
      rho0 = 1;
      Tc = L::TLat;
#pragma unroll
      for (int i1 = 0; i1 < 5; i1++)
#pragma unroll
        for (int i3 = 0; i3 < 5; i3++) f0[i1][i3] = float(lattice_weight_t<POND_D3Q125>(25 * i1 + 5 * j + i3));
    }
    if (a.guess) {
      U[0] = a.guess[idx]; U[1] = a.guess[a.N + idx]; U[2] = a.guess[2 * a.N + idx]; Tc = a.guess[3 * a.N + idx];
    }
    const int pos[3] = {(int)(active ? x : x0), y, z};
    const float* corner = sm.f + ((lz * SY + ly) * SX + n) * NS;  // stencil node (-1, -1, -1) of this lane's node
    int niter = 0;
    bool done = !active, conv = false;
    while (__any_sync(0xffffffffu, !done)) {
      if (!done) niter++;
      const double C = sqrt(Tc / L::TLat);
      // transfer R -> target per axis: G[i][k] = L_i(b + a xi_k), a = c_ref/C, b = (u_ref - U)/C
      const double iC = 1.0 / C;
      const float ga = float(double(cref) * iC);
      float gb[3];
#pragma unroll
      for (int ax = 0; ax < 3; ax++) gb[ax] = float((double(uref[ax]) - U[ax]) * iC);
      // this lane's rows i2 = j and i1 = j of the y and x tables
      {
        float wy[3], wx[3];
        d125t::stencil_weights(pos[1], C, U[1], j, wy);
        d125t::stencil_weights(pos[0], C, U[0], j, wx);
        const d125t::BasisRowT<float> Lj(j);
        __syncwarp();  // the previous iteration's readers are done
#pragma unroll
        for (int k = 0; k < 5; k++) {
          const float ty = finite_or_zero_f(Lj(fmaf(ga, d125t::xi5r<float>(k), gb[1])));
          const float tx = finite_or_zero_f(Lj(fmaf(ga, d125t::xi5r<float>(k), gb[0])));
#pragma unroll
          for (int o = 0; o < 3; o++) {
            sm.gy[warp][n][o][j > 0 ? 4 * k + j - 1 : 20 + k] = wy[o] * ty;
            sm.gx[warp][n][o][j > 0 ? 4 * k + j - 1 : 20 + k] = wx[o] * tx;
          }
        }
        __syncwarp();
      }
      // z weight x transfer of every class, for the whole iteration: pairs over k3,
      // and for k3 = 0 the pair of the first two stencil nodes
      float2 cp[3][5][2], c01[5];
      float c2[5];
      {
        float B[5][5];
        basis5(gb[2], ga, B);
#pragma unroll
        for (int i3 = 0; i3 < 5; i3++) {
          float wz[3];
          d125t::stencil_weights(pos[2], C, U[2], i3, wz);
#pragma unroll
          for (int o = 0; o < 3; o++) {
            cp[o][i3][0] = make_float2(wz[o] * B[i3][1], wz[o] * B[i3][2]);
            cp[o][i3][1] = make_float2(wz[o] * B[i3][3], wz[o] * B[i3][4]);
          }
          c01[i3] = make_float2(wz[0] * B[i3][0], wz[1] * B[i3][0]);
          c2[i3] = wz[2] * B[i3][0];
        }
      }
      Five acc[5];  // [i1], z-classes, of i2 = j
#pragma unroll
      for (int i1 = 0; i1 < 5; i1++) acc[i1].clear();
#pragma unroll 1
      for (int ox = 0; ox < 3; ox++) {
        Five Y[5];  // [i2], z-classes, of k1 = j
#pragma unroll
        for (int i2 = 0; i2 < 5; i2++) Y[i2].clear();
#pragma unroll 1
        for (int oy = 0; oy < 3; oy++) {
          const float* fq = corner + (oy * SX + ox) * NS + 20 * j;
          const float* fs = corner + (oy * SX + ox) * NS + 100 + 5 * j;
          const float* gy = sm.gy[warp][n][oy];
#pragma unroll
          for (int k2 = 0; k2 < 5; k2++) {
            Five v[3];
#pragma unroll
            for (int oz = 0; oz < 3; oz++) v[oz].load(fq + oz * (SX * SY * NS) + 4 * k2, fs + oz * (SX * SY * NS) + k2);
            float z[5];
#pragma unroll
            for (int i3 = 0; i3 < 5; i3++) {
              float2 p = __fmul2_rn(c01[i3], make_float2(v[0].s, v[1].s));
#pragma unroll
              for (int oz = 0; oz < 3; oz++) {
                p = __ffma2_rn(cp[oz][i3][0], v[oz].a, p);
                p = __ffma2_rn(cp[oz][i3][1], v[oz].b, p);
              }
              z[i3] = fmaf(c2[i3], v[2].s, p.x) + p.y;
            }
            Five Z, g;
            Z.a = make_float2(z[1], z[2]); Z.b = make_float2(z[3], z[4]); Z.s = z[0];
            g.load(gy + 4 * k2, gy + 20 + k2);
#pragma unroll
            for (int i2 = 0; i2 < 5; i2++) Y[i2].add(g.get(i2), Z);
          }
        }
#pragma unroll
        for (int i2 = 0; i2 < 5; i2++) Y[i2].store(ex + lane * 28 + 4 * i2, ex + lane * 28 + 20 + i2);
        __syncwarp();
        const float* gx = sm.gx[warp][n][ox];
#pragma unroll
        for (int k1 = 0; k1 < 5; k1++) {
          Five w, g;
          w.load(ex + (5 * n + k1) * 28 + 4 * j, ex + (5 * n + k1) * 28 + 20 + j);
          g.load(gx + 4 * k1, gx + 20 + k1);
#pragma unroll
          for (int i1 = 0; i1 < 5; i1++) acc[i1].add(g.get(i1), w);
        }
        __syncwarp();
      }
      if (!(C >= 1.0e-300)) {  // target T = 0: every transfer term is non-finite and dropped
#pragma unroll
        for (int i1 = 0; i1 < 5; i1++) acc[i1].clear();
      }
      // calcMoments in float64 (structs.cuh:315-342): this lane's share through its
      // sums over i1 and over i3, then the five lanes of the node in a fixed order
      double mv[5] = {0, 0, 0, 0, 0};
      bool ok = true;
      {
        double s1[5] = {0, 0, 0, 0, 0}, s3[5] = {0, 0, 0, 0, 0};
#pragma unroll
        for (int i1 = 0; i1 < 5; i1++)
#pragma unroll
          for (int i3 = 0; i3 < 5; i3++) {
            const double nv = acc[i1].get(i3), ov = f0[i1][i3];
            s1[i1] += nv;
            s3[i3] += nv;
            ok = ok && !(fabs(nv - ov) >= a.tol_abs + a.tol_rel * fabs(nv));
          }
        const double vy = C * d125t::xi5(j) + U[1];
        mv[0] = ((s1[0] + s1[1]) + (s1[2] + s1[3])) + s1[4];
        mv[2] = mv[0] * vy;
        mv[4] = mv[2] * vy;
#pragma unroll
        for (int q = 0; q < 5; q++) {
          const double vx = C * d125t::xi5(q) + U[0], vz = C * d125t::xi5(q) + U[2];
          const double px = s1[q] * vx, pz = s3[q] * vz;
          mv[1] += px;
          mv[3] += pz;
          mv[4] += px * vx + pz * vz;
        }
      }
      double m[5];
#pragma unroll
      for (int q = 0; q < 5; q++) {
        double s = __shfl_sync(0xffffffffu, mv[q], 5 * n);
#pragma unroll
        for (int d = 1; d < 5; d++) s += __shfl_sync(0xffffffffu, mv[q], 5 * n + d);
        m[q] = s;
      }
      const double rho = m[0];
      if (rho != 0) {
        const double ir = 1.0 / rho;
#pragma unroll
        for (int q = 1; q < 5; q++) m[q] *= ir;
      }
      double Tn = (m[4] - m[1] * m[1] - m[2] * m[2] - m[3] * m[3]) * (1.0 / L::Dim);
      if (Tn < 0) Tn = Tc;  // steps.cu:475
#pragma unroll
      for (int q = 0; q < 3; q++) ok = ok && !(fabs(m[1 + q] - U[q]) >= a.tolg_abs + a.tolg_rel * fabs(m[1 + q]));
      ok = ok && !(fabs(Tn - Tc) >= a.tolg_abs + a.tolg_rel * fabs(Tn));
      const unsigned votes = __ballot_sync(0xffffffffu, ok);
      if (!done) {
#pragma unroll
        for (int i1 = 0; i1 < 5; i1++)
#pragma unroll
          for (int i3 = 0; i3 < 5; i3++) f0[i1][i3] = acc[i1].get(i3);
        rho0 = rho; U[0] = m[1]; U[1] = m[2]; U[2] = m[3]; Tc = Tn;
        conv = ((votes >> (5 * n)) & 31u) == 31u;
        done = conv || niter >= a.max_iter;
      }
    }
    // BGK and store (steps.cu:230-248)
    if (worker && active) {
      const float rr = float(rho0), dtau = float(a.dtau);
#pragma unroll
      for (int i1 = 0; i1 < 5; i1++)
#pragma unroll
        for (int i3 = 0; i3 < 5; i3++) {
          const int p = 25 * i1 + 5 * j + i3;
          a.f_out[(long long)p * a.N + idx] =
              f0[i1][i3] + dtau * (rr * float(lattice_weight_t<POND_D3Q125>(p)) - f0[i1][i3]);
        }
      if (j == 0) {
        const float u0 = float(U[0]), u1 = float(U[1]), u2 = float(U[2]), ts = float(Tc);
        a.rho_out[idx] = rr;
        a.g_out[idx] = u0; a.g_out[a.N + idx] = u1; a.g_out[2 * a.N + idx] = u2; a.g_out[3 * a.N + idx] = ts;
        if (a.niter_out) a.niter_out[idx] = niter;
        const double dr = rr, d0 = u0, d1 = u1, d2 = u2, dt = ts;
        const double u2s = d0 * d0 + d1 * d1 + d2 * d2;
        ns.mass += dr; ns.m0 += dr * d0; ns.m1 += dr * d1; ns.m2 += dr * d2;
        ns.enrg += dr * (u2s + L::Dim * dt);
        ns.k += a.kdx * u2s;
        ns.niter += niter; ns.nonconv += conv ? 0 : 1; ns.nmax = max(ns.nmax, niter);
        ns.work += 27ull * niter;
      }
    }
  }
  reduce_and_commit(ns, a.sums);
}

}  // namespace d125r
}  // namespace pond
