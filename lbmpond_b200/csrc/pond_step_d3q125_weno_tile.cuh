// D3Q125 PonD pull step with the centred WENO5 (POND_WENO5_ROW), float32: a
// tile of nodes per CTA, a warp per node at a time.
//
// The arithmetic is pull_weno3d_kernel's centred variant (propagateWENO<3,5>,
// steps.cu:774-825, with the y/z windows centred): three quadratic
// candidates on x nodes fx-2+s .. fx+s, y nodes fy-1 .. fy+1 and z nodes
// fz-1 .. fz+1 (fx = floor(crd.x+0.5), likewise fy, fz), blended with
// Jiang-Shu weights from five transferred values on the row
// (fx-2 .. fx+2, fy, fz).  Organised for the SM:
//
//  * a CTA owns a 4 x 2 x 2 tile and stages it once per step with the halo
//    the windows reach while |v| < 1.5 along every axis: 3 nodes on both
//    sides in x, 2 in y and z (10 x 6 x 6 nodes, node-major, 190 KB: per
//    (k1, k2) the quad k3 = 1..4, then the 25 singles k3 = 0);
//  * every staged node is transferred into the tile's reference gauge R
//    once, five lanes per node (three passes of the 5x5 basis); the transfer
//    of a source node into a target gauge equals R -> target applied to its
//    R-gauge populations, since the 5-point basis reproduces every quartic in
//    the particle velocity;
//  * eight warps step the 16 tile nodes, one node at a time, the lanes
//    splitting the 125 populations by two classes: lane 5 k1 + k2 transfers
//    the z classes of every stencil column, so one 16-byte and one 4-byte
//    load serve the 15 (class, node) products that the column's three-node
//    windows need; the column goes through shared memory to lane 5 k1 + i3,
//    which transfers and weights the target y-classes whose window holds it;
//    the row goes to lane 5 i2 + i3, which transfers the target x-classes and
//    keeps their five window values (weighted in y and z, and the smoothness
//    row); the three candidates and the blend follow at the end.  The windows
//    are the same for the whole warp, so classes a column or row does not
//    serve are skipped by uniform branches, and the usual z windows (the
//    fastest class on each side one node off centre) run as straight-line
//    code;
//  * a warp whose node's windows leave the staged halo runs that iteration
//    from global memory (the group transfer of pull_weno3d_kernel).
//
// What bounds it: an iteration is ~90,000 multiply-adds per node (30 columns of
// 15 (class, node) z products for 25 (k1, k2), against 150 sites each
// transferred for every class before) at two warps per scheduler; staging 360
// nodes for 16 is a fifth of a three-iteration step.  48^3 shock and vortex,
// 2.97 iterations per node: 7.6 ms per step, 1.95 ms per iteration; the form it
// replaces (every class at every site, one scalar shared load per
// multiply-add) took 15.9 and 4.1 ms.
#pragma once
#include <cstddef>

#include "pond_step_d3q125_rows.cuh"
#include "pond_step_d3q125_tile.cuh"
#include "pond_step_weno3d.cuh"

namespace pond {
namespace d125w {

constexpr int TX = 4, TY = 2, TZ = 2;      // tile
constexpr int HXL = 3, HXH = 3, HL = 2, HH = 2;  // halo: x both sides; y and z below / above
constexpr int SX = TX + HXL + HXH, SY = TY + HL + HH, SZ = TZ + HL + HH;
constexpr int SN = SX * SY * SZ;  // 360 staged nodes
constexpr int ROWS = SY * SZ;
constexpr int NS = 132;           // floats per staged node (4 mod 32: the transfer's node groups fall on distinct banks)
constexpr int NODES = TX * TY * TZ;
constexpr int WARPS = 8;  // each warp steps NODES / WARPS tile nodes in turn
constexpr int THREADS = 32 * WARPS;

using d125r::Five;
using d125r::basis5;
using d125r::dot5;

struct alignas(16) WarpTables {  // of the node a warp is stepping, rewritten every iteration
  float ex1[25 * 12]; // lane 5 k1 + k2: the column's z classes, weighted [0..4] and on the middle node [5..9]
  float ex2[25 * 12]; // lane 5 k1 + i3: the row's y classes, the same two
  float t[3][28];     // R -> target transfer of z, y, x: quads [4 i + k - 1], singles [20 + i]
  float w[2][16];     // z and y window weights [3 i + j]
  float lx[5][12];    // x candidate weights [3 s + j]
  double cdist[5];    // departure point to rounded node along x
  int b[3][8];        // window starts of z, y, x, relative to the node
};
struct Smem {
  float f[SN * NS];         // staged populations, then their transfer into R
  float u[3][SN];           // staged velocities (sign-flipped on mirrored axes)
  float c[SN];              // sqrts(T / TLat)
  int g[SN];                // global node (-1: the inflow ghost)
  unsigned char flags[SN];  // mirrored axes (bits 0-2)
  WarpTables wt[WARPS];
};
static_assert(sizeof(Smem) + 4096 <= 232448 && offsetof(Smem, wt) % 16 == 0, "the tile must fit one CTA");

// staged node i -> global node (-1: the inflow ghost) and mirror flags
__device__ __forceinline__ int staged_global(const StepArgs<float>& a, int x0, int y0, int z0, int i, bool rv[3]) {
  const int hx = i % SX, hy = (i / SX) % SY, hz = i / (SX * SY);
  bool ghost = false;
  const int gx = d125t::staged_axis(x0 - HXL + hx, a.nx, a.bc[0], rv[0], ghost);
  const int gy = d125t::staged_axis(y0 - HL + hy, a.ny, a.bc[1], rv[1], ghost);
  const int gz = d125t::staged_axis(z0 - HL + hz, a.nz, a.bc[2], rv[2], ghost);
  if (ghost) { rv[0] = rv[1] = rv[2] = false; return -1; }
  return gx + a.nx * (gy + a.ny * gz);
}

// weno5_blend with its weights over a common denominator: one division.  The
// products stay finite for smoothness indicators up to 1e76 of each other's
// scale; beyond that the separate quotients decide.
__device__ __forceinline__ double blend(const double S[3], const double u[5], double c) {
  const double d0 = (c * c - 3 * c + 2) * (1.0 / 12.0);
  const double d2 = (c * c + 3 * c + 2) * (1.0 / 12.0);
  const double d1 = 1. - d0 - d2;
  const double u1 = u[0], u2 = u[1], u3 = u[2], u4 = u[3], u5 = u[4];
  const double b0 = (10 * u3 * u3 + (11 * u1 - 31 * u2) * u3 + 25 * u2 * u2 - 19 * u1 * u2 + 4 * u1 * u1) * (1.0 / 3.0);
  const double b1 = (4 * u4 * u4 + (5 * u2 - 13 * u3) * u4 + 13 * u3 * u3 - 13 * u2 * u3 + 4 * u2 * u2) * (1.0 / 3.0);
  const double b2 = (4 * u5 * u5 + (11 * u3 - 19 * u4) * u5 + 25 * u4 * u4 - 31 * u3 * u4 + 10 * u3 * u3) * (1.0 / 3.0);
  const double q0 = (1e-6 + b0) * (1e-6 + b0), q1 = (1e-6 + b1) * (1e-6 + b1), q2 = (1e-6 + b2) * (1e-6 + b2);
  const double w0 = d0 * (q1 * q2), w1 = d1 * (q0 * q2), w2 = d2 * (q0 * q1);
  const double ws = w0 + w1 + w2;
  if (!(fabs(ws) < 1e300 && fabs(ws) > 1e-300)) return w3d::weno5_blend(S, u, c);
  return (w0 * S[0] + w1 * S[1] + w2 * S[2]) / ws;
}

__global__ void __launch_bounds__(THREADS, 1) pull_d3q125_weno_tile_kernel(StepArgs<float> a) {
  using L = Lattice<POND_D3Q125>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, z0 = blockIdx.z * TZ;

  // ---- the gauge and the global index of every staged node
  for (int i = tid; i < SN; i += THREADS) {
    bool rv[3];
    const int g = staged_global(a, x0, y0, z0, i, rv);
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
  // ---- the populations: a warp copies the ten nodes of a row times three
  //      planes, row after row
  {
    const int n = lane % SX, j = lane / SX;
    for (int t = warp; t < 42; t += WARPS) {  // planes 3 t + j
      const int p = 3 * t + j;
      if (j >= 3 || p >= 125) continue;
      const int k12 = p / 5, k3 = p % 5;
      float* dst = sm.f + n * NS + (k3 > 0 ? 4 * k12 + k3 - 1 : 100 + k12);
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

  // ---- reference gauge R: the staged gauge of tile node (2, 1, 1)
  //      ((0, 1) if that gauge is not finite or its c is 0)
  float uref[3], cref;
  {
    constexpr int ci = ((1 + HL) * SY + (1 + HL)) * SX + (2 + HXL);
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
  // ---- every staged node into R: lane 5n + j takes x-class j of a node through
  //      the z and y passes of the 5x5 basis, then y-class j through the x pass;
  //      non-finite populations count as 0, a node with a non-finite gauge as all 0
  {
    const bool part = lane < 30;
    const int n = part ? lane / 5 : 5, j = part ? lane % 5 : lane - 30;
    // the exchange (20 floats of each of the 32 lanes) uses this warp's table space
    static_assert(sizeof(WarpTables) >= 32 * 20 * sizeof(float), "room for the transfer's exchange");
    float* ex = reinterpret_cast<float*>(&sm.wt[warp]);
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
      // y-classes 1..4 (quads) go over in one exchange, then y-class 0
      Five y[5];
#pragma unroll
      for (int i2 = 0; i2 < 5; i2++) {
        y[i2].scale(B[i2][0], w[0]);
#pragma unroll
        for (int k2 = 1; k2 < 5; k2++) y[i2].add(B[i2][k2], w[k2]);
      }
#pragma unroll
      for (int i2 = 0; i2 < 5; i2++)
        *reinterpret_cast<float4*>(ex + lane * 20 + 4 * i2) = make_float4(y[i2].a.x, y[i2].a.y, y[i2].b.x, y[i2].b.y);
      __syncwarp();
#pragma unroll
      for (int k1 = 0; k1 < 5; k1++) {
        const float4 q = *reinterpret_cast<const float4*>(ex + (5 * n + k1) * 20 + 4 * j);
        w[k1].a = make_float2(q.x, q.y);
        w[k1].b = make_float2(q.z, q.w);
      }
      __syncwarp();
#pragma unroll
      for (int i2 = 0; i2 < 5; i2++) ex[lane * 5 + i2] = y[i2].s;
      __syncwarp();
#pragma unroll
      for (int k1 = 0; k1 < 5; k1++) w[k1].s = ex[(5 * n + k1) * 5 + j];
      __syncwarp();
      basis5(sq[0], rq[0], B);
#pragma unroll
      for (int i1 = 0; i1 < 5; i1++) {
        Five t;
        t.scale(B[i1][0], w[0]);
#pragma unroll
        for (int k1 = 1; k1 < 5; k1++) t.add(B[i1][k1], w[k1]);
        if (!ok) t.clear();
        if (part) t.store(fi + 20 * i1 + 4 * j, fi + 100 + 5 * i1 + j);
      }
    }
  }
  __syncthreads();

  // ---- one warp per tile node.  Lane 5 h + l: h = k1 and l = k2 along z, h = k1
  //      and l = i3 along y, h = i2 and l = i3 along x and for the output.  Idle
  //      lanes (25..31) compute like lane 20 + l and write nothing.
  const bool worker = lane < 25;
  const int h = worker ? lane / 5 : 4, l = lane % 5;
  const int slot = 5 * h + l;
  WarpTables& wt = sm.wt[warp];
  NodeSums ns = {0, 0, 0, 0, 0, 0, 0ull, 0ull, 0ull, 0};
#pragma unroll 1
  for (int t = warp; t < NODES; t += WARPS) {
    const int lx = t % TX, ly = (t / TX) % TY, lz = t / (TX * TY);
    const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
    if (x < a.nx && y < a.ny && z < a.nz) {  // warp-uniform
      const long long idx = x + (long long)a.nx * (y + (long long)a.ny * z);
      float f0[5];  // [i1] of i2 = h, i3 = l
#pragma unroll
      for (int i1 = 0; i1 < 5; i1++) f0[i1] = a.f_in[(long long)(25 * i1 + slot) * a.N + idx];
      double rho0 = a.rho_in[idx];
      double U[3] = {(double)a.g_in[idx], (double)a.g_in[a.N + idx], (double)a.g_in[2 * a.N + idx]};
      double Tc = a.g_in[3 * a.N + idx];
      if (rho0 == 0 && U[0] == 0 && U[1] == 0 && U[2] == 0 && Tc == 0) {  // set_base(1, TLat)
        rho0 = 1; Tc = L::TLat;
#pragma unroll
        for (int i1 = 0; i1 < 5; i1++) f0[i1] = float(lattice_weight_t<POND_D3Q125>(25 * i1 + slot));
      }
      if (a.guess) {
        U[0] = a.guess[idx]; U[1] = a.guess[a.N + idx]; U[2] = a.guess[2 * a.N + idx]; Tc = a.guess[3 * a.N + idx];
      }
      const float* centre = sm.f + (((lz + HL) * SY + (ly + HL)) * SX + (lx + HXL)) * NS;
      int niter = 0;
      bool conv = false;
      unsigned long long work = 0;
      while (niter < a.max_iter) {
        niter++;
        const double C = sqrt(Tc / L::TLat);
        // transfer R -> target per axis: G[i][k] = L_i(b + a xi_k), a = c_ref/C, b = (u_ref - U)/C;
        // lane 5 i + k writes its entry of the three axes, lanes 0-4 / 5-9 / 10-14 the
        // windows of their z / y / x class
        bool inside = true;
        __syncwarp();  // the previous iteration's readers are done
        {
          const double iC = 1.0 / C;
          const float ga = float(double(cref) * iC);
          const d125t::BasisRowT<float> Lh(h);
          if (worker) {
            const int e = l > 0 ? 4 * h + l - 1 : 20 + h;
#pragma unroll
            for (int ax = 0; ax < 3; ax++) {
              const float gb = float((double(uref[2 - ax]) - U[2 - ax]) * iC);
              wt.t[ax][e] = finite_or_zero_f(Lh(fmaf(ga, d125t::xi5r<float>(l), gb)));
            }
          }
          if (lane < 15) {
            const int ax = lane / 5;  // 0: z, 1: y, 2: x
            const int pos = ax == 0 ? z : ax == 1 ? y : x;
            const double crd = double(pos) - (C * d125t::xi5(l) + (ax == 0 ? U[2] : ax == 1 ? U[1] : U[0]));
            const double fd = floor(crd + 0.5);
            const int b = w3d::clamp_off((int)(fd - (ax == 2 ? 0.0 : 1.0)) - (ax == 2 ? 2 : 0) - pos);
            wt.b[ax][l] = b;
            if (ax == 2) {
              wt.cdist[l] = crd - fd;
#pragma unroll
              for (int s = 0; s < 3; s++) lagr_weights<3, float>(crd - (fd - 2 + s), &wt.lx[l][3 * s]);
              inside = b >= -HXL && b + 4 <= HXH;
            } else {
              lagr_weights<3, float>(crd - (fd - 1), &wt.w[ax][3 * l]);
              inside = b >= -HL && b + 2 <= HH;
            }
          }
        }
        __syncwarp();
        float acc[5];
        if (__all_sync(0xffffffffu, inside)) {
          Five tz[5];
          float wz[5][3];
          int bz[5], by[5];
#pragma unroll
          for (int i = 0; i < 5; i++) {
            tz[i].load(&wt.t[0][4 * i], &wt.t[0][20 + i]);
#pragma unroll
            for (int k = 0; k < 3; k++) wz[i][k] = wt.w[0][3 * i + k];
            bz[i] = wt.b[0][i];
            by[i] = wt.b[1][i];
          }
          int ylo = by[0], yhi = by[0], xlo = wt.b[2][0], xhi = xlo, zlo = bz[0], zhi = bz[0];
#pragma unroll
          for (int i = 1; i < 5; i++) {
            ylo = min(ylo, by[i]); yhi = max(yhi, by[i]);
            zlo = min(zlo, bz[i]); zhi = max(zhi, bz[i]);
            xlo = min(xlo, wt.b[2][i]); xhi = max(xhi, wt.b[2][i]);
          }
          work += (unsigned long long)(xhi - xlo + 5) * (yhi - ylo + 3) * (zhi - zlo + 3);
          const bool usual = bz[0] == -1 && bz[1] == -1 && bz[2] == -1 && bz[3] == -2 && bz[4] == 0;
          float tx5[5][5], ux5[5][5];  // [i1][window node]: weighted in y and z; on the smoothness row
#pragma unroll
          for (int i1 = 0; i1 < 5; i1++)
#pragma unroll
            for (int m = 0; m < 5; m++) tx5[i1][m] = ux5[i1][m] = 0.f;
#pragma unroll 1
          for (int ox = xlo; ox <= xhi + 4; ox++) {
            float Y[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, Yd[5] = {0.f, 0.f, 0.f, 0.f, 0.f};  // [i2] of k1 = h, i3 = l
#pragma unroll 1
            for (int oy = ylo; oy <= yhi + 2; oy++) {
              const float* col = centre + (oy * SX + ox) * NS;
              float A[5], D[5];  // [i3] of k1 = h, k2 = l
              if (usual) {
                Five v[5];
#pragma unroll
                for (int o = 0; o < 5; o++) {
                  const float* q = col + (o - 2) * (SX * SY * NS);
                  v[o].load(q + 4 * slot, q + 100 + slot);
                }
#pragma unroll
                for (int i3 = 0; i3 < 5; i3++) {
                  const int o = i3 == 3 ? 0 : i3 == 4 ? 2 : 1;
                  const float r0 = dot5(tz[i3], v[o]), r1 = dot5(tz[i3], v[o + 1]), r2 = dot5(tz[i3], v[o + 2]);
                  A[i3] = fmaf(wz[i3][2], r2, fmaf(wz[i3][1], r1, wz[i3][0] * r0));
                  D[i3] = r1;
                }
              } else {
#pragma unroll
                for (int i3 = 0; i3 < 5; i3++) A[i3] = D[i3] = 0.f;
#pragma unroll 1
                for (int oz = zlo; oz <= zhi + 2; oz++) {
                  Five v;
                  const float* q = col + oz * (SX * SY * NS);
                  v.load(q + 4 * slot, q + 100 + slot);
#pragma unroll
                  for (int i3 = 0; i3 < 5; i3++) {
                    const int k = oz - bz[i3];
                    if (k >= 0 && k <= 2) {
                      const float r = dot5(tz[i3], v);
                      A[i3] = fmaf(k == 0 ? wz[i3][0] : k == 1 ? wz[i3][1] : wz[i3][2], r, A[i3]);
                      if (k == 1) D[i3] = r;
                    }
                  }
                }
              }
              // to the lanes (k1, i3)
              if (worker) {
                float4* e = reinterpret_cast<float4*>(wt.ex1 + 12 * slot);
                e[0] = make_float4(A[0], A[1], A[2], A[3]);
                e[1] = make_float4(A[4], D[0], D[1], D[2]);
                *reinterpret_cast<float2*>(e + 2) = make_float2(D[3], D[4]);
              }
              __syncwarp();
              Five zc, zd;
              {
                const float* e = wt.ex1 + 12 * (5 * h) + l;
                zc.s = e[0]; zc.a = make_float2(e[12], e[24]); zc.b = make_float2(e[36], e[48]);
                zd.s = e[5]; zd.a = make_float2(e[17], e[29]); zd.b = make_float2(e[41], e[53]);
              }
              __syncwarp();
#pragma unroll
              for (int i2 = 0; i2 < 5; i2++) {
                const int k = oy - by[i2];
                if (k >= 0 && k <= 2) {  // warp-uniform
                  Five ty;
                  ty.load(&wt.t[1][4 * i2], &wt.t[1][20 + i2]);
                  Y[i2] = fmaf(wt.w[1][3 * i2 + k], dot5(ty, zc), Y[i2]);
                  if (k == 1) Yd[i2] = dot5(ty, zd);
                }
              }
            }
            // the row, to the lanes (i2, i3)
            if (worker) {
              float4* e = reinterpret_cast<float4*>(wt.ex2 + 12 * slot);
              e[0] = make_float4(Y[0], Y[1], Y[2], Y[3]);
              e[1] = make_float4(Y[4], Yd[0], Yd[1], Yd[2]);
              *reinterpret_cast<float2*>(e + 2) = make_float2(Yd[3], Yd[4]);
            }
            __syncwarp();
            Five yc, yd;
            {  // [k1] of i2 = h, i3 = l: written by lanes 5 k1 + l
              const float* e = wt.ex2 + 12 * l + h;
              yc.s = e[0]; yc.a = make_float2(e[60], e[120]); yc.b = make_float2(e[180], e[240]);
              yd.s = e[5]; yd.a = make_float2(e[65], e[125]); yd.b = make_float2(e[185], e[245]);
            }
            __syncwarp();
#pragma unroll
            for (int i1 = 0; i1 < 5; i1++) {
              const int k = ox - wt.b[2][i1];
              if (k >= 0 && k <= 4) {  // warp-uniform
                Five tx;
                tx.load(&wt.t[2][4 * i1], &wt.t[2][20 + i1]);
                const float tc = dot5(tx, yc), td = dot5(tx, yd);
#pragma unroll
                for (int m = 0; m < 5; m++) {
                  tx5[i1][m] = k == m ? tc : tx5[i1][m];
                  ux5[i1][m] = k == m ? td : ux5[i1][m];
                }
              }
            }
          }
          // the three candidates and the blend
#pragma unroll
          for (int i1 = 0; i1 < 5; i1++) {
            double S[3], u[5];
#pragma unroll
            for (int s = 0; s < 3; s++) {
              const float* w = &wt.lx[i1][3 * s];
              S[s] = double(fmaf(w[2], tx5[i1][s + 2], fmaf(w[1], tx5[i1][s + 1], w[0] * tx5[i1][s])));
            }
#pragma unroll
            for (int m = 0; m < 5; m++) u[m] = double(ux5[i1][m]);
            acc[i1] = (C >= 1.0e-300) ? float(blend(S, u, wt.cdist[i1])) : 0.f;  // target T = 0: terms dropped
          }
        } else {
          // a window leaves the staged halo: this iteration from global memory, lane (p, k)
          // with every y-class, and over to the lanes (i2, i3) through shared memory
          const int j = h, k = l;
          const double crdx = double(x) - (C * L::xi1(j) + U[0]);
          const double fxd = floor(crdx + 0.5);
          const double cdist = crdx - fxd;
          const int bx = w3d::clamp_off((int)fxd - 2 - x);
          float LX[3][3];
#pragma unroll
          for (int s = 0; s < 3; s++) lagr_weights<3, float>(crdx - (fxd - 2 + s), LX[s]);
          const double crdz = double(z) - (C * L::xi1(k) + U[2]);
          const double fzd = floor(crdz + 0.5) - 1;
          const int bz = w3d::clamp_off((int)fzd - z);
          float WZ[3];
          lagr_weights<3, float>(crdz - fzd, WZ);
          int by[5];
          float WY[5][3];
#pragma unroll
          for (int i2 = 0; i2 < 5; i2++) {
            const double crdy = double(y) - (C * L::xi1(i2) + U[1]);
            const double fyd = floor(crdy + 0.5) - 1;
            by[i2] = w3d::clamp_off((int)fyd - y);
            lagr_weights<3, float>(crdy - fyd, WY[i2]);
          }
          float S[3][5], U5[5][5];
          const float Uc[3] = {float(U[0]), float(U[1]), float(U[2])};
          w3d::accumulate_global<POND_D3Q125, float, true>(a, x, y, z, !worker, 0, j, k, Uc, float(1.0 / C), bx, LX,
                                                           bz, WZ, by, WY, S, U5, work, true);
          __syncwarp();
#pragma unroll
          for (int i2 = 0; i2 < 5; i2++) {
            const double Sd[3] = {double(S[0][i2]), double(S[1][i2]), double(S[2][i2])};
            const double ud[5] = {double(U5[0][i2]), double(U5[1][i2]), double(U5[2][i2]), double(U5[3][i2]),
                                  double(U5[4][i2])};
            if (worker) wt.ex1[25 * j + 5 * i2 + k] = (C >= 1.0e-300) ? float(w3d::weno5_blend(Sd, ud, cdist)) : 0.f;
          }
          __syncwarp();
#pragma unroll
          for (int i1 = 0; i1 < 5; i1++) acc[i1] = wt.ex1[25 * i1 + slot];
        }
        // calcMoments (structs.cuh:315-342) in float64, warp-wide
        double mv[5] = {0, 0, 0, 0, 0};
        if (worker) {
          const double vy = C * d125t::xi5(h) + U[1], vz = C * d125t::xi5(l) + U[2];
#pragma unroll
          for (int i1 = 0; i1 < 5; i1++) {
            const double fv = acc[i1], vx = C * L::xi1(i1) + U[0];
            mv[0] += fv; mv[1] += fv * vx; mv[2] += fv * vy; mv[3] += fv * vz;
            mv[4] += fv * (vx * vx + vy * vy + vz * vz);
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int q = 0; q < 5; q++) mv[q] += __shfl_xor_sync(0xffffffffu, mv[q], o);
        const double rho = mv[0];
        double m[4] = {mv[1], mv[2], mv[3], mv[4]};
        if (rho != 0) {
          const double ir = 1.0 / rho;
#pragma unroll
          for (int q = 0; q < 4; q++) m[q] *= ir;
        }
        double Tn = (m[3] - m[0] * m[0] - m[1] * m[1] - m[2] * m[2]) * (1.0 / L::Dim);
        if (Tn < 0) Tn = Tc;  // steps.cu:475
        bool ok = true;
#pragma unroll
        for (int q = 0; q < 3; q++) ok = ok && !(fabs(m[q] - U[q]) >= a.tolg_abs + a.tolg_rel * fabs(m[q]));
        ok = ok && !(fabs(Tn - Tc) >= a.tolg_abs + a.tolg_rel * fabs(Tn));
        if (worker)
#pragma unroll
          for (int i1 = 0; i1 < 5; i1++) {
            const double nv = acc[i1], ov = f0[i1];
            ok = ok && !(fabs(nv - ov) >= a.tol_abs + a.tol_rel * fabs(nv));
          }
        const bool all_ok = __all_sync(0xffffffffu, ok);
#pragma unroll
        for (int i1 = 0; i1 < 5; i1++) f0[i1] = acc[i1];
        rho0 = rho; U[0] = m[0]; U[1] = m[1]; U[2] = m[2]; Tc = Tn;
        if (all_ok) { conv = true; break; }
      }
      // BGK toward rho*w_i (steps.cu:557-564) and store
      const float rr = float(rho0), dtau = float(a.dtau);
      if (worker)
#pragma unroll
        for (int i1 = 0; i1 < 5; i1++) {
          const int p = 25 * i1 + slot;
          a.f_out[(long long)p * a.N + idx] = f0[i1] + dtau * (rr * float(lattice_weight_t<POND_D3Q125>(p)) - f0[i1]);
        }
      if (lane == 0) {
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
        ns.work += work;
      }
    }
  }
  reduce_and_commit(ns, a.sums);
}

}  // namespace d125w
}  // namespace pond
