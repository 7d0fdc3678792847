// D3Q27 PonD pull step, float32, one thread per node with the stencil tile
// staged in shared memory (the hot kernel of the 256^3 benchmark).
//
// Same arithmetic as pull_point_kernel (steps.cu:356-588 LBMpull with
// propagate<N>, N = 2, 3, 4), organised for the SM:
//
//  * a CTA owns an 8 x 4 x 4 tile of nodes (order 3: 32 x 4 x 2, see Tile) and
//    stages the tile plus a halo of
//    2 nodes per side (12 x 8 x 8 nodes) once per step, node-major: a staged
//    node's 27 populations are contiguous and 16-byte aligned (a 28-float
//    stride, 86 KB), so a lane fetches a stencil node with seven 16-byte
//    loads, and the 28-word stride puts the eight lanes of every 16-byte load
//    phase on distinct banks.  Two CTAs share an SM (110 KB and 128 threads
//    of 255 registers each): one stages while the other iterates, and neither
//    waits for the other's slowest warp.  Each staging thread copies whole
//    nodes with their gauges, all copies in flight at once, and transfers them
//    itself.
//    Boundary resolution (periodic wrap, clamp, mirror with population
//    reversal), the reference's dropping of non-finite terms and the square
//    root of T are applied while staging;
//  * after staging, each staged node's 27 populations are replaced by their
//    transfer into a reference gauge shared by the CTA (the gauge of the
//    tile's centre node).  The transfer of a source node into a target gauge
//    (U, C), sum_b prod_ax L_i(y_b) f_b with y = (v_b - U)/C and L_i the
//    quadratic Lagrange basis over the target classes, is a quadratic in the
//    particle velocity v_b along each axis, so it equals the transfer from
//    the reference gauge to (U, C), G[i][k] = L_i((u_ref + c_ref xi_k - U)/C),
//    applied to the reference-gauge populations.  G depends on the target
//    alone: the interpolation weights and G are contracted against the
//    reference-gauge populations one axis at a time (z per stencil node, y
//    per stencil column, x per stencil row: 81 FMA each) instead of
//    transforming every stencil node into the target gauge (243 FMA);
//  * the fixed-point iteration is warp-synchronous: a warp (an 8 x 4 patch of
//    one z plane) iterates while any of its lanes is unconverged and walks the
//    union of its lanes' stencil offsets, contracting every target class at
//    every offset (a class a lane does not weight there has weight 0), except
//    at the two ends of the usual z window (contract_tile);
//  * once only a few lanes of a warp still iterate, the warp serves their nodes
//    one at a time, a stencil column per lane, with the same roundings: a node
//    that runs to the iteration cap then takes 2 us per iteration instead of 11
//    to 20, which is what the end of a step waited for (128^3 vortex with nodes
//    at the cap, order 3: 4.22 -> 3.88 ms; two steps with energy populations at
//    64^3: 4.11 -> 2.58 ms);
//  * the z and y contractions run as two-wide float32 multiply-adds on pairs
//    of populations that the staged layout keeps in neighbouring registers
//    (slot27): 45 instructions per stencil node instead of 81, for the same
//    81 multiply-adds with the same roundings.
//
// What bounds it: the 128 B/clk of shared memory and, at two warps per
// scheduler, latency.  A stencil node costs 28 wavefronts per warp and 20-23
// cycles of the SM's FMA pipes, so an iteration of 125 nodes takes at least
// 3,500 cycles per warp of its SM: 19 ms of the 27.9 ms that a 256^3 step of a
// half-uniform blast takes (46.1 ms in the earlier form: 32 x 4 x 2 tiles, one
// CTA of 256 threads per SM, scalar multiply-adds, rolled z offsets).  Of that
// the first form of this kernel took 30.0; walking k3 outermost in the column
// node (1.0 ms), copying the gauges with the populations instead of loading
// them node by node (0.4), transferring staged nodes on pairs, keeping the
// tile's own populations while staging and shorter float64 sums (0.3) the rest.
// At 128^3, by ncu, in the first form: shared-memory wavefronts 70 % of peak,
// FMA pipe 52 % (the earlier form 40 %), issue slots 52 %.
#pragma once
#include "pond_step_point.cuh"

namespace pond {
namespace d27 {

constexpr int H = 2;    // halo
constexpr int NS = 28;  // floats per staged node: its 27 R-gauge populations and a pad
// Scratch of a warp for contract_node_by_warp that takes `rows` rows of five
// stencil columns at a time, in floats (27 each, from 16-byte boundaries).
__host__ __device__ constexpr int served_floats(int rows) { return (5 * 27 * rows + 3) / 4 * 4; }

// The tile of order N and its shared memory: the staged nodes (node-major, a
// node's populations contiguous, 16-byte aligned: seven 16-byte loads per
// stencil node; the 28-word stride keeps the eight lanes of each 16-byte load
// phase on distinct banks), the iterate's populations of every lane, the
// warps' scratch and the staged velocities.
//
// Orders 2 and 4: 8 x 4 x 4, two CTAs per SM.  Order 3: 32 x 4 x 2, one CTA of
// eight warps, its velocities staged in the iterates' place.  A quadratic
// window is chosen by rounding (x) and jumps where two windows meet, so a node
// whose iterates cycle between two of them turns the last digit of a transfer
// into 1e-3 of its populations; the reference gauge decides those digits, and
// order 3 keeps the gauge of 32 x 4 x 2 blocks that its results were checked
// with (26 boxes of 26 to 110 nodes a side, 1 to 8 steps: with an 8 x 4 x 4
// tile's gauge two came out 1e-6 and 2.9e-6 off float64 instead of 3e-7, and
// two others 2e-7 instead of 1.5e-6).  The wider tile costs a 128^3 vortex 3.88
// instead of 3.33 ms per step.
template <int N> struct Tile {
  static constexpr int TX = N == 3 ? 32 : 8, TY = 4, TZ = N == 3 ? 2 : 4;
  static constexpr int SX = TX + 2 * H, SY = TY + 2 * H, SZ = TZ + 2 * H;
  static constexpr int SN = SX * SY * SZ;  // staged nodes
  static constexpr int THREADS = TX * TY * TZ, WARPS = THREADS / 32, CTAS = N == 3 ? 1 : 2;
  static constexpr bool kOwnLater = N == 3;
  // the warps' scratch takes the velocities' place, or what is left of the SM's shared memory
  static constexpr int ROWS = N == 3 ? 2 : 5, SERVED = served_floats(ROWS);
  static constexpr int OFF_OWN = NS * SN, OFF_S = OFF_OWN + 27 * THREADS, OFF_U = kOwnLater ? OFF_OWN : OFF_S;
  static constexpr size_t SMEM_BYTES =
      size_t(kOwnLater || 3 * SN < SERVED * WARPS ? OFF_S + SERVED * WARPS : OFF_S + 3 * SN) * sizeof(float);
  static_assert(!kOwnLater || 3 * SN <= 27 * THREADS, "the velocities must fit the iterates' place");
  static_assert(CTAS * (SMEM_BYTES + 1024 + 2432) <= 233472, "the CTAs must fit in the 228 KB of an SM");
  // nodes: a warp takes an 8 x 4 patch of a z plane
  static __device__ __forceinline__ int lx(int tid) { return (tid & 7) + 8 * ((tid >> 5) % (TX / 8)); }
  static __device__ __forceinline__ int ly(int tid) { return (tid >> 3) & 3; }
  static __device__ __forceinline__ int lz(int tid) { return (tid >> 5) / (TX / 8); }
  static __device__ __forceinline__ int thread_of(int x, int y, int z) {
    return (x & 7) + 8 * y + 32 * ((x >> 3) + (TX / 8) * z);
  }
};

// Slot of class (k1, k2, k3) in a staged node: the contractions along z and y
// run on pairs of populations (two-wide float32 multiply-adds), so the
// classes k1 = +, - of each (k2, k3) are neighbours (slots 0-17), the k1 = 0
// classes k2 = +, - of each k3 (slots 18-23) and the three of k2 = 0 are last.
__host__ __device__ constexpr int slot27(int k1, int k2, int k3) {
  return k1 > 0 ? 2 * (3 * k3 + k2) + (k1 - 1) : k2 > 0 ? 18 + 2 * k3 + (k2 - 1) : 24 + k3;
}
__host__ __device__ constexpr int slot27(int t) { return slot27(t / 9, (t / 3) % 3, t % 3); }

// reference population index of tensor class t = 9 cx + 3 cy + cz, for
// lookups with run-time indices (consts.h:20-30 order)
__constant__ int c_ref27[27] = {0, 3, 16, 2, 6, 18, 12, 13, 24, 1, 5, 17, 4, 7, 19, 14, 15, 25,
                                8, 10, 22, 9, 11, 23, 20, 21, 26};

// 4-byte asynchronous global -> shared copy and the wait for all of them
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// class index -> its mirror image along one axis (0 <-> 0, + <-> -)
__device__ __forceinline__ int rev3(int c) { return c == 0 ? 0 : 3 - c; }

// Quadratic Lagrange basis over the classes xi = {0, +1, -1}, evaluated at
// s + r xi_b: B[i][b] = L_i(s + r xi_b) with L_0 = 1 - y^2,
// L_+ = y (y + 1) / 2, L_- = y (y - 1) / 2.  B is the one-axis gauge
// transfer (structs.cuh:343-551) from a gauge (u, c) to (U, C) for
// s = (u - U) / C, r = c / C.
template <typename R> __device__ __forceinline__ void basis_rows(R s, R r, R B[3][3]) {
  const R y[3] = {s, s + r, s - r};
#pragma unroll
  for (int b = 0; b < 3; b++) {
    const R yb = y[b], h = R(0.5) * yb;
    B[0][b] = fma(-yb, yb, R(1));
    B[1][b] = fma(h, yb, h);
    B[2][b] = fma(h, yb, -h);
  }
}

// Transfer of one node's 27 populations (tensor-class order), in place, into
// the gauge (u_ref, c_ref) shared by the CTA: per axis the 3x3 basis with
// s = (u - u_ref) / c_ref, r = c / c_ref.  A transfer into the target gauge
// then equals the transfer of the result from (u_ref, c_ref) to the target,
// because the basis reproduces every quadratic in the particle velocity.
template <typename R> __device__ __forceinline__ void node_to_ref(R v[27], const R s[3], const R r[3]) {
#pragma unroll
  for (int ax = 0; ax < 3; ax++) {
    R B[3][3];
    basis_rows(s[ax], r[ax], B);
    const int st = ax == 0 ? 9 : ax == 1 ? 3 : 1;
#pragma unroll
    for (int o = 0; o < 9; o++) {
      // the two other axes' indices
      const int base = ax == 0 ? o : ax == 1 ? (o / 3) * 9 + (o % 3) : o * 3;
      const R f0 = v[base], fp = v[base + st], fm = v[base + 2 * st];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const R o3 = fma(B[i][2], fm, fma(B[i][1], fp, B[i][0] * f0));
        if (i == 0) v[base] = o3; else if (i == 1) v[base + st] = o3; else v[base + 2 * st] = o3;
      }
    }
  }
}

// node_to_ref of a staged node in its slots, with the same roundings (the
// axes in the same order; a node beyond the halo goes through node_to_ref, and
// nodes whose iterates cycle between two windows turn a last digit into 1e-3):
// non-finite populations count as 0 (all of them when !ok).  Pairs of target
// classes i1 = +, - from the x pass on, pairs i2 = +, - of i1 = 0 from the y
// pass on: 144 instructions for the 243 multiply-adds.  `raw` (null, or the
// node's column of the iterates, `stride` floats apart) gets the populations
// as they were.
__device__ __forceinline__ void staged_to_ref(float* node, bool ok, const float s[3], const float r[3], float* raw,
                                              int stride) {
  float e[28];
  float4* s4 = reinterpret_cast<float4*>(node);
#pragma unroll
  for (int q = 0; q < 7; q++) {
    const float4 w = s4[q];
    e[4 * q] = w.x; e[4 * q + 1] = w.y; e[4 * q + 2] = w.z; e[4 * q + 3] = w.w;
  }
  if (raw)
#pragma unroll
    for (int t = 0; t < 27; t++) raw[t * stride] = e[slot27(t)];
#pragma unroll
  for (int q = 0; q < 27; q++) e[q] = (ok && fabsf(e[q]) <= 3.402823466e38f) ? e[q] : 0.f;
  float B[3][3];
  float2 P[3][3];  // [k2][k3] of i1 = +, -
  float Z[3][3];   // [k2][k3] of i1 = 0
  basis_rows(s[0], r[0], B);
  {
    const float2 c0 = make_float2(B[1][0], B[2][0]), c1 = make_float2(B[1][1], B[2][1]), c2 = make_float2(B[1][2], B[2][2]);
#pragma unroll
    for (int k2 = 0; k2 < 3; k2++)
#pragma unroll
      for (int k3 = 0; k3 < 3; k3++) {
        const float z = e[slot27(0, k2, k3)], p = e[slot27(1, k2, k3)], m = e[slot27(2, k2, k3)];
        Z[k2][k3] = fmaf(B[0][2], m, fmaf(B[0][1], p, B[0][0] * z));
        P[k2][k3] = __ffma2_rn(c2, make_float2(m, m), __ffma2_rn(c1, make_float2(p, p), __fmul2_rn(c0, make_float2(z, z))));
      }
  }
  basis_rows(s[1], r[1], B);
  float2 P2[3][3], Q[3];  // [i2][k3] of i1 = +, -; [k3] of i1 = 0, i2 = +, -
  float S[3];             // [k3] of i1 = i2 = 0
  {
    const float2 c0 = make_float2(B[1][0], B[2][0]), c1 = make_float2(B[1][1], B[2][1]), c2 = make_float2(B[1][2], B[2][2]);
#pragma unroll
    for (int k3 = 0; k3 < 3; k3++) {
#pragma unroll
      for (int i2 = 0; i2 < 3; i2++) {
        const float b0 = B[i2][0], b1 = B[i2][1], b2 = B[i2][2];
        P2[i2][k3] = __ffma2_rn(make_float2(b2, b2), P[2][k3],
                                __ffma2_rn(make_float2(b1, b1), P[1][k3], __fmul2_rn(make_float2(b0, b0), P[0][k3])));
      }
      const float z = Z[0][k3], p = Z[1][k3], m = Z[2][k3];
      S[k3] = fmaf(B[0][2], m, fmaf(B[0][1], p, B[0][0] * z));
      Q[k3] = __ffma2_rn(c2, make_float2(m, m), __ffma2_rn(c1, make_float2(p, p), __fmul2_rn(c0, make_float2(z, z))));
    }
  }
  basis_rows(s[2], r[2], B);
#pragma unroll
  for (int i3 = 0; i3 < 3; i3++) {
    const float b0 = B[i3][0], b1 = B[i3][1], b2 = B[i3][2];
    const auto pair = [&](const float2 v[3], int slot) {
      const float2 o = __ffma2_rn(make_float2(b2, b2), v[2],
                                  __ffma2_rn(make_float2(b1, b1), v[1], __fmul2_rn(make_float2(b0, b0), v[0])));
      e[slot] = o.x;
      e[slot + 1] = o.y;
    };
#pragma unroll
    for (int i2 = 0; i2 < 3; i2++) pair(P2[i2], slot27(1, i2, i3));
    pair(Q, slot27(0, 1, i3));
    e[slot27(0, 0, i3)] = fmaf(b2, S[2], fmaf(b1, S[1], b0 * S[0]));
  }
  e[27] = 0.f;
#pragma unroll
  for (int q = 0; q < 7; q++) s4[q] = make_float4(e[4 * q], e[4 * q + 1], e[4 * q + 2], e[4 * q + 3]);
}

// Queue the copies of global node g's populations into the slots of a staged
// node (`rv`: axes mirrored there, which reverses the classes along them).
__device__ __forceinline__ void copy_node(const float* f, long long N, long long g, const bool rv[3], float* node) {
  if (!(rv[0] || rv[1] || rv[2])) {
    // in the stored order, one addition per population
    constexpr int cls[27] = {0, 9, 3, 1, 12, 10, 4, 13, 18, 21, 19, 22, 6, 7, 15, 16, 2, 11, 5, 14, 24, 25, 20, 23, 8, 17, 26};
    const float* src = f + g;
#pragma unroll
    for (int q = 0; q < 27; q++) {
      cp_async4(node + slot27(cls[q]), src);
      src += N;
    }
    return;
  }
#pragma unroll
  for (int t = 0; t < 27; t++) {
    int cx = t / 9, cy = (t / 3) % 3, cz = t % 3;
    if (rv[0]) cx = rev3(cx);
    if (rv[1]) cy = rev3(cy);
    if (rv[2]) cz = rev3(cz);
    cp_async4(node + slot27(t), f + (long long)c_ref27[cx * 9 + cy * 3 + cz] * N + g);
  }
}

// moments_and_test for the float32 tiles: the node's previous populations lie
// in shared memory (`f0`, `stride` floats apart, replaced by acc).  isConv's
// comparison is float64's: the float32 difference and threshold, each within
// 3e-7 of the exact one, decide where they lie further apart than 1e-6, and the
// float64 ones where they do not, or where the threshold is too small for that.
// Order 3 forms its sums in moments_and_test's order, so that its results stay
// those of the node-by-node sums to the last bit (128^3: 1 % of the step).
template <int N>
__device__ __forceinline__ bool tile_moments_and_test(const StepArgs<float>& a, const float acc[27], float* f0, int stride,
                                                      double C, double& rho0, double U[3], double& T) {
  using L = Lattice<POND_D3Q27>;
  const float ta = float(a.tol_abs), tr = float(a.tol_rel);
  bool ok = true, close = false;
#pragma unroll
  for (int t = 0; t < 27; t++) {
    const float d = fabsf(acc[t] - f0[t * stride]), thr = fmaf(tr, fabsf(acc[t]), ta);
    const bool over = d > 1.000001f * thr, under = d < 0.999999f * thr && thr > 1e-30f;
    ok = ok && !(over && thr > 1e-30f);
    close = close || !(under || (over && thr > 1e-30f));
  }
  if (ok && close)
#pragma unroll
    for (int t = 0; t < 27; t++) {
      const double nv = acc[t], ov = f0[t * stride];
      ok = ok && !(fabs(nv - ov) >= a.tol_abs + a.tol_rel * fabs(nv));
    }
  double m[4] = {0, 0, 0, 0}, rho = 0;
  if constexpr (N == 3) {
#pragma unroll
    for (int t = 0; t < 27; t++) {
      const double fv = acc[t];
      const double vx = C * L::xi1(t / 9) + U[0], vy = C * L::xi1(t / 3 % 3) + U[1], vz = C * L::xi1(t % 3) + U[2];
      rho += fv;
      m[0] += fv * vx; m[1] += fv * vy; m[2] += fv * vz;
      m[3] += fv * (vx * vx + vy * vy + vz * vz);
      f0[t * stride] = acc[t];
    }
  } else {
    // the sums of each class of each axis first: 93 operations instead of 190
    double sx[3] = {0, 0, 0}, sy[3] = {0, 0, 0}, sz[3] = {0, 0, 0};
#pragma unroll
    for (int cx = 0; cx < 3; cx++)
#pragma unroll
      for (int cy = 0; cy < 3; cy++) {
        double row = 0;
#pragma unroll
        for (int cz = 0; cz < 3; cz++) {
          const int t = (cx * 3 + cy) * 3 + cz;
          const double nv = acc[t];
          row += nv;
          sz[cz] += nv;
          f0[t * stride] = acc[t];
        }
        sx[cx] += row;
        sy[cy] += row;
      }
    rho = sx[0] + sx[1] + sx[2];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double vx = C * L::xi1(c) + U[0], vy = C * L::xi1(c) + U[1], vz = C * L::xi1(c) + U[2];
      const double px = sx[c] * vx, py = sy[c] * vy, pz = sz[c] * vz;
      m[0] += px; m[1] += py; m[2] += pz;
      m[3] += px * vx + py * vy + pz * vz;
    }
  }
  if (rho != 0) {
    const double ir = 1.0 / rho;
#pragma unroll
    for (int k = 0; k < 4; k++) m[k] *= ir;
  }
  double Tn = (m[3] - m[0] * m[0] - m[1] * m[1] - m[2] * m[2]) * (1.0 / L::Dim);
  if (Tn < 0) Tn = T;
#pragma unroll
  for (int k = 0; k < 3; k++) ok = ok && !(fabs(m[k] - U[k]) >= a.tolg_abs + a.tolg_rel * fabs(m[k]));
  ok = ok && !(fabs(Tn - T) >= a.tolg_abs + a.tolg_rel * fabs(Tn));
  rho0 = rho; U[0] = m[0]; U[1] = m[1]; U[2] = m[2]; T = Tn;
  return ok;
}

// Z[k1,k2,i3] += sum_k3 w_i3 Gz[i3][k3] F[k1,k2,k3] (F: reference-gauge populations) for the z-classes i3
// flagged in nz (the first contraction, one per stencil node).
template <typename LoadV>
__device__ __forceinline__ void contract_z(const float Gz[3][3], const float wz[3], const bool nz[3], LoadV loadv,
                                           float Z[27]) {
  float g[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int k = 0; k < 3; k++) g[i][k] = wz[i] * Gz[i][k];
#pragma unroll
  for (int k12 = 0; k12 < 9; k12++) {
    const float v0 = loadv(k12 * 3 + 0), v1 = loadv(k12 * 3 + 1), v2 = loadv(k12 * 3 + 2);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      if (!nz[i]) continue;
      float& o = Z[k12 * 3 + i];
      o = fmaf(g[i][2], v2, fmaf(g[i][1], v1, fmaf(g[i][0], v0, o)));
    }
  }
}

// Y[k1,i2,i3] += sum_k2 w_i2 Gy[i2][k2] Z[k1,k2,i3] (one per stencil column)
__device__ __forceinline__ void contract_y(const float Gy[3][3], const float wy[3], const bool ny[3], const float Z[27],
                                           float Y[27]) {
  float g[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int k = 0; k < 3; k++) g[i][k] = wy[i] * Gy[i][k];
#pragma unroll
  for (int k1 = 0; k1 < 3; k1++)
#pragma unroll
    for (int i2 = 0; i2 < 3; i2++) {
      if (!ny[i2]) continue;
#pragma unroll
      for (int i3 = 0; i3 < 3; i3++) {
        float& o = Y[(k1 * 3 + i2) * 3 + i3];
        o = fmaf(g[i2][2], Z[(k1 * 3 + 2) * 3 + i3],
                 fmaf(g[i2][1], Z[(k1 * 3 + 1) * 3 + i3], fmaf(g[i2][0], Z[k1 * 9 + i3], o)));
      }
    }
}

// acc[i1,i2,i3] += sum_k1 w_i1 Gx[i1][k1] Y[k1,i2,i3] (one per stencil row)
__device__ __forceinline__ void contract_x(const float Gx[3][3], const float wx[3], const bool nx[3], const float Y[27],
                                           float acc[27]) {
  float g[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int k = 0; k < 3; k++) g[i][k] = wx[i] * Gx[i][k];
#pragma unroll
  for (int i1 = 0; i1 < 3; i1++) {
    if (!nx[i1]) continue;
#pragma unroll
    for (int i23 = 0; i23 < 9; i23++) {
      float& o = acc[i1 * 9 + i23];
      o = fmaf(g[i1][2], Y[18 + i23], fmaf(g[i1][1], Y[9 + i23], fmaf(g[i1][0], Y[i23], o)));
    }
  }
}

// interpolation weight of relative offset o for a window starting at ro
template <int N, typename R> __device__ __forceinline__ R wpick(const R w[N], int ro, int o) {
  const int j = o - ro;
  R r = R(0);
#pragma unroll
  for (int k = 0; k < N; k++) r = (j == k) ? w[k] : r;
  return r;
}

// Two-wide float32 multiply-add with one factor shared by both halves.
__device__ __forceinline__ float2 fma2(float g, float2 v, float2 o) { return __ffma2_rn(make_float2(g, g), v, o); }

// One z offset of a stencil column: Z[k1,k2,i] += sum_k3 w_i Gz[i][k3] F[k1,k2,k3]
// for the z-classes i in [I0, I1], i = 0 always (I0..I1 = 1..2: all three).
// Zp[i][k2] holds the pair k1 = +, -; Zq[i] the pair k2 = +, - of k1 = 0; Zs[i] the rest.
template <bool kPlus, bool kMinus>
__device__ __forceinline__ void column_node(const float* node, const float Gz[3][3], const float w[3], float2 Zp[3][3],
                                            float2 Zq[3], float Zs[3]) {
  float4 v[7];
  const float4* s4 = reinterpret_cast<const float4*>(node);
#pragma unroll
  for (int q = 0; q < 7; q++) v[q] = s4[q];
  const auto pair = [&](int p) {  // slots 2p, 2p + 1
    return (p & 1) ? make_float2(v[p >> 1].z, v[p >> 1].w) : make_float2(v[p >> 1].x, v[p >> 1].y);
  };
  const float last[3] = {v[6].x, v[6].y, v[6].z};
#pragma unroll
  for (int k3 = 0; k3 < 3; k3++) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
      if ((i == 1 && !kPlus) || (i == 2 && !kMinus)) continue;
      const float g = w[i] * Gz[i][k3];
#pragma unroll
      for (int k2 = 0; k2 < 3; k2++) Zp[i][k2] = fma2(g, pair(3 * k3 + k2), Zp[i][k2]);
      Zq[i] = fma2(g, pair(9 + k3), Zq[i]);
      Zs[i] = fmaf(g, last[k3], Zs[i]);
    }
  }
}

// The populations of one iterate from the staged, R-gauge nodes around `centre`
// (the lane's node): acc[i1,i2,i3] = sum over the stencil offsets of the
// interpolation weights times the transfer from the reference gauge to the
// target, contracted along z per stencil node, y per column, x per row.  The
// offsets walked are wl..wh per axis, the union over the warp's unconverged
// lanes; a class a lane does not weight at an offset has weight 0 there.
// `staggered` (warp-uniform): along z every lane's + class starts at wl and
// its - class one later, wh = wl + N, as for |u_z| < c below one node per
// step; then the first offset skips the - class and the last one the + class,
// and the column is straight-line code.
template <int N>
__device__ __forceinline__ void contract_tile(const float* centre, int sx, int sxy, const int wl[3], const int wh[3],
                                              bool staggered, const int ro[3][3], const float wt[3][3][N],
                                              const float bq[3], float ainv, float acc[27]) {
  float Gz[3][3];  // the z basis is used per stencil node; x and y are rebuilt per row and column
  basis_rows(bq[2], ainv, Gz);
  float wz[N + 1][3];  // z weights of the staggered window, by offset from wl
#pragma unroll
  for (int j = 0; j <= N; j++)
#pragma unroll
    for (int c = 0; c < 3; c++) wz[j][c] = wpick<N>(wt[2][c], ro[2][c], wl[2] + j);
#pragma unroll 1
  for (int ox = wl[0]; ox <= wh[0]; ox++) {
    float2 Yp[3][3];
    float Y0[3][3];
#pragma unroll
    for (int i2 = 0; i2 < 3; i2++)
#pragma unroll
      for (int i3 = 0; i3 < 3; i3++) { Yp[i2][i3] = make_float2(0.f, 0.f); Y0[i2][i3] = 0.f; }
#pragma unroll 1
    for (int oy = wl[1]; oy <= wh[1]; oy++) {
      float2 Zp[3][3], Zq[3];
      float Zs[3];
#pragma unroll
      for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int k2 = 0; k2 < 3; k2++) Zp[i][k2] = make_float2(0.f, 0.f);
        Zq[i] = make_float2(0.f, 0.f);
        Zs[i] = 0.f;
      }
      const float* col = centre + (wl[2] * sxy + oy * sx + ox) * NS;
      if (staggered) {
        column_node<true, false>(col, Gz, wz[0], Zp, Zq, Zs);
#pragma unroll
        for (int j = 1; j < N; j++) column_node<true, true>(col + j * sxy * NS, Gz, wz[j], Zp, Zq, Zs);
        column_node<false, true>(col + N * sxy * NS, Gz, wz[N], Zp, Zq, Zs);
      } else {
#pragma unroll 1
        for (int oz = wl[2]; oz <= wh[2]; oz++) {
          float w[3];
#pragma unroll
          for (int c = 0; c < 3; c++) w[c] = wpick<N>(wt[2][c], ro[2][c], oz);
          column_node<true, true>(col + (oz - wl[2]) * sxy * NS, Gz, w, Zp, Zq, Zs);
        }
      }
      float G[3][3];
      basis_rows(bq[1], ainv, G);
#pragma unroll
      for (int i2 = 0; i2 < 3; i2++) {
        const float w = wpick<N>(wt[1][i2], ro[1][i2], oy);
        const float g0 = w * G[i2][0], g1 = w * G[i2][1], g2 = w * G[i2][2];
#pragma unroll
        for (int i3 = 0; i3 < 3; i3++) {
          Yp[i2][i3] = fma2(g2, Zp[i3][2], fma2(g1, Zp[i3][1], fma2(g0, Zp[i3][0], Yp[i2][i3])));
          Y0[i2][i3] = fmaf(g2, Zq[i3].y, fmaf(g1, Zq[i3].x, fmaf(g0, Zs[i3], Y0[i2][i3])));
        }
      }
    }
    float G[3][3];
    basis_rows(bq[0], ainv, G);
#pragma unroll
    for (int i1 = 0; i1 < 3; i1++) {
      const float w = wpick<N>(wt[0][i1], ro[0][i1], ox);
      const float g0 = w * G[i1][0], g1 = w * G[i1][1], g2 = w * G[i1][2];
#pragma unroll
      for (int i2 = 0; i2 < 3; i2++)
#pragma unroll
        for (int i3 = 0; i3 < 3; i3++) {
          float& o = acc[(i1 * 3 + i2) * 3 + i3];
          o = fmaf(g2, Yp[i2][i3].y, fmaf(g1, Yp[i2][i3].x, fmaf(g0, Y0[i2][i3], o)));
        }
    }
  }
}

// What contract_node_by_warp needs of its node, in the warp's scratch.
template <int N> struct alignas(16) ServedNode {
  float wt[3][3][N], bq[3], ainv;
  int ro[3][3], lo[3], hi[3], centre;
};
static_assert(sizeof(ServedNode<4>) <= served_floats(1) * sizeof(float), "the scratch holds a node's windows");

// The same iterate for one node by the whole warp, with contract_tile's
// roundings: lane 5 (oy + 2) + ox + 2 sums the stencil column at (ox, oy) along
// z; then, ROWS rows of columns at a time, the sums go through shared memory to
// lane 9 k1 + 3 i2 + i3, which takes them along y, and to lane 9 i1 + 3 i2 + i3
// by shuffle along x.  Every sum runs over the same terms in the same order as in
// contract_tile (whose further offsets have weight 0), so a node's result does
// not depend on how many of its neighbours still iterate.  The node comes in
// `scratch` and its populations go there.  Used when few lanes of a warp still
// iterate: the warp's contraction of all its lanes costs the same however few
// they are (about 11,000 instructions at N = 4).  Not inlined: the registers it
// needs would be taken from the contraction of full warps (256^3: 28.5 ms, 31.6
// inlined).  Five rows at a time instead of one: 28.5 -> 28.3 ms there, two steps
// with energy populations at 64^3 2.73 -> 2.65 (three rows).
template <int N, int ROWS>
__device__ __noinline__ void contract_node_by_warp(const float* staged, int sx, int sxy, float* scratch) {
  const int lane = threadIdx.x & 31;
  const ServedNode<N>& node = *reinterpret_cast<const ServedNode<N>*>(scratch);
  const int ox = lane < 25 ? lane % 5 - 2 : 0, oy = lane < 25 ? lane / 5 - 2 : 0;
  const int xlo = max(node.lo[0], -H), xhi = min(node.hi[0], H), ylo = node.lo[1], yhi = node.hi[1];
  float2 Zp[3][3], Zq[3];
  float Zs[3], G[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
#pragma unroll
    for (int k2 = 0; k2 < 3; k2++) Zp[i][k2] = make_float2(0.f, 0.f);
    Zq[i] = make_float2(0.f, 0.f);
    Zs[i] = 0.f;
  }
  const float ainv = node.ainv;
  basis_rows(node.bq[2], ainv, G);
  {
    const float* col = staged + (node.centre + oy * sx + ox) * NS;
    const int zlo = node.lo[2], zhi = node.hi[2];
#pragma unroll
    for (int oz = -H; oz <= H; oz++) {
      if (oz < zlo || oz > zhi) continue;
      float w[3];
#pragma unroll
      for (int c = 0; c < 3; c++) w[c] = wpick<N>(node.wt[2][c], node.ro[2][c], oz);
      column_node<true, true>(col + oz * sxy * NS, G, w, Zp, Zq, Zs);
    }
  }
  // this lane's classes along y and x: the rows i2 and i1 of the bases, the windows and their weights
  const int i1 = min(lane / 9, 2), i2 = (lane / 3) % 3, i3 = lane % 3;
  float Gy[3], Gx[3], wy[N], wx[N];
  const auto row = [](float B[3][3], int i, float out[3]) {
#pragma unroll
    for (int k = 0; k < 3; k++) out[k] = i == 0 ? B[0][k] : i == 1 ? B[1][k] : B[2][k];
  };
  basis_rows(node.bq[1], ainv, G);
  row(G, i2, Gy);
  basis_rows(node.bq[0], ainv, G);
  row(G, i1, Gx);
#pragma unroll
  for (int k = 0; k < N; k++) {
    wy[k] = node.wt[1][i2][k];
    wx[k] = node.wt[0][i1][k];
  }
  const int roy = node.ro[1][i2], rox = node.ro[0][i1];
  __syncwarp();  // the node has been read
  // column slots: pairs [2 (3 i3 + k2) + k1 - 1] of k1 = +, -, then those of k1 = 0 as [18 + 3 i3 + k2]
  const int from = i1 > 0 ? 6 * i3 + i1 - 1 : 18 + 3 * i3, step = i1 > 0 ? 2 : 1;  // k1 = i1 here
  float out = 0.f;
#pragma unroll 1
  for (int p0 = xlo; p0 <= xhi; p0 += ROWS) {
    if (lane < 25 && ox >= p0 && ox < p0 + ROWS) {
      float* col = scratch + (5 * (ox - p0) + oy + H) * 27;
#pragma unroll
      for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int k2 = 0; k2 < 3; k2++) {
          col[2 * (3 * i + k2)] = Zp[i][k2].x;
          col[2 * (3 * i + k2) + 1] = Zp[i][k2].y;
        }
        col[18 + 3 * i] = Zs[i];
        col[18 + 3 * i + 1] = Zq[i].x;
        col[18 + 3 * i + 2] = Zq[i].y;
      }
    }
    __syncwarp();
    float Y[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; r++) Y[r] = 0.f;
#pragma unroll
    for (int py = -H; py <= H; py++) {
      if (py < ylo || py > yhi) continue;  // warp-uniform
      const float* col = scratch + (py + H) * 27 + from;
      const float w = wpick<N>(wy, roy, py);
      const float g0 = w * Gy[0], g1 = w * Gy[1], g2 = w * Gy[2];
#pragma unroll
      for (int r = 0; r < ROWS; r++)  // rows past the last are not used
        Y[r] = fmaf(g2, col[135 * r + 2 * step], fmaf(g1, col[135 * r + step], fmaf(g0, col[135 * r], Y[r])));
    }
    const int at = 3 * i2 + i3;
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      if (p0 + r > xhi) break;
      const float w = wpick<N>(wx, rox, p0 + r);
      const float g0 = w * Gx[0], g1 = w * Gx[1], g2 = w * Gx[2];
      const float y0 = __shfl_sync(0xffffffffu, Y[r], at), y1 = __shfl_sync(0xffffffffu, Y[r], 9 + at),
                  y2 = __shfl_sync(0xffffffffu, Y[r], 18 + at);
      out = fmaf(g2, y2, fmaf(g1, y1, fmaf(g0, y0, out)));
    }
    __syncwarp();
  }
  if (lane < 27) scratch[lane] = out;
  __syncwarp();
}

// The lanes of `live`, one after another, through contract_node_by_warp; each
// gets its node's populations in acc.  `centre`: the lane's staged node;
// `scratch`: served_floats(ROWS) floats of the warp, 16-byte aligned.
template <int N, int ROWS>
__device__ __forceinline__ void contract_live_lanes(unsigned live, const float* staged, int centre, int sx, int sxy,
                                                    const int lo[3], const int hi[3], const int ro[3][3],
                                                    const float wt[3][3][N], const float bq[3], float ainv,
                                                    float* scratch, float acc[27]) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (; live; live &= live - 1) {
    const int src = __ffs(live) - 1;
    if (lane == src) {
      ServedNode<N> node;
#pragma unroll
      for (int ax = 0; ax < 3; ax++) {
        node.lo[ax] = lo[ax]; node.hi[ax] = hi[ax]; node.bq[ax] = bq[ax];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          node.ro[ax][c] = ro[ax][c];
#pragma unroll
          for (int k = 0; k < N; k++) node.wt[ax][c][k] = wt[ax][c][k];
        }
      }
      node.ainv = ainv;
      node.centre = centre;
      *reinterpret_cast<ServedNode<N>*>(scratch) = node;
    }
    __syncwarp();
    contract_node_by_warp<N, ROWS>(staged, sx, sxy, scratch);
    if (lane == src)
#pragma unroll
      for (int t = 0; t < 27; t++) acc[t] = scratch[t];
    __syncwarp();
  }
}

// Live lanes at which the warp serves nodes one by one: the serial iteration
// costs about 11,000 / 6,500 / 3,000 instructions (N = 4 / 3 / 2), a node by
// the warp 1,300 and its exchanges.  4 to 6 lanes (N = 4) and 3 or 4 (N = 3)
// are within 0.7 % of each other from 32^3 to 256^3, 8 lanes 0.5-4 % slower.
template <int N> __host__ __device__ constexpr int few_lanes() { return N == 4 ? 5 : N == 3 ? 3 : 2; }

// Record of a CTA's step sums, written instead of the context's sums when the
// kernel runs without a context.
struct BlockPartial {
  double mass, mom[3], enrg, k;
  unsigned long long niter_sum, nonconv, work;
  int niter_max;
  int pad;
};

// Add the CTA's sums to `sum` (in shared memory), in a fixed order.
template <int WARPS> __device__ __forceinline__ void add_block_partial(NodeSums s, BlockPartial& sum) {
  __shared__ double pd[6][WARPS];
  __shared__ unsigned long long pu[3][WARPS];
  __shared__ int pm[WARPS];
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  double v[6] = {s.mass, s.m0, s.m1, s.m2, s.enrg, s.k};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int q = 0; q < 6; q++) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    s.niter += __shfl_xor_sync(0xffffffffu, s.niter, o);
    s.nonconv += __shfl_xor_sync(0xffffffffu, s.nonconv, o);
    s.work += __shfl_xor_sync(0xffffffffu, s.work, o);
    s.nmax = max(s.nmax, __shfl_xor_sync(0xffffffffu, s.nmax, o));
  }
  if ((tid & 31) == 0) {
    for (int q = 0; q < 6; q++) pd[q][warp] = v[q];
    pu[0][warp] = s.niter; pu[1][warp] = s.nonconv; pu[2][warp] = s.work; pm[warp] = s.nmax;
  }
  __syncthreads();
  if (tid == 0) {
    BlockPartial b = sum;
    for (int w = 0; w < WARPS; w++) {
      b.mass += pd[0][w]; b.mom[0] += pd[1][w]; b.mom[1] += pd[2][w]; b.mom[2] += pd[3][w];
      b.enrg += pd[4][w]; b.k += pd[5][w];
      b.niter_sum += pu[0][w]; b.nonconv += pu[1][w]; b.work += pu[2][w];
      b.niter_max = max(b.niter_max, pm[w]);
    }
    sum = b;
  }
}

// The step of the tile whose first node is (x0, y0, z0), by one CTA; `ns`
// gains this thread's share of the sums.
template <int N>
__device__ __forceinline__ void step_tile(const StepArgs<float>& a, const int x0, const int y0, const int z0, NodeSums& ns) {
  using L = Lattice<POND_D3Q27>;
  using Ti = Tile<N>;
  constexpr int SX = Ti::SX, SY = Ti::SY, SN = Ti::SN, THREADS = Ti::THREADS;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x;
  float* own = sm + Ti::OFF_OWN;
  float* su = sm + Ti::OFF_U;

  // ---- stage: each thread copies whole staged nodes (27 populations, the
  // mirror reversing classes, and the gauge) with asynchronous copies, waits
  // for its own copies and transfers its nodes into the reference gauge;
  // boundary resolution happens in the addresses (mirrored velocity components
  // flip; a node with a non-finite gauge contributes nothing, non-finite
  // populations count as 0)
#pragma unroll 1
  for (int i = tid; i < SN; i += THREADS) {
    const int hx = i % SX, hy = (i / SX) % SY, hz = i / (SX * SY);
    bool rv[3];
    const int gx = resolve_axis(x0 - H + hx, a.nx, a.bc[0], rv[0]);
    const int gy = resolve_axis(y0 - H + hy, a.ny, a.bc[1], rv[1]);
    const int gz = resolve_axis(z0 - H + hz, a.nz, a.bc[2], rv[2]);
    const long long g = gx + (long long)a.nx * (gy + (long long)a.ny * gz);
    copy_node(a.f_in, a.N, g, rv, sm + i * NS);
#pragma unroll
    for (int k = 0; k < 3; k++) cp_async4(su + k * SN + i, a.g_in + (long long)k * a.N + g);
    cp_async4(sm + i * NS + 27, a.g_in + 3 * a.N + g);
  }
  // ---- reference gauge of the CTA: the gauge of the tile's centre node
  //      ((0, 1) if it is not finite or its c is 0)
  float uref[3], icref;
  {
    bool rv[3];
    const int gx = resolve_axis(x0 + Ti::TX / 2, a.nx, a.bc[0], rv[0]);
    const int gy = resolve_axis(y0 + Ti::TY / 2, a.ny, a.bc[1], rv[1]);
    const int gz = resolve_axis(z0 + Ti::TZ / 2, a.nz, a.bc[2], rv[2]);
    const long long g = gx + (long long)a.nx * (gy + (long long)a.ny * gz);
    const float T = a.g_in[3 * a.N + g];
    const float cc = copysignf(sqrtf(fabsf(T) * (float)(1.0 / L::TLat)), T);
    bool ok = fabsf(cc) <= 3.0e38f;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float v = a.g_in[(long long)k * a.N + g];
      uref[k] = rv[k] ? -v : v;
      ok = ok && fabsf(v) <= 3.0e38f;
    }
#pragma unroll
    for (int k = 0; k < 3; k++) uref[k] = ok ? uref[k] : 0.f;
    icref = (ok && fabsf(cc) > 1.0e-20f) ? 1.f / cc : 1.f;
  }
  const float cref = 1.f / icref;
  cp_async_wait_all();
#pragma unroll 1
  for (int i = tid; i < SN; i += THREADS) {
    const int hx = i % SX, hy = (i / SX) % SY, hz = i / (SX * SY);
    // the axes mirrored there (only positions outside the grid can be)
    const int p[3] = {x0 - H + hx, y0 - H + hy, z0 - H + hz}, n[3] = {a.nx, a.ny, a.nz};
    float u[3];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      bool rv = false;
      if (p[k] < 0 || p[k] >= n[k]) resolve_axis(p[k], n[k], a.bc[k], rv);
      const float v = su[k * SN + i];
      u[k] = rv ? -v : v;
      ok = ok && fabsf(v) <= 3.0e38f;
    }
    const float T = sm[i * NS + 27];
    const float c = copysignf(sqrtf(fabsf(T) * (float)(1.0 / L::TLat)), T);
    ok = ok && fabsf(c) <= 3.0e38f;
    const float r = ok ? c * icref : 0.f;
    const float sq[3] = {ok ? (u[0] - uref[0]) * icref : 0.f, ok ? (u[1] - uref[1]) * icref : 0.f,
                         ok ? (u[2] - uref[2]) * icref : 0.f};
    const float rq[3] = {r, r, r};
    // a node of the tile leaves its populations where its thread keeps its iterate
    float* raw = nullptr;
    if constexpr (!Ti::kOwnLater) {
      const int tx = hx - H, ty = hy - H, tz = hz - H;
      if (tx >= 0 && tx < Ti::TX && ty >= 0 && ty < Ti::TY && tz >= 0 && tz < Ti::TZ) raw = own + Ti::thread_of(tx, ty, tz);
    }
    staged_to_ref(sm + i * NS, ok, sq, rq, raw, THREADS);
  }
  __syncthreads();

  const int lx = Ti::lx(tid), ly = Ti::ly(tid), lz = Ti::lz(tid);
  const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
  const bool active = x < a.nx && y < a.ny && z < a.nz;
  const long long idx = active ? x + (long long)a.nx * (y + (long long)a.ny * z) : 0;
  // the node's current populations live in shared memory between iterations,
  // which keeps them out of the loop's registers
  float* f0s = own + tid;
  if constexpr (Ti::kOwnLater) {
#pragma unroll
    for (int t = 0; t < 27; t++) f0s[t * THREADS] = a.f_in[(long long)c_ref27[t] * a.N + idx];
  }
  double rho0 = 1, U[3] = {0, 0, 0}, T = L::TLat;
  if (active) {  // c0.load (steps.cu:360-363); the populations are in f0s already
    rho0 = a.rho_in[idx];
    U[0] = a.g_in[idx]; U[1] = a.g_in[a.N + idx]; U[2] = a.g_in[2 * a.N + idx];
    T = a.g_in[3 * a.N + idx];
    if (rho0 == 0 && U[0] == 0 && U[1] == 0 && U[2] == 0 && T == 0) {  // set_base(1, TLat) of an empty record
      rho0 = 1; T = L::TLat;
#pragma unroll
      for (int t = 0; t < 27; t++) f0s[t * THREADS] = float(lattice_weight_t<POND_D3Q27>(t));
    }
    if (a.guess) {
      U[0] = a.guess[idx]; U[1] = a.guess[a.N + idx]; U[2] = a.guess[2 * a.N + idx]; T = a.guess[3 * a.N + idx];
    }
  }
  const int pos[3] = {x, y, z};
  const int sbase = (lz + H) * SX * SY + (ly + H) * SX + (lx + H);
  bool done = !active;
  bool conv = false;
  int niter = 0;
  unsigned long long work = 0;
  while (__any_sync(0xffffffffu, !done)) {
    if (!done) niter++;
    const double C = sqrt(T * (1.0 / L::TLat));
    // relative window origins and Lagrange weights per axis and class
    int ro[3][3];
    float wt[3][3][N];
    int lo[3], hi[3];
#pragma unroll
    for (int ax = 0; ax < 3; ax++) {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double crd = double(pos[ax]) - (C * L::xi1(c) + U[ax]);
        const int org = window_origin<N>(crd, ax);
        ro[ax][c] = org - pos[ax];
        if (N == 2) { wt[ax][c][0] = float(1 - (crd - org)); wt[ax][c][N - 1] = float(crd - org); }
        else lagr_weights<N, float>(crd - double(org), wt[ax][c]);
      }
      lo[ax] = min(ro[ax][0], min(ro[ax][1], ro[ax][2]));
      hi[ax] = max(ro[ax][0], max(ro[ax][1], ro[ax][2])) + N - 1;
    }
    // transfer from the reference gauge to this iteration's target gauge,
    // per axis: G[i][k] = L_i(b + a xi_k), a = c_ref / C, b = (u_ref - U) / C
    const double iC = 1.0 / C;
    const float ainv = float(double(cref) * iC);
    float bq[3];
#pragma unroll
    for (int ax = 0; ax < 3; ax++) bq[ax] = float((double(uref[ax]) - U[ax]) * iC);
    float acc[27];
#pragma unroll
    for (int t = 0; t < 27; t++) acc[t] = 0.f;
    const bool inside = lo[0] >= -H && lo[1] >= -H && lo[2] >= -H && hi[0] <= H && hi[1] <= H && hi[2] <= H;
    if (__all_sync(0xffffffffu, inside || done)) {
      // warp-uniform offsets: the union of the unconverged lanes' stencils
      int wl[3], wh[3];
#pragma unroll
      for (int ax = 0; ax < 3; ax++) {
        wl[ax] = __reduce_min_sync(0xffffffffu, done ? H : lo[ax]);
        wh[ax] = __reduce_max_sync(0xffffffffu, done ? -H : hi[ax]);
      }
      const unsigned live = __ballot_sync(0xffffffffu, !done);
      if (__popc(live) <= few_lanes<N>()) {
        if (!done) {  // the node's own windows
          const unsigned long long ex = hi[0] - lo[0] + 1, ey = hi[1] - lo[1] + 1, ez = hi[2] - lo[2] + 1;
          work += ex * ey * ez * 171 + ex * ey * 171 + ex * 171;
        }
        contract_live_lanes<N, Ti::ROWS>(live, sm, sbase, SX, SX * SY, lo, hi, ro, wt, bq, ainv,
                                         sm + Ti::OFF_S + (tid >> 5) * Ti::SERVED, acc);
      } else {
        const bool staggered =
            __all_sync(0xffffffffu, done || (ro[2][1] == wl[2] && ro[2][2] == wl[2] + 1 && ro[2][0] >= wl[2] &&
                                             ro[2][0] <= wl[2] + 1)) && wh[2] == wl[2] + N;
        if (!done) {  // floating-point operations of the contractions below
          const unsigned long long ex = wh[0] - wl[0] + 1, ey = wh[1] - wl[1] + 1, ez = wh[2] - wl[2] + 1;
          work += ex * ey * (ez * 171 - (staggered ? 114 : 0)) + ex * ey * 171 + ex * 171;
        }
        contract_tile<N>(sm + sbase * NS, SX, SX * SY, wl, wh, staggered, ro, wt, bq, ainv, acc);
      }
    } else if (!done) {
      // departure points beyond the staged halo: this lane reads global memory
      // and transfers each stencil node into the reference gauge itself
      const unsigned long long ex = window_positions<N, 3>(ro[0]), ey = window_positions<N, 3>(ro[1]),
                               ez = window_positions<N, 3>(ro[2]);
      work += ex * ey * ez * 171 + ex * ey * 171 + ex * 171;
      const bool all3[3] = {true, true, true};
      float Gz[3][3];
      basis_rows(bq[2], ainv, Gz);
      for (int ox = lo[0]; ox <= hi[0]; ox = window_next<N, 3>(ro[0], ox)) {
        bool rv[3] = {false, false, false};
        const int gx = resolve_axis(x + ox, a.nx, a.bc[0], rv[0]);
        float wx[3];
#pragma unroll
        for (int c = 0; c < 3; c++) wx[c] = wpick<N>(wt[0][c], ro[0][c], ox);
        float Yr[27];
#pragma unroll
        for (int t = 0; t < 27; t++) Yr[t] = 0.f;
        for (int oy = lo[1]; oy <= hi[1]; oy = window_next<N, 3>(ro[1], oy)) {
          const int gy = resolve_axis(y + oy, a.ny, a.bc[1], rv[1]);
          float wy[3];
#pragma unroll
          for (int c = 0; c < 3; c++) wy[c] = wpick<N>(wt[1][c], ro[1][c], oy);
          float Zc[27];
#pragma unroll
          for (int t = 0; t < 27; t++) Zc[t] = 0.f;
          for (int oz = lo[2]; oz <= hi[2]; oz = window_next<N, 3>(ro[2], oz)) {
            const int gz = resolve_axis(z + oz, a.nz, a.bc[2], rv[2]);
            float wz[3];
#pragma unroll
            for (int c = 0; c < 3; c++) wz[c] = wpick<N>(wt[2][c], ro[2][c], oz);
            const long long g = gx + (long long)a.nx * (gy + (long long)a.ny * gz);
            const float un[3] = {a.g_in[g], a.g_in[a.N + g], a.g_in[2 * a.N + g]};
            const float Tn = a.g_in[3 * a.N + g];
            const bool ok = fabsf(un[0]) <= 3.0e38f && fabsf(un[1]) <= 3.0e38f && fabsf(un[2]) <= 3.0e38f &&
                            fabsf(Tn) <= 3.0e38f;
            const float cn = copysignf(sqrtf(fabsf(Tn) * (float)(1.0 / L::TLat)), Tn);
            float v[27];  // plain loads: f_in may have been written while this kernel was resident
#pragma unroll
            for (int t = 0; t < 27; t++)
              v[t] = ok ? finite_or_zero_f(a.f_in[(long long)c_ref27[t] * a.N + g]) : 0.f;
            float sq[3], rq[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
              sq[k] = ok ? ((rv[k] ? -un[k] : un[k]) - uref[k]) * icref : 0.f;
              rq[k] = ok ? (rv[k] ? -cn : cn) * icref : 0.f;
            }
            node_to_ref(v, sq, rq);
            contract_z(Gz, wz, all3, [&](int t) { return v[t]; }, Zc);
          }
          float Gy[3][3];
          basis_rows(bq[1], ainv, Gy);
          contract_y(Gy, wy, all3, Zc, Yr);
        }
        float Gx[3][3];
        basis_rows(bq[0], ainv, Gx);
        contract_x(Gx, wx, all3, Yr, acc);
      }
    }
    if (!done) {
      if (!(C >= 1.0e-300)) {  // C <= 0, NaN, or 1/C beyond 1e300
        // target T = 0: every transfer term is non-finite and dropped (structs.cuh:542)
#pragma unroll
        for (int t = 0; t < 27; t++) acc[t] = 0.f;
      }
      conv = tile_moments_and_test<N>(a, acc, f0s, THREADS, C, rho0, U, T);
      if (conv || niter >= a.max_iter) done = true;
    }
  }
  if (active) {
    float f0[27];
#pragma unroll
    for (int t = 0; t < 27; t++) f0[t] = f0s[t * THREADS];
    NodeSums one;
    finish_node<POND_D3Q27, float>(a, idx, f0, rho0, U, T, niter, conv, one);
    ns.mass += one.mass; ns.m0 += one.m0; ns.m1 += one.m1; ns.m2 += one.m2; ns.enrg += one.enrg; ns.k += one.k;
    ns.niter += one.niter; ns.nonconv += one.nonconv; ns.work += work; ns.nmax = max(ns.nmax, one.nmax);
  }
}

template <int N> __global__ void __launch_bounds__(Tile<N>::THREADS, Tile<N>::CTAS) pull_d3q27_tile_kernel(StepArgs<float> a) {
  NodeSums ns = {0, 0, 0, 0, 0, 0, 0ull, 0ull, 0ull, 0};
  // launched while the step before still runs (launch_early): let the next one
  // come, then wait for the step before to be complete and visible
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  step_tile<N>(a, blockIdx.x * Tile<N>::TX, blockIdx.y * Tile<N>::TY, blockIdx.z * Tile<N>::TZ, ns);
  reduce_and_commit(ns, a.sums);
}

// The step without a context: of the nx x ny x .. = `tiles` tiles CTA b takes b,
// b + gridDim.x, .. in turn and writes record b, so that the sums come out the
// same however the CTAs are scheduled.  (Order 3 has a CTA per tile: an accepted
// grid has no more of its tiles than records.)
template <int N>
__global__ void __launch_bounds__(Tile<N>::THREADS, Tile<N>::CTAS)
    pull_d3q27_records_kernel(StepArgs<float> a, int nx, int ny, int tiles, BlockPartial* records) {
  __shared__ BlockPartial sum;
  if (threadIdx.x == 0) sum = {};
  int t = blockIdx.x;
#pragma unroll 1
  do {
    NodeSums ns = {0, 0, 0, 0, 0, 0, 0ull, 0ull, 0ull, 0};
    step_tile<N>(a, t % nx * Tile<N>::TX, t / nx % ny * Tile<N>::TY, t / nx / ny * Tile<N>::TZ, ns);
    add_block_partial<Tile<N>::WARPS>(ns, sum);  // its barrier ends the tile's use of shared memory
    t += gridDim.x;
  } while (N != 3 && t < tiles);
  if (threadIdx.x == 0) records[blockIdx.x] = sum;
}

}  // namespace d27
}  // namespace pond
