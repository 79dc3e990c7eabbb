// hop_f32.cuh -- the FP32 batch hop with one right-hand side a thread, the next
// neighbour term's words loaded before the current term is computed.
//
// Same operator, arithmetic and epilogues as hop_mrhs_kernel with one right-hand side
// a thread on 12-real links (reference Vector::applyDslash, lib/lattice_util.cpp:1158-1213):
// the bits are the same.  A term is 6 spinor words (3 for the diagonal g_4) and 3 link
// words of 16 bytes; two terms' words live in registers, so a thread always has nine loads
// in flight while it multiplies.  Ten 64-thread blocks an SM (96 registers, up to 20 B of spills).
//
// What bounds it: the latency of the gathers, and 9-10 TB/s from L2.  One B200, average of the four hops of a
// solver iteration, against loads issued term by term (also 96 registers):
//   32^3x64, 12 RHS   1.164 -> 1.057 ms      24^3x48, 12 RHS   363 -> 331 us      16^3x32, 12 RHS   78.6 -> 71.8 us
//             1 RHS   125.7 -> 117.2 us                5 RHS   161 -> 147 us                5 RHS   37.6 -> 34.6 us
// A^-1 D alone, 24^3x48 x 5: 0.136 -> 0.130 ms; at eight blocks an SM (128 registers) 0.133, at six 0.150; without
// the early loads twelve or fourteen blocks an SM 0.138 and 0.135 there, 1.03 and 1.02 ms for 32^3x64 x 12 (0.97).
#pragma once
#include "hop_mrhs.cuh"

namespace qkx {

struct F32Term {
  float4 v[6], u[3];
};

// the words of neighbour term D = 2 mu + (backward)
template <int B, bool DAG, int D>
__device__ __forceinline__ void f32_load(F32Term& w, const SpinorF32& in, const GaugeF32x12& U, const Geom& g,
                                         int par, int cb, const int x[4], int s, int stride) {
  constexpr int MU = D >> 1;
  constexpr bool BWD = (D & 1) != 0;
  constexpr int SF = DAG ? +1 : -1;  // forward projector 1 + SF*g
  using PJ = Proj<B, MU, BWD ? -SF : SF>;
  const int Lm = g.L[MU];
  const int n = BWD ? (x[MU] == 0 ? s + (Lm - 1) * stride : s - stride) >> 1
                    : (x[MU] == Lm - 1 ? s - (Lm - 1) * stride : s + stride) >> 1;
  const float4* p = (par ? in.p0 : in.p1) + n;  // neighbours have the other parity
#pragma unroll
  for (int q = 0; q < 6; q++) {
    if (PJ::diag && (PJ::drow == 0 ? q >= 3 : q < 3)) continue;  // the rows a diagonal gamma drops
    w.v[q] = __ldg(p + (size_t)q * g.Vh);
  }
  const float4* u = U.p + (size_t)((BWD ? 1 - par : par) * 4 + MU) * 3 * g.Vh + (BWD ? n : cb);
#pragma unroll
  for (int q = 0; q < 3; q++) w.u[q] = __ldg(u + (size_t)q * g.Vh);
}

// acc += that term
template <int B, bool DAG, int D>
__device__ __forceinline__ void f32_add(const F32Term& w, const Geom& g, const int x[4], Spinor<float>& acc) {
  constexpr int MU = D >> 1;
  constexpr bool BWD = (D & 1) != 0;
  constexpr int SF = DAG ? +1 : -1;
  using PJ = Proj<B, MU, BWD ? -SF : SF>;
  Spinor<float> v;
#pragma unroll
  for (int q = 0; q < 6; q++) {
    if (PJ::diag && (PJ::drow == 0 ? q >= 3 : q < 3)) continue;
    v.c[(2 * q) / 3][(2 * q) % 3] = {w.v[q].x, w.v[q].y};
    v.c[(2 * q + 1) / 3][(2 * q + 1) % 3] = {w.v[q].z, w.v[q].w};
  }
  Link<float> u;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    u.m[(2 * q) / 3][(2 * q) % 3] = {w.u[q].x, w.u[q].y};
    u.m[(2 * q + 1) / 3][(2 * q + 1) % 3] = {w.u[q].z, w.u[q].w};
  }
  rebuild_row2(u);
  HalfSpinor<float> h, uh;
  PJ::project(v, h);
  if constexpr (BWD) mul_link_dag(u, h, uh);
  else mul_link(u, h, uh);
  const bool flip = MU == 3 && g.bc_sign < 0 && x[3] == (BWD ? 0 : g.L[3] - 1);
  PJ::reconstruct_scaled(acc, uh, flip ? -1.f : 1.f);
}

template <int NT, int B, bool DAG, int EPI>
__global__ void __launch_bounds__(NT, 640 / NT) hop_f32_kernel(HopArgs<SpinorF32, GaugeF32x12> A) {
  const int r = blockIdx.x % A.nrhs, blk = blockIdx.x / A.nrhs;
  if (A.active && !A.active[r]) {
    if (A.norm_part && threadIdx.x == 0) A.norm_part[(size_t)r * A.nblk + blk] = 0.0;
    return;
  }
  const int par = A.out_parity;
  const int cb = blk * NT + threadIdx.x;
  double nrm[1] = {0.0};
  if (cb < A.g.Vh) {
    const Geom& g = A.g;
    int x[4];
    cb_coords(g, cb, par, x);
    const int L0 = g.L[0], L01 = L0 * g.L[1], L012 = L01 * g.L[2];
    const int s = x[0] + L0 * x[1] + L01 * x[2] + L012 * x[3];
    const SpinorF32 in = A.in.shift(r);
    Spinor<float> acc;
    zero(acc);
    F32Term a, b;
    f32_load<B, DAG, 0>(a, in, A.gauge, g, par, cb, x, s, 1);
    f32_load<B, DAG, 1>(b, in, A.gauge, g, par, cb, x, s, 1);
    f32_add<B, DAG, 0>(a, g, x, acc);
    f32_load<B, DAG, 2>(a, in, A.gauge, g, par, cb, x, s, L0);
    f32_add<B, DAG, 1>(b, g, x, acc);
    f32_load<B, DAG, 3>(b, in, A.gauge, g, par, cb, x, s, L0);
    f32_add<B, DAG, 2>(a, g, x, acc);
    f32_load<B, DAG, 4>(a, in, A.gauge, g, par, cb, x, s, L01);
    f32_add<B, DAG, 3>(b, g, x, acc);
    f32_load<B, DAG, 5>(b, in, A.gauge, g, par, cb, x, s, L01);
    f32_add<B, DAG, 4>(a, g, x, acc);
    f32_load<B, DAG, 6>(a, in, A.gauge, g, par, cb, x, s, L012);
    f32_add<B, DAG, 5>(b, g, x, acc);
    f32_load<B, DAG, 7>(b, in, A.gauge, g, par, cb, x, s, L012);
    f32_add<B, DAG, 6>(a, g, x, acc);
    f32_add<B, DAG, 7>(b, g, x, acc);
    nrm[0] = mrhs_epilogue<float, B, EPI>(A, r, par, cb, acc);
  }
  if (A.norm_part) block_partials<1, NT>(nrm, A.norm_part, A.nblk, r, A.nrhs, blk);
}

}  // namespace qkx
