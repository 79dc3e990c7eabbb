// hop_mu4.cuh -- the sloppy hop for batches too small to fill the GPU: an output site split
// over four threads, one per direction, one right-hand side a thread.
//
// On a small lattice a hop is not bound by what it moves but by its chain: a thread that
// walks the eight neighbour terms waits for eight round trips to memory one after the other (8^3x16:
// 4,096 sites of one parity, 32 blocks of 128 threads on 148 SMs).  Here warp mu of a 128-thread block takes the
// forward and backward term of direction mu for 32 sites, so there is one round trip and four times as
// many warps; the four partial spinors meet in shared memory, after which warp w owns spin w of the
// sites for the epilogue (it reads the partner spin that gamma5 brings in as well).
// Same operator and epilogues as hop_mrhs_kernel (reference Vector::applyDslash,
// lib/lattice_util.cpp:1158-1213); the partial sums are added in the order of the directions, so
// results differ from its by the rounding of the sum.
#pragma once
#include "hop_mrhs.cuh"

namespace qkx {

constexpr int MU4_NS = 32;  // sites per block

// colours 0..2 of spin sp of one site, in the accessors' storage (scale is the site's largest component)
template <class Ld>
__device__ __forceinline__ void store_spin(const SpinorF16T<Ld>& f, int parity, int cb, int sp, const Cx<float> (&v)[3],
                                           float scale) {
  if (!(scale >= 1.17549435e-38f)) scale = 0.f;  // as SpinorF16::store
  const float inv = scale > 0.f ? 1.f / scale : 0.f;
  uint4* b = (parity ? f.p1 : f.p0) + cb;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int k = sp * 3 + a;
    const __half2 h = __floats2half2_rn(v[a].re * inv, v[a].im * inv);
    reinterpret_cast<uint32_t*>(b + (size_t)(k >> 2) * f.Vh)[k & 3] = *reinterpret_cast<const uint32_t*>(&h);
  }
  if (sp == 0) (parity ? f.n1 : f.n0)[cb] = scale;
}
template <class Ld>
__device__ __forceinline__ void store_spin(const SpinorF32T<Ld>& f, int parity, int cb, int sp, const Cx<float> (&v)[3],
                                           float) {
  float4* b = (parity ? f.p1 : f.p0) + cb;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int k = sp * 3 + a;
    reinterpret_cast<float2*>(b + (size_t)(k >> 1) * f.Vh)[k & 1] = make_float2(v[a].re, v[a].im);
  }
}
template <class Ld>
__device__ __forceinline__ void load_spin(const SpinorF32T<Ld>& f, int parity, int cb, int sp, Cx<float> (&v)[3]) {
  const float4* b = (parity ? f.p1 : f.p0) + cb;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int k = sp * 3 + a;
    const float2 d = Ld::ld(reinterpret_cast<const float2*>(b + (size_t)(k >> 1) * f.Vh) + (k & 1));
    v[a] = {d.x, d.y};
  }
}

// The work of one block of 128 threads: 32 sites from blk * 32, right-hand side r.
template <int EPI, class ARGS>
__device__ __forceinline__ void hop_mu4_block(const ARGS& A, int blk, int r) {
  static_assert(EPI == EPI_TWIST_INV || EPI == EPI_XPAY_G5 || EPI == EPI_XPAY_G5_CGR, "the solver's epilogues");
  using SP = decltype(ARGS::in);
  using GA = decltype(ARGS::gauge);
  __shared__ float sum[4][24][MU4_NS];
  __shared__ float top[4][MU4_NS];
  __shared__ double red[4];
  if (A.active && !A.active[r]) {
    if (A.norm_part && threadIdx.x == 0) A.norm_part[(size_t)r * A.nblk + blk] = 0.0;
    return;
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int par = A.out_parity;
  const bool inside = blk * MU4_NS + lane < A.g.Vh;
  const int cb = inside ? blk * MU4_NS + lane : A.g.Vh - 1;  // spare lanes repeat the last site and store nothing
  {
    int x[4];
    cb_coords(A.g, cb, par, x);
    const int L0 = A.g.L[0], L01 = L0 * A.g.L[1], L012 = L01 * A.g.L[2];
    const int s = x[0] + L0 * x[1] + L01 * x[2] + L012 * x[3];
    const SP in[1] = {A.in.shift(r)};
    const bool act[1] = {true};
    Spinor<float> acc[1];
    zero(acc[0]);
    if (w == 0) hop_dir_m<1, SP, GA, float, 0, false, 0>(in, A.gauge, A.g, par, cb, x, s, 1, act, acc);
    else if (w == 1) hop_dir_m<1, SP, GA, float, 0, false, 1>(in, A.gauge, A.g, par, cb, x, s, L0, act, acc);
    else if (w == 2) hop_dir_m<1, SP, GA, float, 0, false, 2>(in, A.gauge, A.g, par, cb, x, s, L01, act, acc);
    else hop_dir_m<1, SP, GA, float, 0, false, 3>(in, A.gauge, A.g, par, cb, x, s, L012, act, acc);
#pragma unroll
    for (int k = 0; k < 12; k++) {
      sum[w][2 * k][lane] = acc[0].c[k / 3][k % 3].re;
      sum[w][2 * k + 1][lane] = acc[0].c[k / 3][k % 3].im;
    }
  }
  __syncthreads();
  auto total = [&](int c) { return ((sum[0][c][lane] + sum[1][c][lane]) + sum[2][c][lane]) + sum[3][c][lane]; };
  const float c = float(A.c * (A.cvec ? A.cvec[r] : 1.0));
  const int sg = w ^ 2;  // the spin gamma5 exchanges with w
  Cx<float> o[3];
  int so = w;  // the output spin that o is
  if constexpr (EPI == EPI_TWIST_INV) {
    const float sc = float(A.s * (A.svec ? A.svec[r] : 1.0));
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const Cx<float> v = {total((w * 3 + a) * 2), total((w * 3 + a) * 2 + 1)};
      const Cx<float> g = {total((sg * 3 + a) * 2), total((sg * 3 + a) * 2 + 1)};
      o[a] = sc * (v - c * phase<1>(g));
    }
  } else {
    const float a_ = float(A.a);
    const Spinor<float> xv = A.x.shift(r).load(par, cb);
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const Cx<float> v = {total((w * 3 + a) * 2), total((w * 3 + a) * 2 + 1)};
      Cx<float> xw = xv.c[0][a], xg = xv.c[2][a];
#pragma unroll
      for (int q = 1; q < 4; q++)
        if (w == q) xw = xv.c[q][a], xg = xv.c[q ^ 2][a];
      o[a] = a_ * v + (xw + c * phase<1>(xg));
    }
    so = sg;  // times gamma5
  }
  double nrm = 0.0;
  if constexpr (EPI == EPI_XPAY_G5_CGR) {
    if (inside) {
      const auto rr = A.racc32.shift(r);
      const float al = float(A.alpha[r]);
      Cx<float> q[3];
      load_spin(rr, par, cb, so, q);
#pragma unroll
      for (int a = 0; a < 3; a++) {
        q[a].re = q[a].re - al * o[a].re;
        q[a].im = q[a].im - al * o[a].im;
        nrm += double(q[a].re) * double(q[a].re) + double(q[a].im) * double(q[a].im);
      }
      store_spin(rr, par, cb, so, q, 0.f);
    }
  } else {
    float m = 0.f;
    if constexpr (SP::has_norm) {
#pragma unroll
      for (int a = 0; a < 3; a++) m = fmaxf(m, fmaxf(fabsf(o[a].re), fabsf(o[a].im)));
      top[w][lane] = m;
      __syncthreads();
      m = fmaxf(fmaxf(top[0][lane], top[1][lane]), fmaxf(top[2][lane], top[3][lane]));
    }
    if (inside) {
      store_spin(A.out.shift(r), par, cb, so, o, m);
      if (A.norm_part) {
#pragma unroll
        for (int a = 0; a < 3; a++) nrm += double(o[a].re) * double(o[a].re) + double(o[a].im) * double(o[a].im);
      }
    }
  }
  if (A.norm_part) {
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, k);
    if (lane == 0) red[w] = nrm;
    __syncthreads();
    if (threadIdx.x == 0) A.norm_part[(size_t)r * A.nblk + blk] = ((red[0] + red[1]) + red[2]) + red[3];
  }
}

template <class SP, class GA, int EPI>
__global__ void __launch_bounds__(128) hop_mu4_kernel(HopArgs<SP, GA> A) {
  hop_mu4_block<EPI>(A, blockIdx.x / A.nrhs, blockIdx.x % A.nrhs);
}

}  // namespace qkx
