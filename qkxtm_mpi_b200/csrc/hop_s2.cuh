// hop_s2.cuh -- FP64 hopping term with each output site split over two
// threads, one per row of the projected half spinor.
//
// (1 +- g_mu) psi has two independent rows; row s (s = 0, 1) needs only spins s
// and c_s of the neighbour (c_s = gcol(mu, s)), and its product with the link
// contributes only to the same two spins of the output.  Thread (site, s)
// therefore reads half of the neighbour spinor (6 of 12 words; 3 for the
// diagonal g_4), the whole link, and does half of the arithmetic: no spinor
// word is read and no projection computed twice, only the link is shared (the
// second warp finds it in L1).  For x and y the partner spins are crossed
// (c_s = 3 - s) and for z and t straight (s + 2), so the threads exchange that
// accumulator once, through shared memory, between y and z; after the exchange
// a thread holds spins s and s + 2 of its site, which every epilogue (g5, the
// twist) closes on.  The additions per output component come in the order of a
// one-thread kernel, so the split changes no bit of the result.  Same operator
// and epilogues as hop.cuh (reference Vector::applyDslash / applyDslashDag,
// lib/lattice_util.cpp:1158-1213, 1643-1699; 18-real links exactly as given,
// boundary sign included).
//
// What bounds it: latency of the gathers at 16 warps an SM (128 registers a
// thread), with the L1 data path next (3.6 KB pass through it per site).  A split
// over three colour threads, which this replaced, read every spinor word and did
// every projection three times (5.2 KB a site).  Measured on one B200:
//                                              colour threads   this kernel
//   tm, 32^3x64 (both parities, one launch)        0.600 ms       0.463 ms   (4.3 TB/s of algorithmic bytes)
//   tm, 24^3x48                                    0.199 ms       0.157 ms
//   A^-1 D, one parity, 24^3x48                    0.122 ms       0.094 ms   (5.4 TB/s)
//   A^-1 D, one parity, 32^3x64, 12 RHS            3.77 ms        2.36 ms    (NR = 2; 2.60 with NR = 1)
//   tm_xxDagTm_xx, 24^3x48 (four hops)             0.515 ms       0.400 ms
// (the two one-parity times with the fields on the read-only path).  Tried and slower: 96 registers and 20 warps (0.158 ms for the 24^3x48 tm, 2.68 ms
// for the batch), 80 registers with spills, both halves of a site in adjacent lanes
// (0.156 ms, 2.78 ms), 128 sites a block, links past L1 (0.55 ms at 32^3x64), and L2
// prefetches of the blocks to come (0.55-0.66 ms).  A pair of warps per direction on lattices that do not
// fill the GPU is faster alone on it (8^3x16: 15.1 against 19.7 us for tm_xxDagTm_xx) and slower when
// several lattices' calls overlap (12x14x10x18, three in flight: 21.7 against 15.0 us).
//
// NR right-hand sides per thread share the loaded link.  A block covers 32 sites
// (two warps, one per s), so that s is uniform in a warp and the last wave is fine.
// Grid: blockIdx.x = site_block * groups + group (group of NR right-hand sides);
// with both parities the site blocks alternate parity (link reuse through L2).
#pragma once
#include "hop_c3.cuh"
#include "hop_mrhs.cuh"

namespace qkx {

constexpr int S2_NS = 32;  // sites per block

// a + f * phase<PH>(z), f = +-1 (exact)
template <int PH>
__device__ __forceinline__ Cx<double> add_sph(Cx<double> a, double f, Cx<double> z) {
  const Cx<double> w = phase<PH>(z);
  return {fma(f, w.re, a.re), fma(f, w.im, a.im)};
}

// One neighbour term of row s for NR right-hand sides (input spinors nb[j], link words at ub):
// accA is spin s of the output, accB its partner spin.  sg = s ? -1 : 1: where the phases of
// the two rows differ, they differ by a sign.
template <int NR, int B, bool DAG, int MU, bool FW>
__device__ __forceinline__ void hop_side_s2(const double2* const (&in)[NR], int n, const double2* ub, int Vh, int s,
                                            double sg, Cx<double> (&accA)[NR][3], Cx<double> (&accB)[NR][3]) {
  constexpr int SF = DAG ? +1 : -1;
  using P = Proj<B, MU, FW ? SF : -SF>;
  static_assert(((P::p0 - P::p1) & 1) == 0 && ((P::q0 - P::q1) & 1) == 0, "rows differ by a sign at most");
  const double fp = ((P::p0 - P::p1) & 3) == 0 ? 1.0 : sg;
  const double fq = ((P::q0 - P::q1) & 3) == 0 ? 1.0 : sg;
  Cx<double> u[9];
#pragma unroll
  for (int k = 0; k < 9; k++) u[k] = ld_link(ub + (size_t)k * Vh);
#pragma unroll
  for (int j = 0; j < NR; j++) {
    const double2* nb = in[j] + n;
    Cx<double> h[3];
    if constexpr (P::diag) {
      const double2* b = nb + (size_t)((P::drow + s) * 3) * Vh;
#pragma unroll
      for (int a = 0; a < 3; a++) h[a] = 2.0 * ld_field(b + (size_t)a * Vh);
    } else {
      const int cs = P::c0 == 3 ? 3 - s : 2 + s;
      const double2* b0 = nb + (size_t)(s * 3) * Vh;
      const double2* b1 = nb + (size_t)(cs * 3) * Vh;
      Cx<double> w[3];
#pragma unroll
      for (int a = 0; a < 3; a++) h[a] = ld_field(b0 + (size_t)a * Vh);
#pragma unroll
      for (int a = 0; a < 3; a++) w[a] = ld_field(b1 + (size_t)a * Vh);
#pragma unroll
      for (int a = 0; a < 3; a++) h[a] = add_sph<P::p0>(h[a], fp, w[a]);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      Cx<double> t;
      if constexpr (FW) t = cmul(u[3 * a], h[0]) + cmul(u[3 * a + 1], h[1]) + cmul(u[3 * a + 2], h[2]);
      else t = cmulc(u[a], h[0]) + cmulc(u[3 + a], h[1]) + cmulc(u[6 + a], h[2]);
      if constexpr (P::diag) {
        if constexpr (P::drow == 0) accA[j][a] = accA[j][a] + t;
        else accB[j][a] = accB[j][a] + t;
      } else {
        accA[j][a] = accA[j][a] + t;
        accB[j][a] = add_sph<P::q0>(accB[j][a], fq, t);
      }
    }
  }
}

template <int NR, int B, bool DAG, int MU>
__device__ __forceinline__ void hop_dir_s2(const double2* const (&in)[NR], const GaugeF64x18& U, const Geom& g, int par,
                                           int cb, const int x[4], int sl, int stride, int s, double sg,
                                           Cx<double> (&accA)[NR][3], Cx<double> (&accB)[NR][3]) {
  const int Lm = g.L[MU];
  const int Vh = g.Vh;
  {
    const int n = (x[MU] == Lm - 1 ? sl - (Lm - 1) * stride : sl + stride) >> 1;
    hop_side_s2<NR, B, DAG, MU, true>(in, n, U.p + ((size_t)par * 4 + MU) * 9 * Vh + cb, Vh, s, sg, accA, accB);
  }
  {
    const int n = (x[MU] == 0 ? sl + (Lm - 1) * stride : sl - stride) >> 1;
    hop_side_s2<NR, B, DAG, MU, false>(in, n, U.p + ((size_t)(1 - par) * 4 + MU) * 9 * Vh + n, Vh, s, sg, accA, accB);
  }
}

// gamma5 of a site's spins (s, s + 2), colour by colour
template <int B>
__device__ __forceinline__ void g5_pair(Cx<double> lo, Cx<double> hi, Cx<double>& glo, Cx<double>& ghi) {
  if constexpr (B == 0) {
    glo = hi;
    ghi = lo;
  } else {
    glo = lo;
    ghi = -1.0 * hi;
  }
}

// The fused epilogue of thread (site cb of parity par, spins s and s + 2) for right-hand side rhs;
// stores the output (or, for the residual epilogues, the FP32 residual) and returns this
// thread's share of |output|^2 (|residual|^2).
template <int B, int EPI>
__device__ __forceinline__ double s2_epilogue(const HopArgs<SpinorF64, GaugeF64x18>& A, const HopRes& Rz, int rhs,
                                              int par, int cb, int s, const Cx<double> (&accA)[3],
                                              const Cx<double> (&accB)[3]) {
  const double c = A.c * (A.cvec ? A.cvec[rhs] : 1.0);
  const double sc = A.s * (A.svec ? A.svec[rhs] : 1.0);
  const int Vh = A.g.Vh;
  const size_t o0 = (size_t)(s * 3) * Vh, o1 = (size_t)((s + 2) * 3) * Vh;
  double nrm = 0.0;
  // What the epilogue reads, before the first store (a load cannot pass a store that might alias it); x of EPI_XPAY
  // alone is read colour by colour, which is 1% faster there (tm, 32^3x64: 0.468 -> 0.463 ms).
  constexpr bool HAS_X = EPI != EPI_PLAIN && EPI != EPI_TWIST_INV, X_FIRST = EPI != EPI_XPAY;
  constexpr bool HAS_W = EPI == EPI_XPAY_G5_RES || EPI == EPI_XPAY_RES, HAS_R = EPI == EPI_XPAY_CGR;
  double al = 0.0;
  if constexpr (HAS_R) al = A.alpha[rhs];
  Cx<double> xv[2][3], wv[2][3];
  const SpinorF64 xs = A.x.shift(rhs);
  const double2* xb = (par ? xs.p1 : xs.p0) + cb;
  auto load_x = [&](int a) {
    xv[0][a] = ld_field(xb + o0 + (size_t)a * Vh);
    xv[1][a] = ld_field(xb + o1 + (size_t)a * Vh);
  };
  if constexpr (HAS_X && X_FIRST) {
#pragma unroll
    for (int a = 0; a < 3; a++) load_x(a);
  }
  if constexpr (HAS_W || HAS_R) {
    const SpinorF64 ws = HAS_R ? A.racc64.shift(rhs) : Rz.w.shift(rhs);
    const double2* wb = (par ? ws.p1 : ws.p0) + cb;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      wv[0][a] = ld_field(wb + o0 + (size_t)a * Vh);
      wv[1][a] = ld_field(wb + o1 + (size_t)a * Vh);
    }
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const size_t w0 = o0 + (size_t)a * Vh, w1 = o1 + (size_t)a * Vh;
    Cx<double> lo = accA[a], hi = accB[a], q0, q1;
    if constexpr (EPI == EPI_TWIST_INV) {
      g5_pair<B>(accA[a], accB[a], q0, q1);
      lo = sc * (accA[a] - c * phase<1>(q0));
      hi = sc * (accB[a] - c * phase<1>(q1));
    } else if constexpr (EPI != EPI_PLAIN) {
      if constexpr (!X_FIRST) load_x(a);
      const Cx<double> x0 = xv[0][a], x1 = xv[1][a];
      if constexpr (EPI == EPI_XPAY_TWINV || EPI == EPI_XPAY_TWINV_RES) {
        const Cx<double> v0 = A.a * accA[a] + x0, v1 = A.a * accB[a] + x1;
        g5_pair<B>(v0, v1, q0, q1);
        lo = sc * (v0 - c * phase<1>(q0));
        hi = sc * (v1 - c * phase<1>(q1));
        if constexpr (EPI == EPI_XPAY_TWINV_RES) {
          // the residual of the reconstructed sites, v - A o with A = 1 + i c g5
          g5_pair<B>(lo, hi, q0, q1);
          const Cx<double> z0 = v0 - (lo + c * phase<1>(q0)), z1 = v1 - (hi + c * phase<1>(q1));
          nrm += z0.re * z0.re + z0.im * z0.im + z1.re * z1.re + z1.im * z1.im;
        }
      } else {
        g5_pair<B>(x0, x1, q0, q1);
        lo = A.a * accA[a] + (x0 + c * phase<1>(q0));
        hi = A.a * accB[a] + (x1 + c * phase<1>(q1));
        if constexpr (EPI == EPI_XPAY_G5 || EPI == EPI_XPAY_G5_RES) {
          g5_pair<B>(lo, hi, q0, q1);
          lo = q0;
          hi = q1;
        }
      }
    }
    if constexpr (EPI == EPI_XPAY_G5_RES || EPI == EPI_XPAY_RES) {
      // res = w - o in FP64 and its norm; stored (when a target is given) as FP32, complex
      // k = spin*3 + a in half k%2 of float4 word k/2
      const SpinorF32 rs = Rz.res32.shift(rhs);
      float4* rq = par ? rs.p1 : rs.p0;
      float2* rb = rq ? reinterpret_cast<float2*>(rq + cb) : nullptr;
      const Cx<double> z0 = wv[0][a] - lo, z1 = wv[1][a] - hi;
      nrm += z0.re * z0.re + z0.im * z0.im + z1.re * z1.re + z1.im * z1.im;
      const int k0 = s * 3 + a, k1 = (s + 2) * 3 + a;
      if (rb) {
        rb[2 * (size_t)(k0 >> 1) * Vh + (k0 & 1)] = make_float2(float(z0.re), float(z0.im));
        rb[2 * (size_t)(k1 >> 1) * Vh + (k1 & 1)] = make_float2(float(z1.re), float(z1.im));
      }
    } else if constexpr (EPI == EPI_XPAY_CGR) {
      const SpinorF64 rr = A.racc64.shift(rhs);
      double2* rb = (par ? rr.p1 : rr.p0) + cb;
      const double2 z0 = make_double2(wv[0][a].re - al * lo.re, wv[0][a].im - al * lo.im);
      const double2 z1 = make_double2(wv[1][a].re - al * hi.re, wv[1][a].im - al * hi.im);
      rb[w0] = z0;
      rb[w1] = z1;
      nrm += z0.x * z0.x + z0.y * z0.y + z1.x * z1.x + z1.y * z1.y;
    } else {
      const SpinorF64 os = A.out.shift(rhs);
      double2* ob = (par ? os.p1 : os.p0) + cb;
      ob[w0] = make_double2(lo.re, lo.im);
      ob[w1] = make_double2(hi.re, hi.im);
      if constexpr (EPI != EPI_XPAY_TWINV_RES)
        nrm += lo.re * lo.re + lo.im * lo.im + hi.re * hi.re + hi.im * hi.im;
    }
  }
  return nrm;
}

// Registers: 8 blocks an SM at 128 a thread (NR = 1), 6 at 168 (NR = 2).
template <int NR, int B, bool DAG, int EPI>
__global__ void __launch_bounds__(2 * S2_NS, NR == 1 ? 8 : 6)
    hop_s2_kernel(HopArgs<SpinorF64, GaugeF64x18> A, HopRes Rz) {
  pdl_start();
  const int ngrp = (A.nrhs + NR - 1) / NR;
  const int r0 = (blockIdx.x % ngrp) * NR;
  const int blk = blockIdx.x / ngrp;
  // right-hand sides outside the batch or masked read an active one's fields and store nothing
  bool act[NR];
  int alive = -1;
#pragma unroll
  for (int j = 0; j < NR; j++) {
    act[j] = r0 + j < A.nrhs && (!A.active || A.active[r0 + j]);
    if (act[j]) alive = r0 + j;
  }
  if (alive < 0) {
    if (A.norm_part && threadIdx.x < NR && r0 + (int)threadIdx.x < A.nrhs)
      A.norm_part[(size_t)(r0 + threadIdx.x) * A.nblk + blk] = 0.0;
    return;
  }
  const int ls = threadIdx.x % S2_NS, s = threadIdx.x / S2_NS;
  int par, cb;
  if (A.out_parity < 0) {
    par = blk & 1;
    cb = (blk >> 1) * S2_NS + ls;
  } else {
    par = A.out_parity;
    cb = blk * S2_NS + ls;
  }
  const bool inside = cb < A.g.Vh;
  if (!inside) cb = A.g.Vh - 1;  // the spare threads of the last block repeat its last site and store nothing
  if constexpr (NR == 1 && (EPI == EPI_PLAIN || EPI == EPI_XPAY || EPI == EPI_XPAY_G5)) {
    if (A.zero) {  // the parity that the operator leaves out
#pragma unroll
      for (int k = 0; k < 6; k++) A.zero[(size_t)(s * 6 + k) * A.g.Vh + cb] = make_double2(0.0, 0.0);
    }
  }
  const double2* in[NR];
#pragma unroll
  for (int j = 0; j < NR; j++) {
    const SpinorF64 f = A.in.shift(act[j] ? r0 + j : alive);
    in[j] = par ? f.p0 : f.p1;  // neighbours have the other parity
  }
  int x[4];
  cb_coords(A.g, cb, par, x);
  const int L0 = A.g.L[0], L01 = L0 * A.g.L[1], L012 = L01 * A.g.L[2];
  const int sl = x[0] + L0 * x[1] + L01 * x[2] + L012 * x[3];
  const double sg = s ? -1.0 : 1.0;
  Cx<double> accA[NR][3], accB[NR][3];
#pragma unroll
  for (int k = 0; k < 3 * NR; k++) accA[k / 3][k % 3] = accB[k / 3][k % 3] = {0.0, 0.0};
  hop_dir_s2<NR, B, DAG, 0>(in, A.gauge, A.g, par, cb, x, sl, 1, s, sg, accA, accB);
  hop_dir_s2<NR, B, DAG, 1>(in, A.gauge, A.g, par, cb, x, sl, L0, s, sg, accA, accB);
  __shared__ double2 sw[3 * NR][2][S2_NS];
#pragma unroll
  for (int k = 0; k < 3 * NR; k++) sw[k][1 - s][ls] = make_double2(accB[k / 3][k % 3].re, accB[k / 3][k % 3].im);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 3 * NR; k++) {
    const double2 d = sw[k][s][ls];
    accB[k / 3][k % 3] = {d.x, d.y};
  }
  hop_dir_s2<NR, B, DAG, 2>(in, A.gauge, A.g, par, cb, x, sl, L01, s, sg, accA, accB);
  hop_dir_s2<NR, B, DAG, 3>(in, A.gauge, A.g, par, cb, x, sl, L012, s, sg, accA, accB);
  double nrm[NR];
#pragma unroll
  for (int j = 0; j < NR; j++) {
    nrm[j] = 0.0;
    if (inside && act[j]) nrm[j] = s2_epilogue<B, EPI>(A, Rz, r0 + j, par, cb, s, accA[j], accB[j]);
  }
  if (A.norm_part) block_partials<NR, 2 * S2_NS>(nrm, A.norm_part, A.nblk, r0, A.nrhs, blk);
}

inline int s2_blocks_per_rhs(int Vh, int out_parity) {
  const int per_par = (Vh + S2_NS - 1) / S2_NS;
  return out_parity < 0 ? 2 * per_par : per_par;
}

}  // namespace qkx
