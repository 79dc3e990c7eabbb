// contract.cu -- meson, nucleon and decuplet two-point functions from propagators
// (lib/contractions.cpp: Meson::contract :251, Baryon::contract :494,
// Baryon_Dec::contract :768, their fourier(FORWARD) :121 / :356 / :703 and
// createMomenta :37; contractNucleon, lib/lattice_util.cpp:3374) on one B200.
//
// A propagator is [V][4][4][3][3] complex in the host layout (Propagator::M).
// Per site the contraction needs the whole site block (2304 bytes per
// propagator), so blocks stage 8 sites' blocks in shared memory by cp.async
// and then compute with 16 (mesons) or 8 (nucleons) threads a site, see the
// kernels, or one thread per (site, i, gamma, gamma') (decuplet, i the spatial
// C gamma_i).  The spin structure comes from the gamma and charge-conjugation
// matrices of lib/lattice_util.cpp:255-305, tabulated on the host with the
// reference's threshold |value|^2 > 1e-3.
//
// The Fourier transform has the reference's phase convention,
//   F[t][p] = sum_x C(x) exp(-2 pi i sum_mu p_mu (x_mu - x_src_mu) / L_mu),
// pi = 3.14159265359 as in lib/contractions.cpp:5, x - x_src not wrapped; the
// phase is a product over the directions, so it runs as a sum over each (x, y)
// plane for every distinct (p_x, p_y) and then one over z, for all components
// of a call at once.
#include <string.h>

#include <math.h>
#include <stdlib.h>

#include <algorithm>
#include <complex>
#include <vector>

#include "qkx_ctx.cuh"

using namespace qkx;

namespace qkx {
namespace {

constexpr int CT_SITES = 8;            // sites per block
constexpr int CT_STRIDE = 145;         // double2 per staged site: 144 + 1 of padding, so the 8 sites
                                       // of a quarter warp fall on different shared-memory banks
constexpr double REF_PI = 3.14159265359;
using zc = std::complex<double>;

int bad(const char* what) {
  set_error("invalid argument: %s", what);
  return QKX_ERR_INVALID;
}

// ---------------------------------------------------------------- host tables
struct Gammas {
  zc G[5][4][4], C[4][4], Cbar[4][4], CG[5][4][4], CGbar[5][4][4];
  Gammas() {  // std::complex members start at zero
    const zc j(0, 1);
    G[0][0][3] = j, G[0][1][2] = j, G[0][2][1] = -j, G[0][3][0] = -j;
    G[1][0][3] = 1, G[1][1][2] = -1, G[1][2][1] = -1, G[1][3][0] = 1;
    G[2][0][2] = j, G[2][1][3] = -j, G[2][2][0] = -j, G[2][3][1] = j;
    G[3][0][0] = 1, G[3][1][1] = 1, G[3][2][2] = -1, G[3][3][3] = -1;
    G[4][0][2] = 1, G[4][1][3] = 1, G[4][2][0] = 1, G[4][3][1] = 1;
    for (int m = 0; m < 4; m++)
      for (int n = 0; n < 4; n++)
        for (int k = 0; k < 4; k++) C[m][n] += G[1][m][k] * G[3][k][n];
    for (int m = 0; m < 4; m++)
      for (int n = 0; n < 4; n++)
        for (int k = 0; k < 4; k++)
          for (int l = 0; l < 4; l++) Cbar[m][n] += G[3][m][l] * std::conj(C[k][l]) * G[3][k][n];
    for (int i = 0; i < 5; i++)
      for (int m = 0; m < 4; m++)
        for (int n = 0; n < 4; n++)
          for (int k = 0; k < 4; k++) CG[i][m][n] += C[m][k] * G[i][k][n];
    for (int i = 0; i < 5; i++)
      for (int m = 0; m < 4; m++)
        for (int n = 0; n < 4; n++)
          for (int k = 0; k < 4; k++)
            for (int l = 0; l < 4; l++) CGbar[i][m][n] += G[3][m][l] * std::conj(CG[i][k][l]) * G[3][k][n];
  }
};

bool keep(zc v) { return std::norm(v) > 1e-3; }

// ---- mesons (Meson::contract, lib/contractions.cpp:251)
// Every gamma here has one entry per row, in column row ^ m.  The terms of an operator then pair
// the spin block i = (alpha, beta) of the propagator with the block (alpha ^ n, beta ^ n), n = m ^ 2,
// of its conjugate (g5 on either side moves a spin by ^ 2), so an operator is one n and 16 weights.
struct MesonWeights {
  int n[QKX_NUM_MESONS];
  double2 w[QKX_NUM_MESONS][16];  // [alpha*4 + beta]
};

int meson_weights(const Gammas& g, int op, int slot, MesonWeights& t) {
  zc m[4][4] = {};
  if (op == 0) {
    for (int i = 0; i < 4; i++) m[i][i] = 1;
  } else if (op == 1) {
    memcpy((void*)m, g.G[4], sizeof m);
  } else if (op <= 5) {
    memcpy((void*)m, g.G[op - 2], sizeof m);
  } else {
    for (int a = 0; a < 4; a++)
      for (int b = 0; b < 4; b++)
        for (int k = 0; k < 4; k++) m[a][b] += g.G[4][a][k] * g.G[op - 6][k][b];
  }
  int n = -1;
  for (int i = 0; i < 16; i++) t.w[slot][i] = make_double2(0.0, 0.0);
  for (int be = 0; be < 4; be++)
    for (int ga = 0; ga < 4; ga++)
      for (int de = 0; de < 4; de++)
        for (int al = 0; al < 4; al++) {
          const zc v = m[be][ga] * m[de][al];
          if (!keep(v)) continue;
          const int na = al ^ (de ^ 2), nb = be ^ (ga ^ 2);
          if (na != nb || (n >= 0 && n != na)) return QKX_ERR_INVALID;
          n = na;
          t.w[slot][al * 4 + be] = make_double2(v.real(), v.imag());
        }
  t.n[slot] = n;
  return n < 0 ? QKX_ERR_INVALID : QKX_OK;
}

// ---- nucleons (Baryon::contract, lib/contractions.cpp:494).  The diquark's spin matrices (C or C g5 at
// the sink, their bars at the source) have one entry per row, as has the g5 that NTR, RTN and RTR put on
// the third quark: with beta(alpha), beta'(alpha') and the products of the entries f, and (X, Y) the spins
// of the third quark's element for (gamma, gamma'), the sum over spin terms is a sum over alpha, alpha'.
struct BaryonSpin {
  int be[4], bp[4];   // beta of alpha, beta' of alpha'
  int g[4], gp[4];    // gamma of X, gamma' of Y
  double f[4][4];     // [alpha][alpha']
  double w[4][4];     // sign and g5 entries of output [X][Y]
};

int baryon_spin(const Gammas& g, int op, BaryonSpin& t) {
  const zc(*S1)[4] = op < 2 ? g.CG[4] : g.C;
  const zc(*S2)[4] = (op == 0 || op == 2) ? g.CGbar[4] : g.Cbar;
  zc v1[4], v2[4], gx[4], gy[4];
  for (int a = 0; a < 4; a++) {
    int n1 = 0, n2 = 0, nx = 0, ny = 0;
    for (int b = 0; b < 4; b++) {
      if (keep(S1[a][b])) t.be[a] = b, v1[a] = S1[a][b], n1++;
      if (keep(S2[b][a])) t.bp[a] = b, v2[a] = S2[b][a], n2++;
      const zc sink = op >= 2 ? g.G[4][b][a] : zc(b == a), src = (op & 1) ? g.G[4][b][a] : zc(b == a);
      if (keep(sink)) t.g[a] = b, gx[a] = sink, nx++;
      if (keep(src)) t.gp[a] = b, gy[a] = src, ny++;
    }
    if (n1 != 1 || n2 != 1 || nx != 1 || ny != 1) return QKX_ERR_INVALID;
  }
  const double sign = (op == 1 || op == 3) ? -1.0 : 1.0;
  for (int a = 0; a < 4; a++)
    for (int b = 0; b < 4; b++) {
      const zc f = v1[a] * v2[b], w = sign * gx[a] * gy[b];
      if (f.imag() != 0.0 || w.imag() != 0.0) return QKX_ERR_INVALID;
      t.f[a][b] = f.real();
      t.w[a][b] = w.real();
    }
  return QKX_OK;
}

// ---------------------------------------------------------------- device
__device__ __forceinline__ double2 cm(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

// stage the site blocks (144 complex each) of CT_SITES sites into shared memory, site s at
// sp + s * CT_STRIDE, zeros past the lattice; the caller waits (cp.async.wait_all) and synchronizes
__device__ __forceinline__ void stage(double2* sp, const double2* __restrict__ prop, size_t s0, size_t V) {
  for (int i = threadIdx.x; i < CT_SITES * 144; i += blockDim.x) {
    const int ls = i / 144;
    double2* d = sp + ls * CT_STRIDE + i % 144;
    if (s0 + ls < V) cp_async16(d, prop + s0 * 144 + i);
    else *d = make_double2(0.0, 0.0);
  }
}
__device__ __forceinline__ void stage_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// a += x * y
__device__ __forceinline__ void cmac(double2& a, double2 x, double2 y) {
  a.x += x.x * y.x;
  a.x -= x.y * y.y;
  a.y += x.x * y.y;
  a.y += x.y * y.x;
}

// C[op][site], 16 threads a site.  Thread (d, b) of a site forms the four products
// Q_n = sum_colours P[d][b] conj(P[d ^ n][b ^ n]); an operator is a weighted sum of its n's 16
// products.  That is 576 complex multiply-adds a site for any number of operators, where one
// operator summed over its own terms takes 288, and the propagator is read once (ten operators at 24^3x48:
// 1.67 -> 0.43 ms, 3.6 TB/s of that read, 55% of the copy rate: a block loads its sites, waits, then computes).
__global__ void __launch_bounds__(CT_SITES * 16) k_meson_sites(const double2* __restrict__ prop, size_t V, int nop,
                                                               MesonWeights T, double2* __restrict__ C) {
  __shared__ double2 sp[CT_SITES * CT_STRIDE];
  const size_t s0 = (size_t)blockIdx.x * CT_SITES;
  stage(sp, prop, s0, V);
  stage_wait();
  const int ls = threadIdx.x % CT_SITES, k = threadIdx.x / CT_SITES, d = k >> 2, b = k & 3;
  double2* pp = sp + ls * CT_STRIDE;  // [mu][nu][c1][c2] at mu*36 + nu*9 + c1*3 + c2
  double2 own[9], q[4];
#pragma unroll
  for (int u = 0; u < 9; u++) own[u] = pp[k * 9 + u];
#pragma unroll
  for (int n = 0; n < 4; n++) {
    const double2* o = pp + ((d ^ n) * 4 + (b ^ n)) * 9;
    q[n] = make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < 9; u++) {
      const double2 z = n == 0 ? own[u] : o[u];
      cmac(q[n], own[u], make_double2(z.x, -z.y));
    }
  }
  __syncthreads();  // the staged blocks make room for the products
#pragma unroll
  for (int n = 0; n < 4; n++) pp[n * 16 + k] = q[n];
  __syncthreads();
  const size_t site = s0 + ls;
  if (k >= nop || site >= V) return;
  const double2* qn = pp + T.n[k] * 16;
  double2 m = make_double2(0.0, 0.0);
#pragma unroll
  for (int i = 0; i < 16; i++) cmac(m, T.w[k][i], qn[i]);
  C[(size_t)k * V + site] = m;
}

// C[gamma*4 + gamma'][site], 8 threads a site.  With D(A, B, C) = eps_abc eps_a'b'c' A_aa' B_bb' C_cc'
// (symmetric in its arguments) and W = f P2[beta][beta'], the sum of one (X, Y) is
//   sum_{alpha, alpha'} D(P1[alpha][alpha'], W, P1[X][Y]) + D(P1[alpha][Y], W, P1[X][alpha']).
// Thread (h, alpha) builds R[X][alpha] = sum_alpha' P1[X][alpha'] x W[alpha][alpha'] for X = h, h + 2, the
// colour cross product (A x B)_cc' = eps_abc eps_a'b'c' A_aa' B_bb'; both parts come from it:
//   sum_alpha <P1[alpha][Y], R[X][alpha]>  and  <sum_alpha R[alpha][alpha], P1[X][Y]>.
// 3,024 complex products a site against 36,864 when each of the 16 (gamma, gamma') walks its own
// spin and colour terms (24^3x48: 8.40 -> 0.82 ms).  Bound by the shared-memory reads, then by the FP64
// pipe: one X a thread (16 threads a site) read a third more words and took 0.94 ms.
__global__ void __launch_bounds__(CT_SITES * 8, 6) k_baryon_sites(const double2* __restrict__ p1,
                                                                  const double2* __restrict__ p2, size_t V,
                                                                  BaryonSpin T, double2* __restrict__ C) {
  __shared__ double2 s1[CT_SITES * CT_STRIDE], s2[CT_SITES * CT_STRIDE];
  const size_t s0 = (size_t)blockIdx.x * CT_SITES;
  stage(s1, p1, s0, V);
  stage(s2, p2, s0, V);
  stage_wait();
  const int ls = threadIdx.x % CT_SITES, k = threadIdx.x / CT_SITES, h = k >> 2, al = k & 3;
  const double2* q1 = s1 + ls * CT_STRIDE;
  double2* q2 = s2 + ls * CT_STRIDE;
  double2 R[2][9];
#pragma unroll
  for (int u = 0; u < 18; u++) R[u / 9][u % 9] = make_double2(0.0, 0.0);
  const double2* wrow = q2 + T.be[al] * 36;
#pragma unroll 1
  for (int ap = 0; ap < 4; ap++) {
    double2 E[9];
    const double f = T.f[al][ap];
    const double2* w = wrow + T.bp[ap] * 9;
#pragma unroll
    for (int u = 0; u < 9; u++) E[u] = make_double2(f * w[u].x, f * w[u].y);
#pragma unroll
    for (int x = 0; x < 2; x++) {
      const double2* q = q1 + (h + 2 * x) * 36 + ap * 9;
      // element (i, j) of P1[X][alpha'] meets the four E of the other rows and columns
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
          const double2 A = q[i * 3 + j], nA = make_double2(-A.x, -A.y);
          const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
          cmac(R[x][i2 * 3 + j2], A, E[i1 * 3 + j1]);
          cmac(R[x][i1 * 3 + j1], A, E[i2 * 3 + j2]);
          cmac(R[x][i2 * 3 + j1], nA, E[i1 * 3 + j2]);
          cmac(R[x][i1 * 3 + j2], nA, E[i2 * 3 + j1]);
        }
    }
  }
  double2 t[2][4];
#pragma unroll
  for (int Y = 0; Y < 4; Y++) {
    t[0][Y] = t[1][Y] = make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < 9; u++) {
      const double2 v = q1[al * 36 + Y * 9 + u];
      cmac(t[0][Y], v, R[0][u]);
      cmac(t[1][Y], v, R[1][u]);
    }
  }
  // P2's blocks make room for the exchange: t at [X][alpha][Y], then R[alpha][alpha], then their sum
  __syncthreads();
#pragma unroll
  for (int x = 0; x < 2; x++) {
    const int X = h + 2 * x;
#pragma unroll
    for (int Y = 0; Y < 4; Y++) q2[(X * 4 + al) * 4 + Y] = t[x][Y];
    if (X == al) {
#pragma unroll
      for (int u = 0; u < 9; u++) q2[64 + al * 9 + u] = R[x][u];
    }
  }
  __syncthreads();
  for (int u = k; u < 9; u += 8) {
    double2 z = q2[64 + u];
#pragma unroll
    for (int a = 1; a < 4; a++) {
      z.x += q2[64 + a * 9 + u].x;
      z.y += q2[64 + a * 9 + u].y;
    }
    q2[100 + u] = z;
  }
  __syncthreads();
  const size_t site = s0 + ls;
  if (site >= V) return;
  const int Y = al;  // from here thread (h, Y) owns the outputs (h, Y) and (h + 2, Y)
#pragma unroll
  for (int x = 0; x < 2; x++) {
    const int X = h + 2 * x;
    double2 m = make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < 9; u++) cmac(m, q2[100 + u], q1[(X * 4 + Y) * 9 + u]);
#pragma unroll
    for (int a = 0; a < 4; a++) {
      m.x += q2[(X * 4 + a) * 4 + Y].x;
      m.y += q2[(X * 4 + a) * 4 + Y].y;
    }
    const double w = T.w[X][Y];
    C[(size_t)(T.g[X] * 4 + T.gp[Y]) * V + site] = make_double2(w * m.x, w * m.y);
  }
}

// ---- decuplet (Baryon_Dec): per spatial i, the terms (value; alpha, beta, beta', alpha')
// of (C gamma_i)[alpha][beta] (C gamma_i)bar[beta'][alpha'] in tabulateIndices_Delta's
// order (lib/contractions.cpp:743-765)
constexpr int DELTA_MAX_TERMS = 64;
struct DeltaTerms {
  int n[3];
  double2 val[3][DELTA_MAX_TERMS];
  char4 ab[3][DELTA_MAX_TERMS];  // alpha, beta, beta', alpha'
};

int delta_terms(const Gammas& g, DeltaTerms& t) {
  memset(t.n, 0, sizeof t.n);
  for (int i = 0; i < 3; i++)
    for (int al = 0; al < 4; al++)
      for (int be = 0; be < 4; be++)
        for (int bp = 0; bp < 4; bp++)
          for (int ap = 0; ap < 4; ap++) {
            const zc v = g.CG[i][al][be] * g.CGbar[i][bp][ap];
            if (!keep(v)) continue;
            if (t.n[i] >= DELTA_MAX_TERMS) return QKX_ERR_INVALID;
            t.val[i][t.n[i]] = make_double2(v.real(), v.imag());
            t.ab[i][t.n[i]] = make_char4(al, be, bp, ap);
            t.n[i]++;
          }
  return QKX_OK;
}

constexpr int DT_SITES = CT_SITES;  // sites per block of the decuplet kernel (48 threads a site)

// The six permutations (a, b, c) of lib/contractions.cpp:14-19 in their order, two bits a
// colour, six bits a permutation, as one constant (no table in memory); sign +1 for the first
// three, -1 for the others.
constexpr unsigned long long EPS_PACKED =
    (0ull | 1ull << 2 | 2ull << 4) | (2ull | 0ull << 2 | 1ull << 4) << 6 | (1ull | 2ull << 2 | 0ull << 4) << 12 |
    (2ull | 1ull << 2 | 0ull << 4) << 18 | (0ull | 2ull << 2 | 1ull << 4) << 24 | (1ull | 0ull << 2 | 2ull << 4) << 30;
__device__ __forceinline__ int eps_at(int e, int j) { return (int)((EPS_PACKED >> (6 * e + 2 * j)) & 3ull); }

// C[i*16 + gamma*4 + gamma'][site] of Baryon_Dec::contract (lib/contractions.cpp:768-866):
// one thread per (site, i, gamma, gamma'); op 0 DELTA_ISO1 (three quarks of p1),
// 1 DELTA_ISO1O2 (p2 for the odd quark, the reference's weights 1/3 x {4, 2, 1}).
// Each term reads its colour entries from the staged site blocks.
// Every index the kernel takes from its term table is checked before use: a value out of range
// records a code in *err and the term is skipped, so a bad table cannot address outside the
// staged blocks.
__global__ void __launch_bounds__(DT_SITES * 48) k_delta_sites(const double2* __restrict__ p1,
                                                               const double2* __restrict__ p2, size_t V, int op,
                                                               const DeltaTerms* __restrict__ T,
                                                               double2* __restrict__ C, int* __restrict__ err) {
  extern __shared__ double2 sb[];
  double2* s1 = sb;
  double2* s2 = sb + DT_SITES * CT_STRIDE;
  const size_t s0 = (size_t)blockIdx.x * DT_SITES;
  stage(s1, p1, s0, V);
  stage(s2, p2, s0, V);
  stage_wait();
  const int ls = threadIdx.x % DT_SITES, k = threadIdx.x / DT_SITES;  // k = i*16 + gamma*4 + gamma'
  const size_t site = s0 + ls;
  if (site >= V) return;
  const int i = k >> 4, g = (k >> 2) & 3, gp = k & 3;
  const double2* q1 = s1 + ls * CT_STRIDE;
  const double2* q2 = s2 + ls * CT_STRIDE;
  // entry [s1][s2][c1][c2] of propagator q
  auto at = [](const double2* q, int sa, int sb_, int ca, int cb) { return q[sa * 36 + sb_ * 9 + ca * 3 + cb]; };
  double2 m = make_double2(0.0, 0.0);
  int n = T->n[i];
  if (n < 0 || n > DELTA_MAX_TERMS) {
    atomicCAS(err, 0, 1000 + n);
    n = 0;
  }
  for (int idx = 0; idx < n; idx++) {
    const double2 val = T->val[i][idx];
    const char4 ab = T->ab[i][idx];
    const int al = ab.x, be = ab.y, bp = ab.z, ap = ab.w;
    if ((unsigned)al > 3u || (unsigned)be > 3u || (unsigned)bp > 3u || (unsigned)ap > 3u) {
      atomicCAS(err, 0, 2000 + idx);
      continue;
    }
    for (int e1 = 0; e1 < 6; e1++) {
      const int a = eps_at(e1, 0), b = eps_at(e1, 1), c = eps_at(e1, 2);
      for (int e2 = 0; e2 < 6; e2++) {
        const int a1 = eps_at(e2, 0), b1 = eps_at(e2, 1), c1 = eps_at(e2, 2);
        const double f = (e1 < 3) == (e2 < 3) ? 1.0 : -1.0;
        double2 t;
        if (op == 0) {
          const double2 t1 = cm(cm(at(q1, al, gp, a, c1), at(q1, be, bp, b, b1)), at(q1, g, ap, c, a1));
          const double2 t2 = cm(cm(at(q1, al, bp, a, b1), at(q1, be, gp, b, c1)), at(q1, g, ap, c, a1));
          const double2 t3 = cm(cm(at(q1, al, gp, a, c1), at(q1, be, ap, b, a1)), at(q1, g, bp, c, b1));
          const double2 t4 = cm(cm(at(q1, al, ap, a, a1), at(q1, be, gp, b, c1)), at(q1, g, bp, c, b1));
          const double2 t5 = cm(cm(at(q1, al, bp, a, b1), at(q1, be, ap, b, a1)), at(q1, g, gp, c, c1));
          const double2 t6 = cm(cm(at(q1, al, ap, a, a1), at(q1, be, bp, b, b1)), at(q1, g, gp, c, c1));
          t = make_double2(-t1.x + t2.x + t3.x - t4.x - t5.x + t6.x, -t1.y + t2.y + t3.y - t4.y - t5.y + t6.y);
        } else {
          const double2 t1 = cm(cm(at(q1, al, gp, a, c1), at(q2, be, bp, b, b1)), at(q1, g, ap, c, a1));
          const double2 t2 = cm(cm(at(q1, al, bp, a, b1), at(q2, be, gp, b, c1)), at(q1, g, ap, c, a1));
          const double2 t3 = cm(cm(at(q1, al, gp, a, c1), at(q1, be, ap, b, a1)), at(q2, g, bp, c, b1));
          const double2 t4 = cm(cm(at(q1, al, ap, a, a1), at(q1, be, gp, b, c1)), at(q2, g, bp, c, b1));
          const double2 t5 = cm(cm(at(q1, al, ap, a, a1), at(q2, be, gp, b, c1)), at(q1, g, bp, c, b1));
          const double2 t6 = cm(cm(at(q1, al, bp, a, b1), at(q1, be, ap, b, a1)), at(q2, g, gp, c, c1));
          const double2 t7 = cm(cm(at(q1, al, ap, a, a1), at(q1, be, bp, b, b1)), at(q2, g, gp, c, c1));
          const double2 t8 = cm(cm(at(q1, al, ap, a, a1), at(q2, be, bp, b, b1)), at(q1, g, gp, c, c1));
          const double third = 1.0 / 3.0;
          t = make_double2(third * (-4 * t1.x + 2 * t2.x + 2 * t3.x - 2 * t4.x - 2 * t5.x - t6.x + t7.x + 4 * t8.x),
                           third * (-4 * t1.y + 2 * t2.y + 2 * t3.y - 2 * t4.y - 2 * t5.y - t6.y + t7.y + 4 * t8.y));
        }
        const double2 v = cm(make_double2(f * val.x, f * val.y), t);
        m.x += v.x;
        m.y += v.y;
      }
    }
  }
  C[(size_t)k * V + site] = m;
}

// The momenta of a call as its transform uses them: distinct (p_x, p_y) ordered by p_x with the
// phases of x and y, each momentum's pair and p_z, phases exp(-2 pi i n (x - x_src) / L), n = -nm..nm.
struct FourierTables {
  const double2 *ex, *ey, *ez;  // [2 nm + 1][L]
  const int2* mom;              // [nmom] pair, row of ez
  const int* first;             // [2 nm + 2] first pair of every p_x
  const int* py;                // [npair] row of ey
  int nx, npair, nmom;          // nx = 2 nm + 1
};
constexpr int FT_NX = 5;  // p_x values a lane accumulates at once (all of them up to Q^2 = 8)

// G[t][z][pair][k] = sum over the (x, y) plane of C[k][site] ex ey; a warp per (plane, component).
// A lane takes a row y: it sums the row against every p_x (the phases are the same for all lanes),
// then the warp sums the rows against the p_y of each pair.  20 FP64 operations a site and
// component for the 13 pairs up to Q^2 = 4, and C is read once (26 components at 24^3x48: 0.19 ms); a block
// per (t, p) that formed
// sincos and re-read the slice for each momentum took 6.4 ms.
__global__ void __launch_bounds__(256) k_fourier_xy(const double2* __restrict__ C, int K, int planes, size_t V, int Lx,
                                                    int Ly, FourierTables T, double2* __restrict__ G) {
  const int w = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= planes * K) return;
  const int plane = w / K, k = w - plane * K;
  const double2* c = C + (size_t)k * V + (size_t)plane * Lx * Ly;
  double2* g = G + (size_t)plane * T.npair * K + k;
  for (int n0 = 0; n0 < T.nx; n0 += FT_NX) {
    for (int y0 = 0; y0 < Ly; y0 += 32) {
      const int y = y0 + lane;
      double2 acc[FT_NX];
      const double2* ex[FT_NX];
#pragma unroll
      for (int j = 0; j < FT_NX; j++) {
        acc[j] = make_double2(0.0, 0.0);
        ex[j] = T.ex + (size_t)min(n0 + j, T.nx - 1) * Lx;
      }
      if (y < Ly) {
        const double2* row = c + (size_t)y * Lx;
#pragma unroll 4
        for (int x = 0; x < Lx; x++) {
          const double2 v = __ldg(row + x);
#pragma unroll
          for (int j = 0; j < FT_NX; j++) cmac(acc[j], v, __ldg(ex[j] + x));
        }
      }
#pragma unroll
      for (int j = 0; j < FT_NX; j++) {
        if (n0 + j >= T.nx) break;
        for (int p = T.first[n0 + j]; p < T.first[n0 + j + 1]; p++) {
          double2 a = y < Ly ? cm(acc[j], __ldg(T.ey + (size_t)T.py[p] * Ly + y)) : make_double2(0.0, 0.0);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
            a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
          }
          if (lane == 0) {
            double2& d = g[(size_t)p * K];
            d = y0 == 0 ? a : make_double2(d.x + a.x, d.y + a.y);
          }
        }
      }
    }
  }
}

// F[t][p][k] (or F[k][t][p] when k_major) = sum_z G[t][z][pair(p)][k] ez
__global__ void __launch_bounds__(256) k_fourier_z(const double2* __restrict__ G, int K, int Lz, int Lt,
                                                   FourierTables T, int k_major, double2* __restrict__ F) {
  const size_t n = (size_t)Lt * T.nmom * K, i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const int k = (int)(i % K), p = (int)(i / K % T.nmom), t = (int)(i / K / T.nmom);
  const int2 m = T.mom[p];
  double2 a = make_double2(0.0, 0.0);
  for (int z = 0; z < Lz; z++)
    cmac(a, __ldg(G + (((size_t)t * Lz + z) * T.npair + m.x) * K + k), __ldg(T.ez + (size_t)m.y * Lz + z));
  F[k_major ? ((size_t)k * Lt + t) * T.nmom + p : i] = a;
}

int host_momenta(int Q_sq, std::vector<int>& m) {
  m.clear();
  for (int q = 0; q <= Q_sq; q++)
    for (int nx = q; nx >= -q; nx--)
      for (int ny = q; ny >= -q; ny--)
        for (int nz = q; nz >= -q; nz--)
          if (nx * nx + ny * ny + nz * nz == q) m.insert(m.end(), {nx, ny, nz});
  return (int)(m.size() / 3);
}

// a device copy of a host propagator (or the pointer itself for device input)
struct PropIn {
  const double2* d = nullptr;
  void* owned = nullptr;
};

int prop_in(qkx_ctx* c, const double* p, bool host, PropIn& out) {
  if (!host) {
    out.d = (const double2*)p;
    return QKX_OK;
  }
  const size_t bytes = sizeof(double2) * 144 * c->V;
  if (cudaMallocAsync(&out.owned, bytes, c->st) != cudaSuccess) {
    cudaGetLastError();
    set_error("propagator copy: device allocation failed");
    return QKX_ERR_NOMEM;
  }
  QKX_CUDA(cudaMemcpyAsync(out.owned, p, bytes, cudaMemcpyHostToDevice, c->st));
  out.d = (const double2*)out.owned;
  return QKX_OK;
}

// Device memory on the context's stream, released at scope exit.
struct Scratch {
  cudaStream_t st;
  void* p = nullptr;
  explicit Scratch(cudaStream_t s) : st(s) {}
  Scratch(const Scratch&) = delete;
  ~Scratch() {
    if (p) cudaFreeAsync(p, st);
  }
  int alloc(size_t bytes) {
    if (cudaMallocAsync(&p, bytes, st) != cudaSuccess) {
      p = nullptr;
      cudaGetLastError();
      set_error("contraction: device allocation of %zu bytes failed", bytes);
      return QKX_ERR_NOMEM;
    }
    return QKX_OK;
  }
};
// the same for a propagator copied from the host
struct PropCopy : PropIn {
  cudaStream_t st;
  explicit PropCopy(cudaStream_t s) : st(s) {}
  PropCopy(const PropCopy&) = delete;
  ~PropCopy() {
    if (owned) cudaFreeAsync(owned, st);
  }
};

int momenta_of(int Q_sq, std::vector<int>& m) {
  if (Q_sq < 0) return bad("Q_sq < 0");
  if (host_momenta(Q_sq, m) > 1000) return bad("Q_sq gives more than 1000 momenta (MOM_MAX)");
  return QKX_OK;
}

// the Fourier transform of C [K][V] to host memory, [Lt][nmom][K] or [K][Lt][nmom]; waits for it
int fourier_to_host(qkx_ctx* c, const double2* C, int K, const std::vector<int>& m, const int x_src[4], bool k_major,
                    double* out) {
  const int Lx = c->p.L[0], Ly = c->p.L[1], Lz = c->p.L[2], Lt = c->p.L[3];
  const int nmom = (int)(m.size() / 3);
  int nm = 0;
  for (int v : m) nm = std::max(nm, std::abs(v));
  const int nx = 2 * nm + 1;
  // distinct (p_x, p_y), ordered by p_x
  std::vector<int> id((size_t)nx * nx, -1), first(nx + 1, 0), py;
  for (int p = 0; p < nmom; p++) id[(size_t)(m[3 * p] + nm) * nx + m[3 * p + 1] + nm] = 0;
  for (int ix = 0; ix < nx; ix++) {
    for (int iy = 0; iy < nx; iy++)
      if (id[(size_t)ix * nx + iy] == 0) {
        id[(size_t)ix * nx + iy] = (int)py.size();
        py.push_back(iy);
      }
    first[ix + 1] = (int)py.size();
  }
  std::vector<int2> mom(nmom);
  for (int p = 0; p < nmom; p++)
    mom[p] = make_int2(id[(size_t)(m[3 * p] + nm) * nx + m[3 * p + 1] + nm], m[3 * p + 2] + nm);
  const int npair = (int)py.size();
  // one host block for the tables: phases of x, y, z, then the momentum and pair lists
  const size_t nph = (size_t)nx * (Lx + Ly + Lz);
  std::vector<double2> tab(nph + (2 * nmom + nx + 1 + npair + 3) / 4);
  double2* w = tab.data();
  for (int d = 0; d < 3; d++)
    for (int n = -nm; n <= nm; n++)
      for (int x = 0; x < c->p.L[d]; x++) {
        const double th = (((double)n * (x - x_src[d])) / c->p.L[d]) * 2 * REF_PI;
        *w++ = make_double2(cos(th), -sin(th));
      }
  int2* lm = (int2*)(tab.data() + nph);
  std::copy(mom.begin(), mom.end(), lm);
  int* li = (int*)(lm + nmom);
  std::copy(first.begin(), first.end(), li);
  std::copy(py.begin(), py.end(), li + nx + 1);
  const size_t nG = (size_t)Lt * Lz * npair * K, nF = (size_t)Lt * nmom * K;
  Scratch S(c->st);
  QKX_TRY(S.alloc(sizeof(double2) * (tab.size() + nG + nF)));
  double2* dt = (double2*)S.p;
  double2 *dG = dt + tab.size(), *dF = dG + nG;
  QKX_CUDA(cudaMemcpyAsync(dt, tab.data(), sizeof(double2) * tab.size(), cudaMemcpyHostToDevice, c->st));
  FourierTables T;
  T.ex = dt;
  T.ey = T.ex + (size_t)nx * Lx;
  T.ez = T.ey + (size_t)nx * Ly;
  T.mom = (const int2*)(dt + nph);
  T.first = (const int*)(T.mom + nmom);
  T.py = T.first + nx + 1;
  T.nx = nx;
  T.npair = npair;
  T.nmom = nmom;
  const int planes = Lt * Lz;
  k_fourier_xy<<<(unsigned)(((size_t)planes * K + 7) / 8), 256, 0, c->st>>>(C, K, planes, c->V, Lx, Ly, T, dG);
  counted(c);
  QKX_CUDA(cudaGetLastError());
  k_fourier_z<<<(unsigned)((nF + 255) / 256), 256, 0, c->st>>>(dG, K, Lz, Lt, T, k_major ? 1 : 0, dF);
  counted(c);
  QKX_CUDA(cudaGetLastError());
  QKX_CUDA(cudaMemcpyAsync(out, dF, sizeof(double2) * nF, cudaMemcpyDeviceToHost, c->st));
  QKX_CUDA(cudaStreamSynchronize(c->st));
  return QKX_OK;
}

int meson_2pt(qkx_ctx* c, const double* prop, bool host, int nop, const int* ops, int Q_sq, const int x_src[4],
              double* corr) {
  if (!c || !prop || !ops || !x_src || !corr) return bad("NULL argument");
  if (nop < 1 || nop > QKX_NUM_MESONS) return bad("nop must be in 1..10");
  for (int i = 0; i < nop; i++)
    if (ops[i] < 0 || ops[i] >= QKX_NUM_MESONS) return bad("meson operator id");
  std::vector<int> m;
  QKX_TRY(momenta_of(Q_sq, m));
  QKX_CUDA(cudaSetDevice(c->device));
  static const Gammas g;
  MesonWeights T;
  memset(&T, 0, sizeof T);
  for (int i = 0; i < nop; i++)
    if (meson_weights(g, ops[i], i, T) != QKX_OK) return bad("internal: meson spin terms");
  PropCopy pin(c->st);
  QKX_TRY(prop_in(c, prop, host, pin));
  Scratch C(c->st);
  QKX_TRY(C.alloc(sizeof(double2) * nop * c->V));
  const unsigned nb = (unsigned)((c->V + CT_SITES - 1) / CT_SITES);
  k_meson_sites<<<nb, CT_SITES * 16, 0, c->st>>>(pin.d, c->V, nop, T, (double2*)C.p);
  counted(c);
  QKX_CUDA(cudaGetLastError());
  return fourier_to_host(c, (const double2*)C.p, nop, m, x_src, true, corr);  // [op][Lt][Nmom]
}

int baryon_2pt(qkx_ctx* c, const double* p1, const double* p2, bool host, int op, int Q_sq, const int x_src[4],
               double* corr) {
  if (!c || !p1 || !p2 || !x_src || !corr) return bad("NULL argument");
  if (op < 0 || op > 3) return bad("baryon operator id");
  std::vector<int> m;
  QKX_TRY(momenta_of(Q_sq, m));
  QKX_CUDA(cudaSetDevice(c->device));
  static const Gammas g;
  BaryonSpin T;
  if (baryon_spin(g, op, T) != QKX_OK) return bad("internal: nucleon spin terms");
  PropCopy a(c->st), b(c->st);
  QKX_TRY(prop_in(c, p1, host, a));
  QKX_TRY(prop_in(c, p2, host, b));
  Scratch C(c->st);
  QKX_TRY(C.alloc(sizeof(double2) * 16 * c->V));
  const unsigned nb = (unsigned)((c->V + CT_SITES - 1) / CT_SITES);
  k_baryon_sites<<<nb, CT_SITES * 8, 0, c->st>>>(a.d, b.d, c->V, T, (double2*)C.p);
  counted(c);
  QKX_CUDA(cudaGetLastError());
  return fourier_to_host(c, (const double2*)C.p, 16, m, x_src, false, corr);  // Baryon::F [Lt][Nmom][4][4]
}

int delta_2pt(qkx_ctx* c, const double* p1, const double* p2, bool host, int op, int Q_sq, const int x_src[4],
              double* corr) {
  if (!c || !p1 || !p2 || !x_src || !corr) return bad("NULL argument");
  if (op < 0 || op > 1) return bad("decuplet operator id (0 DELTA_ISO1, 1 DELTA_ISO1O2)");
  std::vector<int> m;
  QKX_TRY(momenta_of(Q_sq, m));
  QKX_CUDA(cudaSetDevice(c->device));
  static const Gammas g;
  DeltaTerms T;
  if (delta_terms(g, T) != QKX_OK) return bad("internal: too many spin terms");
  PropCopy a(c->st), b(c->st);
  QKX_TRY(prop_in(c, p1, host, a));
  QKX_TRY(prop_in(c, p2, host, b));
  Scratch C(c->st), tab(c->st);
  QKX_TRY(C.alloc(sizeof(double2) * 48 * c->V));
  QKX_TRY(tab.alloc(sizeof(DeltaTerms) + sizeof(double)));  // the term table, then the error word
  DeltaTerms* dT = (DeltaTerms*)tab.p;
  int* derr = (int*)(dT + 1);
  QKX_CUDA(cudaMemsetAsync(derr, 0, sizeof(int), c->st));
  QKX_CUDA(cudaMemcpyAsync(dT, &T, sizeof(DeltaTerms), cudaMemcpyHostToDevice, c->st));
  const int smem = (int)(sizeof(double2) * 2 * DT_SITES * CT_STRIDE);
  const unsigned nb = (unsigned)((c->V + DT_SITES - 1) / DT_SITES);
  k_delta_sites<<<nb, DT_SITES * 48, smem, c->st>>>(a.d, b.d, c->V, op, dT, (double2*)C.p, derr);
  counted(c);
  QKX_CUDA(cudaGetLastError());
  int herr = 0;
  QKX_CUDA(cudaMemcpyAsync(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost, c->st));
  QKX_CUDA(cudaStreamSynchronize(c->st));
  if (herr != 0) {
    set_error("decuplet kernel: bad spin-term table entry (code %d)", herr);
    return QKX_ERR_CUDA;
  }
  return fourier_to_host(c, (const double2*)C.p, 48, m, x_src, false, corr);  // Baryon_Dec::F [Lt][Nmom][3][4][4]
}

}  // namespace
}  // namespace qkx

extern "C" {

int qkx_momenta(int Q_sq, int* mom, int max) {
  if (Q_sq < 0) return bad("Q_sq < 0");
  std::vector<int> m;
  const int n = host_momenta(Q_sq, m);
  if (mom)
    for (int i = 0; i < std::min(n, max) * 3; i++) mom[i] = m[i];
  return n;
}

int qkx_meson_2pt(qkx_ctx* c, const double* prop_host, int nop, const int* ops, int Q_sq, const int x_src[4],
                  double* corr) {
  return meson_2pt(c, prop_host, true, nop, ops, Q_sq, x_src, corr);
}
int qkx_meson_2pt_dev(qkx_ctx* c, const double* prop_dev, int nop, const int* ops, int Q_sq, const int x_src[4],
                      double* corr) {
  return meson_2pt(c, prop_dev, false, nop, ops, Q_sq, x_src, corr);
}
int qkx_baryon_2pt(qkx_ctx* c, const double* prop1_host, const double* prop2_host, int op, int Q_sq,
                   const int x_src[4], double* corr) {
  return baryon_2pt(c, prop1_host, prop2_host, true, op, Q_sq, x_src, corr);
}
int qkx_baryon_2pt_dev(qkx_ctx* c, const double* prop1_dev, const double* prop2_dev, int op, int Q_sq,
                       const int x_src[4], double* corr) {
  return baryon_2pt(c, prop1_dev, prop2_dev, false, op, Q_sq, x_src, corr);
}
int qkx_delta_2pt(qkx_ctx* c, const double* prop1_host, const double* prop2_host, int op, int Q_sq,
                  const int x_src[4], double* corr) {
  return delta_2pt(c, prop1_host, prop2_host, true, op, Q_sq, x_src, corr);
}
int qkx_delta_2pt_dev(qkx_ctx* c, const double* prop1_dev, const double* prop2_dev, int op, int Q_sq,
                      const int x_src[4], double* corr) {
  return delta_2pt(c, prop1_dev, prop2_dev, false, op, Q_sq, x_src, corr);
}
// contractNucleon's spin terms (its explicit C gamma5 table, lib/lattice_util.cpp:3418-3428,
// times the table's bar) are Baryon::contract NTN's term for term: C gamma5 there is minus
// the C gamma_5 of the constructor's tables, and the signs cancel in the product
int qkx_nucleon_2pt(qkx_ctx* c, const double* prop1_host, const double* prop2_host, int Q_sq, const int x_src[4],
                    double* corr) {
  return baryon_2pt(c, prop1_host, prop2_host, true, 0, Q_sq, x_src, corr);
}
int qkx_nucleon_2pt_dev(qkx_ctx* c, const double* prop1_dev, const double* prop2_dev, int Q_sq,
                        const int x_src[4], double* corr) {
  return baryon_2pt(c, prop1_dev, prop2_dev, false, 0, Q_sq, x_src, corr);
}

}  // extern "C"
