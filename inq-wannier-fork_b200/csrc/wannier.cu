// TD-MLWF: the Wannier transformation applied after each real-time step
// (src/observables/mlwf_properties.hpp:28-44, src/wannier/tdmlwf_trans.hpp,
// src/wannier/jade_complex.hpp).
//
//   gram     split over points: Z_d[m][n] = sum_p conj(psi_m) e^{i theta_d} psi_n for the
//            three directions (theta_d = 2 pi r_d / |a_d|), one partial per slab of points
//            (FP64 slabs in FP64; FP32 slabs of 1024 points in the mixed precision)
//   finish   sum of the slabs, normalisation 1/(|psi_m| |psi_n|), and the six matrices
//            of tdmlwf_trans::update: cos = (Z + Z^H)/2, sin = (Z - Z^H)/(2i)
//   jade     per pair and rotation step (up to 128 states: all of them in one cluster; else
//            one CTA per pair, one launch per step): the 18 pair elements, the 3 x 3
//            Jacobi eigenproblem, the plane rotation of the pair's rows of the six
//            matrices and of u, and the step's change of the traces.  The reference
//            multiplies dense M x M rotation matrices (7 GEMMs per step); the pairs are
//            disjoint, so rotating two rows per pair is the same product in O(M) per pair.
//   adiag    adiag[k][i] = sum_j conj(a_k[i][j]) u[i][j]
//   rotate   psi <- psi u^H (operations::rotate), tiled through shared memory; complex128
//            orbitals by the rotation kernel of observables.cu
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "dft.cuh"
#include "dmma.cuh"
#include "inqb_internal.h"
#include "observables.h"
#include "wannier.h"

namespace inqb {

namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

// ------------------------------------------------------------------ gram
// Axis lengths are those of the FFT size table, N below 2^31.
// FP64 contexts accumulate in FP64 over the CTA's slab (few slabs).  The mixed context
// accumulates FP32 products in FP32 over a slab of at most kSlabF32 points and keeps one
// FP32 partial per slab; the finish kernel adds the slabs in FP64 (the FP32 rounding of
// a slab sum is about 6e-8 sqrt(kSlabF32) of its size, about 1e-7 of the total after the
// FP64 sum over slabs).
constexpr long kSlabF32 = 1024;    // points per slab in the mixed precision

struct GramGeom {
  int nr[3];
  double frac_to_theta[3][3];  // theta_d / pi = sum_j f_j frac_to_theta[d][j]
};

template <typename T>
struct GramCfg;
template <>
struct GramCfg<double> {
  static constexpr int TILE_M = kDT, TILE_N = kDT, GP = kDK;  // GP: points per staged chunk
  using P = double2;                                          // partial type
};
template <>
struct GramCfg<float> {
  static constexpr int TMX = 4, TNX = 2, TILE_M = 16 * TMX, TILE_N = 16 * TNX, GP = 16;
  using P = float2;
};

// e^{i theta_d} factorises over the axes: axis table entry [d][j][n] = exp(i pi
// frac_to_theta[d][j] f_j(n)), n a grid index of axis j (at most kAxisMax of them).
constexpr int kAxisMax = 256;
__global__ void k_mlwf_axis(GramGeom geo, double2* __restrict__ tab) {
  const int j = blockIdx.x % 3, d = blockIdx.x / 3;
  for (int n = threadIdx.x; n < geo.nr[j]; n += blockDim.x) {
    const int sy = (n >= (geo.nr[j] + 1) / 2) ? n - geo.nr[j] : n;
    double sn, cs;
    sincospi(geo.frac_to_theta[d][j] * ((double)sy / geo.nr[j]), &sn, &cs);
    tab[(d * 3 + j) * kAxisMax + n] = make_double2(cs, sn);
  }
}

__device__ __forceinline__ double2 gram_weight(const GramGeom& geo, const double2* tab, int d, long point) {
  const unsigned p = (unsigned)point;
  const unsigned iz = p % geo.nr[2], r = p / geo.nr[2], iy = r % geo.nr[1], ix = r / geo.nr[1];
  const double2* t = tab + d * 3 * kAxisMax;
  return cmul(cmul(t[ix], t[kAxisMax + iy]), t[2 * kAxisMax + iz]);
}

// FP64: grid (tiles_m * tiles_n, nslab, 3), a 64 x 64 tile of one direction on the FP64
// tensor instruction (DmmaTile), the weight multiplied into the left operand as it is read
// (conj(a) w = conj(a conj(w))).  4 x 2 outputs a thread of the three directions on FMAs
// waited for their shared loads and did a narrow tile's padding (whole TD-MLWF step at 48^3:
// 8 states 463 -> 319 us, 64 states 1905 -> 1790 us).
__global__ void __launch_bounds__(kDThreads, 2)
    k_mlwf_gram_dmma(const cplx<double>* __restrict__ pa, long lda, int Ma, const cplx<double>* __restrict__ pb,
                     long ldb, int Mb, long N, GramGeom geo, const double2* __restrict__ tab, long pts_per_slab,
                     double2* __restrict__ partial) {
  __shared__ DmmaBuf sa[2], sb[2];
  __shared__ double2 sw[2][kDK];
  const int tiles_m = (Ma + kDT - 1) / kDT, d = blockIdx.z;
  const int m0 = (blockIdx.x % tiles_m) * kDT, n0 = (blockIdx.x / tiles_m) * kDT;
  const long p_beg = (long)blockIdx.y * pts_per_slab, p_end = min(N, p_beg + pts_per_slab);
  DmmaTile t;
  t.clear();
  const int rows = min(8, (Ma - m0 + 7) / 8), hi = min(8, (Mb - n0 + 7) / 8);
  DmmaOperand<double, false> oa, ob;
  auto load = [&](long pc, int buf) {
    oa.load(sa[buf], pa, [&](int q, int j) { return pc + q < p_end && m0 + j < Ma ? (pc + q) * lda + m0 + j : -1L; });
    ob.load(sb[buf], pb, [&](int q, int j) { return pc + q < p_end && n0 + j < Mb ? (pc + q) * ldb + n0 + j : -1L; });
    dmma_commit();
    if (threadIdx.x < kDK) sw[buf][threadIdx.x] = gram_weight(geo, tab, d, min(pc + (long)threadIdx.x, N - 1));
  };
  load(p_beg, 0);
  int buf = 0;
  for (long pc = p_beg; pc < p_end; pc += kDK, buf ^= 1) {
    dmma_arrived();
    __syncthreads();  // chunk pc is complete, and every warp has left the other buffer
    if (pc + kDK < p_end) load(pc + kDK, buf ^ 1);
    t.mul_block<kConjX>(sa[buf], sb[buf], rows, hi, [&](double2 u, int k) { return cmul(u, cconj(sw[buf][k])); });
  }
  // partial[slab][d][m][n], m < Ma, n < Mb
  double2* out = partial + ((size_t)blockIdx.y * 3 + d) * Ma * Mb;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int m = m0 + 8 * DmmaTile::row_block(a) + (lane >> 2), n = n0 + 8 * c + 2 * (lane & 3);
      if (m < Ma && n < Mb) out[(size_t)m * Mb + n] = make_double2(t.re[a][c].x, t.im[a][c].x);
      if (m < Ma && n + 1 < Mb) out[(size_t)m * Mb + n + 1] = make_double2(t.re[a][c].y, t.im[a][c].y);
    }
}

// FP32: grid (tiles_m * tiles_n, nslab), 256 threads as 16 x 16; thread (tm, tn) holds outputs
// m = m0 + tm + 16 a (a < TMX), n = n0 + tn + 16 b (b < TNX) for the three directions.  Bound
// by the FP32 units: 4 x 2 outputs of three directions take 96 fused multiply-adds for 10
// shared loads.  The next chunk's orbitals are fetched into registers and its weights formed
// from the axis tables while the current chunk is summed.
__global__ void __launch_bounds__(256, 3)
    k_mlwf_gram(const cplx<float>* __restrict__ pa, long lda, int Ma, const cplx<float>* __restrict__ pb, long ldb,
                int Mb, long N, GramGeom geo, const double2* __restrict__ tab, long pts_per_slab,
                float2* __restrict__ partial) {
  using R = float;
  constexpr int TMX = GramCfg<R>::TMX, TNX = GramCfg<R>::TNX, kGP = GramCfg<R>::GP;
  constexpr int TILE_M = GramCfg<R>::TILE_M, TILE_N = GramCfg<R>::TILE_N;
  constexpr int PA = kGP * TILE_M / 256, PB = kGP * TILE_N / 256;
  __shared__ cplx<R> sA[kGP][TILE_M];
  __shared__ cplx<R> sB[3][kGP][TILE_N];
  __shared__ cplx<R> sW[2][3][kGP];
  const int tiles_m = (Ma + TILE_M - 1) / TILE_M;
  const int m0 = (blockIdx.x % tiles_m) * TILE_M, n0 = (blockIdx.x / tiles_m) * TILE_N;
  const long p_beg = (long)blockIdx.y * pts_per_slab, p_end = min(N, p_beg + pts_per_slab);
  // a warp is 8 x 4 of the 16 x 16 thread grid (its shared loads take one wavefront each)
  const int tm = threadIdx.x / 128 * 8 + threadIdx.x % 8, tn = (threadIdx.x / 32) % 4 * 4 + threadIdx.x % 32 / 8;
  R acc[3][TMX][TNX][2];
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int a = 0; a < TMX; ++a)
#pragma unroll
      for (int b = 0; b < TNX; ++b) acc[d][a][b][0] = acc[d][a][b][1] = (R)0;
  cplx<R> va[PA], vb[PB];
  auto fetch = [&](long pc) {
#pragma unroll
    for (int u = 0; u < PA; ++u) {
      const int i = threadIdx.x + 256 * u, q = i / TILE_M, j = i % TILE_M;
      va[u] = (pc + q < p_end && m0 + j < Ma) ? pa[(pc + q) * lda + m0 + j] : mk<R>(0, 0);
    }
#pragma unroll
    for (int u = 0; u < PB; ++u) {
      const int i = threadIdx.x + 256 * u, q = i / TILE_N, j = i % TILE_N;
      vb[u] = (pc + q < p_end && n0 + j < Mb) ? pb[(pc + q) * ldb + n0 + j] : mk<R>(0, 0);
    }
  };
  // weights of a chunk's points, e^{i theta_d}
  auto weights = [&](long pc, int buf) {
    if (threadIdx.x >= 3 * kGP) return;
    const int d = threadIdx.x / kGP, q = threadIdx.x % kGP;
    const double2 w = gram_weight(geo, tab, d, min(pc + q, N - 1));
    sW[buf][d][q] = mk<R>((R)w.x, (R)w.y);
  };
  fetch(p_beg);
  weights(p_beg, 0);
  __syncthreads();
  int buf = 0;
  for (long pc = p_beg; pc < p_end; pc += kGP, buf ^= 1) {
#pragma unroll
    for (int u = 0; u < PA; ++u) {
      const int i = threadIdx.x + 256 * u;
      sA[i / TILE_M][i % TILE_M] = va[u];
    }
#pragma unroll
    for (int u = 0; u < PB; ++u) {
      const int i = threadIdx.x + 256 * u, q = i / TILE_N;
#pragma unroll
      for (int d = 0; d < 3; ++d) sB[d][q][i % TILE_N] = sW[buf][d][q] * vb[u];
    }
    __syncthreads();
    if (pc + kGP < p_end) {
      fetch(pc + kGP);
      weights(pc + kGP, buf ^ 1);
    }
#pragma unroll 2
    for (int q = 0; q < kGP; ++q) {
      cplx<R> av[TMX];
#pragma unroll
      for (int a = 0; a < TMX; ++a) av[a] = sA[q][tm + 16 * a];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        cplx<R> bv[TNX];
#pragma unroll
        for (int b = 0; b < TNX; ++b) bv[b] = sB[d][q][tn + 16 * b];
#pragma unroll
        for (int a = 0; a < TMX; ++a)
#pragma unroll
          for (int b = 0; b < TNX; ++b) {
            // conj(a) * b
            acc[d][a][b][0] = fma(av[a].x, bv[b].x, fma(av[a].y, bv[b].y, acc[d][a][b][0]));
            acc[d][a][b][1] = fma(av[a].x, bv[b].y, fma(-av[a].y, bv[b].x, acc[d][a][b][1]));
          }
      }
    }
    __syncthreads();
  }
  // partial[slab][d][m][n], m < Ma, n < Mb
  const size_t MM = (size_t)Ma * Mb;
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int a = 0; a < TMX; ++a)
#pragma unroll
      for (int b = 0; b < TNX; ++b) {
        const int m = m0 + tm + 16 * a, n = n0 + tn + 16 * b;
        if (m < Ma && n < Mb)
          partial[((size_t)blockIdx.y * 3 + d) * MM + (size_t)m * Mb + n] =
              make_float2(acc[d][a][b][0], acc[d][a][b][1]);
      }
}

// Z[e] = sum over the slabs of partial[slab][e] in FP64, e = (d, m, n).  A block holds 32
// elements x 8 parts: part k adds the slabs k, k + 8, ... in order, four loads in flight, and
// the parts are added in order (a fixed order; one thread per element left most SMs idle).
template <typename P>
__global__ void __launch_bounds__(256) k_mlwf_slab_sum(const P* __restrict__ partial, int nslab, long n, double2* __restrict__ Z) {
  __shared__ double2 red[8][32];
  const int part = threadIdx.x / 32, el = threadIdx.x % 32;
  const long e = (long)blockIdx.x * 32 + el;
  double zx = 0.0, zy = 0.0;
  if (e < n) {
    for (int s0 = part; s0 < nslab; s0 += 32) {
      P v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = (s0 + 8 * u < nslab) ? partial[(size_t)(s0 + 8 * u) * n + e] : P{0, 0};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        zx += (double)v[u].x;
        zy += (double)v[u].y;
      }
    }
  }
  red[part][el] = make_double2(zx, zy);
  __syncthreads();
  if (part == 0 && e < n) {
    for (int k = 1; k < 8; ++k) {
      zx += red[k][el].x;
      zy += red[k][el].y;
    }
    Z[e] = make_double2(zx, zy);
  }
}

// a[2d][m][n] = (Z + Z^H)/2, a[2d+1][m][n] = (Z - Z^H)/(2i), Z the slab sum (FP64) divided
// by |psi_m| |psi_n|: norms[ns m + ns - 1] = sum_p |psi_m|^2 (ns = 3: the band sums; 1: plain)
__global__ void k_mlwf_finish(const double2* __restrict__ Z, int M, const double* __restrict__ norms, int ns,
                              double2* __restrict__ a) {
  const size_t MM = (size_t)M * M;
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < 3 * (long)MM; e += (long)gridDim.x * blockDim.x) {
    const int d = (int)(e / MM);
    const int m = (int)((e % MM) / M), n = (int)(e % M);
    const double2 x = Z[(size_t)d * MM + (size_t)m * M + n];
    const double2 y = Z[(size_t)d * MM + (size_t)n * M + m];
    const double zx = x.x, zy = x.y, tx = y.x, ty = y.y;
    const double sc = 1.0 / sqrt(norms[ns * m + ns - 1] * norms[ns * n + ns - 1]);
    // conj(Z[n][m]) = (tx, -ty)
    a[(2 * d) * MM + (size_t)m * M + n] = make_double2(0.5 * sc * (zx + tx), 0.5 * sc * (zy - ty));
    // (Z - conj(Z[n][m])) / (2i) = (v - i u) / 2 with u + i v = Z - conj(Z[n][m])
    const double ur = zx - tx, vi = zy + ty;
    a[(2 * d + 1) * MM + (size_t)m * M + n] = make_double2(0.5 * sc * vi, -0.5 * sc * ur);
  }
}

// ------------------------------------------------------------------ jade
// Symmetric 3x3 eigenproblem by cyclic Jacobi rotations (the method of
// wannier/jacobi_eigenvalue.hpp; the oracle restates the same steps); returns the
// eigenvector of the largest eigenvalue with the sign the iteration leaves.
__device__ void jacobi3_top(double S[3][3], double out[3]) {
  double V[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
  double d[3] = {S[0][0], S[1][1], S[2][2]};
  double base[3] = {d[0], d[1], d[2]};
  double inc[3] = {0, 0, 0};
  for (int pass = 1; pass <= 10000; pass++) {
    double off = 0.0;
#pragma unroll
    for (int q = 0; q < 3; q++)
#pragma unroll
      for (int p = 0; p < q; p++) off += S[p][q] * S[p][q];
    // converged once every rotation left is below 2^-60: it would change no digit of V (the
    // iteration's last passes only drive the off-diagonal to an exact zero), nor does a
    // non-finite matrix go on (reported by the sweep's change)
    constexpr double tiny = 8.7e-19;
    if (fabs(S[0][1]) <= tiny * fabs(d[1] - d[0]) && fabs(S[0][2]) <= tiny * fabs(d[2] - d[0]) &&
        fabs(S[1][2]) <= tiny * fabs(d[2] - d[1]))
      break;
    const double thresh = sqrt(off) / 12.0;
    if (!(thresh > 0.0)) break;
#pragma unroll
    for (int p = 0; p < 3; p++)
#pragma unroll
      for (int q = p + 1; q < 3; q++) {
        const double big = 10.0 * fabs(S[p][q]);
        if (pass > 4 && big + fabs(d[p]) == fabs(d[p]) && big + fabs(d[q]) == fabs(d[q])) {
          S[p][q] = 0.0;
          continue;
        }
        if (fabs(S[p][q]) < thresh) continue;
        // t = tan of the rotation angle, the smaller root: 2 S / (h +- sqrt(h^2 + 4 S^2))
        // with the sign of h S (+ for h = 0); c, s = 1, t over sqrt(1 + t^2); tau = s / (1 + c)
        double h = d[q] - d[p];
        const double e2 = 2.0 * fabs(S[p][q]), dd = fabs(h) + sqrt(fma(h, h, e2 * e2));
        const double sg = (h != 0.0 && (h < 0.0) != (S[p][q] < 0.0)) ? -1.0 : 1.0;
        const double rn = rsqrt(fma(dd, dd, e2 * e2));
        const double t = sg * (e2 / dd), c = dd * rn, s = sg * (e2 * rn), tau = s / (1.0 + c);
        h = t * S[p][q];
        inc[p] -= h;
        inc[q] += h;
        d[p] -= h;
        d[q] += h;
        S[p][q] = 0.0;
#define INQB_JROT(x, y)                   \
  {                                       \
    const double g_ = (x), h_ = (y);      \
    (x) = g_ - s * (h_ + g_ * tau);       \
    (y) = h_ + s * (g_ - h_ * tau);       \
  }
#pragma unroll
        for (int j = 0; j < p; j++) INQB_JROT(S[j][p], S[j][q])
#pragma unroll
        for (int j = p + 1; j < q; j++) INQB_JROT(S[p][j], S[j][q])
#pragma unroll
        for (int j = q + 1; j < 3; j++) INQB_JROT(S[p][j], S[q][j])
#pragma unroll
        for (int j = 0; j < 3; j++) INQB_JROT(V[j][p], V[j][q])
#undef INQB_JROT
      }
#pragma unroll
    for (int i = 0; i < 3; i++) {
      base[i] += inc[i];
      d[i] = base[i];
      inc[i] = 0.0;
    }
  }
  // the column that an ascending selection sort of d leaves last (constant indices, so that
  // everything stays in registers)
  const int m = (d[1] < d[0]) ? (d[2] < d[1] ? 2 : 1) : (d[2] < d[0] ? 2 : 0);
  const bool two = m == 2;                        // the two left are (1, 0), else (m == 1 ? 0 : 1, 2)
  const double da = (m == 1) ? d[0] : d[1], db = two ? d[0] : d[2];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double va = (m == 1) ? V[i][0] : V[i][1], vb = two ? V[i][0] : V[i][2];
    out[i] = db < da ? va : vb;
  }
}

constexpr int kJT = 128;  // threads of a pair's CTA

// one CTA per pair of this rotation step; a [6][M][M], u [M][M]
__global__ void __launch_bounds__(kJT)
    k_jade_step(double2* __restrict__ a, double2* __restrict__ u, int M, const int2* __restrict__ pairs,
                double* __restrict__ delta) {
  __shared__ double red[kJT / 32][36];
  __shared__ double rot[3];  // c, Re s, Im s
  __shared__ double old_diag;
  const int2 pq = pairs[blockIdx.x];
  const int p = pq.x, q = pq.y;
  if (p >= M || q >= M) {
    if (threadIdx.x == 0) delta[blockIdx.x] = 0.0;
    return;
  }
  const size_t MM = (size_t)M * M;
  // the 18 pair elements: (sum conj(a_k[p][i]) u[q][i], sum conj(a_k[p][i]) u[p][i],
  // sum conj(a_k[q][i]) u[q][i]) for k < 6
  double s[36];
#pragma unroll
  for (int i = 0; i < 36; ++i) s[i] = 0.0;
  for (int i = threadIdx.x; i < M; i += blockDim.x) {
    const double2 up = u[(size_t)p * M + i], uq = u[(size_t)q * M + i];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const double2 ap = cconj(a[k * MM + (size_t)p * M + i]), aq = cconj(a[k * MM + (size_t)q * M + i]);
      const double2 x0 = cmul(ap, uq), x1 = cmul(ap, up), x2 = cmul(aq, uq);
      s[6 * k + 0] += x0.x;
      s[6 * k + 1] += x0.y;
      s[6 * k + 2] += x1.x;
      s[6 * k + 3] += x1.y;
      s[6 * k + 4] += x2.x;
      s[6 * k + 5] += x2.y;
    }
  }
#pragma unroll
  for (int i = 0; i < 36; ++i)
    for (int o = 16; o > 0; o >>= 1) s[i] += __shfl_down_sync(0xffffffffu, s[i], o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < 36; ++i) red[w][i] = s[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double G[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    double od = 0.0;
    for (int k = 0; k < 6; ++k) {
      double e[6];
      for (int i = 0; i < 6; ++i) {
        double v = 0.0;
        for (int ww = 0; ww < kJT / 32; ++ww) v += red[ww][6 * k + i];
        e[i] = v;
      }
      const double2 aij = make_double2(e[0], e[1]), aii = make_double2(e[2], e[3]), ajj = make_double2(e[4], e[5]);
      // h = (aii - ajj, aij + conj(aij), i (aij - conj(aij))) = (.., (2 Re aij, 0), (-2 Im aij, 0))
      const double2 h[3] = {make_double2(aii.x - ajj.x, aii.y - ajj.y), make_double2(2.0 * aij.x, 0.0),
                            make_double2(-2.0 * aij.y, 0.0)};
      for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) G[r][c] += h[r].x * h[c].x + h[r].y * h[c].y;
      od += a[k * MM + (size_t)p * M + p].x + a[k * MM + (size_t)q * M + q].x;
    }
    double v[3];
    jacobi3_top(G, v);
    double x = v[0], y = v[1], z = v[2];
    if (v[0] < 0.0) {
      x = -x;
      y = -y;
    }
    const double r = sqrt((x + 1.0) / 2.0);
    rot[0] = r;
    rot[1] = y / (2.0 * r);
    rot[2] = -z / (2.0 * r);
    old_diag = od;
  }
  __syncthreads();
  const double c = rot[0];
  const double2 sv = make_double2(rot[1], rot[2]), sc = cconj(sv);
  // rows p, q of a_k and u: row_p <- c row_p + conj(s) row_q, row_q <- -s row_p + c row_q
  for (int e = threadIdx.x; e < 7 * M; e += blockDim.x) {
    const int k = e / M, i = e % M;
    double2* base = (k < 6) ? a + k * MM : u;
    double2& rp = base[(size_t)p * M + i];
    double2& rq = base[(size_t)q * M + i];
    const double2 xv = rp, yv = rq;
    const double2 t1 = cmul(sc, yv), t2 = cmul(sv, xv);
    rp = make_double2(c * xv.x + t1.x, c * xv.y + t1.y);
    rq = make_double2(c * yv.x - t2.x, c * yv.y - t2.y);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double nd = 0.0;
    for (int k = 0; k < 6; ++k) nd += a[k * MM + (size_t)p * M + p].x + a[k * MM + (size_t)q * M + q].x;
    delta[blockIdx.x] = nd - old_diag;
  }
}

// out = sum_steps 2 |sum_pairs delta[step][pair]| (one block, fixed order)
__global__ void k_jade_change(const double* __restrict__ delta, int nsteps, int np, double* __restrict__ out) {
  __shared__ double part[256];
  double acc = 0.0;
  for (int s = threadIdx.x; s < nsteps; s += blockDim.x) {
    double t = 0.0;
    for (int i = 0; i < np; ++i) t += delta[(size_t)s * np + i];
    acc += 2.0 * fabs(t);
  }
  part[threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < (int)blockDim.x; ++i) t += part[i];
    out[0] = t;
  }
}

// ------------------------------------------------------------------ jade in one cluster
// jacobi3_top with its iteration in FP32 and the eigenvector then refined in FP64.  The
// serial chain of FP64 roots and divisions made the Jacobi iteration the longest part of a
// rotation step (5100 of 13200 cycles at 64 states).  The FP32 iteration makes the same
// rotations, so it leaves the eigenvector in the same column with the same sign; then
// v += sum_i v_i (v_i . (A - lambda) v) / (lambda - lambda_i) + v (1 - |v|^2) / 2, three times
// (the column form of Ogita and Aishima's refinement, Japan J. Indust. Appl. Math. 35, 2018).
// v_1, v_2 and the gaps keep their FP32 errors, up to 1e-5 with gaps of 2% and more, so a step
// leaves about 1e-5 of v's error: 1e-5 -> 1e-10 -> 1e-15 -> rounding.  The last residual
// subtracts lambda from the diagonal first, where the difference is exact for a close
// eigenvalue; A v - lambda v rounds at |A| and ended 1.7 times as far off as the FP64
// iteration at gaps of 2 to 4%, this form is nearer than that iteration at every gap.
// Where FP32 could choose differently (a rotation near 45 degrees that involves a large
// eigenvalue) or the top eigenvalue is not well separated, the FP64 iteration runs instead.
__device__ void top3(const double G[3][3], double out[3]) {
  const double scale = fmax(G[0][0], fmax(G[1][1], G[2][2]));
  bool ok = scale > 0.0 && scale < 1e300;
  // a power of two, so that A is G to the last bit (1 / scale rounded every entry)
  const double inv = ok ? __longlong_as_double((2046LL - (__double_as_longlong(scale) >> 52)) << 52) : 0.0;
  double A[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) A[i][j] = G[i][j] * inv;
  float S[3][3], d[3], V[3][3] = {{1.f, 0.f, 0.f}, {0.f, 1.f, 0.f}, {0.f, 0.f, 1.f}};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    d[i] = (float)A[i][i];
#pragma unroll
    for (int j = 0; j < 3; ++j) S[i][j] = (float)A[i][j];
  }
  for (int pass = 0; pass < 8 && ok; ++pass) {
    const float off = S[0][1] * S[0][1] + S[0][2] * S[0][2] + S[1][2] * S[1][2];
    if (!(off > 1e-16f)) break;
    const float thresh = sqrtf(off) * (1.f / 12.f);
#pragma unroll
    for (int p = 0; p < 3; p++)
#pragma unroll
      for (int q = p + 1; q < 3; q++) {
        if (fabsf(S[p][q]) < thresh) continue;
        const float h = d[q] - d[p], big = fmaxf(fabsf(d[p]), fabsf(d[q]));
        if (fabsf(h) < 1e-3f * big && big > 0.05f) ok = false;
        const float e2 = 2.f * fabsf(S[p][q]), dd = fabsf(h) + sqrtf(h * h + e2 * e2);
        const float sg = (h != 0.f && (h < 0.f) != (S[p][q] < 0.f)) ? -1.f : 1.f;
        const float rn = rsqrtf(dd * dd + e2 * e2);
        const float t = sg * __fdividef(e2, dd), c = dd * rn, s = sg * (e2 * rn), tau = __fdividef(s, 1.f + c);
        d[p] -= t * S[p][q];
        d[q] += t * S[p][q];
        S[p][q] = 0.f;
#define INQB_FROT(x, y)                  \
  {                                      \
    const float g_ = (x), h_ = (y);      \
    (x) = g_ - s * (h_ + g_ * tau);      \
    (y) = h_ + s * (g_ - h_ * tau);      \
  }
#pragma unroll
        for (int j = 0; j < p; j++) INQB_FROT(S[j][p], S[j][q])
#pragma unroll
        for (int j = p + 1; j < q; j++) INQB_FROT(S[p][j], S[j][q])
#pragma unroll
        for (int j = q + 1; j < 3; j++) INQB_FROT(S[p][j], S[q][j])
#pragma unroll
        for (int j = 0; j < 3; j++) INQB_FROT(V[j][p], V[j][q])
#undef INQB_FROT
      }
  }
  // the top column v and the other two, v1 and v2
  const int m = (d[1] > d[0]) ? (d[2] > d[1] ? 2 : 1) : (d[2] > d[0] ? 2 : 0);
  const float dm = m == 0 ? d[0] : m == 1 ? d[1] : d[2];
  const float g1 = dm - (m == 0 ? d[1] : d[0]), g2 = dm - (m == 2 ? d[1] : d[2]);
  if (!(ok && g1 > 0.02f * dm && g2 > 0.02f * dm)) {
    double B[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) B[i][j] = G[i][j];
    jacobi3_top(B, out);
    return;
  }
  const double i1 = (double)(1.f / g1), i2 = (double)(1.f / g2);
  double v[3], v1[3], v2[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    v[j] = m == 0 ? V[j][0] : m == 1 ? V[j][1] : V[j][2];
    v1[j] = m == 0 ? V[j][1] : V[j][0];
    v2[j] = m == 2 ? V[j][1] : V[j][2];
  }
#pragma unroll
  for (int it = 0; it < 3; ++it) {
    double w[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) w[j] = fma(A[j][0], v[0], fma(A[j][1], v[1], A[j][2] * v[2]));
    const double vv = fma(v[0], v[0], fma(v[1], v[1], v[2] * v[2]));
    const double lam = fma(v[0], w[0], fma(v[1], w[1], v[2] * w[2])) * (2.0 - vv);  // Rayleigh, |v| near 1
    double e1 = 0.0, e2 = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      double res = fma(-lam, v[j], w[j]);
      if (it == 2) {
        const int p = (j + 1) % 3, q = (j + 2) % 3;
        res = fma(A[j][j] - lam, v[j], fma(A[j][p], v[p], A[j][q] * v[q]));
      }
      e1 = fma(v1[j], res, e1);
      e2 = fma(v2[j], res, e2);
    }
    e1 *= i1;
    e2 *= i2;
    const double em = 0.5 * (1.0 - vv);
#pragma unroll
    for (int j = 0; j < 3; ++j) v[j] += fma(em, v[j], fma(e1, v1[j], e2 * v2[j]));
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) out[j] = v[j];
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// The aligned forms want every lane of the warp at the instruction together, which loops over
// the lanes' rows and branches on one lane do not leave by themselves.
__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// All sweeps in one launch of one thread-block cluster whose shared memory holds the six
// matrices and u.  A rotation step is bound by latency, not by bytes: as a launch of its
// own it gathered rows from L2 and paid a launch around the serial eigenproblem.  Here the
// rows sit where they are rotated: slot j of the tournament holds the rows (top[j], bot[j])
// of the seven matrices, CTA r the slots r SP .. r SP + SP - 1, and a rotated row is stored
// straight into the slot that has it in the next step (remote stores, no remote load: with
// rows at home and read over distributed shared memory a step took 13200 cycles, 4800 of
// them the reads).  Two cluster barriers a step: all rows are read before any is
// overwritten (arrived at after the reads, waited for after the eigenproblem), and all are
// written before the next step reads.  Seven warps a slot: warp k sums and rotates matrix
// k (warp 6: u); E elements of a row per lane (M <= 32 E); GMAX slots per CTA at most.
constexpr int kJG = 7 * 32, kJadeCtas = 16;

struct JadeShared {
  double red[6][6];   // warp k: Re, Im of the pair elements (pq, pp, qq) of matrix k
  double diag[6][2];  // warp k: change of the two diagonal elements
  double rot[3];      // c, Re s, Im s
  int id[2];          // the rows of the slot (M and above: none)
};

template <int E, int GMAX>
__global__ void __launch_bounds__(GMAX * kJG)
    k_jade_cluster(double2* __restrict__ a, double2* __restrict__ u, int M, const int2* __restrict__ pairs, int np,
                   int steps, int maxsweep, double tol, double* delta, double* __restrict__ out) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) double2 rows[];  // [slot of this CTA][top, bot][7][M]
  __shared__ JadeShared sh[GMAX];
  __shared__ double part[GMAX * kJG];
  const size_t MM = (size_t)M * M;
  const int g = threadIdx.x / kJG, k = (threadIdx.x % kJG) / 32, lane = threadIdx.x & 31;
  const int SP = blockDim.x / kJG, slot = (int)cluster.block_rank() * SP + g;
  const bool on = slot < np, lead = threadIdx.x % kJG == 0;
  JadeShared& q = sh[g];
  double2* rp = rows + ((size_t)(2 * g) * 7 + k) * M;
  double2* rq = rp + (size_t)7 * M;
  // the two rows of the first step; dummy rows (odd M) are zero
  const int2 first = on ? pairs[slot] : make_int2(M, M);
  if (lead) {
    q.id[0] = first.x;
    q.id[1] = first.y;
  }
  if (on)
    for (int i = lane; i < M; i += 32) {
      const double2* src = a + (size_t)min(k, 5) * MM;
      rp[i] = first.x >= M ? make_double2(0, 0)
              : k < 6      ? src[(size_t)first.x * M + i]
                           : make_double2(first.x == i ? 1.0 : 0.0, 0.0);
      rq[i] = first.y >= M ? make_double2(0, 0)
              : k < 6      ? src[(size_t)first.y * M + i]
                           : make_double2(first.y == i ? 1.0 : 0.0, 0.0);
    }
  // where the slot's rows go after a step: top 0 stays, the other tops move up one slot and
  // the last one turns to the bottom row; the bottoms move down and the first turns up
  const int ts = (slot == 0 || slot == np - 1) ? slot : slot + 1, tw = (slot > 0 && slot == np - 1) ? 1 : 0;
  const int bs = np == 1 ? slot : slot == 0 ? 1 : slot - 1, bw = (np > 1 && slot == 0) ? 0 : 1;
  double2* tdst = nullptr;
  double2* bdst = nullptr;
  int *tid_dst = nullptr, *bid_dst = nullptr;
  if (on) {
    tdst = cluster.map_shared_rank(rows, ts / SP) + ((size_t)(2 * (ts % SP) + tw) * 7 + k) * M;
    bdst = cluster.map_shared_rank(rows, bs / SP) + ((size_t)(2 * (bs % SP) + bw) * 7 + k) * M;
    tid_dst = cluster.map_shared_rank(&sh[0].id[0], ts / SP) + (sizeof(JadeShared) / sizeof(int)) * (ts % SP) + tw;
    bid_dst = cluster.map_shared_rank(&sh[0].id[0], bs / SP) + (sizeof(JadeShared) / sizeof(int)) * (bs % SP) + bw;
  }
  cluster_arrive();
  int nsweep = 0;
  double change = 0.0;
  for (;;) {
    ++nsweep;
    for (int st = 0; st < steps; ++st) {
      cluster_wait();  // the rows of this step are in place
      // the step before's change of the diagonal, complete since that barrier
      if (on && lead && st > 0) {
        double d = 0.0;
        for (int kk = 0; kk < 6; ++kk) d += q.diag[kk][0] + q.diag[kk][1];
        delta[(size_t)(st - 1) * np + slot] = d;
      }
      const int p0 = q.id[0], q0 = q.id[1];
      const bool live = on && p0 < M && q0 < M;
      double2 xp[E], xq[E];
#pragma unroll
      for (int t = 0; t < E; ++t) {
        const int i = lane + 32 * t;
        xp[t] = xq[t] = make_double2(0.0, 0.0);
        if (on && i < M) {
          xp[t] = rp[i];
          xq[t] = rq[i];
        }
      }
      if (live && k < 6) {
        // sums of conj(a_p) u_q, conj(a_p) u_p, conj(a_q) u_q
        double s[6] = {0, 0, 0, 0, 0, 0};
        const double2 *up = rows + ((size_t)(2 * g) * 7 + 6) * M, *uq = up + (size_t)7 * M;
#pragma unroll
        for (int t = 0; t < E; ++t) {
          const int i = lane + 32 * t;
          if (i < M) {
            const double2 y = up[i], z = uq[i];
            const double2 x0 = cmul(cconj(xp[t]), z), x1 = cmul(cconj(xp[t]), y), x2 = cmul(cconj(xq[t]), z);
            s[0] += x0.x;
            s[1] += x0.y;
            s[2] += x1.x;
            s[3] += x1.y;
            s[4] += x2.x;
            s[5] += x2.y;
          }
        }
#pragma unroll
        for (int v = 0; v < 6; ++v) s[v] = warp_sum(s[v]);
        if (lane == 0) {
#pragma unroll
          for (int v = 0; v < 6; ++v) q.red[k][v] = s[v];
        }
      }
      cluster_arrive();  // this warp has read its rows
      asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(kJG) : "memory");
      if (live && k == 0) {
        double G[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
        for (int kk = 0; kk < 6; ++kk) {
          const double* e = q.red[kk];
          // h = (aii - ajj, aij + conj(aij), i (aij - conj(aij))), as in k_jade_step
          const double h0 = e[2] - e[4], h0i = e[3] - e[5], h1 = 2.0 * e[0], h2 = -2.0 * e[1];
          G[0][0] += h0 * h0 + h0i * h0i;
          G[0][1] += h0 * h1;
          G[0][2] += h0 * h2;
          G[1][1] += h1 * h1;
          G[1][2] += h1 * h2;
          G[2][2] += h2 * h2;
        }
        G[1][0] = G[0][1];
        G[2][0] = G[0][2];
        G[2][1] = G[1][2];
        double v[3];
        top3(G, v);
        const double x = fabs(v[0]), y = v[0] < 0.0 ? -v[1] : v[1];
        const double r = sqrt((x + 1.0) / 2.0);
        if (lane == 0) {
          q.rot[0] = r;
          q.rot[1] = y / (2.0 * r);
          q.rot[2] = -v[2] / (2.0 * r);
        }
      }
      __syncwarp();
      asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(kJG) : "memory");
      cluster_wait();  // every row is read
      if (on) {
        const double c = live ? q.rot[0] : 1.0;
        const double2 sv = live ? make_double2(q.rot[1], q.rot[2]) : make_double2(0.0, 0.0), sc = cconj(sv);
        if (k < 6 && lane < 2 && !live) q.diag[k][lane] = 0.0;
#pragma unroll
        for (int t = 0; t < E; ++t) {
          const int i = lane + 32 * t;
          if (i >= M) continue;
          const double2 t1 = cmul(sc, xq[t]), t2 = cmul(sv, xp[t]);
          const double2 yp = make_double2(c * xp[t].x + t1.x, c * xp[t].y + t1.y);
          const double2 yq = make_double2(c * xq[t].x - t2.x, c * xq[t].y - t2.y);
          tdst[i] = yp;
          bdst[i] = yq;
          if (live && k < 6 && i == p0) q.diag[k][0] = yp.x - xp[t].x;
          if (live && k < 6 && i == q0) q.diag[k][1] = yq.x - xq[t].x;
        }
        if (lead) {
          *tid_dst = p0;
          *bid_dst = q0;
        }
      }
      cluster_arrive();
    }
    cluster_wait();
    if (on && lead) {
      double d = 0.0;
      for (int kk = 0; kk < 6; ++kk) d += q.diag[kk][0] + q.diag[kk][1];
      delta[(size_t)(steps - 1) * np + slot] = d;
    }
    // sum over the steps of 2 |sum over the pairs of the trace change|, in the same order
    // by every CTA, so all take the same decision
    __threadfence();
    cluster_arrive();
    cluster_wait();
    double acc = 0.0;
    for (int st = threadIdx.x; st < steps; st += blockDim.x) {
      double t = 0.0;
      for (int i = 0; i < np; ++i) t += __ldcg(delta + (size_t)st * np + i);
      acc += 2.0 * fabs(t);
    }
    part[threadIdx.x] = acc;
    __syncthreads();
    change = 0.0;
    for (int i = 0; i < min((int)blockDim.x, steps); ++i) change += part[i];
    cluster_arrive();  // every CTA has read the deltas
    if (!isfinite(change) || fabs(change) < tol || nsweep >= maxsweep) break;
  }
  cluster_wait();
  // a sweep's moves bring every row back to its first slot
  for (int w = 0; w < 2 && on; ++w) {
    const int r = q.id[w];
    if (r >= M) continue;
    double2* dst = (k < 6 ? a + (size_t)k * MM : u) + (size_t)r * M;
    for (int i = lane; i < M; i += 32) dst[i] = (w ? rq : rp)[i];
  }
  if (cluster.block_rank() == 0 && threadIdx.x == 0) {
    out[0] = change;
    out[1] = (double)nsweep;
  }
}

__global__ void k_identity(double2* __restrict__ u, int M) {
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < (long)M * M; e += (long)gridDim.x * blockDim.x)
    u[e] = make_double2((e / M == e % M) ? 1.0 : 0.0, 0.0);
}

// adiag[k][i] = sum_j conj(a_k[i][j]) u[i][j]; grid (M, 6)
__global__ void __launch_bounds__(128)
    k_jade_adiag(const double2* __restrict__ a, const double2* __restrict__ u, int M, double2* __restrict__ adiag) {
  __shared__ double red[4][2];
  const int i = blockIdx.x, k = blockIdx.y;
  const size_t MM = (size_t)M * M;
  double sr = 0.0, si = 0.0;
  for (int j = threadIdx.x; j < M; j += blockDim.x) {
    const double2 x = cmul(cconj(a[k * MM + (size_t)i * M + j]), u[(size_t)i * M + j]);
    sr += x.x;
    si += x.y;
  }
  for (int o = 16; o > 0; o >>= 1) {
    sr += __shfl_down_sync(0xffffffffu, sr, o);
    si += __shfl_down_sync(0xffffffffu, si, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5][0] = sr;
    red[threadIdx.x >> 5][1] = si;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0, im = 0.0;
    for (int w = 0; w < 4; ++w) {
      r += red[w][0];
      im += red[w][1];
    }
    adiag[(size_t)k * M + i] = make_double2(r, im);
  }
}

// ------------------------------------------------------------------ rotate
// out[p][i] = sum_j psi[p][j] conj(u[i][j]) in FP32 (complex128 orbitals: launch_rotate_adjoint);
// 64 x 64 output tiles, 256 threads with 4 x 4 outputs each, j in chunks of 8 through shared
// memory.
constexpr int kRT = 64, kRK = 8;

__global__ void __launch_bounds__(256)
    k_mlwf_rotate(const cplx<float>* __restrict__ psi, long ld, int M, long N, const double2* __restrict__ u,
                  cplx<float>* __restrict__ out, long ldo) {
  using R = float;
  __shared__ cplx<R> sP[kRK][kRT + 1];  // [j][point]
  __shared__ cplx<R> sU[kRK][kRT];      // [j][i] = conj(u[i][j])
  const long p0 = (long)blockIdx.x * kRT;
  const int i0 = blockIdx.y * kRT;
  const int ti = threadIdx.x / 128 * 8 + threadIdx.x % 8, tp = (threadIdx.x / 32) % 4 * 4 + threadIdx.x % 32 / 8;
  cplx<R> acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = mk<R>(0, 0);
  for (int j0 = 0; j0 < M; j0 += kRK) {
    for (int e = threadIdx.x; e < kRK * kRT; e += blockDim.x) {
      const int jj = e % kRK, pp = e / kRK;
      const long p = p0 + pp;
      const int j = j0 + jj;
      sP[jj][pp] = (p < N && j < M) ? psi[p * ld + j] : mk<R>(0, 0);
      const int ii = e / kRK;  // same decomposition for u: [i][j] rows
      const int i = i0 + ii;
      if (i < M && j < M) {
        const double2 x = u[(size_t)i * M + j];
        sU[jj][ii] = mk<R>((R)x.x, (R)(-x.y));
      } else {
        sU[jj][ii] = mk<R>(0, 0);
      }
    }
    __syncthreads();
#pragma unroll
    for (int jj = 0; jj < kRK; ++jj) {
      cplx<R> pv[4], uv[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) pv[a] = sP[jj][tp + 16 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) uv[b] = sU[jj][ti + 16 * b];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          acc[a][b].x = fma(pv[a].x, uv[b].x, fma(-pv[a].y, uv[b].y, acc[a][b].x));
          acc[a][b].y = fma(pv[a].x, uv[b].y, fma(pv[a].y, uv[b].x, acc[a][b].y));
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const long p = p0 + tp + 16 * a;
      const int i = i0 + ti + 16 * b;
      if (p < N && i < M) out[p * ldo + i] = acc[a][b];
    }
}

}  // namespace

namespace {
template <typename T>
long gram_slabs(long N, int Ma, int Mb) {
  if (sizeof(T) == 4) return std::max<long>(1, (N + kSlabF32 - 1) / kSlabF32);
  constexpr int TM = GramCfg<T>::TILE_M, TN = GramCfg<T>::TILE_N;
  const long tiles = 3L * ((Ma + TM - 1) / TM) * ((Mb + TN - 1) / TN);
  const long chunks = (N + GramCfg<T>::GP - 1) / GramCfg<T>::GP;
  return std::max<long>(1, std::min<long>(chunks, 148L * 4 / tiles));  // two waves of 2 CTAs an SM
}
size_t slab_bytes(long N, int Ma, int Mb) {
  const size_t MM = (size_t)Ma * Mb;
  return std::max((size_t)gram_slabs<double>(N, Ma, Mb) * 3 * MM * sizeof(double2),
                  (size_t)gram_slabs<float>(N, Ma, Mb) * 3 * MM * sizeof(float2));
}
}  // namespace

// the slabs of the larger layout, then Z [3][Ma][Mb] (FP64) at a 256-byte boundary and the
// axis tables
size_t mlwf_partial_bytes(long N, int Ma, int Mb) {
  return (slab_bytes(N, Ma, Mb) + 255) / 256 * 256 + (3 * (size_t)Ma * Mb + 9 * kAxisMax) * sizeof(double2);
}
size_t mlwf_partial_bytes(long N, int M) { return mlwf_partial_bytes(N, M, M); }

// Z [3][Ma][Mb] = sum_p conj(a_m) e^{i theta_d} b_n (FP64 sums of the slabs), in the
// partial buffer after the slabs; returns Z
template <typename T>
static int gram_impl(const void* pa, long lda, int Ma, const void* pb, long ldb, int Mb, long N, const GramGeom& g,
                     void* partial, double2** Zout, cudaStream_t st) {
  using P = typename GramCfg<T>::P;
  constexpr int TM = GramCfg<T>::TILE_M, TN = GramCfg<T>::TILE_N, kGP = GramCfg<T>::GP;
  const long slabs = gram_slabs<T>(N, Ma, Mb);
  const long per = ((N + slabs - 1) / slabs + kGP - 1) / kGP * kGP;
  const long nslab = (N + per - 1) / per;
  const unsigned tiles = (unsigned)(((Ma + TM - 1) / TM) * ((Mb + TN - 1) / TN));
  double2* Z = reinterpret_cast<double2*>(static_cast<char*>(partial) + (slab_bytes(N, Ma, Mb) + 255) / 256 * 256);
  double2* tab = Z + 3 * (size_t)Ma * Mb;
  k_mlwf_axis<<<9, 128, 0, st>>>(g, tab);
  if constexpr (sizeof(T) == 8)
    k_mlwf_gram_dmma<<<dim3(tiles, (unsigned)nslab, 3), kDThreads, 0, st>>>(
        (const cplx<T>*)pa, lda, Ma, (const cplx<T>*)pb, ldb, Mb, N, g, tab, per, (P*)partial);
  else
    k_mlwf_gram<<<dim3(tiles, (unsigned)nslab), 256, 0, st>>>((const cplx<T>*)pa, lda, Ma, (const cplx<T>*)pb, ldb,
                                                              Mb, N, g, tab, per, (P*)partial);
  INQB_CUDA_TRY(cudaGetLastError());
  const long work = 3L * Ma * Mb;
  k_mlwf_slab_sum<P><<<(unsigned)((work + 31) / 32), 256, 0, st>>>((const P*)partial, (int)nslab, work, Z);
  INQB_CUDA_TRY(cudaGetLastError());
  *Zout = Z;
  return INQB_OK;
}

static GramGeom gram_geom(const int nr[3], const double lat[3][3]) {
  GramGeom g;
  double len[3];
  for (int d = 0; d < 3; ++d) {
    g.nr[d] = nr[d];
    len[d] = sqrt(lat[d][0] * lat[d][0] + lat[d][1] * lat[d][1] + lat[d][2] * lat[d][2]);
  }
  // theta_d / pi = 2 r_d / |a_d|, r = sum_j f_j a_j
  for (int d = 0; d < 3; ++d)
    for (int j = 0; j < 3; ++j) g.frac_to_theta[d][j] = 2.0 * lat[j][d] / len[d];
  return g;
}

int launch_mlwf_gram(int precision, const void* psi, long ld, int M, long N, const int nr[3], const double lat[3][3],
                     const double* sums, void* partial, double2* a, void* stream) {
  const GramGeom g = gram_geom(nr, lat);
  cudaStream_t st = (cudaStream_t)stream;
  double2* Z = nullptr;
  INQB_TRY(precision == INQB_FP64 ? gram_impl<double>(psi, ld, M, psi, ld, M, N, g, partial, &Z, st)
                                  : gram_impl<float>(psi, ld, M, psi, ld, M, N, g, partial, &Z, st));
  return launch_mlwf_finish(Z, M, sums, 3, a, stream);
}

int launch_mlwf_gram_block(int precision, const void* pa, long lda, int Ma, const void* pb, long ldb, int Mb, long N,
                           const int nr[3], const double lat[3][3], void* partial, double2* Z, void* stream) {
  const GramGeom g = gram_geom(nr, lat);
  cudaStream_t st = (cudaStream_t)stream;
  double2* Zw = nullptr;
  INQB_TRY(precision == INQB_FP64 ? gram_impl<double>(pa, lda, Ma, pb, ldb, Mb, N, g, partial, &Zw, st)
                                  : gram_impl<float>(pa, lda, Ma, pb, ldb, Mb, N, g, partial, &Zw, st));
  INQB_CUDA_TRY(cudaMemcpyAsync(Z, Zw, sizeof(double2) * 3 * (size_t)Ma * Mb, cudaMemcpyDeviceToDevice, st));
  return INQB_OK;
}

int launch_mlwf_finish(const double2* Z, int M, const double* norms, int norm_stride, double2* a, void* stream) {
  const long work = 3L * M * M;
  k_mlwf_finish<<<(unsigned)std::min<long>((work + 255) / 256, 148L * 8), 256, 0, (cudaStream_t)stream>>>(
      Z, M, norms, norm_stride, a);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

int launch_identity(double2* u, int M, void* stream) {
  k_identity<<<(unsigned)std::min<long>(((long)M * M + 255) / 256, 1024), 256, 0, (cudaStream_t)stream>>>(u, M);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

int launch_jade_step(double2* a, double2* u, int M, const int2* pairs, int np, double* delta, void* stream) {
  k_jade_step<<<np, kJT, 0, (cudaStream_t)stream>>>(a, u, M, pairs, delta);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

template <int E, int GMAX>
static int jade_cluster_launch(double2* a, double2* u, int M, const int2* pairs, int np, int steps, int maxsweep,
                               double tol, double* delta, double* out, bool* done, cudaStream_t st) {
  const int slots = (np + kJadeCtas - 1) / kJadeCtas;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kJadeCtas);
  cfg.blockDim = dim3(slots * kJG);
  cfg.dynamicSmemBytes = (size_t)slots * 2 * 7 * M * sizeof(double2);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kJadeCtas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  INQB_CUDA_TRY(cudaFuncSetAttribute(k_jade_cluster<E, GMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     GMAX * 2 * 7 * 32 * E * (int)sizeof(double2)));
  INQB_CUDA_TRY(cudaFuncSetAttribute(k_jade_cluster<E, GMAX>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  int fit = 0;
  if (cudaOccupancyMaxActiveClusters(&fit, k_jade_cluster<E, GMAX>, &cfg) != cudaSuccess || fit < 1) {
    cudaGetLastError();  // no place for such a cluster: the step launches
    return INQB_OK;
  }
  INQB_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_jade_cluster<E, GMAX>, a, u, M, pairs, np, steps, maxsweep, tol, delta, out));
  *done = true;
  return INQB_OK;
}

// All sweeps in one launch (a and u on the device; u is set, not read).  done: whether they ran
// so, which takes at most 128 states and a GPU that places a cluster of 16 CTAs.  out[0], out[1]:
// the last sweep's trace change, the sweeps.
int launch_jade_cluster(double2* a, double2* u, int M, const int2* pairs, int np, int steps, int maxsweep, double tol,
                        double* delta, double* out, bool* done, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  *done = false;
  // a slot's seven warps must all be resident, so at most four slots per CTA: 128 states
  if (M <= 64) return jade_cluster_launch<2, 2>(a, u, M, pairs, np, steps, maxsweep, tol, delta, out, done, st);
  if (M <= 128) return jade_cluster_launch<4, 4>(a, u, M, pairs, np, steps, maxsweep, tol, delta, out, done, st);
  return INQB_OK;
}

int launch_jade_change(const double* delta, int nsteps, int np, double* out, void* stream) {
  k_jade_change<<<1, 256, 0, (cudaStream_t)stream>>>(delta, nsteps, np, out);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

int launch_jade_adiag(const double2* a, const double2* u, int M, double2* adiag, void* stream) {
  k_jade_adiag<<<dim3(M, 6), 128, 0, (cudaStream_t)stream>>>(a, u, M, adiag);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

int launch_mlwf_rotate(int precision, const void* psi, long ld, int M, long N, const double2* u, void* out, long ldo,
                       void* stream) {
  if (precision == INQB_FP64) return launch_rotate_adjoint(psi, ld, M, u, out, ldo, N, stream);
  const dim3 grid((unsigned)((N + kRT - 1) / kRT), (unsigned)((M + kRT - 1) / kRT));
  k_mlwf_rotate<<<grid, 256, 0, (cudaStream_t)stream>>>((const cplx<float>*)psi, ld, M, N, u, (cplx<float>*)out, ldo);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

}  // namespace inqb
