// Observables and FP64 orbital linear algebra on the device:
//   density   rho[p] = sum_m occ[m] |psi[p][m]|^2       (src/observables/density.hpp:23-33)
//   dipole    dV sum_p r_p rho[p]                         (src/observables/dipole.hpp:23-40)
//   overlap   S = dV psi^H psi, FP64 arithmetic            (src/operations/overlap.hpp:41)
//   cholesky  S = U^H U, U upper                          (src/matrix/cholesky.hpp:28-89)
//   rotate    psi <- psi U^-1                             (src/operations/rotate.hpp:147-157)
// Input orbitals may be complex64 (mixed) or complex128; every sum is FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "dft.cuh"
#include "dmma.cuh"
#include "inqb_internal.h"
#include "observables.h"

namespace inqb {

// A group of LPP lanes per grid point (16 where M <= 16, so that no lane idles), four points
// at a time: their loads are in flight together, which the one-point loop's reduction
// chain prevented.
template <typename T, int LPP>
__global__ void __launch_bounds__(256)
    k_density(const cplx<T>* __restrict__ psi, long ld, int M, long N, const double* __restrict__ occ,
              double* __restrict__ rho) {
  constexpr int PTS = 4;
  const int lane = threadIdx.x & (LPP - 1);
  const long grp = ((long)blockIdx.x * blockDim.x + threadIdx.x) / LPP;
  const long ngrp = ((long)gridDim.x * blockDim.x) / LPP;
  // every lane of a warp runs the same number of iterations (the shuffles below)
  const long step = ngrp * PTS, pend = (N + step - 1) / step * step;
  for (long p0 = grp * PTS; p0 < pend; p0 += step) {
    double acc[PTS] = {0.0, 0.0, 0.0, 0.0};
    for (int m = lane; m < M; m += LPP) {
      cplx<T> v[PTS];
#pragma unroll
      for (int u = 0; u < PTS; ++u) v[u] = (p0 + u < N) ? psi[(p0 + u) * ld + m] : mk<T>(0, 0);
      const double o = occ[m];
#pragma unroll
      for (int u = 0; u < PTS; ++u) acc[u] += o * ((double)v[u].x * (double)v[u].x + (double)v[u].y * (double)v[u].y);
    }
#pragma unroll
    for (int o = LPP / 2; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < PTS; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
#pragma unroll
    for (int u = 0; u < PTS; ++u)
      if (lane == u && p0 + u < N) rho[p0 + u] = acc[u];
  }
}

struct LatticeView {
  double lat[3][3];
  int nr[3];
};

__device__ __forceinline__ void rvector(const LatticeView& g, long p, double r[3]) {
  const int nyz = g.nr[1] * g.nr[2];
  int ii[3] = {(int)(p / nyz), (int)((p / g.nr[2]) % g.nr[1]), (int)(p % g.nr[2])};
  double c[3];
  for (int d = 0; d < 3; d++) {
    int s = (ii[d] >= (g.nr[d] + 1) / 2) ? ii[d] - g.nr[d] : ii[d];
    c[d] = s * (1.0 / g.nr[d]);
  }
  for (int k = 0; k < 3; k++) r[k] = g.lat[0][k] * c[0] + g.lat[1][k] * c[1] + g.lat[2][k] * c[2];
}

__global__ void k_dipole(const double* __restrict__ rho, long N, LatticeView g, double* __restrict__ out) {
  double acc[3] = {0, 0, 0};
  for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (long)gridDim.x * blockDim.x) {
    double r[3];
    rvector(g, p, r);
    const double d = rho[p];
    for (int k = 0; k < 3; k++) acc[k] += r[k] * d;
  }
  __shared__ double red[3][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = 0; k < 3; k++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (lane == 0) red[k][warp] = acc[k];
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    for (int k = 0; k < 3; k++) {
      double v = lane < nw ? red[k][lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) atomicAdd(&out[k], v);
    }
  }
}

// ---------------------------------------------------------------- overlap
// 256 threads as a 16 x 16 grid, a warp 4 x 8 of it: a warp's 16-byte shared loads then
// touch 64 bytes of the row operand and 128 of the column operand, one wavefront each (as
// 2 x 16 the column operand took two or more, and the loads bound the kernel at 59% of the
// FP64 rate).
__device__ __forceinline__ int grid_row() { return (threadIdx.x / 32) % 4 * 4 + threadIdx.x % 32 / 8; }
__device__ __forceinline__ int grid_col() { return threadIdx.x / 128 * 8 + threadIdx.x % 8; }

// tile t of the tiles on and above the diagonal: (0, 0..), (1, 1..), ...
__device__ __forceinline__ void overlap_tile(int t, int tiles_j, bool upper, int& bi, int& bj) {
  if (upper) {
    bi = 0;
    while (t >= tiles_j - bi) t -= tiles_j - bi++;
    bj = bi + t;
  } else {
    bi = t / tiles_j;
    bj = t % tiles_j;
  }
}

// S[i][j] += dV sum_{p in slab} conj(a[p][i]) b[p][j], FP64 products and sums.
// The square overlap (upper) computes the tiles on and above the diagonal only, which is
// all the Cholesky factorisation reads.
//
// Tiles of 16 and 32 outputs a side (TM = 1, 2), for blocks of at most 32 orbitals: 256
// threads as 16 x 16, TM x TM outputs a thread (outputs ti + 16 a, tj + 16 b) over the
// CTA's slab of points; KP points are staged at a time, the next ones fetched into
// registers meanwhile.
template <int TM>
struct OverlapCfg {
  static constexpr int KP = TM == 2 ? 16 : 32;
  static constexpr int CTAS = 4;  // per SM
};

template <typename T, int TM>
__global__ void __launch_bounds__(256, OverlapCfg<TM>::CTAS)
    k_overlap(const cplx<T>* __restrict__ pa, long lda, int Ma, const cplx<T>* __restrict__ pb, long ldb, int Mb,
              long N, long slab, double dV, double2* __restrict__ S, long lds, int upper) {
  constexpr int TILE = 16 * TM, KP = OverlapCfg<TM>::KP, PER = TILE * KP / 256;
  __shared__ double2 sa[KP][TILE], sb[KP][TILE];
  const int tiles_j = (Mb + TILE - 1) / TILE;
  int bi, bj;
  overlap_tile(blockIdx.x, tiles_j, upper, bi, bj);
  const int i0 = bi * TILE, j0 = bj * TILE;
  const bool diag = upper && bi == bj;  // one block serves both sides
  const int ti = grid_row(), tj = grid_col();
  const long p0 = (long)blockIdx.y * slab, p1 = min(N, p0 + slab);
  double re[TM][TM], im[TM][TM];
#pragma unroll
  for (int a = 0; a < TM; ++a)
#pragma unroll
    for (int b = 0; b < TM; ++b) re[a][b] = im[a][b] = 0.0;
  cplx<T> va[PER], vb[PER];
  auto fetch = [&](long pc) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = threadIdx.x + 256 * u, q = e / TILE, j = e % TILE;
      const long p = pc + q;
      va[u] = (p < p1 && i0 + j < Ma) ? pa[p * lda + i0 + j] : mk<T>(0, 0);
      if (!diag) vb[u] = (p < p1 && j0 + j < Mb) ? pb[p * ldb + j0 + j] : mk<T>(0, 0);
    }
  };
  fetch(p0);
  const double2(*sbv)[TILE] = diag ? sa : sb;
  for (long pc = p0; pc < p1; pc += KP) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = threadIdx.x + 256 * u, q = e / TILE, j = e % TILE;
      sa[q][j] = make_double2(va[u].x, va[u].y);
      if (!diag) sb[q][j] = make_double2(vb[u].x, vb[u].y);
    }
    __syncthreads();
    if (pc + KP < p1) fetch(pc + KP);
#pragma unroll 4
    for (int q = 0; q < KP; ++q) {
      double2 x[TM], y[TM];
#pragma unroll
      for (int a = 0; a < TM; ++a) x[a] = sa[q][ti + 16 * a];
#pragma unroll
      for (int b = 0; b < TM; ++b) y[b] = sbv[q][tj + 16 * b];
      // a tile on the diagonal needs its 16-wide blocks a <= b only
#pragma unroll
      for (int a = 0; a < TM; ++a)
#pragma unroll
        for (int b = 0; b < TM; ++b) {
          if (a > b && diag) continue;
          re[a][b] = fma(x[a].x, y[b].x, fma(x[a].y, y[b].y, re[a][b]));
          im[a][b] = fma(x[a].x, y[b].y, fma(-x[a].y, y[b].x, im[a][b]));
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < TM; ++a)
#pragma unroll
    for (int b = 0; b < TM; ++b) {
      const int i = i0 + ti + 16 * a, j = j0 + tj + 16 * b;
      if (i < Ma && j < Mb && !(upper && i > j)) {
        atomicAdd(&S[(long)i * lds + j].x, dV * re[a][b]);
        atomicAdd(&S[(long)i * lds + j].y, dV * im[a][b]);
      }
    }
}

// Slabs of points per tile in proportion to its work, so that the CTAs of a wave end
// together: a tile takes the time of its busiest warp (8-wide blocks: 16, on the diagonal 9,
// less at the edges) and one more for the chunk's loads and barrier.
struct OverlapShare {
  long ctas, total, most;  // CTAs of the launch, sum of the weights, slabs a tile may have
  __host__ __device__ static int weight(int bi, int bj, int Ma, int Mb, bool upper) {
    const int ra = (Ma - bi * kDT + 7) / 8, rb = (Mb - bj * kDT + 7) / 8;
    const int rows = ra < 8 ? ra : 8, cols = rb < 8 ? rb : 8;
    if (upper && bi == bj) return (cols < 8 ? cols : 9) + 1;
    return cols * (rows > 4 ? 2 : 1) + 1;
  }
  __host__ __device__ int slabs(int bi, int bj, int Ma, int Mb, bool upper) const {
    const long n = ctas * weight(bi, bj, Ma, Mb, upper) / total;
    return (int)(n < 1 ? 1 : n < most ? n : most);
  }
};

// The same overlap with tiles of 64 on the FP64 tensor instruction: a warp's 64 products of
// a staged quad of points take 10 shared loads, where 4 x 4 outputs a thread on FMAs took 8
// loads for 64 FMAs and waited for them (64^3 points x 128 orbitals complex128: 1.19 ->
// 0.69 ms).  Bound by the FP64 pipe, 81% busy.
template <typename T>
__global__ void __launch_bounds__(kDThreads, 2)
    k_overlap_dmma(const cplx<T>* __restrict__ pa, long lda, int Ma, const cplx<T>* __restrict__ pb, long ldb, int Mb,
                   long N, OverlapShare share, double dV, double2* __restrict__ S, long lds, int upper) {
  __shared__ DmmaBuf sa[2], sb[2];
  int bi = 0, bj = 0, first = 0, slabs = share.slabs(0, 0, Ma, Mb, upper);
  while ((int)blockIdx.x >= first + slabs) {  // the tile whose slabs hold this CTA
    first += slabs;
    if (++bj * kDT >= Mb) bj = upper ? ++bi : (++bi, 0);
    slabs = share.slabs(bi, bj, Ma, Mb, upper);
  }
  const long slab = ((N + slabs - 1) / slabs + kDK - 1) / kDK * kDK;
  const int i0 = bi * kDT, j0 = bj * kDT;
  const bool diag = upper && bi == bj;  // one block serves both sides
  const long p0 = (blockIdx.x - first) * slab, p1 = min(N, p0 + slab);
  if (p0 >= N) return;
  DmmaTile t;
  t.clear();
  const int rows = min(8, (Ma - i0 + 7) / 8), hi = min(8, (Mb - j0 + 7) / 8);
  DmmaOperand<T, false> oa, ob;
  auto load = [&](long pc, int buf) {
    oa.load(sa[buf], pa, [&](int q, int j) { return pc + q < p1 && i0 + j < Ma ? (pc + q) * lda + i0 + j : -1L; });
    if (!diag)
      ob.load(sb[buf], pb, [&](int q, int j) { return pc + q < p1 && j0 + j < Mb ? (pc + q) * ldb + j0 + j : -1L; });
    dmma_commit();
  };
  auto store = [&](int buf) {
    oa.store(sa[buf]);
    if (!diag) ob.store(sb[buf]);
  };
  load(p0, 0);
  store(0);
  int buf = 0;
  for (long pc = p0; pc < p1; pc += kDK, buf ^= 1) {
    dmma_arrived();
    __syncthreads();  // chunk pc is complete, and every warp has left the other buffer
    const bool more = pc + kDK < p1;
    if (more) load(pc + kDK, buf ^ 1);
    if (diag)
      t.mul_upper<kConjX>(sa[buf], sa[buf], hi, DmmaNoWeight());
    else
      t.mul_block<kConjX>(sa[buf], sb[buf], rows, hi, DmmaNoWeight());
    if (more) store(buf ^ 1);
  }
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int i = i0 + 8 * DmmaTile::row_block(a) + (lane >> 2), j = j0 + 8 * c + 2 * (lane & 3);
      auto add = [&](int jj, double x, double y) {
        if (i < Ma && jj < Mb && !(upper && i > jj)) {
          atomicAdd(&S[(long)i * lds + jj].x, dV * x);
          atomicAdd(&S[(long)i * lds + jj].y, dV * y);
        }
      };
      add(j, t.re[a][c].x, t.im[a][c].x);
      add(j + 1, t.re[a][c].y, t.im[a][c].y);
    }
}

// ---------------------------------------------------------------- Cholesky factor and its inverse
// S = U^H U by blocks of kNB, one launch per block row: launch k (k = -1 first) finishes
// block row k and updates the trailing blocks, and the CTA of the next diagonal block also
// factors it, so the serial part (32 pivots in shared memory) runs inside the same launch.
//   S[k][k] holds W_k = U_kk^-1 after its factorisation, U[k][j] (in X) = W_k^H S[k][j];
//   trailing S[i][j] -= U[k][i]^H U[k][j], each CTA forming both panels itself.
// The factorisation leaves a pivot row unscaled until the end (D[i][j] -= conj(D[k][i])
// D[k][j] / d_k reads the row as it is), so a pivot costs one barrier.
constexpr int kNB = 32;

// thread (r, c0): row r = tid / 8, columns c0 + 8 m for m < 4, c0 = tid % 8
struct Quad {
  double2 v[4];
};
__device__ __forceinline__ Quad quad_zero() {
  Quad q;
#pragma unroll
  for (int m = 0; m < 4; ++m) q.v[m] = make_double2(0.0, 0.0);
  return q;
}
__device__ __forceinline__ void quad_store(double2 (*d)[kNB], const Quad& q) {
  const int r = threadIdx.x / 8, c0 = threadIdx.x % 8;
#pragma unroll
  for (int m = 0; m < 4; ++m) d[r][c0 + 8 * m] = q.v[m];
}
// block (bi, bj) of an M x M matrix; outside the matrix: the identity (one) or zero
__device__ __forceinline__ Quad quad_load(const double2* A, long lda, int M, int bi, int bj, bool one) {
  const int r = threadIdx.x / 8, c0 = threadIdx.x % 8;
  Quad q;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int i = bi * kNB + r, j = bj * kNB + c0 + 8 * m;
    q.v[m] = (i < M && j < M) ? A[(long)i * lda + j] : make_double2(one && i == j ? 1.0 : 0.0, 0.0);
  }
  return q;
}
__device__ __forceinline__ void quad_write(double2* A, long lda, int M, int bi, int bj, const Quad& q) {
  const int r = threadIdx.x / 8, c0 = threadIdx.x % 8;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int i = bi * kNB + r, j = bj * kNB + c0 + 8 * m;
    if (i < M && j < M) A[(long)i * lda + j] = q.v[m];
  }
}
// acc += s A^H B (ADJ) or s A B of two blocks in shared memory
template <bool ADJ>
__device__ __forceinline__ void quad_mul(Quad& acc, double s, const double2 (*A)[kNB], const double2 (*B)[kNB]) {
  const int r = threadIdx.x / 8, c0 = threadIdx.x % 8;
#pragma unroll 4
  for (int q = 0; q < kNB; ++q) {
    double2 a = ADJ ? A[q][r] : A[r][q];
    a = make_double2(s * a.x, ADJ ? -s * a.y : s * a.y);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const double2 b = B[q][c0 + 8 * m];
      acc.v[m].x = fma(a.x, b.x, fma(-a.y, b.y, acc.v[m].x));
      acc.v[m].y = fma(a.x, b.y, fma(a.y, b.x, acc.v[m].y));
    }
  }
}

// Factor the block in D (upper triangle) and write U_kk to U, W_k = U_kk^-1 (zero below
// the diagonal) to S; info gets the first failing pivot + 1.  W is scratch.
__device__ void chol_diag(double2 (*D)[kNB], double2 (*W)[kNB], double2* S, long lds, double2* U, int M, int k,
                          int* info) {
  const int r = threadIdx.x / 8, c0 = threadIdx.x % 8;
  const int first = *info;  // a failed pivot of an earlier block stays the first
  for (int p = 0; p < kNB; ++p) {
    const double d = D[p][p].x;
    if (!(d > 0.0)) {
      if (threadIdx.x == 0 && first == 0) *info = k * kNB + p + 1;
      return;
    }
    if (r > p) {
      const double2 x = D[p][r];
      const double2 f = make_double2(x.x / d, -x.y / d);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int c = c0 + 8 * m;
        if (c < r) continue;
        const double2 y = D[p][c];
        D[r][c].x -= f.x * y.x - f.y * y.y;
        D[r][c].y -= f.x * y.y + f.y * y.x;
      }
    }
    __syncthreads();
  }
  // U[r][c] = D[r][c] / sqrt(d_r); W starts as the identity
  const double d = D[r][r].x, u = sqrt(d);
  Quad q;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int c = c0 + 8 * m;
    const double2 y = D[r][c];
    q.v[m] = c > r ? make_double2(y.x / u, y.y / u) : make_double2(c == r ? u : 0.0, 0.0);
    W[r][c] = make_double2(c == r ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  quad_store(D, q);
  quad_write(U, M, M, k, k, q);
  __syncthreads();
  // rows from the last up: W[q] / U[q][q] is final, then W[r] -= U[r][q] W[q] / U[q][q]
  for (int p = kNB - 1; p > 0; --p) {
    if (r < p) {
      const double inv = 1.0 / D[p][p].x;
      const double2 f = make_double2(D[r][p].x * inv, D[r][p].y * inv);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int c = c0 + 8 * m;
        if (c < p) continue;
        const double2 y = W[p][c];
        W[r][c].x -= f.x * y.x - f.y * y.y;
        W[r][c].y -= f.x * y.y + f.y * y.x;
      }
    }
    __syncthreads();
  }
  const double inv = 1.0 / D[r][r].x;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const double2 y = W[r][c0 + 8 * m];
    q.v[m] = make_double2(y.x * inv, y.y * inv);
  }
  quad_write(S, lds, M, k, k, q);
}

__global__ void __launch_bounds__(256)
    k_chol_step(double2* S, long lds, double2* U, int M, int k, int* info) {
  __shared__ double2 A[kNB][kNB], B[kNB][kNB], W[kNB][kNB];
  if (k < 0) {
    quad_store(A, quad_load(S, lds, M, 0, 0, true));
    __syncthreads();
    chol_diag(A, W, S, lds, U, M, 0, info);
    return;
  }
  const int nb = (M + kNB - 1) / kNB;
  int t = blockIdx.x, i = k + 1;
  while (t >= nb - i) t -= nb - i++;
  const int j = i + t;
  // panels U[k][i], U[k][j] = W_k^H S[k][i], W_k^H S[k][j]
  quad_store(W, quad_load(S, lds, M, k, k, false));
  quad_store(A, quad_load(S, lds, M, k, i, false));
  quad_store(B, quad_load(S, lds, M, k, j, false));
  __syncthreads();
  Quad pi = quad_zero(), pj = quad_zero();
  quad_mul<true>(pi, 1.0, W, A);
  if (i != j) quad_mul<true>(pj, 1.0, W, B);
  __syncthreads();
  if (i == j) {
    pj = pi;
    quad_write(U, M, M, k, j, pj);
  }
  quad_store(A, pi);
  quad_store(B, pj);
  __syncthreads();
  Quad s = quad_load(S, lds, M, i, j, i == j);
  quad_mul<true>(s, -1.0, A, B);
  if (i == k + 1 && j == k + 1) {
    __syncthreads();
    quad_store(A, s);
    __syncthreads();
    chol_diag(A, W, S, lds, U, M, i, info);
  } else {
    quad_write(S, lds, M, i, j, s);
  }
}

// X = U^-1 in place of S: CTA j solves block column j from the diagonal up,
// X[i][j] = -W_i sum_{i < q <= j} U[i][q] X[q][j], and zeroes it below the diagonal.
__global__ void __launch_bounds__(256) k_chol_inverse(double2* S, long lds, const double2* __restrict__ U, int M) {
  __shared__ double2 A[kNB][kNB], B[kNB][kNB];
  const int j = blockIdx.x, nb = (M + kNB - 1) / kNB;
  for (int i = j + 1; i < nb; ++i) quad_write(S, lds, M, i, j, quad_zero());
  for (int i = j - 1; i >= 0; --i) {
    Quad acc = quad_zero();
    for (int q = i + 1; q <= j; ++q) {
      __syncthreads();
      quad_store(A, quad_load(U, M, M, i, q, false));
      quad_store(B, quad_load(S, lds, M, q, j, false));
      __syncthreads();
      quad_mul<false>(acc, 1.0, A, B);
    }
    __syncthreads();
    quad_store(A, quad_load(S, lds, M, i, i, false));
    quad_store(B, acc);
    __syncthreads();
    Quad x = quad_zero();
    quad_mul<false>(x, -1.0, A, B);
    quad_write(S, lds, M, i, j, x);
  }
}

// ---------------------------------------------------------------- rotation
// out[p][j] = sum_i a[p][i] R[i][j], FP64 arithmetic.  A CTA owns 64 points and a block of
// columns at a time; eight orbitals i are staged at a time, the next ones fetched into
// registers meanwhile.
// UPPER: R is upper triangular and out may be a.  The CTA walks its columns from the last
// block down: a block of outputs reads only the input columns up to itself, so it may
// overwrite its own input columns once they are read.
//
// At most 32 columns: (16 TN) of them, 256 threads as 16 x 16 with 4 x TN outputs each.
template <typename T, int TN, bool UPPER>
__global__ void __launch_bounds__(256, 3)
    k_rotate(const cplx<T>* a, long lda, int Ma, const double2* __restrict__ R, long ldr, int Mo, cplx<T>* out,
             long ldo, long N) {
  constexpr int TP = 4, PTS = 16 * TP, COLS = 16 * TN, KP = 8;
  constexpr int PA = PTS * KP / 256, PB = (COLS * KP + 255) / 256;
  __shared__ double2 sa[KP][PTS + 1];  // [i][point]; the odd row spreads the transposing stores
  __shared__ double2 sr[KP][COLS];
  const int tp = grid_row(), tj = grid_col();
  const long p0 = (long)blockIdx.x * PTS;
  const int nblk = (Mo + COLS - 1) / COLS;
  const int b_hi = UPPER ? nblk - 1 : (int)blockIdx.y, b_lo = UPPER ? 0 : (int)blockIdx.y;
  for (int jb = b_hi; jb >= b_lo; --jb) {
    const int j0 = jb * COLS;
    const int kend = UPPER ? min(Ma, j0 + COLS) : Ma;
    double re[TP][TN], im[TP][TN];
#pragma unroll
    for (int u = 0; u < TP; ++u)
#pragma unroll
      for (int v = 0; v < TN; ++v) re[u][v] = im[u][v] = 0.0;
    cplx<T> va[PA];
    double2 vr[PB];
    auto fetch = [&](int k0) {
#pragma unroll
      for (int u = 0; u < PA; ++u) {
        const int e = threadIdx.x + 256 * u, i = k0 + e % KP;
        const long p = p0 + e / KP;
        va[u] = (p < N && i < kend) ? a[p * lda + i] : mk<T>(0, 0);
      }
#pragma unroll
      for (int u = 0; u < PB; ++u) {
        const int e = threadIdx.x + 256 * u, i = k0 + e / COLS, j = j0 + e % COLS;
        vr[u] = (e < KP * COLS && i < kend && j < Mo) ? R[(long)i * ldr + j] : make_double2(0.0, 0.0);
      }
    };
    fetch(0);
    for (int k0 = 0; k0 < kend; k0 += KP) {
#pragma unroll
      for (int u = 0; u < PA; ++u) {
        const int e = threadIdx.x + 256 * u;
        sa[e % KP][e / KP] = make_double2(va[u].x, va[u].y);
      }
#pragma unroll
      for (int u = 0; u < PB; ++u) {
        const int e = threadIdx.x + 256 * u;
        if (e < KP * COLS) sr[e / COLS][e % COLS] = vr[u];
      }
      __syncthreads();
      if (k0 + KP < kend) fetch(k0 + KP);
      const int vmin = UPPER ? max(0, (k0 - j0) / 16) : 0;
#pragma unroll 4
      for (int q = 0; q < KP; ++q) {
        double2 x[TP], y[TN];
#pragma unroll
        for (int u = 0; u < TP; ++u) x[u] = sa[q][tp + 16 * u];
#pragma unroll
        for (int v = 0; v < TN; ++v) y[v] = sr[q][tj + 16 * v];
        // UPPER: R[i][j] = 0 for the 16-wide column blocks left of row i
#pragma unroll
        for (int v = 0; v < TN; ++v) {
          if (UPPER && v < vmin) continue;
#pragma unroll
          for (int u = 0; u < TP; ++u) {
            re[u][v] = fma(x[u].x, y[v].x, fma(-x[u].y, y[v].y, re[u][v]));
            im[u][v] = fma(x[u].x, y[v].y, fma(x[u].y, y[v].x, im[u][v]));
          }
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < TP; ++u)
#pragma unroll
      for (int v = 0; v < TN; ++v) {
        const long p = p0 + tp + 16 * u;
        const int j = j0 + tj + 16 * v;
        if (p < N && j < Mo) out[p * ldo + j] = mk<T>((T)re[u][v], (T)im[u][v]);
      }
  }
}

// More columns: 64 at a time on the FP64 tensor instruction, a warp 16 points x 64 columns
// (64^3 points x 128 orbitals complex128, triangular: 1.00 -> 0.77 ms; FP64 pipe 69% busy).
// The chunks of all column blocks are one pipeline.
// ADJ: the factor is R^H instead.
template <typename T, bool UPPER, bool ADJ>
__global__ void __launch_bounds__(kDThreads, 2)
    k_rotate_dmma(const cplx<T>* a, long lda, int Ma, const double2* __restrict__ R, long ldr, int Mo, cplx<T>* out,
                  long ldo, long N) {
  __shared__ DmmaBuf sa[2], sr[2];  // [i][point], [i][column]
  const cplx<double>* Rc = reinterpret_cast<const cplx<double>*>(R);
  const long p0 = (long)blockIdx.x * kDT;
  const int nblk = (Mo + kDT - 1) / kDT;
  const int b_hi = UPPER ? nblk - 1 : (int)blockIdx.y, b_lo = UPPER ? 0 : (int)blockIdx.y;
  DmmaOperand<T, true> oa;
  DmmaOperand<double, ADJ> orr;
  auto depth = [&](int jb) { return UPPER ? min(Ma, (jb + 1) * kDT) : Ma; };  // input columns of block jb
  auto load = [&](int jb, int k0, int buf) {
    const int j0 = jb * kDT, kend = depth(jb);
    oa.load(sa[buf], a, [&](int q, int p) { return p0 + p < N && k0 + q < kend ? (p0 + p) * lda + k0 + q : -1L; });
    orr.load(sr[buf], Rc, [&](int q, int j) {
      return k0 + q < kend && j0 + j < Mo ? (ADJ ? (j0 + j) * ldr + k0 + q : (k0 + q) * ldr + j0 + j) : -1L;
    });
    dmma_commit();
  };
  load(b_hi, 0, 0);
  oa.store(sa[0]);
  int buf = 0;
  for (int jb = b_hi; jb >= b_lo; --jb) {
    const int j0 = jb * kDT, kend = depth(jb);
    const int hi = min(8, (Mo - j0 + 7) / 8);
    DmmaTile t;
    t.clear();
    for (int k0 = 0; k0 < kend; k0 += kDK, buf ^= 1) {
      dmma_arrived();
      __syncthreads();  // chunk k0 is complete, and every warp has left the other buffer
      // the next chunk, or the first of the next block: columns that this block does not write
      const bool last = k0 + kDK >= kend, more = !last || jb > b_lo;
      if (more) load(last ? jb - 1 : jb, last ? 0 : k0 + kDK, buf ^ 1);
      // UPPER: R[i][j] = 0 for the 8-wide column blocks left of row i
      const int first = UPPER ? max(0, (k0 - j0) / 8) : 0;
      t.mul_right<ADJ ? kConjY : kConjNone>(sa[buf], sr[buf], first, hi, DmmaNoWeight());
      if (more) oa.store(sa[buf ^ 1]);
    }
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const long p = p0 + 8 * DmmaTile::row_block(r) + (lane >> 2);
        const int j = j0 + 8 * c + 2 * (lane & 3);
        if (p < N && j < Mo) out[p * ldo + j] = mk<T>((T)t.re[r][c].x, (T)t.im[r][c].x);
        if (p < N && j + 1 < Mo) out[p * ldo + j + 1] = mk<T>((T)t.re[r][c].y, (T)t.im[r][c].y);
      }
  }
}

// ---------------------------------------------------------------- launchers
template <typename T>
static int density_impl(const void* psi, long ld, int M, long N, const double* occ, double* rho, cudaStream_t st) {
  const int lpp = M <= 16 ? 16 : 32;
  const int blocks = (int)std::min<long>((N * lpp + 1023) / 1024, 148L * 8);
  if (M <= 16)
    k_density<T, 16><<<blocks, 256, 0, st>>>((const cplx<T>*)psi, ld, M, N, occ, rho);
  else
    k_density<T, 32><<<blocks, 256, 0, st>>>((const cplx<T>*)psi, ld, M, N, occ, rho);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

int launch_density(int precision, const void* psi, long ld, int M, long N, const double* occ, double* rho,
                   void* stream) {
  return precision == INQB_FP64 ? density_impl<double>(psi, ld, M, N, occ, rho, (cudaStream_t)stream)
                                : density_impl<float>(psi, ld, M, N, occ, rho, (cudaStream_t)stream);
}

// acc[3 m .. 3 m + 2] += (Re, Im) sum_p conj(hpsi) psi and sum_p |psi|^2 over this
// block's points (overlap_diagonal.hpp:118-127).  Block: 32 orbitals (lanes) x 8
// point lanes, reduced in shared memory before one FP64 atomic per orbital and sum.
template <typename T>
__global__ void __launch_bounds__(256)
    k_band_sums(const cplx<T>* __restrict__ psi, const cplx<T>* __restrict__ hpsi, long ld, int M, long N,
                long pts_per_block, double* __restrict__ acc) {
  __shared__ double red[8][32][3];
  const int tm = threadIdx.x & 31, tp = threadIdx.x >> 5;
  const int m = blockIdx.y * 32 + tm;
  const long p0 = (long)blockIdx.x * pts_per_block, p1 = min(N, p0 + pts_per_block);
  double vr = 0.0, vi = 0.0, nn = 0.0;
  if (m < M) {
#pragma unroll 4
    for (long p = p0 + tp; p < p1; p += 8) {
      const cplx<T> a = hpsi[p * ld + m], b = psi[p * ld + m];
      const double ax = a.x, ay = a.y, bx = b.x, by = b.y;
      vr += ax * bx + ay * by;
      vi += ax * by - ay * bx;
      nn += bx * bx + by * by;
    }
  }
  red[tp][tm][0] = vr;
  red[tp][tm][1] = vi;
  red[tp][tm][2] = nn;
  __syncthreads();
  if (tp < 3 && m < M) {
    double v = 0.0;
    for (int k = 0; k < 8; k++) v += red[k][tm][tp];
    atomicAdd(&acc[3 * m + tp], v);
  }
}

template <typename T>
static int band_sums_impl(const void* psi, const void* hpsi, long ld, int M, long N, double* acc, cudaStream_t st) {
  INQB_CUDA_TRY(cudaMemsetAsync(acc, 0, sizeof(double) * 3 * (size_t)M, st));
  const int ym = (M + 31) / 32;
  // about 8 blocks per SM over the points
  const long nblk = std::max<long>(1, std::min<long>(N / 64 + 1, 148L * 8 / ym + 1));
  const long per = (N + nblk - 1) / nblk;
  k_band_sums<T><<<dim3((unsigned)((N + per - 1) / per), ym), 256, 0, st>>>(
      (const cplx<T>*)psi, (const cplx<T>*)hpsi, ld, M, N, per, acc);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

int launch_band_sums(int precision, const void* psi, const void* hpsi, long ld, int M, long N, double* acc,
                     void* stream) {
  return precision == INQB_FP64 ? band_sums_impl<double>(psi, hpsi, ld, M, N, acc, (cudaStream_t)stream)
                                : band_sums_impl<float>(psi, hpsi, ld, M, N, acc, (cudaStream_t)stream);
}

int launch_dipole(const double* rho, long N, const double lat[3][3], const int nr[3], double* out_dev,
                  void* stream) {
  LatticeView g;
  for (int i = 0; i < 3; i++) {
    g.nr[i] = nr[i];
    for (int j = 0; j < 3; j++) g.lat[i][j] = lat[i][j];
  }
  cudaStream_t st = (cudaStream_t)stream;
  INQB_CUDA_TRY(cudaMemsetAsync(out_dev, 0, 3 * sizeof(double), st));
  const int blocks = (int)std::min<long>((N + 255) / 256, 148L * 4);
  k_dipole<<<blocks, 256, 0, st>>>(rho, N, g, out_dev);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

// tiles of the output and slabs of points (at least 512 each) so that the CTAs fill the GPU
template <typename T, int TM>
static int overlap_launch(const void* a, long lda, int Ma, const void* b, long ldb, int Mb, long N, double dV,
                          double2* S, long lds, bool upper, cudaStream_t st) {
  constexpr int TILE = 16 * TM, KP = OverlapCfg<TM>::KP;
  const long ti = (Ma + TILE - 1) / TILE, tj = (Mb + TILE - 1) / TILE;
  const long tiles = upper ? ti * (ti + 1) / 2 : ti * tj;
  long slabs = std::max<long>(1, std::min<long>(N / 512, 148L * OverlapCfg<TM>::CTAS / tiles));
  const long slab = ((N + slabs - 1) / slabs + KP - 1) / KP * KP;
  slabs = (N + slab - 1) / slab;
  k_overlap<T, TM><<<dim3((unsigned)tiles, (unsigned)slabs), 256, 0, st>>>(
      (const cplx<T>*)a, lda, Ma, (const cplx<T>*)b, ldb, Mb, N, slab, dV, S, lds, upper);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

template <typename T>
static int overlap_dmma_launch(const void* a, long lda, int Ma, const void* b, long ldb, int Mb, long N, double dV,
                               double2* S, long lds, bool upper, cudaStream_t st) {
  const int ti = (Ma + kDT - 1) / kDT, tj = (Mb + kDT - 1) / kDT;
  // one wave of CTAs for one tile, else two (64^3 x 64, 128, 256 orbitals, whole call: one wave
  // 529, 1542, 5327 us, two 560, 1531, 5224)
  OverlapShare share = {ti * tj == 1 ? 148 * 2 : 148 * 4, 0, std::max<long>(1, N / 512)};
  for (int i = 0; i < ti; i++)
    for (int j = upper ? i : 0; j < tj; j++) share.total += OverlapShare::weight(i, j, Ma, Mb, upper);
  unsigned blocks = 0;
  for (int i = 0; i < ti; i++)
    for (int j = upper ? i : 0; j < tj; j++) blocks += share.slabs(i, j, Ma, Mb, upper);
  k_overlap_dmma<T><<<blocks, kDThreads, 0, st>>>((const cplx<T>*)a, lda, Ma, (const cplx<T>*)b, ldb, Mb, N, share, dV,
                                                  S, lds, upper);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

// the tile follows the larger block: a 16- or 32-wide tile where a 64-wide one would be
// mostly padding
template <typename T>
static int overlap_any(const void* a, long lda, int Ma, const void* b, long ldb, int Mb, long N, double dV,
                       double2* S, long lds, bool upper, cudaStream_t st) {
  const int M = std::max(Ma, Mb);
  if (M <= 16) return overlap_launch<T, 1>(a, lda, Ma, b, ldb, Mb, N, dV, S, lds, upper, st);
  if (M <= 32) return overlap_launch<T, 2>(a, lda, Ma, b, ldb, Mb, N, dV, S, lds, upper, st);
  return overlap_dmma_launch<T>(a, lda, Ma, b, ldb, Mb, N, dV, S, lds, upper, st);
}

// S (upper triangle of a Hermitian matrix) <- U^-1; X: M x M scratch (receives U)
static int cholesky_inverse_launch(double2* S, int M, long lds, double2* X, int* info, cudaStream_t st) {
  const int nb = (M + kNB - 1) / kNB;
  INQB_CUDA_TRY(cudaMemsetAsync(info, 0, sizeof(int), st));
  for (int k = -1; k + 1 < nb; k++) {
    const int n = nb - 1 - k;
    k_chol_step<<<k < 0 ? 1 : n * (n + 1) / 2, 256, 0, st>>>(S, lds, X, M, k, info);
  }
  k_chol_inverse<<<nb, 256, 0, st>>>(S, lds, X, M);
  INQB_CUDA_TRY(cudaGetLastError());
  int h_info = 0;
  INQB_CUDA_TRY(cudaMemcpyAsync(&h_info, info, sizeof(int), cudaMemcpyDeviceToHost, st));
  INQB_CUDA_TRY(cudaStreamSynchronize(st));
  if (h_info != 0)
    return fail(INQB_ERR_NOT_POSITIVE_DEFINITE,
                "overlap matrix is not positive definite at pivot " + std::to_string(h_info - 1));
  return INQB_OK;
}

template <typename T, int TN, bool UPPER>
static int rotate_launch(const void* a, long lda, int Ma, const double2* R, long ldr, int Mo, void* out, long ldo,
                         long N, cudaStream_t st) {
  const dim3 grid((unsigned)((N + 63) / 64), UPPER ? 1u : (unsigned)((Mo + 16 * TN - 1) / (16 * TN)));
  k_rotate<T, TN, UPPER><<<grid, 256, 0, st>>>((const cplx<T>*)a, lda, Ma, R, ldr, Mo, (cplx<T>*)out, ldo, N);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

template <typename T, bool UPPER>
static int rotate_any(const void* a, long lda, int Ma, const double2* R, long ldr, int Mo, void* out, long ldo, long N,
                      cudaStream_t st) {
  if (Mo <= 16) return rotate_launch<T, 1, UPPER>(a, lda, Ma, R, ldr, Mo, out, ldo, N, st);
  if (Mo <= 32) return rotate_launch<T, 2, UPPER>(a, lda, Ma, R, ldr, Mo, out, ldo, N, st);
  const dim3 grid((unsigned)((N + kDT - 1) / kDT), UPPER ? 1u : (unsigned)((Mo + kDT - 1) / kDT));
  k_rotate_dmma<T, UPPER, false><<<grid, kDThreads, 0, st>>>((const cplx<T>*)a, lda, Ma, R, ldr, Mo, (cplx<T>*)out, ldo, N);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

template <typename T>
static int orthonormalize_impl(void* psi, long ld, int M, long N, double dV, double2* S, double2* X, int* info,
                               cudaStream_t st) {
  INQB_CUDA_TRY(cudaMemsetAsync(S, 0, sizeof(double2) * (size_t)M * M, st));
  INQB_TRY(overlap_any<T>(psi, ld, M, psi, ld, M, N, dV, S, M, true, st));
  INQB_TRY(cholesky_inverse_launch(S, M, M, X, info, st));
  INQB_TRY((rotate_any<T, true>(psi, ld, M, S, M, M, psi, ld, N, st)));
  INQB_CUDA_TRY(cudaStreamSynchronize(st));
  return INQB_OK;
}

int launch_orthonormalize(int precision, void* psi, long ld, int M, long N, double dV, double2* S, double2* X,
                          int* info, void* stream) {
  return precision == INQB_FP64
             ? orthonormalize_impl<double>(psi, ld, M, N, dV, S, X, info, (cudaStream_t)stream)
             : orthonormalize_impl<float>(psi, ld, M, N, dV, S, X, info, (cudaStream_t)stream);
}

// ---------------------------------------------------------------- orbital-sharded orthonormalisation
// The pieces of operations::orthogonalize over a states communicator: blocks of the
// overlap, the Cholesky factor's inverse of the summed matrix, and blocks of the
// rotation.  The caller moves the blocks between ranks.
template <typename T>
static int overlap_block_impl(const void* a, long lda, int Ma, const void* b, long ldb, int Mb, long N, double dV,
                              double2* S, long lds, cudaStream_t st) {
  INQB_CUDA_TRY(cudaMemset2DAsync(S, sizeof(double2) * lds, 0, sizeof(double2) * Mb, Ma, st));
  return overlap_any<T>(a, lda, Ma, b, ldb, Mb, N, dV, S, lds, false, st);
}

int launch_overlap_block(int precision, const void* a, long lda, int Ma, const void* b, long ldb, int Mb, long N,
                         double dV, double2* S, long lds, void* stream) {
  return precision == INQB_FP64
             ? overlap_block_impl<double>(a, lda, Ma, b, ldb, Mb, N, dV, S, lds, (cudaStream_t)stream)
             : overlap_block_impl<float>(a, lda, Ma, b, ldb, Mb, N, dV, S, lds, (cudaStream_t)stream);
}

int launch_cholesky_inverse(double2* S, int M, long lds, double2* X, int* info, void* stream) {
  return cholesky_inverse_launch(S, M, lds, X, info, (cudaStream_t)stream);
}

int launch_rotate_block(int precision, const void* a, long lda, int Ma, const double2* R, long ldr, int Mo,
                        void* out, long ldo, long N, void* stream) {
  return precision == INQB_FP64
             ? rotate_any<double, false>(a, lda, Ma, R, ldr, Mo, out, ldo, N, (cudaStream_t)stream)
             : rotate_any<float, false>(a, lda, Ma, R, ldr, Mo, out, ldo, N, (cudaStream_t)stream);
}

// out[p][j] = sum_i psi[p][i] conj(u[j][i]) for complex128 orbitals, u M x M
int launch_rotate_adjoint(const void* psi, long ld, int M, const double2* u, void* out, long ldo, long N,
                          void* stream) {
  const dim3 grid((unsigned)((N + kDT - 1) / kDT), (unsigned)((M + kDT - 1) / kDT));
  k_rotate_dmma<double, false, true><<<grid, kDThreads, 0, (cudaStream_t)stream>>>(
      (const cplx<double>*)psi, ld, M, u, M, M, (cplx<double>*)out, ldo, N);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

// ---------------------------------------------------------------- orthonormalisation without allocation
// The same kernels as launch_orthonormalize, with their scratch (overlap S, inverse
// factor X, pivot status) taken from a fixed array in device memory rather than from
// cudaMalloc, for callers that may not allocate device memory.
namespace {
constexpr size_t kNoAllocMat = (size_t)kOrthoNoAllocMaxStates * kOrthoNoAllocMaxStates;
// S (M x M) | X (M x M) | status: 2 MiB plus a little, held by every GPU that loads
// the library until the process exits.  All calls on a device share it.
static __device__ __align__(256) double2 g_orth_scratch[2 * kNoAllocMat + 16];
std::mutex g_orth_scratch_mutex;
double2* g_orth_scratch_ptr[64] = {};
}  // namespace

int orthonormalize_noalloc(int precision, int device, void* psi, long ld, int M, long N, double dV, void* stream) {
  if (M > kOrthoNoAllocMaxStates)
    return fail(INQB_ERR_UNSUPPORTED, "allocation-free orthonormalisation takes at most " +
                                          std::to_string(kOrthoNoAllocMaxStates) + " orbitals, got " +
                                          std::to_string(M));
  if (device < 0 || device >= 64) return fail(INQB_ERR_INVALID, "device index out of range");
  double2* base = nullptr;
  {
    // once per device, with that device current: the device address of the array
    std::lock_guard<std::mutex> lock(g_orth_scratch_mutex);
    if (!g_orth_scratch_ptr[device]) {
      void* p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_orth_scratch);
      if (e != cudaSuccess)
        return fail(INQB_ERR_CUDA, std::string("cudaGetSymbolAddress of the orthonormalisation scratch: ") +
                                       cudaGetErrorString(e));
      g_orth_scratch_ptr[device] = static_cast<double2*>(p);
    }
    base = g_orth_scratch_ptr[device];
  }
  // launch_orthonormalize zeroes S and the status before accumulating into them
  return launch_orthonormalize(precision, psi, ld, M, N, dV, base, base + kNoAllocMat,
                               reinterpret_cast<int*>(base + 2 * kNoAllocMat), stream);
}

}  // namespace inqb
