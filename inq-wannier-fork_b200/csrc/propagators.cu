// Kernels of the Crank-Nicolson step (src/real_time/crank_nicolson.hpp:22-114):
// the per-orbital reductions and the update of solvers::steepest_descent
// (src/solvers/steepest_descent.hpp:22-80) without preconditioner.
//
//   sums     per block and orbital: sum_p (|hsd|^2, conj(r) hsd (re, im), |r|^2)
//   update   lambda_m = cc / qq from those sums, phi += lambda_m r, normres[m] = |cc|
//
// Both run on the device, so a sweep of five steps needs no host round trip.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "dft.cuh"
#include "inqb_internal.h"
#include "propagators.h"

namespace inqb {

// Block: 32 orbitals (lanes) x 8 point lanes; the point lanes' partial sums meet in shared
// memory, those of a cluster's blocks in its first block, which writes one partial per
// orbital and sum, partial[cluster][4][M].  The update adds the partials in order: no
// atomics (a thousand blocks adding to the same 4 M words took 47 us at 40^3 x 24 orbitals),
// and few enough that every update block can add them all.
namespace cg = cooperative_groups;
constexpr int kSdCluster = 8;

template <typename T>
__global__ void __cluster_dims__(kSdCluster) __launch_bounds__(256)
    k_sd_sums(const cplx<T>* __restrict__ r, const cplx<T>* __restrict__ hsd, long ld, int M, long N,
              long pts_per_block, double* __restrict__ partial) {
  __shared__ double red[8][32][5];
  const int tm = threadIdx.x & 31, tp = threadIdx.x >> 5;
  const int m = blockIdx.y * 32 + tm;
  const long p0 = (long)blockIdx.x * pts_per_block, p1 = min(N, p0 + pts_per_block);
  double hh = 0.0, rhr = 0.0, rhi = 0.0, rr = 0.0;
  if (m < M) {
#pragma unroll 8
    for (long p = p0 + tp; p < p1; p += 8) {
      const cplx<T> a = r[p * ld + m], b = hsd[p * ld + m];
      const double ax = a.x, ay = a.y, bx = b.x, by = b.y;
      hh += bx * bx + by * by;
      rhr += ax * bx + ay * by;
      rhi += ax * by - ay * bx;
      rr += ax * ax + ay * ay;
    }
  }
  red[tp][tm][0] = hh;
  red[tp][tm][1] = rhr;
  red[tp][tm][2] = rhi;
  red[tp][tm][3] = rr;
  __syncthreads();
  if (tp < 4) {
    double v = 0.0;
    for (int k = 0; k < 8; k++) v += red[k][tm][tp];
    red[0][tm][tp] = v;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (cluster.block_rank() == 0 && tp < 4 && m < M) {
    double v = 0.0;
    for (int c = 0; c < kSdCluster; c++) v += *cluster.map_shared_rank(&red[0][tm][tp], c);
    partial[((long)(blockIdx.x / kSdCluster) * 4 + tp) * M + m] = v;
  }
  cluster.sync();  // no block leaves while its sums may still be read
}

// The step length of steepest_descent.hpp:48-58 in complex FP64: ca = <hsd|hsd>,
// cb = 4 Re <r|hsd>, cc = <r|r> (all times dV); qq = -(cb + sign sqrt(cb^2 - 4 ca cc)) / 2
// with the sign of Re(conj(cb) (cb^2 - 4 ca cc)); lambda = cc / qq.
__device__ __forceinline__ double2 sd_lambda(const double* a, double dV, double* normres) {
  const double ca = dV * a[0];
  const double cb = 4.0 * dV * a[1];
  const double cc = dV * a[3];
  *normres = fabs(cc);
  // ca and cc are exact norms, so in the reference's complex arithmetic the
  // discriminant cb^2 - 4 ca cc is real with imaginary part -0 (a real minus a
  // complex with +0 imaginary part); its principal square root is sqrt(disc) or,
  // below zero, -i sqrt(-disc) (C99 csqrt takes the sign of the imaginary zero)
  const double disc = cb * cb - 4.0 * ca * cc;
  const double signb = (cb * disc >= 0.0) ? 1.0 : -1.0;
  double qr, qi;
  if (disc >= 0.0) {
    qr = -0.5 * (cb + signb * sqrt(disc));
    qi = 0.0;
  } else {
    qr = -0.5 * cb;
    qi = 0.5 * signb * sqrt(-disc);
  }
  const double den = qr * qr + qi * qi;
  return make_double2(cc * qr / den, -cc * qi / den);
}

// Block: 32 orbitals (lanes) x 8 point lanes, as the sums.  The block first adds the sums'
// partials of its orbitals (point lane t the partials t, t + 8, ..., then the lanes in
// order), and forms each step length (a square root and divisions in FP64) once.
template <typename T>
__global__ void __launch_bounds__(256)
    k_sd_update(cplx<T>* __restrict__ phi, long ldp, const cplx<T>* __restrict__ r, long ldr, int M, long N,
                long pts_per_block, const double* __restrict__ partial, int npart, double dV,
                double* __restrict__ normres) {
  __shared__ double red[8][32][5];
  __shared__ double2 step[32];
  const int tm = threadIdx.x & 31, tp = threadIdx.x >> 5;
  const int m = blockIdx.y * 32 + tm;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  if (m < M) {
#pragma unroll 4
    for (int b = tp; b < npart; b += 8)
#pragma unroll
      for (int k = 0; k < 4; k++) s[k] += partial[((long)b * 4 + k) * M + m];
  }
#pragma unroll
  for (int k = 0; k < 4; k++) red[tp][tm][k] = s[k];
  __syncthreads();
  if (tp == 0 && m < M) {
    for (int b = 1; b < 8; b++)
#pragma unroll
      for (int k = 0; k < 4; k++) s[k] += red[b][tm][k];
    double nr;
    step[tm] = sd_lambda(s, dV, &nr);
    if (blockIdx.x == 0) normres[m] = nr;
  }
  __syncthreads();
  if (m >= M) return;
  const double2 lam = step[tm];
  const long p0 = (long)blockIdx.x * pts_per_block, p1 = min(N, p0 + pts_per_block);
#pragma unroll 4
  for (long p = p0 + tp; p < p1; p += 8) {
    const cplx<T> rv = r[p * ldr + m];
    cplx<T>& d = phi[p * ldp + m];
    d.x = (T)((double)d.x + lam.x * rv.x - lam.y * rv.y);
    d.y = (T)((double)d.y + lam.x * rv.y + lam.y * rv.x);
  }
}

// Blocks of the sums over the points: about two per SM, whole clusters.
static long sd_blocks(long N, int M) {
  const int ym = (M + 31) / 32;
  const long want = std::max<long>(1, std::min<long>(N / 64, 148L * 2 / ym));
  return (want + kSdCluster - 1) / kSdCluster * kSdCluster;
}

template <typename T>
static int sd_sums_impl(const void* r, const void* hsd, long ld, int M, long N, double* partial, cudaStream_t st) {
  const int ym = (M + 31) / 32;
  const long nblk = sd_blocks(N, M), per = (N + nblk - 1) / nblk;
  k_sd_sums<T><<<dim3((unsigned)nblk, ym), 256, 0, st>>>((const cplx<T>*)r, (const cplx<T>*)hsd, ld, M, N, per, partial);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

int launch_sd_sums(int precision, const void* r, const void* hsd, long ld, int M, long N, double* partial,
                   void* stream) {
  return precision == INQB_FP64 ? sd_sums_impl<double>(r, hsd, ld, M, N, partial, (cudaStream_t)stream)
                                : sd_sums_impl<float>(r, hsd, ld, M, N, partial, (cudaStream_t)stream);
}

template <typename T>
static int sd_update_impl(void* phi, long ldp, const void* r, long ldr, int M, long N, const double* partial, double dV,
                          double* normres, cudaStream_t st) {
  const int ym = (M + 31) / 32;
  const long nblk = std::max<long>(1, std::min<long>(N / 64, 148L * 4 / ym)), per = (N + nblk - 1) / nblk;
  k_sd_update<T><<<dim3((unsigned)((N + per - 1) / per), ym), 256, 0, st>>>(
      (cplx<T>*)phi, ldp, (const cplx<T>*)r, ldr, M, N, per, partial, (int)(sd_blocks(N, M) / kSdCluster), dV, normres);
  INQB_CUDA_TRY(cudaGetLastError());
  return INQB_OK;
}

int launch_sd_update(int precision, void* phi, long ldp, const void* r, long ldr, int M, long N, const double* partial,
                     double dV, double* normres, void* stream) {
  return precision == INQB_FP64
             ? sd_update_impl<double>(phi, ldp, r, ldr, M, N, partial, dV, normres, (cudaStream_t)stream)
             : sd_update_impl<float>(phi, ldp, r, ldr, M, N, partial, dV, normres, (cudaStream_t)stream);
}

size_t sd_partial_doubles(int M) { return (size_t)(148 * 2 / kSdCluster + 1) * 4 * M; }

}  // namespace inqb
