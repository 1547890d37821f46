// Dense FP64 tiles on the FP64 tensor instruction: the overlap, rotation and Gram kernels.
#pragma once
#include "dft.cuh"

namespace inqb {

// The FP64 tensor instruction D = A B + C on 8 x 4 x 8 (FP64 has no tcgen05 kind): lane l
// holds A[l / 4][l % 4], B[l % 4][l / 4] and C[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double2& c, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c.x), "+d"(c.y)
      : "d"(a), "d"(b));
}

constexpr int kDT = 64, kDK = 8, kDS = kDT + 2, kDThreads = 128;
using DmmaBuf = double2[kDK][kDS];

// One operand of a chunk: kDK rows of kDT columns in shared memory as complex128.  The eight
// lanes of a quarter warp read 4 rows x 2 neighbours, and kDS % 8 = 2 puts these into eight
// different 16-byte banks.  complex128 sources are copied asynchronously (zeros outside the
// matrix), complex64 ones wait in registers while the chunk before is multiplied.
// TR: the source runs along the rows, so eight lanes take 4 rows of 2 columns and the
// transposing store meets eight banks.
template <typename T, bool TR>
struct DmmaOperand {
  static constexpr int PER = kDT * kDK / kDThreads;
  cplx<T> v[sizeof(T) == 8 ? 1 : PER];
  __device__ static __forceinline__ int row(int u) {
    const int e = threadIdx.x + kDThreads * u;
    return TR ? e % 4 + e / (4 * kDT) * 4 : e / kDT;
  }
  __device__ static __forceinline__ int col(int u) {
    const int e = threadIdx.x + kDThreads * u;
    return TR ? e / 4 % kDT : e % kDT;
  }
  // offset(row, col) of an element from src, negative outside the matrix
  template <typename F>
  __device__ __forceinline__ void load(DmmaBuf& dst, const cplx<T>* src, F offset) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const long o = offset(row(u), col(u));
      if constexpr (sizeof(T) == 8) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(&dst[row(u)][col(u)]);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src + (o < 0 ? 0 : o)),
                     "r"(o < 0 ? 0 : 16)
                     : "memory");
      } else {
        v[u] = o < 0 ? mk<T>(0, 0) : src[o];
      }
    }
  }
  __device__ __forceinline__ void store(DmmaBuf& dst) const {
    if constexpr (sizeof(T) != 8) {
#pragma unroll
      for (int u = 0; u < PER; ++u) dst[row(u)][col(u)] = make_double2(v[u].x, v[u].y);
    }
  }
};
__device__ __forceinline__ void dmma_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void dmma_arrived() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Four warps hold a 64 x 64 tile of complex outputs in registers, warp w the 8-high row
// blocks w and 7 - w over all eight 8-wide column blocks: on a diagonal tile, where only
// the column blocks from the row block on are wanted, every warp then has nine.
enum DmmaConj { kConjNone, kConjX, kConjY };
struct DmmaTile {
  double2 re[2][8], im[2][8];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int c = 0; c < 8; ++c) re[a][c] = im[a][c] = make_double2(0.0, 0.0);
  }
  __device__ static __forceinline__ int row_block(int a) { return a == 0 ? threadIdx.x / 32 : 7 - threadIdx.x / 32; }
  // += sum_k x[k][row] y[k][col], x or y conjugated and weight(x, k) in place of x, of the
  // column blocks [LO0, hi) of the first row block and [LO1, hi) of the second.  The first
  // column blocks are compile-time: a conditional product compiles to a predicated
  // instruction, and the FP64 pipe is as long busy with it where the predicate is off (87%
  // busy for 62% of wanted products).  ALL: hi is 8, and the loads of y run ahead of the
  // products; else a tile that is mostly padding loads little.
  template <DmmaConj C, int LO0, int LO1, bool ALL, typename W>
  __device__ __forceinline__ void mul(const DmmaBuf& x, const DmmaBuf& y, int hi, W weight) {
    constexpr int LO = LO0 < LO1 ? LO0 : LO1;
    const int lane = threadIdx.x & 31, k = lane & 3, n = lane >> 2;
#pragma unroll
    for (int q = 0; q < kDK; q += 4) {
      double2 u[2], v[8];
#pragma unroll
      for (int a = 0; a < 2; ++a)
        if ((a == 0 ? LO0 : LO1) < 8) u[a] = weight(x[q + k][8 * row_block(a) + n], q + k);
      if (ALL)
#pragma unroll
        for (int c = LO; c < 8; ++c) v[c] = y[q + k][8 * c + n];
#pragma unroll
      for (int c = LO; c < 8; ++c) {
        if (!ALL && c >= hi) break;
        if (!ALL) v[c] = y[q + k][8 * c + n];
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
          for (int a = 0; a < 2; ++a)
            if (c >= (a == 0 ? LO0 : LO1)) {
              if (half == 0) {
                dmma(re[a][c], u[a].x, v[c].x);
                dmma(im[a][c], C == kConjY ? -u[a].x : u[a].x, v[c].y);
              } else {
                dmma(re[a][c], C == kConjNone ? -u[a].y : u[a].y, v[c].y);
                dmma(im[a][c], C == kConjX ? -u[a].y : u[a].y, v[c].x);
              }
            }
      }
    }
  }
  template <DmmaConj C, int LO, typename W>
  __device__ __forceinline__ void mul_from(const DmmaBuf& x, const DmmaBuf& y, int hi, W weight) {
    if (hi == 8)
      mul<C, LO, LO, true>(x, y, hi, weight);
    else
      mul<C, LO, LO, false>(x, y, hi, weight);
  }
  // the first `rows` row blocks and first `hi` column blocks
  template <DmmaConj C, typename W>
  __device__ __forceinline__ void mul_block(const DmmaBuf& x, const DmmaBuf& y, int rows, int hi, W weight) {
    if (row_block(1) < rows)
      mul_from<C, 0>(x, y, hi, weight);
    else if (row_block(0) < rows)
      mul<C, 0, 8, false>(x, y, hi, weight);
  }
  // on and above the diagonal, the first hi of both
  template <DmmaConj C, typename W>
  __device__ __forceinline__ void mul_upper(const DmmaBuf& x, const DmmaBuf& y, int hi, W weight) {
    switch (threadIdx.x / 32 + (hi < 8 ? 4 : 0)) {
      case 0: return mul<C, 0, 7, true>(x, y, hi, weight);
      case 1: return mul<C, 1, 6, true>(x, y, hi, weight);
      case 2: return mul<C, 2, 5, true>(x, y, hi, weight);
      case 3: return mul<C, 3, 4, true>(x, y, hi, weight);
      case 4: return mul<C, 0, 7, false>(x, y, hi, weight);
      case 5: return mul<C, 1, 6, false>(x, y, hi, weight);
      case 6: return mul<C, 2, 5, false>(x, y, hi, weight);
      default: return mul<C, 3, 4, false>(x, y, hi, weight);
    }
  }
  // all rows, column blocks [lo, hi)
  template <DmmaConj C, typename W>
  __device__ __forceinline__ void mul_right(const DmmaBuf& x, const DmmaBuf& y, int lo, int hi, W weight) {
    switch (lo) {
      case 0: return mul_from<C, 0>(x, y, hi, weight);
      case 1: return mul_from<C, 1>(x, y, hi, weight);
      case 2: return mul_from<C, 2>(x, y, hi, weight);
      case 3: return mul_from<C, 3>(x, y, hi, weight);
      case 4: return mul_from<C, 4>(x, y, hi, weight);
      case 5: return mul_from<C, 5>(x, y, hi, weight);
      case 6: return mul_from<C, 6>(x, y, hi, weight);
      default: return mul_from<C, 7>(x, y, hi, weight);
    }
  }
};
struct DmmaNoWeight {
  __device__ __forceinline__ double2 operator()(double2 u, int) const { return u; }
};

}  // namespace inqb
