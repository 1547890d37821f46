// Complex arithmetic and fully unrolled in-register DFTs for the plane/line FFT
// kernels.  Forward transforms use exp(-2 pi i / R) (FFTW sign -1, the sign of
// INQ's to_fourier); inverse transforms use exp(+2 pi i / R) and are unscaled.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>
#include <utility>

#include "twiddles.cuh"

namespace inqb {

template <typename T>
struct alignas(2 * sizeof(T)) cplx {
  T x, y;
};

template <typename T>
__host__ __device__ __forceinline__ cplx<T> mk(T a, T b) {
  return cplx<T>{a, b};
}
template <typename T>
__device__ __forceinline__ cplx<T> operator+(cplx<T> a, cplx<T> b) {
  return {a.x + b.x, a.y + b.y};
}
template <typename T>
__device__ __forceinline__ cplx<T> operator-(cplx<T> a, cplx<T> b) {
  return {a.x - b.x, a.y - b.y};
}
template <typename T>
__device__ __forceinline__ cplx<T> operator*(cplx<T> a, cplx<T> b) {
  return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
template <typename T>
__device__ __forceinline__ cplx<T> operator*(T s, cplx<T> a) {
  return {s * a.x, s * a.y};
}
template <typename T>
__device__ __forceinline__ cplx<T> conj(cplx<T> a) {
  return {a.x, -a.y};
}
// acc += a * b
template <typename T>
__device__ __forceinline__ void fma_acc(cplx<T>& acc, cplx<T> a, cplx<T> b) {
  acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}

// ---------------------------------------------------------------- lanes
// The transforms work on lanes, usually of 16 bytes: one complex128 value (cplx<double>), or
// the complex64 values of two neighbouring orbitals as (re, re | im, im) in two packed FP32
// pairs (cplx<F2>); long FP32 axes use one complex64 (cplx<float>, TileGeom in tiles.cuh).
// Every operation of the transforms is the same for the orbitals of a lane, so
// a packed f32x2 instruction (sm_100: add, sub, mul, fma; each half rounded to nearest
// like the scalar form) does the work of two, and shared memory, HBM and the index
// arithmetic see one 16-byte access per lane in both precisions.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2_get(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }

// the value c in every part of a lane component
template <typename P>
__device__ __forceinline__ P splat(double c);
template <>
__device__ __forceinline__ double splat<double>(double c) { return c; }
template <>
__device__ __forceinline__ F2 splat<F2>(double c) { return f2((float)c, (float)c); }
template <>
__device__ __forceinline__ float splat<float>(double c) { return (float)c; }
// the same of a value in the tile precision
template <typename P, typename T>
__device__ __forceinline__ P splat_of(T c) { return c; }
template <>
__device__ __forceinline__ F2 splat_of<F2, float>(float c) { return f2(c, c); }
template <typename P>
__device__ __forceinline__ P vneg(P a) { return splat<P>(-1.0) * a; }
template <>
__device__ __forceinline__ double vneg<double>(double a) { return -a; }
template <>
__device__ __forceinline__ float vneg<float>(float a) { return -a; }

template <typename T>
struct LaneOf;
template <>
struct LaneOf<float> { using P = F2; };
template <>
struct LaneOf<double> { using P = double; };
template <typename T>
using LaneP = typename LaneOf<T>::P;
template <typename T>
using Lane = cplx<LaneP<T>>;

// Between the orbital layout (re, im of each orbital) and the lane layout: in FP32 the
// middle two words of the 16 bytes change places (its own inverse), in FP64 nothing does.
__device__ __forceinline__ cplx<F2> flip(cplx<F2> a) {
  const float2 p = f2_get(a.x), q = f2_get(a.y);
  return {f2(p.x, q.x), f2(p.y, q.y)};
}
__device__ __forceinline__ cplx<double> flip(cplx<double> a) { return a; }
__device__ __forceinline__ cplx<float> flip(cplx<float> a) { return a; }
// value of orbital k of a lane
__device__ __forceinline__ cplx<float> lane_get(cplx<F2> a, int k) {
  const float2 p = f2_get(a.x), q = f2_get(a.y);
  return k ? mk<float>(p.y, q.y) : mk<float>(p.x, q.x);
}
__device__ __forceinline__ cplx<double> lane_get(cplx<double> a, int) { return a; }
__device__ __forceinline__ cplx<float> lane_get(cplx<float> a, int) { return a; }
template <typename P, typename T>
__device__ __forceinline__ cplx<P> lane_splat(cplx<T> a) { return {splat_of<P>(a.x), splat_of<P>(a.y)}; }
__device__ __forceinline__ cplx<F2> lane_shfl_xor(cplx<F2> a, int o) {
  return {F2{__shfl_xor_sync(0xffffffffu, a.x.v, o)}, F2{__shfl_xor_sync(0xffffffffu, a.y.v, o)}};
}
template <typename P>
__device__ __forceinline__ cplx<P> lane_shfl_xor(cplx<P> a, int o) {
  return {__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o)};
}

// a b and a conj(b) of lanes (b: a twiddle, the same value for both orbitals)
template <typename P>
__device__ __forceinline__ cplx<P> lmul(cplx<P> a, cplx<P> b) {
  return {vfma(a.x, b.x, a.y * vneg(b.y)), vfma(a.x, b.y, a.y * b.x)};
}
template <typename P>
__device__ __forceinline__ cplx<P> lmul_conj(cplx<P> a, cplx<P> b) {
  return {vfma(a.x, b.x, a.y * b.y), vfma(a.y, b.x, a.x * vneg(b.y))};
}
// a + i b, a - i b
template <typename P>
__device__ __forceinline__ cplx<P> add_i(cplx<P> a, cplx<P> b) {
  return {a.x - b.y, a.y + b.x};
}
template <typename P>
__device__ __forceinline__ cplx<P> sub_i(cplx<P> a, cplx<P> b) {
  return {a.x + b.y, a.y - b.x};
}

// Compile-time loop: f(std::integral_constant<int, I>{}) for I in [0, N).
template <typename F, int... Is>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, Is...>) {
  (f(std::integral_constant<int, Is>{}), ...);
}
template <int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  static_for_impl(f, std::make_integer_sequence<int, N>{});
}

// a * exp(-+ 2 pi i K / R) with K, R compile time (forward: minus sign).
template <int R, int K, bool INV, typename P>
__device__ __forceinline__ cplx<P> rot(cplx<P> a) {
  constexpr int k = K % R;
  if constexpr (k == 0) {
    return a;
  } else if constexpr (2 * k == R) {
    return {vneg(a.x), vneg(a.y)};
  } else if constexpr (4 * k == R || 4 * k == 3 * R) {
    if constexpr (INV == (4 * k == R)) return {vneg(a.y), a.x};
    return {a.y, vneg(a.x)};
  } else {
    const P c = splat<P>(RootsOfUnity<R>::re[k]);
    constexpr double sd = INV ? RootsOfUnity<R>::im[k] : -RootsOfUnity<R>::im[k];
    const P s = splat<P>(sd), ns = splat<P>(-sd);
    return {vfma(a.x, c, a.y * ns), vfma(a.x, s, a.y * c)};
  }
}

constexpr int first_factor(int r) {
  return (r % 4 == 0 && r != 8) ? 4 : (r % 2 == 0) ? 2 : (r % 3 == 0) ? 3 : (r % 5 == 0) ? 5 : r;
}

// In-place DFT of R lanes held in registers, natural order in and out.
template <int R, bool INV, typename P>
struct DFT {
  static_assert(first_factor(R) != R, "prime radix without a specialisation");
  static constexpr int A = first_factor(R);
  static constexpr int B = R / A;
  __device__ __forceinline__ static void run(cplx<P>* v) {
    // n = b + B a ; k = k1 + A k2 (four-step inside the registers)
    cplx<P> y[R];
    static_for<B>([&](auto bI) {
      constexpr int b = decltype(bI)::value;
      cplx<P> u[A];
#pragma unroll
      for (int a = 0; a < A; ++a) u[a] = v[b + B * a];
      DFT<A, INV, P>::run(u);
      static_for<A>([&](auto kI) {
        constexpr int k1 = decltype(kI)::value;
        y[b * A + k1] = rot<R, b * k1, INV>(u[k1]);
      });
    });
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      cplx<P> w[B];
#pragma unroll
      for (int b = 0; b < B; ++b) w[b] = y[b * A + k1];
      DFT<B, INV, P>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = w[k2];
    }
  }
};

template <bool INV, typename P>
struct DFT<1, INV, P> {
  __device__ __forceinline__ static void run(cplx<P>*) {}
};

template <bool INV, typename P>
struct DFT<2, INV, P> {
  __device__ __forceinline__ static void run(cplx<P>* v) {
    cplx<P> a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
  }
};

template <bool INV, typename P>
struct DFT<3, INV, P> {
  __device__ __forceinline__ static void run(cplx<P>* v) {
    constexpr double sd = INV ? 0.8660254037844386 : -0.8660254037844386;  // sin(+-2 pi / 3)
    const P c = splat<P>(-0.5), s = splat<P>(sd), ns = splat<P>(-sd);
    cplx<P> a = v[1] + v[2], d = v[1] - v[2];
    cplx<P> m = {vfma(c, a.x, v[0].x), vfma(c, a.y, v[0].y)};
    v[0] = v[0] + a;
    v[1] = {vfma(ns, d.y, m.x), vfma(s, d.x, m.y)};  // m + i s d
    v[2] = {vfma(s, d.y, m.x), vfma(ns, d.x, m.y)};
  }
};

template <bool INV, typename P>
struct DFT<4, INV, P> {
  __device__ __forceinline__ static void run(cplx<P>* v) {
    cplx<P> t0 = v[0] + v[2], t1 = v[0] - v[2], t2 = v[1] + v[3], t3 = v[1] - v[3];
    v[0] = t0 + t2;
    v[2] = t0 - t2;
    v[1] = INV ? add_i(t1, t3) : sub_i(t1, t3);
    v[3] = INV ? sub_i(t1, t3) : add_i(t1, t3);
  }
};

template <bool INV, typename P>
struct DFT<5, INV, P> {
  __device__ __forceinline__ static void run(cplx<P>* v) {
    const P c1 = splat<P>(0.30901699437494745);   // cos(2 pi / 5)
    const P c2 = splat<P>(-0.80901699437494734);  // cos(4 pi / 5)
    constexpr double s1d = INV ? 0.95105651629515353 : -0.95105651629515353;
    constexpr double s2d = INV ? 0.58778525229247314 : -0.58778525229247314;
    const P s1 = splat<P>(s1d), s2 = splat<P>(s2d), ns1 = splat<P>(-s1d);
    cplx<P> a1 = v[1] + v[4], b1 = v[1] - v[4], a2 = v[2] + v[3], b2 = v[2] - v[3];
    cplx<P> m1 = {vfma(c2, a2.x, vfma(c1, a1.x, v[0].x)), vfma(c2, a2.y, vfma(c1, a1.y, v[0].y))};
    cplx<P> m2 = {vfma(c1, a2.x, vfma(c2, a1.x, v[0].x)), vfma(c1, a2.y, vfma(c2, a1.y, v[0].y))};
    const cplx<P> n1 = {vfma(s2, b2.x, s1 * b1.x), vfma(s2, b2.y, s1 * b1.y)};
    const cplx<P> n2 = {vfma(ns1, b2.x, s2 * b1.x), vfma(ns1, b2.y, s2 * b1.y)};
    v[0] = v[0] + a1 + a2;
    v[1] = add_i(m1, n1);
    v[4] = sub_i(m1, n1);
    v[2] = add_i(m2, n2);
    v[3] = sub_i(m2, n2);
  }
};

// DFT_8 written out as the split 8 = 2 x 4 (the generic form above with the same
// factors): a_n = v_n + v_{n+4} gives the even outputs as a DFT_4, b_n = v_n - v_{n+4}
// twiddled by w^n the odd ones, w = exp(-+ 2 pi i / 8).  The products with +-i are
// exchanges of components inside the sums, and the two products with sqrt(1/2) ride in
// the last sums as fused multiply-adds: 52 instructions per lane transform.
template <bool INV, typename P>
struct DFT<8, INV, P> {
  __device__ __forceinline__ static void run(cplx<P>* v) {
    const P h = splat<P>(0.70710678118654752), nh = splat<P>(-0.70710678118654752);  // 1/sqrt(2)
    cplx<P> a[4], b[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      a[n] = v[n] + v[n + 4];
      b[n] = v[n] - v[n + 4];
    }
    // even outputs: DFT_4 of a
    DFT<4, INV, P>::run(a);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[2 * k] = a[k];
    // odd outputs: DFT_4 of c_n = b_n w^n.  e = c0 + c2, f = c0 - c2 (c2 = +-i b2);
    // c1 = h p1, c3 = h p3 with p1 = b1 (1 +- i), p3 = b3 (-1 +- i): s = p1 + p3, d = p1 - p3
    const cplx<P> e = INV ? add_i(b[0], b[2]) : sub_i(b[0], b[2]);
    const cplx<P> f = INV ? sub_i(b[0], b[2]) : add_i(b[0], b[2]);
    const P m1 = b[1].x - b[1].y, q1 = b[1].x + b[1].y;
    const P m3 = b[3].x - b[3].y, q3 = b[3].x + b[3].y;
    cplx<P> s, d;
    if (INV) {
      s = {m1 - q3, q1 + m3};
      d = {m1 + q3, q1 - m3};
    } else {  // p1 = (q1, -m1), p3 = (-m3, -q3); s and d negated in y, folded below
      s = {q1 - m3, m1 + q3};
      d = {q1 + m3, m1 - q3};
    }
    const P hy = INV ? h : nh, nhy = INV ? nh : h;
    v[1] = {vfma(h, s.x, e.x), vfma(hy, s.y, e.y)};
    v[5] = {vfma(nh, s.x, e.x), vfma(nhy, s.y, e.y)};
    // X3 = f +- i h d, X7 = f -+ i h d (upper signs inverse)
    if (INV) {
      v[3] = {vfma(nh, d.y, f.x), vfma(h, d.x, f.y)};
      v[7] = {vfma(h, d.y, f.x), vfma(nh, d.x, f.y)};
    } else {  // d.y is negated: -i h (d.x - i d.y) = (-h d.y, -h d.x)
      v[3] = {vfma(nh, d.y, f.x), vfma(nh, d.x, f.y)};
      v[7] = {vfma(h, d.y, f.x), vfma(h, d.x, f.y)};
    }
  }
};

}  // namespace inqb
