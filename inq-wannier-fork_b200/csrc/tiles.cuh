// Six-step tiles of H|psi> (src/hamiltonian/ks_hamiltonian.hpp:132-152).
//
// The y axis is split NY = Y2 * Y1 (the four-step split of the size table):
// y = y1 + Y1 * y2 and ky = ka + Y2 * kb.  Then
//   X[ka + Y2 kb] = sum_y1 w_Y1^{y1 kb} [ w_NY^{y1 ka} sum_y2 w_Y2^{y2 ka} x[y1 + Y1 y2] ]
// so a tile (x-plane ix, row class y1) of Y2 rows x NZ points finishes the z
// transform and the inner y stage on its own, and the outer y stage lands in
// the x-line pass.  Every tile moves whole 64-byte runs of G orbitals per grid
// point (G = 8 complex64 or 4 complex128; 32-byte runs for the long rows of
// 144^3), so the orbital-fastest layout [point][orbital] is read and written in
// full sectors.
//
//   pass A  k_tile_fwd  CTA (group, ix, share of the y1 classes), loops over y1: psi
//           rows -> KB projection (plane accumulators in shared memory, flushed
//           once per CTA) ->
//           z FFT -> inner y stage -> tmp[g][ka][kz][ix][y1][G]
//   pass B  k_tile_x    CTA (ka, kz, group): contiguous [ix][y1][G] block ->
//           outer y stage -> x FFT -> 1/2 |G + k + A|^2 / N -> inverse x ->
//           inverse outer y stage, in place
//   pass C  k_tile_inv  CTA (group, ix, y1): inverse inner y stage -> inverse z
//           -> nonlocal scatter -> alpha (K + V + V_nl) psi + beta base - minus
#pragma once

#include "fft_tile.cuh"

namespace inqb {

// ---------------------------------------------------------------- cp.async
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(PENDING) : "memory");
}

// The three passes of an apply are launched with programmatic dependence: a pass may be
// scheduled while the one before it drains, fills its tables (which no pass writes) and
// waits here before it touches anything the passes exchange.  The next pass is let in as
// the CTAs of this one exit; letting it in earlier (launch_dependents) parks its CTAs in
// the slots of running ones and measured slower (64^3 x 128 mixed: 548 -> 595 us).
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Loads of data another CTA of the same launch wrote (the Fourier intermediate, the
// projection partial sums and results): through L2 (ld.global.cg), never a line an
// earlier load left in this SM's L1, so one persistent launch can run the passes.
__device__ __forceinline__ cplx<F2> ld_l2(const cplx<F2>* p) {
  const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(p));
  return {F2{v.x}, F2{v.y}};
}
__device__ __forceinline__ cplx<double> ld_l2(const cplx<double>* p) {
  const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
  return mk<double>(v.x, v.y);
}
__device__ __forceinline__ cplx<float> ld_l2(const cplx<float>* p) {
  const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
  return mk<float>(v.x, v.y);
}
__device__ __forceinline__ double2 ld_l2(const double2* p) { return __ldcg(p); }

// ---------------------------------------------------------------- geometry
template <typename T, int NX, int NY, int NZ>
struct TileGeom {
  using AX = Axis<Split<NX>::N1, Split<NX>::N2>;
  using AY = Axis<Split<NY>::N1, Split<NY>::N2>;
  using AZ = Axis<Split<NZ>::N1, Split<NZ>::N2>;
  static constexpr int Y2 = AY::N1;  // rows per tile
  static constexpr int Y1 = AY::N2;  // tiles per x-plane
  static constexpr int ZS = AZ::SLOTS;  // padded z slots per row
  // orbitals per tile: one 64-byte run per grid point, or in FP32 one 32-byte sector
  // where a 64-byte tile would pass 80 KB (long rows: 144^3), which buys a second CTA
  // per SM (measured: FP32 144^3 apply 75 -> 65 ms; FP64 is faster with 64 bytes)
  static constexpr int RUN = (sizeof(T) == 4 && Y2 * ZS * 64 > 80 * 1024) ? 32 : 64;
  static constexpr int G = RUN / (int)sizeof(cplx<T>);
  // A lane holds 16 bytes, except in FP32 where a transform step is longer than 12 values:
  // 16 lanes of two orbitals take 64 registers, which leaves two CTAs of 256 threads per SM;
  // with one orbital per lane twice the threads fit (144^3 x 64 orbitals, two orbitals ->
  // one: pass A 1964 -> 1777 us, B 1176 -> 1099 us, C 2487 -> 2273 us).
  static constexpr int cmin(int a, int b) { return a < b ? a : b; }
  static constexpr int cmax(int a, int b) { return a > b ? a : b; }
  static constexpr int RZ = cmax(AZ::N1, AZ::N2), RX = cmax(AX::N1, AX::N2);
  static constexpr bool NARROW = sizeof(T) == 4 && cmax(cmax(RZ, RX), cmax(Y1, Y2)) > 12;
  using P = std::conditional_t<NARROW, T, LaneP<T>>;
  using V = cplx<P>;
  static constexpr int PV = (int)(sizeof(V) / sizeof(cplx<T>));  // orbitals per lane
  static constexpr int VP = G / PV;                               // lanes per point
  static constexpr int CH = RUN / 16, LC = 16 / (int)sizeof(V);   // 16-byte copies of a point, lanes of one
  // the sizes below count lanes
  static constexpr int TILE = Y2 * ZS * VP;  // a tile in shared memory
  static constexpr int PTS = Y2 * NZ;        // grid points of a tile
  static constexpr int XS = (Y1 + 1) * VP;   // x-slot stride of the x-line block (one point of padding)
  static constexpr int XBLK = AX::SLOTS * XS;
  static constexpr int BLK = NX * Y1 * VP;   // one tmp block [ix][y1][G]
  static constexpr size_t SMEM_MAX = 227 * 1024;  // dynamic shared memory a CTA may have
  static constexpr size_t smem_fwd(int acc_atoms, int rec_cap) {
    return sizeof(V) * ((size_t)TILE + NY + NZ) + sizeof(double2) * (size_t)acc_atoms * LMAX * G +
           sizeof(EntRec<T>) * (size_t)rec_cap;
  }
  // The second pass copies a block of 32 KB or more to shared memory before its first stage
  // (outer_y_load), the H pass only with at most 8 row classes.
  // Measured (straight -> staged, us): H pass 64^3 x 128 mixed 144 -> 137, FP64 313 -> 259;
  // 72^3 mixed 218 -> 211, 128^3 x 64 821 -> 613, FP64 x 16 330 -> 313; 96^3 even; 144^3
  // (9 classes) 1104 -> 1115, FP64 549 -> 596.  Forward FFT (two passes) 64^3 x 128 232 -> 226,
  // FP64 517 -> 444; 128^3 x 16 418 -> 384, 663 -> 620; 144^3 554 -> 534, 982 -> 925; below
  // 32 KB 48^3 x 64 60 -> 62, 60^3 x 37 127 -> 130, 40^3 x 24 FP64 27 -> 29.
  static constexpr bool FFT_STAGED = sizeof(V) * (size_t)BLK >= 32 * 1024;
  static constexpr bool H_STAGED = FFT_STAGED && Y1 <= 8;
  static constexpr size_t SMEM_X = sizeof(V) * ((size_t)XBLK + NX) + sizeof(T) * 2 * Y1;
  static constexpr size_t TILE_BYTES = sizeof(V) * (size_t)TILE;
  // CTAs of 256 threads per SM that a pass asks the compiler for: four where the radices
  // fit 64 registers a thread (up to 8 lanes of a transform), three (80 registers) up to
  // 12, two (128) beyond, and no more than the tiles in shared memory allow
  static constexpr int radix_ctas(int r) { return r * (int)sizeof(V) <= 128 ? 4 : r * (int)sizeof(V) <= 192 ? 3 : 2; }
  static constexpr int fit(size_t bytes) { return (int)(SMEM_MAX / (bytes + 1024)); }
  // 512 threads in the z passes where the tile lets one CTA on an SM, or two of narrow lanes
  // (144^3 x 16 orbitals FP64, 256 -> 512 threads: pass A 885 -> 537 us, C 2149 -> 924 us)
  static constexpr int THREADS = 256, ZT = (NARROW || fit(TILE_BYTES) < 2) ? 512 : 256;
  static constexpr int FWD_MIN_CTAS = NARROW ? 2 : cmax(1, cmin(cmin(3, radix_ctas(cmax(RZ, Y2))), fit(TILE_BYTES)));
  static constexpr int X_MIN_CTAS = cmax(1, cmin(radix_ctas(cmax(RX, Y1)), fit(SMEM_X)));
  static constexpr int INV_MIN_CTAS = NARROW ? 2 : cmax(1, cmin(radix_ctas(cmax(RZ, Y2)), fit(TILE_BYTES)));
  // lanes per atom segment of pass C's staged projections [l][orbital]: 64 bytes of
  // padding, so that consecutive segments start in opposite halves of the
  // shared-memory banks
  static constexpr int PT_STRIDE = LMAX * VP + 64 / (int)sizeof(V);
  static constexpr size_t smem_inv(int seg_cap) {
    return sizeof(V) * ((size_t)TILE + NY + NZ + (size_t)seg_cap * PT_STRIDE);
  }
  // Pass A default: the CTAs that share an x-plane.  Each walks its tiles one after the
  // other, so fewer tiles per CTA end the launch more evenly; more CTAs add partial sums of
  // the projection.  Measured (mixed; CTAs per plane: us of the pass): 144^3 1: 2487,
  // 3: 2223, 9: 2104 (two-orbital lanes); 128^3 2: 735, 4: 608, 8: 626; 96^3 2: 315, 4: 275, 8: 280; 60^3 1: 118,
  // 5: 95; 40^3 1: 25.8, 5: 18.7; 32^3 2: 14.1, 4: 10.7; 24^3 1: 18.7, 3: 12.3; but 64^3 2: 184,
  // 4: 193, 8: 187 and 72^3 2: 135, 8: 136.
  static constexpr int YSPLIT = (Y1 % 2 == 1 || Y1 <= 4) ? Y1 : Y1 == 6 ? 3 : (TILE_BYTES > 40 * 1024) ? 4 : 2;
  // default threads of the passes: the columns of a pass's stages in as few equal rounds as
  // its register budget suggests (blockDim need not match; idle lanes in the last round of
  // every stage do cost).  Measured (mixed, us): pass B 144^3 256 threads 1302, 160 1111;
  // 96^3 256 242, 192 232; 60^3 256 57, 128 52; 48^3 256 36.8, 192 34.8; pass C 40^3 256 22.7,
  // 160 20.1; 36^3 256 31, 160 28.7.
  static constexpr int round_threads(int cols, int most) {
    const int rounds = (cols + most - 1) / most;
    return cmin(THREADS, cmax(64, ((cols + rounds - 1) / rounds + 31) / 32 * 32));
  }
  static constexpr int X_THREADS =
      round_threads(NX * VP, sizeof(T) == 8 ? 192 : (cmax(RX, Y1) > 8 || NX * VP > 256) ? 192 : 256);
  static constexpr int Z_THREADS = (NZ * VP > 128 && NZ * VP <= 192) ? round_threads(NZ * VP, 192) : ZT;
};

// Entry records staged in shared memory per tile; a tile with more entries
// reads its records from global memory.
constexpr int kRecCapMax = 1024;

// Start the cp.async copy of tile `tile`'s entry records (from `recs`) into R
// (cap records).  Returns the records to index with (e - roff): R when staged,
// else global memory.
template <typename T>
__device__ __forceinline__ const EntRec<T>* stage_entries(const ProjView<T>& pj, const EntRec<T>* recs, int tile,
                                                          int cap, EntRec<T>* R, int& roff) {
  const int e0 = pj.seg_ent[pj.seg_ptr[tile]], e1 = pj.seg_ent[pj.seg_ptr[tile + 1]];
  if (e1 - e0 > cap) {
    roff = 0;
    return recs;
  }
  constexpr int V = (int)(sizeof(EntRec<T>) / 16);
  const float4* src = reinterpret_cast<const float4*>(recs + e0);
  float4* dst = reinterpret_cast<float4*>(R);
  for (int q = threadIdx.x; q < (e1 - e0) * V; q += blockDim.x) cp_async16(dst + q, src + q);
  roff = e0;
  return R;
}

// Plane accumulators held in shared memory by pass A; atoms beyond this many per
// plane accumulate straight into global memory.
constexpr int kAccAtomsMax = 192;
// Atom segments of a tile whose projections pass C stages in shared memory; a tile with
// more reads its projections from global memory.
constexpr int kSegMax = 320;

// ---------------------------------------------------------------- pass A
// The body of one CTA (bx, by) of the pass; k_tile_fwd runs it at (blockIdx.x,
// blockIdx.y), the persistent batch kernel at the coordinates of a work item.
template <typename T, int NX, int NY, int NZ>
__device__ __forceinline__ void tile_fwd_body(int bx, int by, const cplx<T>* __restrict__ in, long ld, int M,
                                              typename TileGeom<T, NX, NY, NZ>::V* __restrict__ tmp, const cplx<T>* __restrict__ tw_y,
                                              const cplx<T>* __restrict__ tw_z, ProjView<T> pj, int acc_cap,
                                              int rec_cap, int ysplit, int vec) {
  using TG = TileGeom<T, NX, NY, NZ>;
  using AZ = typename TG::AZ;
  using V = typename TG::V;
  using P = typename TG::P;
  constexpr int G = TG::G, PV = TG::PV, VP = TG::VP, Y1 = TG::Y1, Y2 = TG::Y2, ZS = TG::ZS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* S = reinterpret_cast<V*>(smem_raw);
  V* twy = S + TG::TILE;
  V* twz = twy + NY;
  double2* acc = reinterpret_cast<double2*>(twz + NZ);  // [acc_cap][LMAX][G]
  EntRec<T>* R = reinterpret_cast<EntRec<T>*>(acc + acc_cap * LMAX * G);  // [rec_cap]

  // ysplit CTAs share plane ix, each taking Y1 / ysplit row classes
  const int YS = ysplit, YPER = Y1 / ysplit;
  const int grp = bx, ix = by / YS, yh = by % YS;
  const int m0 = grp * G;
  const int gcount = min(G, M - m0);
  const bool v16 = vec && gcount == G;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const bool proj_on = pj.nproj > 0;
  for (int i = threadIdx.x; i < NY; i += blockDim.x) twy[i] = lane_splat<P>(tw_y[i]);
  for (int i = threadIdx.x; i < NZ; i += blockDim.x) twz[i] = lane_splat<P>(tw_z[i]);
  if (proj_on)
    for (int i = threadIdx.x; i < acc_cap * LMAX * G; i += blockDim.x) acc[i] = make_double2(0.0, 0.0);
  chain_wait();
  // slots of the plane's atoms beyond the shared-memory accumulators start at zero
  if (proj_on) {
    const int a0 = pj.plane_ptr[ix], na = pj.plane_ptr[ix + 1] - a0;
    for (int i = threadIdx.x; i < max(0, na - acc_cap) * LMAX * G; i += blockDim.x) {
      const int j = i % G, l = (i / G) % LMAX, sl = acc_cap + i / (G * LMAX);
      if (j < gcount) pj.slots[(((long)(a0 + sl) * YS + yh) * LMAX + l) * M + m0 + j] = make_double2(0.0, 0.0);
    }
  }

  // rows y1 + Y1 r of plane ix, G orbitals per point, in the orbital layout, and the tile's
  // entry records: the copies of tile y1
  int roff = 0;
  const EntRec<T>* rec = pj.ent_rec;
  auto load_tile = [&](int y1) {
    if (v16) {
#pragma unroll 1
      for (int q = threadIdx.x; q < TG::PTS * TG::CH; q += blockDim.x) {
        const int c = q % TG::CH * TG::LC, pt = q / TG::CH;
        const int z = pt % NZ, r = pt / NZ;
        const long p = ((long)ix * NY + y1 + Y1 * r) * NZ + z;
        cp_async16(S + (r * ZS + AZ::slot(z)) * VP + c, in + p * ld + m0 + c * PV);
      }
    } else {
      cplx<T>* Sj = reinterpret_cast<cplx<T>*>(S);
      for (int q = threadIdx.x; q < TG::PTS * G; q += blockDim.x) {
        const int j = q % G, pt = q / G;
        const int z = pt % NZ, r = pt / NZ;
        const long p = ((long)ix * NY + y1 + Y1 * r) * NZ + z;
        Sj[(r * ZS + AZ::slot(z)) * G + j] = (j < gcount) ? in[p * ld + m0 + j] : mk<T>(0, 0);
      }
    }
    if (proj_on) rec = stage_entries(pj, pj.ent_rec, ix * Y1 + y1, rec_cap, R, roff);
    cp_async_commit();
  };
  load_tile(yh * YPER);

  for (int y1 = yh * YPER; y1 < (yh + 1) * YPER; ++y1) {
    cp_async_wait<0>();
    __syncthreads();

    // -- KB projection of the tile (projector_all.hpp:104-165).  A group of 4 VP lanes
    // walks one atom segment: lane = (orbital lane v, entry lane e of four).  The four
    // entry lanes' sums meet in two exchange steps that leave entry lane e with
    // projector l = e, which adds it to the plane accumulators.
    if (proj_on) {
      static_assert(LMAX == 4, "an entry lane ends with one projector");
      constexpr int SGRP = 32 / (4 * VP);
      const int v = lane % VP, el = (lane / VP) % 4, sg = lane / (4 * VP);
      const int tile = ix * Y1 + y1;
      const int s0 = pj.seg_ptr[tile], s1 = pj.seg_ptr[tile + 1];
      for (int sb = s0 + warp * SGRP; sb < s1; sb += nw * SGRP) {
        const int s = sb + sg;
        const int e1 = s < s1 ? pj.seg_ent[s + 1] : 0;
        V a[LMAX];
#pragma unroll
        for (int l = 0; l < LMAX; ++l) a[l] = {splat<P>(0.0), splat<P>(0.0)};
        auto add = [&](const EntRec<T>& re) {
          const V u = flip(S[re.off * VP + v]);
          const P pr = splat_of<P>(re.ph[0]), pi = splat_of<P>(re.ph[1]), npi = splat_of<P>(-re.ph[1]);
          const V x = {vfma(u.x, pr, u.y * npi), vfma(u.x, pi, u.y * pr)};
#pragma unroll
          for (int l = 0; l < LMAX; ++l) {
            const P b = splat_of<P>(re.beta[l]);
            a[l].x = vfma(b, x.x, a[l].x);
            a[l].y = vfma(b, x.y, a[l].y);
          }
        };
        int e = s < s1 ? pj.seg_ent[s] + el : 0;
        if constexpr (TG::TILE_BYTES > 40 * 1024) {
          // a tile this large seldom has its records staged: the next one is fetched ahead
          EntRec<T> nx;
          if (e < e1) nx = rec[e - roff];
          for (; e < e1; e += 4) {
            const EntRec<T> re = nx;
            if (e + 4 < e1) nx = rec[e + 4 - roff];
            add(re);
          }
        } else {
#pragma unroll 1
          for (; e < e1; e += 4) add(rec[e - roff]);
        }
        __syncwarp();
        // entry lanes 0, 1 keep l = 0, 1 and 2, 3 keep l = 2, 3; then one each
        const bool hi = (el & 2) != 0, odd = (el & 1) != 0;
        const V b0 = (hi ? a[2] : a[0]) + lane_shfl_xor(hi ? a[0] : a[2], 2 * VP);
        const V b1 = (hi ? a[3] : a[1]) + lane_shfl_xor(hi ? a[1] : a[3], 2 * VP);
        const V c = (odd ? b1 : b0) + lane_shfl_xor(odd ? b0 : b1, VP);
        if (s < s1) {
          const int sl = pj.seg_local[s], l = el;
#pragma unroll
          for (int k = 0; k < PV; ++k) {
            const int j = v * PV + k;
            const cplx<T> w = lane_get(c, k);
            if (j >= gcount) continue;
            if (sl < acc_cap) {
              // one segment per atom in a tile, tiles separated by barriers: no race
              double2& d = acc[(sl * LMAX + l) * G + j];
              d.x += (double)w.x;
              d.y += (double)w.y;
            } else {
              // beyond the shared-memory accumulators: this CTA's own slot in global
              // memory (zeroed at the start), the same ownership
              double2* d = pj.slots + (((long)(pj.plane_ptr[ix] + sl) * YS + yh) * LMAX + l) * M + m0 + j;
              double2 o = ld_l2(d);
              o.x += (double)w.x;
              o.y += (double)w.y;
              *d = o;
            }
          }
        }
      }
      __syncthreads();
    }

    // -- z lines: (r, v), element stride VP; the first step leaves the lane layout
    step1<AZ, false, true>(S, Y2 * VP * AZ::N2, twz, [](int it, int& base, int& es, int& j2) {
      const int v = it % VP, rest = it / VP;
      j2 = rest % AZ::N2;
      base = (rest / AZ::N2) * ZS * VP + v;
      es = VP;
    });
    __syncthreads();
    step2<AZ, false>(S, Y2 * VP * AZ::N1, [](int it, int& base, int& es, int& k1) {
      const int v = it % VP, rest = it / VP;
      k1 = rest % AZ::N1;
      base = (rest / AZ::N1) * ZS * VP + v;
      es = VP;
    });
    __syncthreads();

    // -- inner y stage: DFT_Y2 over the rows, twiddle w_NY^{y1 ka}, written straight
    // to tmp[g][ka][kz][ix][y1][G] (lanes along v write whole 64-byte runs).  (Starting the
    // next tile's copies once the columns are in registers, before they are transformed and
    // stored, spilled and measured slower: 64^3 x 128 mixed 178 -> 193 us.)
    for (int it0 = 0; it0 < NZ * VP; it0 += blockDim.x) {
      const int it = it0 + threadIdx.x;
      if (it >= NZ * VP) continue;
      const int v = it % VP, kz = it / VP;
      const int base = AZ::slot_of_freq(kz) * VP + v;
      V u[Y2];
#pragma unroll
      for (int r = 0; r < Y2; ++r) u[r] = S[base + r * ZS * VP];
      DFT<Y2, false, P>::run(u);
#pragma unroll
      for (int ka = 1; ka < Y2; ++ka) u[ka] = lmul(u[ka], twy[ka * Y1 + y1]);
      V* dst = tmp + (((long)grp * Y2 * NZ + kz) * NX + ix) * (Y1 * VP) + y1 * VP + v;
#pragma unroll
      for (int ka = 0; ka < Y2; ++ka) dst[(long)ka * NZ * TG::BLK] = u[ka];
    }
    __syncthreads();
    if (y1 + 1 < (yh + 1) * YPER) load_tile(y1 + 1);
  }

  // -- flush the plane accumulators into this CTA's slots, which the second pass adds per
  // atom in a fixed order
  if (proj_on) {
    const int a0 = pj.plane_ptr[ix];
    const int na = min(pj.plane_ptr[ix + 1] - a0, acc_cap);
    for (int i = threadIdx.x; i < na * LMAX * G; i += blockDim.x) {
      const int j = i % G, l = (i / G) % LMAX, sl = i / (G * LMAX);
      if (j >= gcount) continue;
      pj.slots[(((long)(a0 + sl) * YS + yh) * LMAX + l) * M + m0 + j] = acc[i];
    }
  }
}

template <typename T, int NX, int NY, int NZ>
__global__ void __launch_bounds__(TileGeom<T, NX, NY, NZ>::ZT, TileGeom<T, NX, NY, NZ>::FWD_MIN_CTAS)
    k_tile_fwd(const cplx<T>* __restrict__ in, long ld, int M, typename TileGeom<T, NX, NY, NZ>::V* __restrict__ tmp,
               const cplx<T>* __restrict__ tw_y, const cplx<T>* __restrict__ tw_z, ProjView<T> pj, int acc_cap,
               int rec_cap, int ysplit, int vec) {
  tile_fwd_body<T, NX, NY, NZ>(blockIdx.x, blockIdx.y, in, ld, M, tmp, tw_y, tw_z, pj, acc_cap, rec_cap, ysplit,
                               vec);
}

// ---------------------------------------------------------------- projection finish
// proj[a][l][m] = dV ekb[a][l] sum over the atom's (plane, CTA of the plane) slots: pass A
// wrote one partial per slot, no atomics.  Eight lanes (kFinParts) share an item
// i = (a * L + l) * M + m: part k adds the slots k, k + 8, ... in order and the parts meet
// by shuffles, so the sum has one fixed order and a chain of only slots / 8 loads (one
// thread per item: 24^3, 57 slots an atom, pass B 12 -> 19 us).  Lanes of a warp: four
// items next to each other in m, eight parts; every lane of the warp calls it.
constexpr int kFinParts = 8;
template <typename T>
__device__ __forceinline__ void proj_finish_item(const ProjView<T>& pj, int M, int ysplit, unsigned i, bool on) {
  const int part = (threadIdx.x & 31) / (32 / kFinParts);
  const unsigned al = i / M;
  const int m = (int)(i - al * M), a = on ? (int)(al / pj.L) : 0, l = (int)(al % pj.L);
  const int q0 = pj.aslot_ptr[a] * ysplit, q1 = on ? pj.aslot_ptr[a + 1] * ysplit : 0;
  double sx = 0.0, sy = 0.0;
  for (int qb = q0 + part; qb < q1; qb += 4 * kFinParts) {
    double2 v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int q = qb + u * kFinParts;
      v[u] = make_double2(0.0, 0.0);
      if (q < q1) {
        const long slot = (long)pj.aslot[q / ysplit] * ysplit + q % ysplit;
        v[u] = ld_l2(pj.slots + (slot * LMAX + l) * M + m);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      sx += v[u].x;
      sy += v[u].y;
    }
  }
  __syncwarp();
#pragma unroll
  for (int o = 32 / kFinParts; o < 32; o *= 2) {
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
    sy += __shfl_xor_sync(0xffffffffu, sy, o);
  }
  if (on && part == 0) {
    const double sc = pj.scale[a * pj.L + l];
    pj.proj[i] = make_double2(sc * sx, sc * sy);
  }
}
// the item of this thread among the warps' groups of four: thread t of a run of threads
// handles item (t / 32) * 4 + t % 4
__device__ __forceinline__ long finish_item(long t) { return t / 32 * (32 / kFinParts) + t % (32 / kFinParts); }

// The forward outer y stage y1 -> kb of one block [ix][y1][G] into the x slots.  Straight
// from HBM a thread loads the Y1 lanes of its (ix, v) column (neighbouring threads read
// whole runs) and writes it to shared memory once; STAGED copies the block to shared memory
// first, with more bytes in flight a thread.
template <typename TG, bool STAGED>
__device__ __forceinline__ void outer_y_load(typename TG::V* X, const typename TG::V* blk) {
  using AX = typename TG::AX;
  constexpr int NX = TG::AX::N, Y1 = TG::Y1, VP = TG::VP, XS = TG::XS;
  if (STAGED) {
    for (int q = threadIdx.x; q < NX * Y1 * TG::CH; q += blockDim.x) {
      const int c = q % TG::CH * TG::LC, r = q / TG::CH;
      cp_async16(X + AX::slot(r / Y1) * XS + r % Y1 * VP + c, blk + r * VP + c);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
  }
  for (int it = threadIdx.x; it < NX * VP; it += blockDim.x) {
    const int v = it % VP, ix = it / VP;
    const int base = AX::slot(ix) * XS + v;
    typename TG::V u[Y1];
#pragma unroll
    for (int y = 0; y < Y1; ++y) u[y] = STAGED ? X[base + y * VP] : ld_l2(blk + (ix * Y1 + y) * VP + v);
    DFT<Y1, false, typename TG::P>::run(u);
#pragma unroll
    for (int y = 0; y < Y1; ++y) X[base + y * VP] = u[y];
  }
}

// ---------------------------------------------------------------- pass B
// One contiguous block tmp[g][ka][kz] = [ix][y1][G]; in shared memory the x
// index goes to padded slots of stride XS and (y1, j) stays contiguous.  With
// fin.slots set, the first CTAs also finish the fused projection (pass C reads it):
// four items a warp (proj_finish_item), the warps of the launch in order, so the few CTAs
// that carry the finish run beside thousands that do not.
template <typename T, int NX, int NY, int NZ>
__device__ __forceinline__ void tile_x_body(int bx, int by, typename TileGeom<T, NX, NY, NZ>::V* __restrict__ tmp,
                                            const cplx<T>* __restrict__ tw_x, KinParams<T> kp,
                                            cplx<T>* __restrict__ fout) {
  using TG = TileGeom<T, NX, NY, NZ>;
  using AX = typename TG::AX;
  using V = typename TG::V;
  using P = typename TG::P;
  constexpr int VP = TG::VP, Y1 = TG::Y1, Y2 = TG::Y2, XS = TG::XS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* X = reinterpret_cast<V*>(smem_raw);
  V* twx = X + TG::XBLK;
  T* kinB = reinterpret_cast<T*>(twx + NX);  // [Y1] linear and [Y1] constant term per kb
  T* kinC = kinB + Y1;

  const int kz = bx % NZ, ka = bx / NZ, grp = by;
  V* blk = tmp + ((long)(grp * Y2 + ka) * NZ + kz) * TG::BLK;
  for (int i = threadIdx.x; i < NX; i += blockDim.x) twx[i] = lane_splat<P>(tw_x[i]);
  // Along an x line 1/2 |G + k + A|^2 / N = kA2 n0^2 + kinB n0 + kinC with
  // q = n1 b1 + n2 b2 + k + A:  kA2 = |b0|^2 / 2N, kinB = b0.q / N, kinC = |q|^2 / 2N
  if (threadIdx.x < Y1) {
    const int kb = threadIdx.x;
    const T n1 = (T)sym_freq(ka + Y2 * kb, NY), n2 = (T)sym_freq(kz, NZ);
    T q[3], bq = 0, qq = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      q[d] = n1 * kp.b[1][d] + n2 * kp.b[2][d] + kp.kA[d];
      bq += kp.b[0][d] * q[d];
      qq += q[d] * q[d];
    }
    kinB[kb] = kp.scale * bq;
    kinC[kb] = (T)0.5 * kp.scale * qq;
  }
  const T kinA = (T)0.5 * kp.scale *
                 (kp.b[0][0] * kp.b[0][0] + kp.b[0][1] * kp.b[0][1] + kp.b[0][2] * kp.b[0][2]);

  chain_wait();
  outer_y_load<TG, TG::H_STAGED>(X, blk);
  __syncthreads();

  auto map1 = [](int it, int& base, int& es, int& j2) {
    const int v = it % VP, rest = it / VP;
    j2 = rest % AX::N2;
    base = (rest / AX::N2) * VP + v;
    es = XS;
  };
  auto map2 = [](int it, int& base, int& es, int& k1) {
    const int v = it % VP, rest = it / VP;
    k1 = rest % AX::N1;
    base = (rest / AX::N1) * VP + v;
    es = XS;
  };
  const int n2 = sym_freq(kz, NZ);
  step1<AX, false>(X, Y1 * VP * AX::N2, twx, map1);
  __syncthreads();
  // fout (optional): the forward coefficients of this block, before the kinetic
  // factor, as [kx][kb][G] in the orbital layout (the adjoint's velocity terms read them)
  V* fblk = fout ? reinterpret_cast<V*>(fout) + ((long)(grp * Y2 + ka) * NZ + kz) * TG::BLK : nullptr;
  step2_fwd_op_inv<AX>(X, Y1 * VP * AX::N1, twx, map2, [&](int it, int kx, V v) -> V {
    const int kb = (it / VP) / AX::N1;
    if (fblk) fblk[(kx * Y1 + kb) * VP + it % VP] = flip(v);
    const int n0 = sym_freq(kx, NX);
    const T f0 = (T)n0;
    T k = fma(fma(kinA, f0, kinB[kb]), f0, kinC[kb]);
    if (kp.mask) k = outside_sphere(kp.nr, n0, sym_freq(ka + Y2 * kb, NY), n2) ? (T)0 : k - kp.shift;
    if (kp.pois != (T)0) k = ((T)2 * k < (T)1e-6) ? (T)0 : kp.pois / k;
    const P ks = splat_of<P>(k);
    return {ks * v.x, ks * v.y};
  });
  __syncthreads();
  step1_inv_transposed<AX>(X, Y1 * VP * AX::N2, map1);
  __syncthreads();

  // inverse outer y stage kb -> y1, written straight back to HBM
  for (int it = threadIdx.x; it < NX * VP; it += blockDim.x) {
    const int v = it % VP, ix = it / VP;
    const int base = AX::slot(ix) * XS + v;
    V u[Y1];
#pragma unroll
    for (int y = 0; y < Y1; ++y) u[y] = X[base + y * VP];
    DFT<Y1, true, P>::run(u);
#pragma unroll
    for (int y = 0; y < Y1; ++y) blk[(ix * Y1 + y) * VP + v] = u[y];
  }
}

template <typename T, int NX, int NY, int NZ>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? TileGeom<T, NX, NY, NZ>::X_MIN_CTAS : 1)
    k_tile_x(typename TileGeom<T, NX, NY, NZ>::V* __restrict__ tmp, const cplx<T>* __restrict__ tw_x, KinParams<T> kp,
             cplx<T>* __restrict__ fout, ProjView<T> fin, int fin_M, int fin_ysplit) {
  if (fin.slots) {
    const long n = (long)fin.nproj * fin.L * fin_M;
    const long stride = (long)gridDim.x * gridDim.y * blockDim.x;
    chain_wait();
    for (long t = ((long)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x; finish_item(t) < n; t += stride) {
      const long i = finish_item(t + threadIdx.x);
      proj_finish_item(fin, fin_M, fin_ysplit, i < n ? (unsigned)i : 0u, i < n);
    }
  }
  tile_x_body<T, NX, NY, NZ>(blockIdx.x, blockIdx.y, tmp, tw_x, kp, fout);
}

// ---------------------------------------------------------------- pass B of the plain FFTs
// DIR = 0 (to_fourier): block tmp[g][ka][kz] -> outer y stage -> forward x ->
//   out[kx][ky][kz][m] in natural frequency order (transform.hpp:115-188, sign -1).
// DIR = 1 (to_real, first half): in[kx][ky][kz][m] -> inverse x -> inverse outer
//   y stage -> block tmp[g][ka][kz]; pass C finishes with the inner y and z stages
//   and the 1/N (transform.hpp:250-332).
template <typename T, int NX, int NY, int NZ, int DIR>
__global__ void __launch_bounds__(256, TileGeom<T, NX, NY, NZ>::X_MIN_CTAS)
    k_tile_x_fft(typename TileGeom<T, NX, NY, NZ>::V* __restrict__ tmp, const cplx<T>* __restrict__ in, cplx<T>* __restrict__ out, long ld,
                 int M, const cplx<T>* __restrict__ tw_x, int vec) {
  using TG = TileGeom<T, NX, NY, NZ>;
  using AX = typename TG::AX;
  using V = typename TG::V;
  using P = typename TG::P;
  constexpr int G = TG::G, PV = TG::PV, VP = TG::VP, Y1 = TG::Y1, Y2 = TG::Y2, XS = TG::XS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* X = reinterpret_cast<V*>(smem_raw);
  V* twx = X + TG::XBLK;

  const int kz = blockIdx.x % NZ, ka = blockIdx.x / NZ, grp = blockIdx.y;
  const int m0 = grp * G;
  const int gcount = min(G, M - m0);
  const bool v16 = vec && gcount == G;
  V* blk = tmp + ((long)(grp * Y2 + ka) * NZ + kz) * TG::BLK;
  // point of frequency (kx, ka + Y2 kb, kz) in the orbital layout
  auto point = [&](int kx, int kb) { return ((long)kx * NY + ka + Y2 * kb) * NZ + kz; };
  auto map1 = [](int it, int& base, int& es, int& j2) {
    const int v = it % VP, rest = it / VP;
    j2 = rest % AX::N2;
    base = (rest / AX::N2) * VP + v;
    es = XS;
  };
  auto map2 = [](int it, int& base, int& es, int& k1) {
    const int v = it % VP, rest = it / VP;
    k1 = rest % AX::N1;
    base = (rest / AX::N1) * VP + v;
    es = XS;
  };
  for (int i = threadIdx.x; i < NX; i += blockDim.x) twx[i] = lane_splat<P>(tw_x[i]);
  chain_wait();

  if (DIR == 0) {
    outer_y_load<TG, TG::FFT_STAGED>(X, blk);
    __syncthreads();
    step1<AX, false>(X, Y1 * VP * AX::N2, twx, map1);
    __syncthreads();
    step2<AX, false>(X, Y1 * VP * AX::N1, map2);
    __syncthreads();
    // kx sits in slot_of_freq(kx)
    for (int q = threadIdx.x; q < NX * Y1 * VP; q += blockDim.x) {
      const int v = q % VP, r = q / VP;
      const int kb = r % Y1, kx = r / Y1;
      const V w = X[AX::slot_of_freq(kx) * XS + kb * VP + v];
      cplx<T>* dst = out + point(kx, kb) * ld + m0 + v * PV;
      if (v16) {
        *reinterpret_cast<V*>(dst) = flip(w);
      } else {
#pragma unroll
        for (int k = 0; k < PV; ++k)
          if (v * PV + k < gcount) dst[k] = lane_get(w, k);
      }
    }
  } else {
    // natural kx into slot(kx); the inverse from natural order leaves ix in slot_of_freq(ix)
    if (v16) {
      for (int q = threadIdx.x; q < NX * Y1 * TG::CH; q += blockDim.x) {
        const int c = q % TG::CH * TG::LC, r = q / TG::CH;
        const int kb = r % Y1, kx = r / Y1;
        cp_async16(X + AX::slot(kx) * XS + kb * VP + c, in + point(kx, kb) * ld + m0 + c * PV);
      }
      cp_async_commit();
      cp_async_wait<0>();
    } else {
      cplx<T>* Xj = reinterpret_cast<cplx<T>*>(X);
      for (int q = threadIdx.x; q < NX * Y1 * G; q += blockDim.x) {
        const int j = q % G, r = q / G;
        const int kb = r % Y1, kx = r / Y1;
        Xj[(AX::slot(kx) * XS + kb * VP) * PV + j] = (j < gcount) ? in[point(kx, kb) * ld + m0 + j] : mk<T>(0, 0);
      }
    }
    __syncthreads();
    step1<AX, true, true>(X, Y1 * VP * AX::N2, twx, map1);
    __syncthreads();
    step2<AX, true>(X, Y1 * VP * AX::N1, map2);
    __syncthreads();
    // inverse outer y stage kb -> y1, written straight to HBM
    for (int it = threadIdx.x; it < NX * VP; it += blockDim.x) {
      const int v = it % VP, ix = it / VP;
      const int base = AX::slot_of_freq(ix) * XS + v;
      V u[Y1];
#pragma unroll
      for (int y = 0; y < Y1; ++y) u[y] = X[base + y * VP];
      DFT<Y1, true, P>::run(u);
#pragma unroll
      for (int y = 0; y < Y1; ++y) blk[(ix * Y1 + y) * VP + v] = u[y];
    }
  }
}

// ---------------------------------------------------------------- pass C
// The (ka, kz) runs of the tile come by cp.async; the nonlocal term is added to the
// transformed tile in shared memory, and the epilogue reads the input orbitals (for V psi)
// straight from HBM, four lanes a thread in flight.
// MODE_H = 1: the H epilogue; 0: out = alpha * (inverse transform), the second
// half of to_real (alpha = 1/N), reading neither orbitals, V nor projectors.
template <typename T, int NX, int NY, int NZ, int MODE_H>
__device__ __forceinline__ void tile_inv_body(int bx, int by, const typename TileGeom<T, NX, NY, NZ>::V* __restrict__ tmp,
                                              const cplx<T>* __restrict__ in, long ld_in, cplx<T>* __restrict__ out,
                                              long ld_out, int M, const cplx<T>* __restrict__ tw_y,
                                              const cplx<T>* __restrict__ tw_z, const ProjView<T>& pj,
                                              const EpiParams<T>& ep, int seg_cap, int vec) {
  using TG = TileGeom<T, NX, NY, NZ>;
  using AZ = typename TG::AZ;
  using V = typename TG::V;
  using P = typename TG::P;
  constexpr int G = TG::G, PV = TG::PV, VP = TG::VP, Y1 = TG::Y1, Y2 = TG::Y2, ZS = TG::ZS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* S = reinterpret_cast<V*>(smem_raw);
  V* twy = S + TG::TILE;
  V* twz = twy + NY;
  V* PT = twz + NZ;  // [seg_cap][PT_STRIDE] projections

  const int grp = bx, ix = by / Y1, y1 = by % Y1;
  const int m0 = grp * G;
  const int gcount = min(G, M - m0);
  // vec: bit 0, the input and output blocks take 16-byte accesses; bits 1 and 2, the base
  // and the subtracted block do
  const bool v16 = (vec & 1) && gcount == G, b16 = (vec & 2) && gcount == G, s16 = (vec & 4) && gcount == G;

  for (int i = threadIdx.x; i < NY; i += blockDim.x) twy[i] = lane_splat<P>(tw_y[i]);
  for (int i = threadIdx.x; i < NZ; i += blockDim.x) twz[i] = lane_splat<P>(tw_z[i]);
  // where the tile's segments and records lie (set with the projectors, no pass writes it)
  const bool proj_on = MODE_H && pj.nproj > 0;
  const int tile = ix * Y1 + y1;
  const int s0 = proj_on ? pj.seg_ptr[tile] : 0, nseg = proj_on ? pj.seg_ptr[tile + 1] - s0 : 0;
  const int k0 = proj_on ? pj.rk_ptr[tile] : 0, k1 = proj_on ? pj.rk_ptr[tile + 1] : 0;
  const int e_first = k0 < k1 ? pj.rk_start[k0] + (int)threadIdx.x / VP : 0;
  chain_wait();
  // the (ka, kz) runs of this tile
  for (int q = threadIdx.x; q < TG::PTS * TG::CH; q += blockDim.x) {
    const int c = q % TG::CH * TG::LC, pt = q / TG::CH;
    const int kz = pt % NZ, ka = pt / NZ;
    cp_async16(S + (ka * ZS + AZ::slot(kz)) * VP + c,
               tmp + (((long)(grp * Y2 + ka) * NZ + kz) * NX + ix) * (Y1 * VP) + y1 * VP + c);
  }
  cp_async_commit();
  // the tile's atom projections, in the tile precision, as [segment][l][orbital lane]
  // with a segment stride of PT_STRIDE: the lanes of one grid point read one contiguous
  // run per l
  const bool pt_staged = nseg <= seg_cap;
  // projection l of atom at, orbital lane v (two orbitals in FP32)
  auto projection = [&](int at, int l, int v) -> V {
    cplx<T> w[PV];
#pragma unroll
    for (int k = 0; k < PV; ++k) {
      w[k] = mk<T>(0, 0);
      if (l < pj.L && v * PV + k < gcount) {
        const double2 d = ld_l2(pj.proj + ((long)at * pj.L + l) * M + m0 + v * PV + k);
        w[k] = mk<T>((T)d.x, (T)d.y);
      }
    }
    V r;
    memcpy(&r, w, sizeof(V));
    return flip(r);
  };
  if (proj_on && pt_staged) {
    for (int i = threadIdx.x; i < nseg * LMAX * VP; i += blockDim.x) {
      const int v = i % VP, l = (i / VP) % LMAX, ts = i / (VP * LMAX);
      PT[ts * TG::PT_STRIDE + l * VP + v] = projection(pj.seg_atom[s0 + ts], l, v);
    }
  }
  cp_async_wait<0>();
  __syncthreads();

  // inverse inner y stage: conj twiddle, inverse DFT_Y2 over ka -> rows
  for (int it = threadIdx.x; it < NZ * VP; it += blockDim.x) {
    const int v = it % VP, zi = it / VP;
    const int base = AZ::slot(zi) * VP + v;
    V u[Y2];
#pragma unroll
    for (int ka = 0; ka < Y2; ++ka) u[ka] = S[base + ka * ZS * VP];
#pragma unroll
    for (int ka = 1; ka < Y2; ++ka) u[ka] = lmul_conj(u[ka], twy[ka * Y1 + y1]);
    DFT<Y2, true, P>::run(u);
#pragma unroll
    for (int r = 0; r < Y2; ++r) S[base + r * ZS * VP] = u[r];
  }
  __syncthreads();
  // inverse z from natural order: element z ends in slot_of_freq(z)
  step1<AZ, true>(S, Y2 * VP * AZ::N2, twz, [](int it, int& base, int& es, int& j2) {
    const int v = it % VP, rest = it / VP;
    j2 = rest % AZ::N2;
    base = (rest / AZ::N2) * ZS * VP + v;
    es = VP;
  });
  __syncthreads();
  step2<AZ, true>(S, Y2 * VP * AZ::N1, [](int it, int& base, int& es, int& k1) {
    const int v = it % VP, rest = it / VP;
    k1 = rest % AZ::N1;
    base = (rest / AZ::N1) * ZS * VP + v;
    es = VP;
  });

  // nonlocal term, added to the tile in shared memory: V_nl psi(r) = sum over the entries
  // at r of conj(exp(i (k+A).r_e)) sum_l beta_e[l] proj[a_e][l] (projector_all.hpp:182-232).
  // A group of VP threads takes an entry.  The tile's records are in rank order (the first
  // entry of every point, then the second ones, ...): within a rank no two entries share a
  // point, and a barrier ends each rank, so every point adds its entries in a fixed order.
  // A thread's next record, of this rank or the next one, is on its way while it works on
  // the current (a dense shell of atoms has a dozen ranks of one or two records a thread).
  if (proj_on) {
    const int v = threadIdx.x % VP, eg = blockDim.x / VP, t0 = threadIdx.x / VP;
    int e = e_first, e1 = k0 < k1 ? pj.rk_start[k0 + 1] : 0;
    EntRec<T> re;
    if (e < e1) re = pj.ent_rec_rk[e];
    for (int k = k0; k < k1; ++k) {
      const int next = e1 + t0, next_end = k + 1 < k1 ? pj.rk_start[k + 2] : e1;
      __syncthreads();
      if (e >= e1 && next < next_end) re = pj.ent_rec_rk[next];
      while (e < e1) {
        const EntRec<T> cur = re;
        e += eg;
        if (e < e1 || next < next_end) re = pj.ent_rec_rk[e < e1 ? e : next];
        // t = sum over l in increasing order of beta[l] proj[l]
        V t = {splat<P>(0.0), splat<P>(0.0)};
        const V* pt = PT + cur.tseg * TG::PT_STRIDE + v;
#pragma unroll
        for (int l = 0; l < LMAX; ++l) {
          // more atom segments in this tile than staged: projections from global memory
          const V pv = pt_staged ? pt[l * VP] : projection(pj.seg_atom[s0 + cur.tseg], l, v);
          const P b = splat_of<P>(cur.beta[l]);
          t.x = vfma(b, pv.x, t.x);
          t.y = vfma(b, pv.y, t.y);
        }
        const P pr = splat_of<P>(cur.ph[0]), pi = splat_of<P>(cur.ph[1]), npi = splat_of<P>(-cur.ph[1]);
        V* dst = S + cur.off * VP + v;
        const V h = *dst;
        *dst = {h.x + vfma(t.x, pr, t.y * pi), h.y + vfma(t.y, pr, t.x * npi)};
      }
      e = next;
      e1 = next_end;
    }
  }
  __syncthreads();

  // epilogue: out = alpha (K psi + (V + vshift) psi + V_nl psi) + beta base - minus
  // BE lanes per thread whose loads are issued together
  constexpr int BE = 4;
  const P ar = splat_of<P>(ep.alpha.x), ai = splat_of<P>(ep.alpha.y), nai = splat_of<P>(-ep.alpha.y);
  // a lane of the output (orbital layout) at point p, orbitals m0 + jb ..
  auto store = [&](long p, int jb, V w) {
    cplx<T>* dst = out + p * ld_out + m0 + jb;
    if (v16) {
      *reinterpret_cast<V*>(dst) = flip(w);
    } else {
#pragma unroll
      for (int k = 0; k < PV; ++k)
        if (jb + k < gcount) dst[k] = lane_get(w, k);
    }
  };
  // a lane of an orbital block at point p
  auto load = [&](const cplx<T>* src, long ld, long p, int jb, bool wide) -> V {
    V r;
    if (wide) {
      r = *reinterpret_cast<const V*>(src + p * ld + m0 + jb);
    } else {
      cplx<T> w[PV];
#pragma unroll
      for (int k = 0; k < PV; ++k) w[k] = (jb + k < gcount) ? src[p * ld + m0 + jb + k] : mk<T>(0, 0);
      memcpy(&r, w, sizeof(V));
    }
    return r;
  };
  const bool own = ep.base == in && ep.ld_base == ld_in;
  if constexpr (!MODE_H) {
    for (int q = threadIdx.x; q < TG::PTS * VP; q += blockDim.x) {
      const int v = q % VP, pt = q / VP;
      const int z = pt % NZ, r = pt / NZ;
      const long p = ((long)ix * NY + y1 + Y1 * r) * NZ + z;
      const V h = S[(r * ZS + AZ::slot_of_freq(z)) * VP + v];
      store(p, v * PV, {vfma(h.x, ar, h.y * nai), vfma(h.x, ai, h.y * ar)});
    }
  } else
  for (int q0 = threadIdx.x; q0 < TG::PTS * VP; q0 += BE * blockDim.x) {
    V x[BE];
    T vp[BE];
#pragma unroll
    for (int b = 0; b < BE; ++b) {
      const int q = q0 + b * blockDim.x;
      if (q >= TG::PTS * VP) continue;
      const int v = q % VP, pt = q / VP;
      const int z = pt % NZ, r = pt / NZ;
      const long p = ((long)ix * NY + y1 + Y1 * r) * NZ + z;
      vp[b] = ep.V[p] + ep.vshift;
      x[b] = load(in, ld_in, p, v * PV, v16);
    }
#pragma unroll
    for (int b = 0; b < BE; ++b) {
      const int q = q0 + b * blockDim.x;
      if (q >= TG::PTS * VP) continue;
      const int v = q % VP, pt = q / VP;
      const int z = pt % NZ, r = pt / NZ;
      const long p = ((long)ix * NY + y1 + Y1 * r) * NZ + z;
      V h = S[(r * ZS + AZ::slot_of_freq(z)) * VP + v];
      const V xv = flip(x[b]);
      const P vs = splat_of<P>(vp[b]);
      h = {vfma(vs, xv.x, h.x), vfma(vs, xv.y, h.y)};
      V o = {vfma(h.x, ar, h.y * nai), vfma(h.x, ai, h.y * ar)};
      if (ep.base) {
        // base the input block itself (a Taylor series' first term, 1 + c H): already here
        const V bb = own ? xv : flip(load(ep.base, ep.ld_base, p, v * PV, b16));
        const P br = splat_of<P>(ep.beta.x), bi = splat_of<P>(ep.beta.y), nbi = splat_of<P>(-ep.beta.y);
        o.x = o.x + vfma(bb.x, br, bb.y * nbi);
        o.y = o.y + vfma(bb.x, bi, bb.y * br);
      }
      if (ep.minus) o = o - flip(load(ep.minus, ep.ld_minus, p, v * PV, s16));
      store(p, v * PV, o);
    }
  }
}

template <typename T, int NX, int NY, int NZ, int MODE_H = 1>
__global__ void __launch_bounds__(TileGeom<T, NX, NY, NZ>::ZT, TileGeom<T, NX, NY, NZ>::INV_MIN_CTAS)
    k_tile_inv(const typename TileGeom<T, NX, NY, NZ>::V* __restrict__ tmp, const cplx<T>* __restrict__ in, long ld_in,
               cplx<T>* __restrict__ out, long ld_out, int M, const cplx<T>* __restrict__ tw_y,
               const cplx<T>* __restrict__ tw_z, ProjView<T> pj, EpiParams<T> ep, int seg_cap, int vec) {
  tile_inv_body<T, NX, NY, NZ, MODE_H>(blockIdx.x, blockIdx.y, tmp, in, ld_in, out, ld_out, M, tw_y, tw_z, pj, ep,
                                       seg_cap, vec);
}

}  // namespace inqb
