// Shared-memory FFT passes of the pressure solve
// (the device replacement of PoissonSolverPeriodic's FFTW r2c / _solve / c2r,
// source/poisson/PoissonSolverPeriodic.cpp:15-146).
//
// The wide Laplacian couples a cell only with cells two apart, so along each
// axis the even and the odd cells are two independent periodic lines of
// M = N/2 cells. Packed as z[m] = x[2m] + i x[2m+1] they take ONE complex FFT
// of length M and nothing else: the spectral factor depends on cos(2 pi k / M)
// alone, so it multiplies the packed bin k as it stands, and the even/odd
// split that a real transform of length N would need (with its twiddles and
// its two extra passes through shared memory) cancels between the forward and
// the inverse transform. Along x the pair is one element of memory, along y
// and z it is two rows of a column tile; the three axes are separate
// real-linear maps, so every pass is in place on the Nx*Ny*Nz array of reals.
// The 8 null modes of the reference (k in {0, N/2} on every axis) are the one
// packed mode k = 0.
//
// Plan of a length-M line (R2 threads): m = t + R2 r,
//   A  radix R1 over r, times W_M^(t k1)     (thread t, all k1)
//   B  radix R2 over t                        (thread t: k1 = t + R2 b)
// Both stages write where they read, element (k1, q) of B's output at position
// R2 k1 + q, which holds bin k1 + R1 q: the spectrum stays in that order (the
// factor's cosine tables are permuted to it on the host) and the inverse runs
// the stages backwards (B, then A), so nothing is reordered, one exchange
// through shared memory is left per transform, and the z pass goes from the
// forward B through the factor to the inverse B in registers. The inverse is
// the forward arithmetic on (im, re).
//
// Measured at 256^3 (one B200, passes in sequence) against the Hartley passes
// of dht.cuh, which every solve ran before and the FP64 handles of
// amplifies_rounding still run: FP64 RHS + x 187 -> 102 us, y 49 ->
// 43, z with the divide 80 -> 53, y 49 -> 44, x 53 -> 45; mixed correction solve
// x 38 -> 27, y 27 -> 22, z 58 -> 45, y 49 -> 44, x + p 74 -> 65.5. The column
// passes now move their 16 B/cell at 5-6 TB/s (82-95 % of the measured copy
// bandwidth); RHS + x waits on its loads of u, v, w (32 B/cell, 5.3 TB/s).
#pragma once

#include "common.cuh"
#include "dht.cuh"
#include "ops.cuh"

namespace cup {

template <int M>
struct PPlan {
  static constexpr int R1 = M == 128 ? 16 : 8;
  static constexpr int R2 = M / R1;   // also the threads per line
  static constexpr int NB = R1 / R2;  // radix-R2 butterflies per thread in B
  // bin held at position pos of a transformed line
  static constexpr int bin(int pos) { return pos / R2 + R1 * (pos % R2); }
  // rows: element (k1, q) sits at R2 k1 + (q ^ (k1 mod R2)), which spreads B's
  // accesses (lanes k1, stride R2) over the banks
  static __host__ __device__ constexpr int row_pos(int k1, int q) { return R2 * k1 + (q ^ (k1 & (R2 - 1))); }
  static constexpr int row_bin(int pos) { return pos / R2 + R1 * ((pos % R2) ^ ((pos / R2) & (R2 - 1))); }
};
template <typename R2_>
struct DFT<1, R2_> {
  __device__ __forceinline__ static void run(R2_*) {}
};

template <typename R2>
__device__ __forceinline__ R2 swap_ri(R2 a) {
  R2 r;
  r.x = a.y;
  r.y = a.x;
  return r;
}

// A pair of float columns that go through one instruction stream (f32x2).
struct F2 {
  float2 v;
  __device__ __forceinline__ F2() {}
  __device__ __forceinline__ F2(float2 a) : v(a) {}
  __device__ __forceinline__ explicit F2(double a) : v(make_float2((float)a, (float)a)) {}
};
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return F2(__ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v)); }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return F2(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 operator-(F2 a) { return F2(make_float2(-a.v.x, -a.v.y)); }
struct F2c {
  F2 x, y;
};
// complex times a scalar twiddle
__device__ __forceinline__ F2c tmul(F2c a, float2 w) {
  const float2 wr = make_float2(w.x, w.x), wi = make_float2(w.y, w.y), mwi = make_float2(-w.y, -w.y);
  F2c r;
  r.x = F2(__ffma2_rn(a.y.v, mwi, __fmul2_rn(a.x.v, wr)));
  r.y = F2(__ffma2_rn(a.y.v, wr, __fmul2_rn(a.x.v, wi)));
  return r;
}
__device__ __forceinline__ float2 tmul(float2 a, float2 w) { return cmul(a, w); }
__device__ __forceinline__ double2 tmul(double2 a, double2 w) { return cmul(a, w); }

// Lane types of a column tile: what one thread's column element is, its complex
// pair and the scalar type of the tile and its twiddles.
template <typename L>
struct Lane;
template <>
struct Lane<double> {
  using S = double;
  using C = double2;
  static constexpr int COLS = 1;
};
template <>
struct Lane<float> {
  using S = float;
  using C = float2;
  static constexpr int COLS = 1;
};
template <>
struct Lane<F2> {
  using S = float;
  using C = F2c;
  static constexpr int COLS = 2;
};

// Column of a tile: row n of the column at base + n stride (stride in scalars).
template <typename L>
struct PCol {
  using S = typename Lane<L>::S;
  using C = typename Lane<L>::C;
  S* base;
  int stride;
  __device__ __forceinline__ C ld(int pos) const {
    C c;
    c.x = *reinterpret_cast<const L*>(base + (2 * pos) * stride);
    c.y = *reinterpret_cast<const L*>(base + (2 * pos + 1) * stride);
    return c;
  }
  __device__ __forceinline__ void st(int pos, C c) const {
    *reinterpret_cast<L*>(base + (2 * pos) * stride) = c.x;
    *reinterpret_cast<L*>(base + (2 * pos + 1) * stride) = c.y;
  }
};

// Forward stage A of thread t, in place. tw[k1 R2 + t] = W_M^(k1 t).
template <int M, class Col, typename TW>
__device__ __forceinline__ void pcol_fwd_a(const Col& c, const TW* tw, int t) {
  using P = PPlan<M>;
  typename Col::C v[P::R1];
#pragma unroll
  for (int r = 0; r < P::R1; ++r) v[r] = c.ld(P::R2 * r + t);
  DFT<P::R1, typename Col::C>::run(v);
#pragma unroll
  for (int r = 0; r < P::R1; ++r) {
    if (r > 0 && P::R2 > 1) v[r] = tmul(v[r], tw[r * P::R2 + t]);
    c.st(P::R2 * r + t, v[r]);
  }
}
// Inverse stage A of thread t (data as (im, re)), in place, output as (re, im).
template <int M, class Col, typename TW>
__device__ __forceinline__ void pcol_inv_a(const Col& c, const TW* tw, int t) {
  using P = PPlan<M>;
  typename Col::C v[P::R1];
#pragma unroll
  for (int r = 0; r < P::R1; ++r) {
    v[r] = c.ld(P::R2 * r + t);
    if (r > 0 && P::R2 > 1) v[r] = tmul(v[r], tw[r * P::R2 + t]);
  }
  DFT<P::R1, typename Col::C>::run(v);
#pragma unroll
  for (int r = 0; r < P::R1; ++r) c.st(P::R2 * r + t, swap_ri(v[r]));
}
// Stage B of thread t, in place: forward, or inverse on (re, im) giving (im, re).
template <int M, bool INV, class Col>
__device__ __forceinline__ void pcol_b(const Col& c, int t) {
  using P = PPlan<M>;
#pragma unroll
  for (int b = 0; b < P::NB; ++b) {
    const int k1 = t + P::R2 * b;
    typename Col::C z[P::R2];
#pragma unroll
    for (int q = 0; q < P::R2; ++q) {
      z[q] = c.ld(P::R2 * k1 + q);
      if constexpr (INV) z[q] = swap_ri(z[q]);
    }
    DFT<P::R2, typename Col::C>::run(z);
#pragma unroll
    for (int q = 0; q < P::R2; ++q) c.st(P::R2 * k1 + q, z[q]);
  }
}

// Planes of a y tile / rows of a z tile: short lines take several so that a CTA has 128 threads.
template <int M, typename L, int W>
struct PTile {
  static constexpr int LANES = W / Lane<L>::COLS;
  static constexpr int TPL = PPlan<M>::R2;
  static constexpr int P = LANES * TPL >= 128 ? 1 : 128 / (LANES * TPL);
  static constexpr int THREADS = LANES * TPL * P;
};

// ---------------------------------------------------------------------------
// y pass: persistent CTAs walk tiles of W x-columns by the whole y line by P
// planes through NB buffers. Tile t is x0 = (t % ntiles_x) W, planes
// (t / ntiles_x) P. The next tile's TMA load is issued after stage A, when the
// store that still reads its buffer is done.
template <int M, typename L, bool INV, int W, int NB>
__global__ void __launch_bounds__(PTile<M, L, W>::THREADS)
    k_pfft_y(const __grid_constant__ CUtensorMap map, int ntiles_x, int ntiles, int rev,
             const typename Cplx<typename Lane<L>::S>::T* tw_g, int* err, const int* skip) {
  pdl_entry();
  if (skip && *skip) return;
  using S = typename Lane<L>::S;
  using TW = typename Cplx<S>::T;
  using Tile = PTile<M, L, W>;
  static_assert(NB >= 2, "the refill follows the wait: one buffer would wait for a load never issued");
  constexpr int N = 2 * M, P = Tile::P;
  constexpr int ELEMS = N * W * P;
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  S* tiles = reinterpret_cast<S*>(smem_raw);  // [NB][P][N][W]
  TW* tw = reinterpret_cast<TW*>(tiles + (size_t)NB * ELEMS);
  uint64_t* bar = reinterpret_cast<uint64_t*>(tw + M);
  const int tid = threadIdx.x;
  const int my = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  if (tid == 0) {
    for (int b = 0; b < NB; ++b) mbar_init(&bar[b], 1);
    mbar_fence_init();
  }
  __syncthreads();
  auto tile_of = [&](int i) {
    const int t = blockIdx.x + i * gridDim.x;
    return rev ? ntiles - 1 - t : t;
  };
  auto issue = [&](int i) {
    const int t = tile_of(i), b = i % NB;
    mbar_arrive_expect_tx(&bar[b], (uint32_t)(ELEMS * sizeof(S)));
    tma_load_3d(tiles + (size_t)b * ELEMS, &map, (t % ntiles_x) * W, 0, (t / ntiles_x) * P, &bar[b]);
  };
  int issued = 0;
  if (tid == 0)
    for (; issued < min(NB, my); ++issued) issue(issued);
  for (int i = tid; i < M; i += blockDim.x) tw[i] = tw_g[i];
  __syncthreads();
  const int lane = tid % (Tile::LANES * P), t = tid / (Tile::LANES * P);
  const int off = (lane / Tile::LANES) * N * W + (lane % Tile::LANES) * Lane<L>::COLS;
  bool ok = true;
  int done = 0;
  for (int i = 0; i < my; ++i) {
    const int b = i % NB;
    S* tile = tiles + (size_t)b * ELEMS;
    const PCol<L> c{tile + off, W};
    ok = mbar_wait(&bar[b], (i / NB) & 1, err);
    if (ok) {
      if constexpr (INV) pcol_b<M, true>(c, t);
      else pcol_fwd_a<M>(c, tw, t);
    }
    ok = __syncthreads_and(ok);
    if (!ok) break;
    // refill the buffer of tile i - 1 once its store has read it
    if (tid == 0 && i > 0 && issued < my) {
      bulk_wait_read<0>();
      issue(issued++);
    }
    if constexpr (INV) pcol_inv_a<M>(c, tw, t);
    else pcol_b<M, false>(c, t);
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      const int tt = tile_of(i);
      tma_store_3d(&map, (tt % ntiles_x) * W, 0, (tt / ntiles_x) * P, tile);
      bulk_commit();
    }
    done = i + 1;
  }
  if (tid == 0) {
    bulk_wait_all();
    // after a timed-out wait: bounded drain of the loads still in flight
    if (!ok)
      for (int r = done; r < issued; ++r) mbar_wait(&bar[r % NB], (r / NB) & 1, nullptr);
  }
}

// Spectral factor of PoissonSolverPeriodic::_solve (grid-consistent branch,
// source/poisson/PoissonSolverPeriodic.cpp:23-61) in the packed order: cx, cy,
// cz hold cos(2 pi k / M) of the bin at each position.
struct PSpectral {
  const double *cx, *cy, *cz;
  double nf;  // 4 / h / (Mx My Mz): the transforms are unnormalised
};

// Factors of the R2 bins of one B butterfly: nf / (2 (cos_x + cos_y + cos_z) - 6),
// zero for the null mode (null, q = 0). FP64: one division serves four factors
// (the products of the denominators, in [1e-4, 12] each, are far from overflow).
template <int N_>
__device__ __forceinline__ void p_factors(double (&f)[N_], double cxy, const double* cz, double nf, bool null0) {
#pragma unroll
  for (int q = 0; q < N_; ++q) f[q] = 2 * (cxy + cz[q]) - 6;
  if (null0) f[0] = 1.0;
  constexpr int G = N_ >= 4 ? 4 : N_;
#pragma unroll
  for (int g = 0; g < N_; g += G) {
    if constexpr (G == 4) {
      const double ab = f[g] * f[g + 1], cd = f[g + 2] * f[g + 3];
      const double inv = nf / (ab * cd);
      const double iab = inv * cd, icd = inv * ab;
      const double a = iab * f[g + 1], b = iab * f[g], c = icd * f[g + 3], d = icd * f[g + 2];
      f[g] = a, f[g + 1] = b, f[g + 2] = c, f[g + 3] = d;
    } else {
#pragma unroll
      for (int q = g; q < g + G; ++q) f[q] = nf / f[q];
    }
  }
  if (null0) f[0] = 0.0;
}
// The correction solve of the defect-correction loop: the denominator in FP64
// (it cancels to 2 (1 - cos(2 pi / M)) at the lowest modes), the quotient in
// FP32. A factor with relative error e changes its mode of the correction by
// 1 + e and leaves a residual of relative size e, as the FP32 transform does.
template <int N_>
__device__ __forceinline__ void p_factors(float (&f)[N_], double cxy, const double* cz, double nf, bool null0) {
#pragma unroll
  for (int q = 0; q < N_; ++q) f[q] = __fdividef((float)nf, (float)(2 * (cxy + cz[q]) - 6));
  if (null0) f[0] = 0.f;
}

// z pass: forward transform, spectral divide and inverse of every z line. T:
// the forward's type (float: the mixed correction solve, whose inverse and
// output are FP64). Tiles of W x-columns by P rows by the whole z line. FP64:
// NB buffers, in place. Mixed: NB narrow FP32 buffers and one FP64 buffer; the
// forward runs in the narrow one and B hands over in registers.
template <int M, typename T, int W, int NB>
__global__ void __launch_bounds__(PTile<M, T, W>::THREADS)
    k_pfft_z(const __grid_constant__ CUtensorMap map_in, const __grid_constant__ CUtensorMap map_out, int ntiles_x,
             int ntiles, const typename Cplx<T>::T* tw_in_g, const double2* tw_g, PSpectral sp, int* err,
             const int* skip) {
  pdl_entry();
  if (skip && *skip) return;
  using TW = typename Cplx<T>::T;
  using Tile = PTile<M, T, W>;
  using Pl = PPlan<M>;
  constexpr bool MIXED = sizeof(T) == 4;
  static_assert(MIXED || NB >= 2, "the refill follows the wait: one buffer would wait for a load never issued");
  constexpr int N = 2 * M, P = Tile::P, WP = W * P;
  constexpr int ELEMS = N * WP;
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  T* tiles = reinterpret_cast<T*>(smem_raw);                                // [NB][N][P][W]
  double* wide = reinterpret_cast<double*>(tiles + (size_t)NB * ELEMS);      // (mixed) [N][P][W]
  double2* tw = reinterpret_cast<double2*>(wide + (MIXED ? ELEMS : 0));
  double* cz = reinterpret_cast<double*>(tw + M);
  TW* tw_in = MIXED ? reinterpret_cast<TW*>(cz + M) : reinterpret_cast<TW*>(tw);
  uint64_t* bar = reinterpret_cast<uint64_t*>(cz + M + (MIXED ? M : 0));
  const int tid = threadIdx.x;
  const int my = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  if (tid == 0) {
    for (int b = 0; b < NB; ++b) mbar_init(&bar[b], 1);
    mbar_fence_init();
  }
  __syncthreads();
  auto coords = [&](int i, int& x0, int& y0) {
    const int t = blockIdx.x + i * gridDim.x;
    x0 = (t % ntiles_x) * W;
    y0 = (t / ntiles_x) * P;
  };
  auto issue = [&](int i) {
    int x0, y0;
    coords(i, x0, y0);
    const int b = i % NB;
    mbar_arrive_expect_tx(&bar[b], (uint32_t)(ELEMS * sizeof(T)));
    tma_load_3d(tiles + (size_t)b * ELEMS, &map_in, x0, y0, 0, &bar[b]);
  };
  int issued = 0;
  if (tid == 0)
    for (; issued < min(NB, my); ++issued) issue(issued);
  for (int i = tid; i < M; i += blockDim.x) {
    tw[i] = tw_g[i];
    cz[i] = sp.cz[i];
    if constexpr (MIXED) tw_in[i] = tw_in_g[i];
  }
  __syncthreads();
  const int lane = tid % WP, t = tid / WP;
  bool ok = true;
  int done = 0;
  for (int i = 0; i < my; ++i) {
    const int b = i % NB;
    T* tile = tiles + (size_t)b * ELEMS;
    const PCol<T> ci{tile + lane, WP};
    double* otile = MIXED ? wide : reinterpret_cast<double*>(tile);
    const PCol<double> co{otile + lane, WP};
    int x0, y0;
    coords(i, x0, y0);
    const int cx = (x0 + lane % W) >> 1, cy = (y0 + lane / W) >> 1;
    const double cxy = __ldg(sp.cx + cx) + __ldg(sp.cy + cy);
    const bool null_col = cx == 0 && cy == 0;
    ok = mbar_wait(&bar[b], (i / NB) & 1, err);
    if (ok) pcol_fwd_a<M>(ci, tw_in, t);
    // mixed: the store of tile i - 1 must have read the FP64 buffer before B writes it
    if (MIXED && tid == 0 && i > 0) bulk_wait_read<0>();
    ok = __syncthreads_and(ok);
    if (!ok) break;
    if (!MIXED && tid == 0 && i > 0 && issued < my) {
      bulk_wait_read<0>();
      issue(issued++);
    }
#pragma unroll
    for (int bb = 0; bb < Pl::NB; ++bb) {
      const int k1 = t + Pl::R2 * bb;
      TW z[Pl::R2];
      T f[Pl::R2];
#pragma unroll
      for (int q = 0; q < Pl::R2; ++q) z[q] = ci.ld(Pl::R2 * k1 + q);
      p_factors<Pl::R2>(f, cxy, cz + Pl::R2 * k1, sp.nf, null_col && k1 == 0);
      DFT<Pl::R2, TW>::run(z);
      double2 o[Pl::R2];
#pragma unroll
      for (int q = 0; q < Pl::R2; ++q) {  // from here on (im, re)
        o[q].x = (double)(z[q].y * f[q]);
        o[q].y = (double)(z[q].x * f[q]);
      }
      DFT<Pl::R2, double2>::run(o);
#pragma unroll
      for (int q = 0; q < Pl::R2; ++q) co.st(Pl::R2 * k1 + q, o[q]);
    }
    if constexpr (MIXED) fence_proxy_async_smem();  // the narrow tile was written in place
    __syncthreads();
    // mixed: every read of the narrow tile is done
    if (MIXED && tid == 0 && issued < my) issue(issued++);
    pcol_inv_a<M>(co, tw, t);
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      tma_store_3d(&map_out, x0, y0, 0, otile);
      bulk_commit();
    }
    done = i + 1;
  }
  if (tid == 0) {
    bulk_wait_all();
    // after a timed-out wait: bounded drain of the loads still in flight
    if (!ok)
      for (int r = done; r < issued; ++r) mbar_wait(&bar[r % NB], (r / NB) & 1, nullptr);
  }
}

// ---------------------------------------------------------------------------
// x passes. A line's R2 threads sit in one warp, so the exchange between the
// stages needs no block barrier: every warp walks its own tiles of 32 / R2
// consecutive rows through its own buffers and barriers.
template <int M>
struct PRows {
  static constexpr int TPL = PPlan<M>::R2;
  static constexpr int ROWS = 32 / TPL;         // rows of a warp's tile
  static constexpr int ELEMS = ROWS * 2 * M;    // reals of a tile
};

// Forward stages of a row whose elements m = t + R2 r are in v; the spectrum
// goes to row (complex, swizzled positions).
template <int M, typename C, typename TW>
__device__ __forceinline__ void prow_fwd(C (&v)[PPlan<M>::R1], C* row, const TW* tw, int t) {
  using P = PPlan<M>;
  DFT<P::R1, C>::run(v);
  __syncwarp();  // the row may hold the input other lanes read
#pragma unroll
  for (int r = 0; r < P::R1; ++r) {
    if (r > 0 && P::R2 > 1) v[r] = cmul(v[r], tw[r * P::R2 + t]);
    row[P::row_pos(r, t)] = v[r];
  }
  if constexpr (P::R2 > 1) {
    __syncwarp();
#pragma unroll
    for (int b = 0; b < P::NB; ++b) {
      const int k1 = t + P::R2 * b;
      C z[P::R2];
#pragma unroll
      for (int q = 0; q < P::R2; ++q) z[q] = row[P::row_pos(k1, q)];
      DFT<P::R2, C>::run(z);
#pragma unroll
      for (int q = 0; q < P::R2; ++q) row[P::row_pos(k1, q)] = z[q];
    }
  }
}
// Inverse stages of a row; v[r] = element m = t + R2 r, (re, im).
template <int M, typename C, typename TW>
__device__ __forceinline__ void prow_inv(C (&v)[PPlan<M>::R1], C* row, const TW* tw, int t) {
  using P = PPlan<M>;
  if constexpr (P::R2 > 1) {
#pragma unroll
    for (int b = 0; b < P::NB; ++b) {
      const int k1 = t + P::R2 * b;
      C z[P::R2];
#pragma unroll
      for (int q = 0; q < P::R2; ++q) z[q] = swap_ri(row[P::row_pos(k1, q)]);
      DFT<P::R2, C>::run(z);
#pragma unroll
      for (int q = 0; q < P::R2; ++q) row[P::row_pos(k1, q)] = z[q];
    }
    __syncwarp();
  }
#pragma unroll
  for (int r = 0; r < P::R1; ++r) {
    v[r] = row[P::row_pos(r, t)];
    if constexpr (P::R2 == 1) v[r] = swap_ri(v[r]);
    if (r > 0 && P::R2 > 1) v[r] = cmul(v[r], tw[r * P::R2 + t]);
  }
  DFT<P::R1, C>::run(v);
#pragma unroll
  for (int r = 0; r < P::R1; ++r) v[r] = swap_ri(v[r]);
}

enum { PROW_FWD = 0, PROW_INV = 1, PROW_INV_ADDP = 2 };

// x pass over an array: MODE forward or inverse from `in` to `out` (may be the
// same), or the inverse added into out = p minus the parity-class means of p
// (the last pass of a correction solve; the p rows ride in the tile's buffer).
// out2: a second copy of the output (nullptr: none).
template <int M, typename S, int MODE, int NB, int WARPS, bool LATE = false>
__global__ void __launch_bounds__(32 * WARPS) k_pfft_x(const S* in, S* out, S* out2, const double* cmean, int log2ny,
                                                      int ntiles, int rev, const typename Cplx<S>::T* tw_g, int* err,
                                                      const int* skip) {
  pdl_entry();
  if (skip && *skip) return;
  using C = typename Cplx<S>::T;
  using P = PPlan<M>;
  using Rw = PRows<M>;
  constexpr bool ADDP = MODE == PROW_INV_ADDP;
  static_assert(NB >= 2, "the refill follows the wait: one buffer would wait for a load never issued");
  constexpr int BUF = Rw::ELEMS * (ADDP ? 2 : 1);
  constexpr uint32_t BYTES = (uint32_t)(Rw::ELEMS * sizeof(S));
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  S* bufs = reinterpret_cast<S*>(smem_raw) + (size_t)warp * NB * BUF;  // [warp][NB][rows (, p rows)]
  C* tw = reinterpret_cast<C*>(reinterpret_cast<S*>(smem_raw) + (size_t)WARPS * NB * BUF);
  uint64_t* bar = reinterpret_cast<uint64_t*>(tw + M) + warp * NB;
  double* cms = reinterpret_cast<double*>(reinterpret_cast<uint64_t*>(tw + M) + WARPS * NB);
  const int first = blockIdx.x * WARPS + warp, step = gridDim.x * WARPS;
  const int my = first < ntiles ? (ntiles - 1 - first) / step + 1 : 0;
  if (tid < WARPS * NB) mbar_init(reinterpret_cast<uint64_t*>(tw + M) + tid, 1);
  if (tid < WARPS * NB) mbar_fence_init();
  for (int i = tid; i < M; i += blockDim.x) tw[i] = tw_g[i];
  if (ADDP && tid < 8) cms[tid] = cmean[tid];
  __syncthreads();
  auto tile_of = [&](int i) { return rev ? ntiles - 1 - (first + i * step) : first + i * step; };
  auto issue = [&](int i) {
    const size_t o = (size_t)tile_of(i) * Rw::ELEMS;
    S* d = bufs + (size_t)(i % NB) * BUF;
    mbar_arrive_expect_tx(&bar[i % NB], ADDP ? 2 * BYTES : BYTES);
    bulk_load(d, in + o, BYTES, &bar[i % NB]);
    if constexpr (ADDP) bulk_load(d + Rw::ELEMS, out + o, BYTES, &bar[i % NB]);
  };
  int issued = 0;
  if (lane == 0)
    for (; issued < min(NB, my); ++issued) issue(issued);
  const int l = lane / P::R2, t = lane % P::R2;
  int done = 0;
  bool ok = true;
  for (int i = 0; i < my; ++i) {
    // refill: the buffer of tile i - 1 takes tile i - 1 + NB once its store has read it
    if (!LATE && lane == 0 && i > 0 && issued < my) {
      bulk_wait_read<0>();
      issue(issued++);
    }
    ok = __all_sync(0xffffffffu, mbar_wait(&bar[i % NB], (i / NB) & 1, err));
    if (!ok) break;
    S* buf = bufs + (size_t)(i % NB) * BUF;
    C* row = reinterpret_cast<C*>(buf) + l * M;
    C v[P::R1];
    const int tile = tile_of(i);
    S* src = buf;
    if constexpr (MODE == PROW_FWD) {
#pragma unroll
      for (int r = 0; r < P::R1; ++r) v[r] = row[P::R2 * r + t];
      prow_fwd<M>(v, row, tw, t);
    } else {
      prow_inv<M>(v, row, tw, t);
      if constexpr (ADDP) {
        C* prow = reinterpret_cast<C*>(buf + Rw::ELEMS) + l * M;
        const int rr = tile * Rw::ROWS + l;  // (y, z) = (rr mod ny, rr / ny)
        const int cls = ((rr & 1) << 1) | (((rr >> log2ny) & 1) << 2);
        const S c0 = (S)cms[cls], c1 = (S)cms[cls | 1];
#pragma unroll
        for (int r = 0; r < P::R1; ++r) {
          C q = prow[P::R2 * r + t];
          q.x = q.x + v[r].x - c0;
          q.y = q.y + v[r].y - c1;
          prow[P::R2 * r + t] = q;
        }
        src = buf + Rw::ELEMS;
      } else {
        __syncwarp();
#pragma unroll
        for (int r = 0; r < P::R1; ++r) row[P::R2 * r + t] = v[r];
      }
    }
    if (LATE && lane == 0 && i > 0 && issued < my) {
      bulk_wait_read<0>();
      issue(issued++);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      bulk_store(out + (size_t)tile * Rw::ELEMS, src, BYTES);
      if (out2) bulk_store(out2 + (size_t)tile * Rw::ELEMS, src, BYTES);
      bulk_commit();
    }
    done = i + 1;
  }
  if (lane == 0) {
    bulk_wait_all();
    // after a timed-out wait: bounded drain of the loads still in flight
    if (!ok)
      for (int r = done; r < issued; ++r) mbar_wait(&bar[r % NB], (r / NB) & 1, nullptr);
  }
}

// Forward x pass of the pressure RHS b = (h^2 / 2 dt) div u* (KernelPressureRHS,
// source/operators/PressureRHS.cpp:51-76), which never goes to HBM: a thread
// forms the elements m = t + R2 r of its row (cells 2m, 2m+1) from paired loads
// of u, v, w, straight into stage A's registers. bdelta (may be nullptr): the
// obstacle's RHS terms on its box, added there.
// The launch bound of one CTA per SM lets the compiler hold all of a row's loads in
// registers (254 at M = 128); without it, it keeps to 102 and waits for them (12 FP64
// steps at 256^3 10170 -> 10320 us).
template <int M, typename T, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 1) k_pfft_x_rhs(const T* __restrict__ u, const T* __restrict__ v_,
                                                          const T* __restrict__ w, double* __restrict__ out, DtArg dt,
                                                          double h, int ny, int nz, int ntiles,
                                                          const double2* tw_g, const Box box, const double* bdelta) {
  pdl_entry();
  using P = PPlan<M>;
  using Rw = PRows<M>;
  using T2 = typename Cplx<T>::T;
  constexpr int N = 2 * M;
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* buf = reinterpret_cast<double*>(smem_raw) + (size_t)warp * Rw::ELEMS;
  double2* tw = reinterpret_cast<double2*>(reinterpret_cast<double*>(smem_raw) + (size_t)WARPS * Rw::ELEMS);
  for (int i = tid; i < M; i += blockDim.x) tw[i] = tw_g[i];
  __syncthreads();
  const int l = lane / P::R2, t = lane % P::R2;
  const double fac = 0.5 * h * h / dt.get();
  const int tile = blockIdx.x * WARPS + warp;
  if (tile >= ntiles) return;
  const int r0 = tile * Rw::ROWS + l;
  const int y = r0 % ny, z = r0 / ny;
  const T* U = u + (size_t)r0 * N;
  const T2* VN = reinterpret_cast<const T2*>(v_ + gidx(0, wrapi(y + 1, ny), z, N, ny));
  const T2* VS = reinterpret_cast<const T2*>(v_ + gidx(0, wrapi(y - 1, ny), z, N, ny));
  const T2* WB = reinterpret_cast<const T2*>(w + gidx(0, y, wrapi(z + 1, nz), N, ny));
  const T2* WF = reinterpret_cast<const T2*>(w + gidx(0, y, wrapi(z - 1, nz), N, ny));
  double2 a[P::R1];
#pragma unroll
  for (int r = 0; r < P::R1; ++r) {
    const int m = t + P::R2 * r;
    const T2 u0 = *reinterpret_cast<const T2*>(U + 2 * m);
    const double uW = U[(2 * m - 1) & (N - 1)], uE = U[(2 * m + 2) & (N - 1)];
    const T2 vN = VN[m], vS = VS[m], wB = WB[m], wF = WF[m];
    a[r].x = fac * ((double)u0.y - uW + (double)vN.x - (double)vS.x + (double)wB.x - (double)wF.x);
    a[r].y = fac * (uE - (double)u0.x + (double)vN.y - (double)vS.y + (double)wB.y - (double)wF.y);
  }
  if (bdelta) {
    int dy = y - box.lo[1], dz = z - box.lo[2];
    dy += dy < 0 ? ny : 0;
    dz += dz < 0 ? nz : 0;
    if (dy < box.n[1] && dz < box.n[2]) {
      const double* bd = bdelta + (size_t)box.n[0] * (dy + (size_t)box.n[1] * dz);
#pragma unroll
      for (int r = 0; r < P::R1; ++r) {
        const int d0 = (2 * (t + P::R2 * r) - box.lo[0]) & (N - 1), d1 = (d0 + 1) & (N - 1);
        if (d0 < box.n[0]) a[r].x += bd[d0];
        if (d1 < box.n[0]) a[r].y += bd[d1];
      }
    }
  }
  prow_fwd<M>(a, reinterpret_cast<double2*>(buf) + l * M, tw, t);
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    bulk_store(out + (size_t)tile * Rw::ELEMS, buf, (uint32_t)(Rw::ELEMS * sizeof(double)));
    bulk_commit();
    bulk_wait_all();
  }
}

}  // namespace cup
