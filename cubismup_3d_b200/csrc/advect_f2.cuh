// FP32 upwind3 + RK2 stages with Blackwell's packed FP32x2 arithmetic.
//
// Same streaming structure as k_advect_zq (TMA ring of planes, register
// z-queues, one x/y partial), but each
// thread owns PPT pairs of x-adjacent cells and every arithmetic instruction
// works on a pair (fma/add/mul .f32x2). The upwind term uses the branch-free
// identity
//   a up3(a; f) = 1/2 (a S(f) + |a| Q(f)),
//   S = f-2 - 8 f-1 + 8 f+1 - f+2,  Q = f-2 - 4 f-1 + 6 f0 - 4 f+1 + f+2,
// which is the same operator as the sign-selected stencil (at a = 0 both
// give 0), so both cells of a pair follow one instruction stream.
#pragma once

#include "advect.cuh"

namespace cup {

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 splat2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 abs2(float2 a) { return make_float2(fabsf(a.x), fabsf(a.y)); }

// The five weights of one direction of the update, for a pair: with
// facA = -dt / (12 h) and facD = nu dt / h^2,
//   facA (a S(f) + |a| Q(f)) + facD (f-1 + f+1 - 2 f0) = m2 f-2 + m1 f-1 + c0 f0 + p1 f+1 + p2 f+2,
//   m2 = A1 + A2, p2 = A2 - A1, m1 = -8 A1 - 4 A2 + facD, p1 = 8 A1 - 4 A2 + facD,
//   c0 = 6 A2 - 2 facD,  A1 = facA a, A2 = facA |a|.
// They depend on the advecting velocity only, so the three components of a
// cell share them (five FMAs per component and direction).
struct Weights5 {
  float2 m2, m1, c0, p1, p2;
};
__device__ __forceinline__ Weights5 weights5(float2 a, float2 facA, float2 facD, float2 m2FacD) {
  const float2 A1 = mul2(facA, a), A2 = mul2(facA, abs2(a));
  const float2 t = fma2(splat2(-4.f), A2, facD);
  Weights5 k;
  k.m2 = add2(A1, A2);
  k.p2 = sub2(A2, A1);
  k.m1 = fma2(splat2(-8.f), A1, t);
  k.p1 = fma2(splat2(8.f), A1, t);
  k.c0 = fma2(splat2(6.f), A2, m2FacD);
  return k;
}
__device__ __forceinline__ float2 apply5(const Weights5& k, float2 fm2, float2 fm1, float2 f0, float2 fp1, float2 fp2,
                                         float2 acc) {
  return fma2(k.m2, fm2, fma2(k.m1, fm1, fma2(k.c0, f0, fma2(k.p1, fp1, fma2(k.p2, fp2, acc)))));
}
__device__ __forceinline__ float2 apply5(const Weights5& k, float2 fm2, float2 fm1, float2 f0, float2 fp1, float2 fp2) {
  return fma2(k.m2, fm2, fma2(k.m1, fm1, fma2(k.c0, f0, fma2(k.p1, fp1, mul2(k.p2, fp2)))));
}

struct AdvectF2Maps {
  RowMaps f[3];         // stencil fields
  CUtensorMap base[3];  // (stage 2) point-wise fields, box {nx, TY, 1}
};

// Ring bytes: TY + 4 rows of the three fields per slot, in stage 2 also TY rows of u^n.
template <bool STAGE2, int TY, int NS>
constexpr size_t advect_f2_smem_bytes(int nx) {
  return (size_t)NS * (3 * (TY + 4) + (STAGE2 ? 3 * TY : 0)) * nx * sizeof(float) + PlaneRing<NS, 1, STAGE2 ? 6 : 3>::kBytes;
}

// STAGE2 false: out = f + dt A(f); true: out = 1/2 (f^n + f1 + dt A(f1)).
// blockDim.x * PPT * 2 == TY * nx (<= 512 threads).
// NXC: nx fixed at compile time (0: read from g): every shared-memory offset of
// the stencil is then an immediate on a per-thread base register.
template <bool STAGE2, int TY, int NS, int PPT, int NXC = 0>
__global__ void __launch_bounds__(512) k_advect_zq_f2(const __grid_constant__ AdvectF2Maps maps, const StreamGeom g,
                                                     float* __restrict__ ou, float* __restrict__ ov,
                                                     float* __restrict__ ow, DtArg dt, double h, double nu, double ux,
                                                     double uy, double uz, int* err) {
  pdl_entry();
  constexpr int G = 2;
  constexpr int ROWS = TY + 2 * G;
  constexpr int Q = 2 * G + 1;
  static_assert(TY >= G, "tile height must cover the halo depth");
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  const int nx = NXC ? NXC : g.nx, ny = g.ny, nz = g.nz, zc = g.zc;
  const int field_elems = ROWS * nx;
  const int stencil_elems = 3 * field_elems;
  const int slot_elems = stencil_elems + (STAGE2 ? 3 * TY * nx : 0);
  float* slots = reinterpret_cast<float*>(smem_raw);
  PlaneRing<NS, 1, STAGE2 ? 6 : 3> ring(smem_raw + (size_t)NS * slot_elems * sizeof(float), err);
  const int tid = threadIdx.x;
  const int PL = zc + 2 * G;
  auto issue = [&](int l, int s, int j, const ItemPos& p) {
    float* dst = slots + s * slot_elems;
    if (l < 3) {
      int z = p.z0 - G + j;
      z = z < 0 ? z + nz : (z >= nz ? z - nz : z);
      mbar_arrive_expect_tx(&ring.full[s], (uint32_t)(field_elems * sizeof(float)));
      tma_load_rows<G, TY>(dst + l * field_elems, maps.f[l], nx, ny, p.y0, z, &ring.full[s]);
    } else if (j >= 2 * G) {
      // u^n of the output plane completed by this load (< nz)
      mbar_arrive_expect_tx(&ring.full[s], (uint32_t)(TY * nx * sizeof(float)));
      tma_load_3d(dst + stencil_elems + (l - 3) * TY * nx, &maps.base[l - 3], 0, p.y0, p.z0 + j - 2 * G, &ring.full[s]);
    } else {
      mbar_arrive(&ring.full[s]);
    }
  };
  ring.start(item_pos(g, blockIdx.x, TY, zc), issue);

  const int mask = nx - 1;
  const int half = nx >> 1;
  int px[PPT], cy[PPT];  // even x of the pair, tile row
  int ctr[PPT], xl[PPT], xr[PPT];  // slot offsets: centre row, pairs at x -+ 2 in that row
#pragma unroll
  for (int i = 0; i < PPT; ++i) {
    const int pi = tid + i * blockDim.x;
    px[i] = (pi % half) * 2;
    cy[i] = pi / half;
    ctr[i] = (G + cy[i]) * nx + px[i];
    xl[i] = (G + cy[i]) * nx + ((px[i] - 2) & mask);
    xr[i] = (G + cy[i]) * nx + ((px[i] + 2) & mask);
  }
  const size_t plane = (size_t)nx * ny;
  const double dtv = dt.get();
  const float2 facA = splat2((float)(-dtv / (12 * h)));  // the 1/2 of the symmetric form folded in
  const float2 facD = splat2((float)((nu / h) * (dtv / h)));
  const float2 m2facD = splat2(-2.f * (float)((nu / h) * (dtv / h)));
  const float2 uinf[3] = {splat2((float)ux), splat2((float)uy), splat2((float)uz)};

  float2 qv[3][Q][PPT];
  float2 part[3][PPT];
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int d = 0; d < Q; ++d)
#pragma unroll
      for (int i = 0; i < PPT; ++i) qv[f][d][i] = splat2(0.f);
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int i = 0; i < PPT; ++i) part[f][i] = splat2(0.f);

  bool ok = true;
  ItemPos pos = item_pos(g, blockIdx.x, TY, zc);
  for (int item = blockIdx.x; item < g.n_items; item += gridDim.x) {
    const bool more = item + gridDim.x < g.n_items;
    const ItemPos nextp = item_pos(g, item + gridDim.x, TY, zc);
    size_t o[PPT];  // output index of the pair in the next plane
#pragma unroll
    for (int i = 0; i < PPT; ++i) o[i] = gidx(px[i], pos.y0 + cy[i], pos.z0, nx, ny);
    for (int j0 = 0; j0 < PL; j0 += Q) {
#pragma unroll
      for (int jj = 0; jj < Q; ++jj) {
        const int j = j0 + jj;
        if (j >= PL) break;
        if (ok) ok = ring.wait();
        if (ok) {
          const float* sl = slots + ring.slot * slot_elems;
          const int QN = jj;
#pragma unroll
          for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int i = 0; i < PPT; ++i)
              qv[f][QN][i] = *reinterpret_cast<const float2*>(sl + f * field_elems + ctr[i]);
          if (j >= 2 * G) {
            const int QC = (jj + 3 * Q - G) % Q;
            const int QM1 = (jj + 3 * Q - G - 1) % Q, QP1 = (jj + 3 * Q - G + 1) % Q;
            const int QM2 = (jj + 3 * Q - G - 2) % Q, QP2 = (jj + 3 * Q - G + 2) % Q;
#pragma unroll
            for (int i = 0; i < PPT; ++i) {
              const Weights5 kz = weights5(add2(qv[2][QC][i], uinf[2]), facA, facD, m2facD);
              float2 outv[3];
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                const float2 f0 = qv[f][QC][i];
                outv[f] = apply5(kz, qv[f][QM2][i], qv[f][QM1][i], f0, qv[f][QP1][i], qv[f][QP2][i],
                                 add2(f0, part[f][i]));
              }
              if constexpr (STAGE2) {
                const float* bs = sl + stencil_elems + cy[i] * nx + px[i];
#pragma unroll
                for (int f = 0; f < 3; ++f)
                  outv[f] = mul2(splat2(0.5f), add2(*reinterpret_cast<const float2*>(bs + f * TY * nx), outv[f]));
              }
              *reinterpret_cast<float2*>(ou + o[i]) = outv[0];
              *reinterpret_cast<float2*>(ov + o[i]) = outv[1];
              *reinterpret_cast<float2*>(ow + o[i]) = outv[2];
              o[i] += plane;
            }
          }
          // x/y partial of plane j - 1 (output plane j - 2G + 1)
          if (j >= 2 * G - 1 && j < PL - 1) {
            const float* sp = slots + ring.slot_back(1) * slot_elems;
            const int QX = (jj + Q - 1) % Q;
#pragma unroll
            for (int i = 0; i < PPT; ++i) {
              const Weights5 kx = weights5(add2(qv[0][QX][i], uinf[0]), facA, facD, m2facD);
              const Weights5 ky = weights5(add2(qv[1][QX][i], uinf[1]), facA, facD, m2facD);
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                const float* F = sp + f * field_elems;
                const float* Fc = F + ctr[i];
                const float2 c0 = qv[f][QX][i];
                const float2 A = *reinterpret_cast<const float2*>(F + xl[i]);
                const float2 B = *reinterpret_cast<const float2*>(F + xr[i]);
                const float2 ym2 = *reinterpret_cast<const float2*>(Fc - 2 * nx);
                const float2 ym1 = *reinterpret_cast<const float2*>(Fc - nx);
                const float2 yp1 = *reinterpret_cast<const float2*>(Fc + nx);
                const float2 yp2 = *reinterpret_cast<const float2*>(Fc + 2 * nx);
                // x: the pairs at x -+ 1 straddle A|c0 and c0|B, so their two
                // weights go in as scalar FMAs (no register shuffle)
                float2 acc = fma2(kx.m2, A, fma2(kx.c0, c0, fma2(kx.p2, B, apply5(ky, ym2, ym1, c0, yp1, yp2))));
                acc.x = fmaf(kx.m1.x, A.y, fmaf(kx.p1.x, c0.y, acc.x));
                acc.y = fmaf(kx.m1.y, c0.x, fmaf(kx.p1.y, B.x, acc.y));
                part[f][i] = acc;
              }
            }
          }
        }
        ring.step(ok, ring.n & 1, j, PL, pos, nextp, more, issue);
      }
    }
    pos = nextp;
  }
  ring.drain(ok);
}

}  // namespace cup
