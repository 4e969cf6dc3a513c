// Discrete adjoint of one explicit advection-diffusion stage
// S(f) = f + facA sum_d a_d D_d(f) + facD Lap(f), a_d = f_d + uinf_d, the stage
// of KernelAdvectDiffuse (source/operators/AdvectionDiffusion.cpp:111-144) or
// of the upwind3 + RK2 scheme. The reference has no adjoint; this is new.
//
// For upwind3, a D(f) with the sign-selected stencil equals
// 1/2 (a S(f) + |a| Q(f)), S(f) = f-2 - 8f-1 + 8f+1 - f+2 (antisymmetric) and
// Q(f) = f-2 - 4f-1 + 6f0 - 4f+1 + f+2 (symmetric), so with the signs frozen at
// the base state the transpose of the transport part is
// 1/2 (-S(a g) + Q(|a| g)): a stencil of point-wise products, no scatter.
// For the central scheme a D(f) = a (f+1 - f-1) and its transpose is
// (a g)-1 - (a g)+1. With g the adjoint of the stage output:
//   S'(f)^T g = g + facD Lap(g) + facA sum_d T_d^T(a_d g)
//               + facA e_q sum_q' g_q' D_q(f_q')        (a_q's own adjoint)
// and the kernel writes out = alpha lam + beta S'(f)^T g (lam point-wise).
//
// Structure as k_advect_zq: TMA ring of planes (base f and g with G halo
// rows), register queues of the last 2G+1 planes of f and g, one x/y partial,
// z terms at output; lam is loaded at the end of the plane before its use.
#pragma once

#include "advect.cuh"

namespace cup {

struct AdjointMaps {
  RowMaps f[6];         // f (3) then g (3)
};

template <typename T, int SCHEME, int TY, int NS>
constexpr size_t adjoint_smem_bytes(int nx) {
  constexpr int G = SCHEME == 0 ? 1 : 2;
  return (size_t)NS * 6 * (TY + 2 * G) * nx * sizeof(T) + PlaneRing<NS, G - 1, 6>::kBytes;
}

// transpose of the transport stencil at one point from the 5 products
// h(o) = a(o) g(o) and k(o) = |a(o)| g(o), o = -2..2 (upwind3) or the 2 products
// h(-1), h(+1) (central).
template <typename T>
__device__ __forceinline__ T tabs(T x) {
  return x < (T)0 ? -x : x;
}

// Derivative of a up3(a; f) with respect to a (the adjoint of the advecting
// velocity): up3(a; f) off a = 0; at a = 0, where the one-sided derivatives
// are the two upwind stencils, their mean (f-2 - 8 f-1 + 8 f+1 - f+2) / 2, the
// value central differences see (a flow started from rest has a_y = a_z = 0
// in every cell of its first step).
template <typename T>
__device__ __forceinline__ T up3_da(T a, T fm2, T fm1, T f0, T fp1, T fp2) {
  if (a == (T)0) return (T)0.5 * (fm2 - (T)8 * fm1 + (T)8 * fp1 - fp2);
  return up3(a, fm2, fm1, f0, fp1, fp2);
}

template <typename T>
__device__ __forceinline__ T tr_up3(T hm2, T hm1, T hp1, T hp2, T km2, T km1, T k0, T kp1, T kp2) {
  return (T)0.5 * ((-hm2 + (T)8 * hm1 - (T)8 * hp1 + hp2) + (km2 - (T)4 * km1 + (T)6 * k0 - (T)4 * kp1 + kp2));
}

template <typename T, int SCHEME, bool LAM, int TY, int NS, int CPT>
__global__ void __launch_bounds__(512) k_adjoint_zq(const __grid_constant__ AdjointMaps maps, const StreamGeom g,
                                                   const T* lu, const T* lv, const T* lw, T* ou, T* ov, T* ow,
                                                   T alpha, T beta, DtArg dt, double h, double nu, double ux,
                                                   double uy, double uz, int* err) {
  pdl_entry();
  constexpr int G = SCHEME == 0 ? 1 : 2;
  constexpr int ROWS = TY + 2 * G;
  constexpr int Q = 2 * G + 1;
  // a G-row halo box starting at y0 - G (wrapped) stays inside [0, ny) only if y0 is a multiple of TY >= G
  static_assert(TY >= G, "tile height must cover the halo depth");
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  const int nx = g.nx, ny = g.ny, nz = g.nz, zc = g.zc;
  static_assert(NS > G, "the ring must hold the planes in use and one in flight");
  const int field_elems = ROWS * nx;
  const int slot_elems = 6 * field_elems;
  T* slots = reinterpret_cast<T*>(smem_raw);
  PlaneRing<NS, G - 1, 6> ring(smem_raw + (size_t)NS * slot_elems * sizeof(T), err);
  const int tid = threadIdx.x;
  const int PL = zc + 2 * G;
  auto issue = [&](int f, int s, int j, const ItemPos& p) {
    int z = p.z0 - G + j;
    z = z < 0 ? z + nz : (z >= nz ? z - nz : z);
    mbar_arrive_expect_tx(&ring.full[s], (uint32_t)(field_elems * sizeof(T)));
    tma_load_rows<G, TY>(slots + s * slot_elems + f * field_elems, maps.f[f], nx, ny, p.y0, z, &ring.full[s]);
  };
  ring.start(item_pos(g, blockIdx.x, TY, zc), issue);

  const int mask = nx - 1;
  int cx[CPT], cy[CPT];
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int c = tid + i * blockDim.x;
    cx[i] = c & mask;
    cy[i] = c >> g.log2nx;
  }
  const double dtv = dt.get();
  const T facA = (T)(SCHEME == 0 ? -dtv / (2 * h) : -dtv / (6 * h));
  const T facD = (T)((nu / h) * (dtv / h));
  const T uinf[3] = {(T)ux, (T)uy, (T)uz};

  T qf[3][Q][CPT];  // base field centre values, plane j in slot j % Q
  T qg[3][Q][CPT];  // adjoint input centre values
  T part[3][CPT];
  T lam[LAM ? 3 : 1][CPT];  // point-wise lam of the next output plane
  const T* lsrc[3] = {lu, lv, lw};
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int d = 0; d < Q; ++d)
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        qf[f][d][i] = (T)0;
        qg[f][d][i] = (T)0;
      }
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int i = 0; i < CPT; ++i) part[f][i] = (T)0;

  bool ok = true;
  ItemPos pos = item_pos(g, blockIdx.x, TY, zc);
  for (int item = blockIdx.x; item < g.n_items; item += gridDim.x) {
    const bool more = item + gridDim.x < g.n_items;
    const ItemPos nextp = item_pos(g, item + gridDim.x, TY, zc);
    size_t o[CPT];  // output index of the next plane
#pragma unroll
    for (int i = 0; i < CPT; ++i) o[i] = gidx(cx[i], pos.y0 + cy[i], pos.z0, nx, ny);
    for (int j0 = 0; j0 < PL; j0 += Q) {
#pragma unroll
      for (int jj = 0; jj < Q; ++jj) {
        const int j = j0 + jj;
        if (j >= PL) break;
        if (ok) ok = ring.wait();
        if (ok) {
          const T* sl = slots + ring.slot * slot_elems;
          const int QN = jj;
#pragma unroll
          for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int i = 0; i < CPT; ++i) {
              const int off = (G + cy[i]) * nx + cx[i];
              qf[f][QN][i] = sl[f * field_elems + off];
              qg[f][QN][i] = sl[(3 + f) * field_elems + off];
            }
          // z terms and output of plane k = j - 2G
          if (j >= 2 * G) {
            const int QC = (jj + 3 * Q - G) % Q;
            const int QM1 = (jj + 3 * Q - G - 1) % Q, QP1 = (jj + 3 * Q - G + 1) % Q;
            const int QM2 = (jj + 3 * Q - G - 2) % Q, QP2 = (jj + 3 * Q - G + 2) % Q;
#pragma unroll
            for (int i = 0; i < CPT; ++i) {
              const T azc = qf[2][QC][i] + uinf[2];
              // adjoint of a_z at the cell: sum_q' g_q' D_z(f_q')
              T advz = (T)0;
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                T dz;
                if constexpr (SCHEME == 0) dz = qf[f][QP1][i] - qf[f][QM1][i];
                else dz = up3_da(azc, qf[f][QM2][i], qf[f][QM1][i], qf[f][QC][i], qf[f][QP1][i], qf[f][QP2][i]);
                advz += qg[f][QC][i] * dz;
              }
              T outv[3];
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                const T g0 = qg[f][QC][i];
                T tz;
                if constexpr (SCHEME == 0) {
                  tz = (qf[2][QM1][i] + uinf[2]) * qg[f][QM1][i] - (qf[2][QP1][i] + uinf[2]) * qg[f][QP1][i];
                } else {
                  const T am2 = qf[2][QM2][i] + uinf[2], am1 = qf[2][QM1][i] + uinf[2];
                  const T ap1 = qf[2][QP1][i] + uinf[2], ap2 = qf[2][QP2][i] + uinf[2];
                  tz = tr_up3(am2 * qg[f][QM2][i], am1 * qg[f][QM1][i], ap1 * qg[f][QP1][i], ap2 * qg[f][QP2][i],
                              tabs(am2) * qg[f][QM2][i], tabs(am1) * qg[f][QM1][i], tabs(azc) * g0,
                              tabs(ap1) * qg[f][QP1][i], tabs(ap2) * qg[f][QP2][i]);
                }
                T v = part[f][i] + facD * (qg[f][QM1][i] + qg[f][QP1][i] - g0 * 6) + facA * tz;
                if (f == 2) v += facA * advz;
                outv[f] = v;
              }
              if constexpr (LAM) {
#pragma unroll
                for (int f = 0; f < 3; ++f) outv[f] = alpha * lam[f][i] + beta * outv[f];
              } else {
#pragma unroll
                for (int f = 0; f < 3; ++f) outv[f] = beta * outv[f];
              }
              ou[o[i]] = outv[0];
              ov[o[i]] = outv[1];
              ow[o[i]] = outv[2];
              o[i] += (size_t)nx * ny;
            }
          }
          // x/y partial of plane j - G + 1 (output plane j - 2G + 1)
          if (j >= 2 * G - 1 && j < PL - 1) {
            const T* sp = slots + ring.slot_back(G - 1) * slot_elems;
            const int QX = (jj + Q - G + 1) % Q;
#pragma unroll
            for (int i = 0; i < CPT; ++i) {
              const int x = cx[i], r = G + cy[i];
              const int xm1 = (x - 1) & mask, xp1 = (x + 1) & mask, xm2 = (x - 2) & mask, xp2 = (x + 2) & mask;
              const T* Fx = sp;                    // base u (advects in x)
              const T* Fy = sp + field_elems;      // base v (advects in y)
              const T ax0 = qf[0][QX][i] + uinf[0], ay0 = qf[1][QX][i] + uinf[1];
              // adjoints of a_x, a_y at the cell: sum_q' g_q' D(f_q')
              T advx = (T)0, advy = (T)0;
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                const T* F = sp + f * field_elems;
                const T f0 = qf[f][QX][i], gq = qg[f][QX][i];
                T dx, dy;
                if constexpr (SCHEME == 0) {
                  dx = F[r * nx + xp1] - F[r * nx + xm1];
                  dy = F[(r + 1) * nx + x] - F[(r - 1) * nx + x];
                } else {
                  dx = up3_da(ax0, F[r * nx + xm2], F[r * nx + xm1], f0, F[r * nx + xp1], F[r * nx + xp2]);
                  dy = up3_da(ay0, F[(r - 2) * nx + x], F[(r - 1) * nx + x], f0, F[(r + 1) * nx + x], F[(r + 2) * nx + x]);
                }
                advx += gq * dx;
                advy += gq * dy;
              }
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                const T* Gf = sp + (3 + f) * field_elems;
                const T g0 = qg[f][QX][i];
                const T gxm1 = Gf[r * nx + xm1], gxp1 = Gf[r * nx + xp1];
                const T gym1 = Gf[(r - 1) * nx + x], gyp1 = Gf[(r + 1) * nx + x];
                T tx, ty;
                if constexpr (SCHEME == 0) {
                  tx = (Fx[r * nx + xm1] + uinf[0]) * gxm1 - (Fx[r * nx + xp1] + uinf[0]) * gxp1;
                  ty = (Fy[(r - 1) * nx + x] + uinf[1]) * gym1 - (Fy[(r + 1) * nx + x] + uinf[1]) * gyp1;
                } else {
                  const T gxm2 = Gf[r * nx + xm2], gxp2 = Gf[r * nx + xp2];
                  const T gym2 = Gf[(r - 2) * nx + x], gyp2 = Gf[(r + 2) * nx + x];
                  const T axm2 = Fx[r * nx + xm2] + uinf[0], axm1 = Fx[r * nx + xm1] + uinf[0];
                  const T axp1 = Fx[r * nx + xp1] + uinf[0], axp2 = Fx[r * nx + xp2] + uinf[0];
                  const T aym2 = Fy[(r - 2) * nx + x] + uinf[1], aym1 = Fy[(r - 1) * nx + x] + uinf[1];
                  const T ayp1 = Fy[(r + 1) * nx + x] + uinf[1], ayp2 = Fy[(r + 2) * nx + x] + uinf[1];
                  tx = tr_up3(axm2 * gxm2, axm1 * gxm1, axp1 * gxp1, axp2 * gxp2, tabs(axm2) * gxm2,
                              tabs(axm1) * gxm1, tabs(ax0) * g0, tabs(axp1) * gxp1, tabs(axp2) * gxp2);
                  ty = tr_up3(aym2 * gym2, aym1 * gym1, ayp1 * gyp1, ayp2 * gyp2, tabs(aym2) * gym2,
                              tabs(aym1) * gym1, tabs(ay0) * g0, tabs(ayp1) * gyp1, tabs(ayp2) * gyp2);
                }
                T v = g0 + facD * (gyp1 + gym1 + gxp1 + gxm1) + facA * (tx + ty);
                if (f == 0) v += facA * advx;
                if (f == 1) v += facA * advy;
                part[f][i] = v;
              }
            }
            if constexpr (LAM) {
              // of output plane j - 2G + 1, finished by the next plane
#pragma unroll
              for (int i = 0; i < CPT; ++i)
#pragma unroll
                for (int f = 0; f < 3; ++f) lam[f][i] = lsrc[f][o[i]];
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
