// Discrete adjoint of one upwind3 stage in FP32 on x-pairs of cells with
// Blackwell's packed FP32x2 arithmetic: the operator of k_adjoint_zq (SCHEME 1)
// with the structure of k_advect_zq_f2.
//
// For a stage S(f) = f + facA sum_d a_d D_d(f) + facD Lap f with the adjoint g of
// its output (see adjoint.cuh), per cell and component q:
//   out_q = g_q + facD Lap(g_q) + facA sum_d T_d(a_d g_q, |a_d| g_q)
//           + facA sum_q' g_q' D'_q(f_q')            (the adjoint of a_q, q = d)
// with, along one direction and h(o) = a(o) g(o), k(o) = |a(o)| g(o):
//   2 T = (-h-2 + 8 h-1 - 8 h+1 + h+2) + (k-2 - 4 k-1 + 6 k0 - 4 k+1 + k+2)
// (as weights of the g, see TrW),
//   2 D'(f) = S(f) + sgn(a) Q(f),  S = f-2 - 8 f-1 + 8 f+1 - f+2,
//                                  Q = f-2 - 4 f-1 + 6 f0 - 4 f+1 + f+2,
// sgn(0) = 0 (the mean of the two one-sided slopes at the kink, as in
// up3_da). The 1/2 is folded into facA. A thread owns PPT pairs (x, x+1) of a
// TY x nx tile and marches down z: TMA ring of planes of the six fields (base
// f, adjoint input g; G = 2 halo rows), register queues of the last 5 planes
// of both, one x/y partial and the z part a plane later; LAM: out = alpha lam +
// beta (...), lam loaded at the end of the plane before its use. In x, the pairs at x -+ 2 come in whole and the values at
// x -+ 1 straddle two pairs, so the terms at -+1 go in as scalar FMAs.
#pragma once

#include "advect_f2.cuh"
#include "adjoint.cuh"

namespace cup {

// sgn(a) per lane: 1, -1 or 0
__device__ __forceinline__ float2 sgn2(float2 a) {
  return make_float2(a.x > 0.f ? 1.f : (a.x < 0.f ? -1.f : 0.f), a.y > 0.f ? 1.f : (a.y < 0.f ? -1.f : 0.f));
}

// The weights of 2 T along one direction. With h(o) = a(o) g(o) and k(o) =
// |a(o)| g(o), each sample enters as a weight of its own a alone times its g:
//   2 T = P-2 g-2 + P-1 g-1 + P0 g0 + P+1 g+1 + P+2 g+2,
//   P-2 = |a| - a, P-1 = 8 a - 4 |a|, P0 = 6 |a|, P+1 = -8 a - 4 |a|, P+2 = |a| + a,
// so the weights are formed once for the three components: 7 + 3 x 5 packed
// operations a direction where the products h and k took 3 x 16. The pass is
// bound by issue and the latency of its chains at 4 warps a scheduler: a
// 16-step gradient at 128^3 (32 such passes of 43 us) 7.70 -> 7.52 ms.
struct TrW {
  float2 m2, m1, c, p1, p2;
};
__device__ __forceinline__ TrW tr2_weights(float2 am2, float2 am1, float2 a0, float2 ap1, float2 ap2) {
  TrW w;
  w.m2 = sub2(abs2(am2), am2);
  w.m1 = fma2(splat2(-4.f), abs2(am1), mul2(splat2(8.f), am1));
  w.c = mul2(splat2(6.f), abs2(a0));
  w.p1 = fma2(splat2(-4.f), abs2(ap1), mul2(splat2(-8.f), ap1));
  w.p2 = add2(abs2(ap2), ap2);
  return w;
}
// 2 T along a direction whose five samples are whole pairs (y, z); the
// large weights first, whose partial sums cancel.
__device__ __forceinline__ float2 tr2_pairs(const TrW& w, float2 gm2, float2 gm1, float2 g0, float2 gp1, float2 gp2) {
  float2 t = fma2(w.p1, gp1, mul2(w.c, g0));
  t = fma2(w.m1, gm1, t);
  t = fma2(w.p2, gp2, t);
  return fma2(w.m2, gm2, t);
}

// S and Q of a field along a direction whose samples are whole pairs.
__device__ __forceinline__ void sq_pairs(float2 fm2, float2 fm1, float2 f0, float2 fp1, float2 fp2, float2& S,
                                         float2& Qs) {
  S = fma2(splat2(8.f), sub2(fp1, fm1), sub2(fm2, fp2));
  Qs = fma2(splat2(6.f), f0, fma2(splat2(-4.f), add2(fm1, fp1), add2(fm2, fp2)));
}

template <int TY, int NS>
constexpr size_t adjoint_f2_smem_bytes(int nx) {
  return (size_t)NS * 6 * (TY + 4) * nx * sizeof(float) + PlaneRing<NS, 1, 6>::kBytes;
}

// blockDim.x * PPT * 2 == TY * nx (<= 512 threads). NXC: nx fixed at compile
// time (0: read from g).
template <bool LAM, int TY, int NS, int PPT, int NXC = 0>
__global__ void __launch_bounds__(512) k_adjoint_zq_f2(const __grid_constant__ AdjointMaps maps, const StreamGeom g,
                                                      const float* lu, const float* lv, const float* lw, float* ou,
                                                      float* ov, float* ow, float alpha, float beta, DtArg dt,
                                                      double h, double nu, double ux, double uy, double uz, int* err) {
  pdl_entry();
  constexpr int G = 2;
  constexpr int ROWS = TY + 2 * G;
  constexpr int Q = 2 * G + 1;
  static_assert(TY >= G, "tile height must cover the halo depth");
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  const int nx = NXC ? NXC : g.nx, ny = g.ny, nz = g.nz, zc = g.zc;
  const int field_elems = ROWS * nx;
  const int slot_elems = 6 * field_elems;
  float* slots = reinterpret_cast<float*>(smem_raw);
  PlaneRing<NS, 1, 6> ring(smem_raw + (size_t)NS * slot_elems * sizeof(float), err);
  const int tid = threadIdx.x;
  const int PL = zc + 2 * G;
  auto issue = [&](int f, int s, int j, const ItemPos& p) {
    int z = p.z0 - G + j;
    z = z < 0 ? z + nz : (z >= nz ? z - nz : z);
    mbar_arrive_expect_tx(&ring.full[s], (uint32_t)(field_elems * sizeof(float)));
    tma_load_rows<G, TY>(slots + s * slot_elems + f * field_elems, maps.f[f], nx, ny, p.y0, z, &ring.full[s]);
  };
  ring.start(item_pos(g, blockIdx.x, TY, zc), issue);

  const int mask = nx - 1;
  const int half = nx >> 1;
  int px[PPT], cy[PPT];
  int ctr[PPT], xl[PPT], xr[PPT];  // slot offsets: the pair, the pairs at x -+ 2
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
  const float2 facA = splat2((float)(-dtv / (12 * h)));  // facA of the stage with the 1/2 of T and D' folded in
  const float2 facD = splat2((float)((nu / h) * (dtv / h)));
  const float2 uinf[3] = {splat2((float)ux), splat2((float)uy), splat2((float)uz)};
  const float2 alpha2 = splat2(alpha), beta2 = splat2(beta);

  float2 qf[3][Q][PPT];  // base field pairs, plane j in slot j % Q
  float2 qg[3][Q][PPT];  // adjoint input pairs
  float2 part[3][PPT];
  float2 lam[LAM ? 3 : 1][PPT];  // point-wise lam of the next output plane
  const float* lsrc[3] = {lu, lv, lw};
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int d = 0; d < Q; ++d)
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        qf[f][d][i] = splat2(0.f);
        qg[f][d][i] = splat2(0.f);
      }
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int i = 0; i < PPT; ++i) part[f][i] = splat2(0.f);

  bool ok = true;
  ItemPos pos = item_pos(g, blockIdx.x, TY, zc);
  for (int item = blockIdx.x; item < g.n_items; item += gridDim.x) {
    const bool more = item + gridDim.x < g.n_items;
    const ItemPos nextp = item_pos(g, item + gridDim.x, TY, zc);
    size_t o[PPT];  // output index of the next plane
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
            for (int i = 0; i < PPT; ++i) {
              qf[f][QN][i] = *reinterpret_cast<const float2*>(sl + f * field_elems + ctr[i]);
              qg[f][QN][i] = *reinterpret_cast<const float2*>(sl + (3 + f) * field_elems + ctr[i]);
            }
          // z terms and output of plane k = j - 2G
          if (j >= 2 * G) {
            const int QC = (jj + 3 * Q - G) % Q;
            const int QM1 = (jj + 3 * Q - G - 1) % Q, QP1 = (jj + 3 * Q - G + 1) % Q;
            const int QM2 = (jj + 3 * Q - G - 2) % Q, QP2 = (jj + 3 * Q - G + 2) % Q;
#pragma unroll
            for (int i = 0; i < PPT; ++i) {
              const float2 am2 = add2(qf[2][QM2][i], uinf[2]), am1 = add2(qf[2][QM1][i], uinf[2]);
              const float2 a0 = add2(qf[2][QC][i], uinf[2]);
              const float2 ap1 = add2(qf[2][QP1][i], uinf[2]), ap2 = add2(qf[2][QP2][i], uinf[2]);
              // adjoint of a_z at the cell: sum_q' g_q' D'_z(f_q')
              float2 sS = splat2(0.f), sQ = splat2(0.f);
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                float2 S, Qs;
                sq_pairs(qf[f][QM2][i], qf[f][QM1][i], qf[f][QC][i], qf[f][QP1][i], qf[f][QP2][i], S, Qs);
                sS = fma2(qg[f][QC][i], S, sS);
                sQ = fma2(qg[f][QC][i], Qs, sQ);
              }
              const float2 advz = fma2(sgn2(a0), sQ, sS);
              const TrW wz = tr2_weights(am2, am1, a0, ap1, ap2);
              float2 outv[3];
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                const float2 g0 = qg[f][QC][i];
                const float2 tz = tr2_pairs(wz, qg[f][QM2][i], qg[f][QM1][i], g0, qg[f][QP1][i], qg[f][QP2][i]);
                // Lap_z with the centre's -6 g0
                const float2 lz = fma2(splat2(-6.f), g0, add2(qg[f][QM1][i], qg[f][QP1][i]));
                float2 v = fma2(facD, lz, fma2(facA, tz, part[f][i]));
                if (f == 2) v = fma2(facA, advz, v);
                outv[f] = v;
              }
              if constexpr (LAM) {
#pragma unroll
                for (int f = 0; f < 3; ++f) outv[f] = fma2(alpha2, lam[f][i], mul2(beta2, outv[f]));
              } else {
#pragma unroll
                for (int f = 0; f < 3; ++f) outv[f] = mul2(beta2, outv[f]);
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
              const float* Fx = sp;                // base u (advects in x)
              const float* Fy = sp + field_elems;  // base v (advects in y)
              const int c = ctr[i];
              // advecting velocities: x at x-2..x+3 (pairs A, C, B), y at rows -2..2
              const float2 axA = add2(*reinterpret_cast<const float2*>(Fx + xl[i]), uinf[0]);
              const float2 axC = add2(qf[0][QX][i], uinf[0]);
              const float2 axB = add2(*reinterpret_cast<const float2*>(Fx + xr[i]), uinf[0]);
              const float2 aym2 = add2(*reinterpret_cast<const float2*>(Fy + c - 2 * nx), uinf[1]);
              const float2 aym1 = add2(*reinterpret_cast<const float2*>(Fy + c - nx), uinf[1]);
              const float2 ay0 = add2(qf[1][QX][i], uinf[1]);
              const float2 ayp1 = add2(*reinterpret_cast<const float2*>(Fy + c + nx), uinf[1]);
              const float2 ayp2 = add2(*reinterpret_cast<const float2*>(Fy + c + 2 * nx), uinf[1]);
              // in x the samples at -+1 straddle two pairs: m1, p1 are the weights of each lane's own
              const float2 w0 = mul2(splat2(6.f), abs2(axC));
              const float2 wm2 = sub2(abs2(axA), axA), wp2 = add2(abs2(axB), axB);
              const float2 wm1 = make_float2(fmaf(-4.f, fabsf(axA.y), 8.f * axA.y), fmaf(-4.f, fabsf(axC.x), 8.f * axC.x));
              const float2 wp1 = make_float2(fmaf(-4.f, fabsf(axC.y), -8.f * axC.y), fmaf(-4.f, fabsf(axB.x), -8.f * axB.x));
              const TrW wy = tr2_weights(aym2, aym1, ay0, ayp1, ayp2);
              // adjoints of a_x, a_y at the cell: sum_q' g_q' D'(f_q'), as S and Q sums
              float2 sSx = splat2(0.f), sQx = splat2(0.f), sSy = splat2(0.f), sQy = splat2(0.f);
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                const float* F = sp + f * field_elems;
                const float2 fA = *reinterpret_cast<const float2*>(F + xl[i]);
                const float2 fC = qf[f][QX][i];
                const float2 fB = *reinterpret_cast<const float2*>(F + xr[i]);
                const float2 gq = qg[f][QX][i];
                // x: S = f-2 - 8 f-1 + 8 f+1 - f+2, Q = f-2 - 4 f-1 + 6 f0 - 4 f+1 + f+2
                float2 Sx = sub2(fA, fB);  // the -+2 terms of each lane
                Sx.x = fmaf(8.f, fC.y - fA.y, Sx.x);
                Sx.y = fmaf(8.f, fB.x - fC.x, Sx.y);
                float2 Qx = fma2(splat2(6.f), fC, add2(fA, fB));
                Qx.x = fmaf(-4.f, fA.y + fC.y, Qx.x);
                Qx.y = fmaf(-4.f, fC.x + fB.x, Qx.y);
                float2 Sy, Qy;
                sq_pairs(*reinterpret_cast<const float2*>(F + c - 2 * nx), *reinterpret_cast<const float2*>(F + c - nx),
                         fC, *reinterpret_cast<const float2*>(F + c + nx),
                         *reinterpret_cast<const float2*>(F + c + 2 * nx), Sy, Qy);
                sSx = fma2(gq, Sx, sSx);
                sQx = fma2(gq, Qx, sQx);
                sSy = fma2(gq, Sy, sSy);
                sQy = fma2(gq, Qy, sQy);
              }
              const float2 advx = fma2(sgn2(axC), sQx, sSx);
              const float2 advy = fma2(sgn2(ay0), sQy, sSy);
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                const float* Gf = sp + (3 + f) * field_elems;
                const float2 gA = *reinterpret_cast<const float2*>(Gf + xl[i]);
                const float2 g0 = qg[f][QX][i];
                const float2 gB = *reinterpret_cast<const float2*>(Gf + xr[i]);
                const float2 gym2 = *reinterpret_cast<const float2*>(Gf + c - 2 * nx);
                const float2 gym1 = *reinterpret_cast<const float2*>(Gf + c - nx);
                const float2 gyp1 = *reinterpret_cast<const float2*>(Gf + c + nx);
                const float2 gyp2 = *reinterpret_cast<const float2*>(Gf + c + 2 * nx);
                // x transport
                float2 tx = mul2(w0, g0);
                tx.x = fmaf(wp1.x, g0.y, tx.x);
                tx.y = fmaf(wp1.y, gB.x, tx.y);
                tx.x = fmaf(wm1.x, gA.y, tx.x);
                tx.y = fmaf(wm1.y, g0.x, tx.y);
                tx = fma2(wm2, gA, fma2(wp2, gB, tx));
                const float2 ty = tr2_pairs(wy, gym2, gym1, g0, gyp1, gyp2);
                // Lap in x and y without the centre (the z part adds -6 g0)
                float2 lxy = add2(add2(gym1, gyp1), make_float2(gA.y + g0.y, g0.x + gB.x));
                float2 v = fma2(facD, lxy, fma2(facA, add2(tx, ty), g0));
                if (f == 0) v = fma2(facA, advx, v);
                if (f == 1) v = fma2(facA, advy, v);
                part[f][i] = v;
              }
            }
            if constexpr (LAM) {
              // of output plane j - 2G + 1, finished by the next plane
#pragma unroll
              for (int i = 0; i < PPT; ++i)
#pragma unroll
                for (int f = 0; f < 3; ++f) lam[f][i] = *reinterpret_cast<const float2*>(lsrc[f] + o[i]);
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
