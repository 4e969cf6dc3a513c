// KernelGradP (source/operators/PressureProjection.cpp:38-50) in the z-queue
// form: out = in - dt / 2h grad_c p, p FP64, the velocity in the storage type T
// (out may be in). Planes of p (TY + 2 rows) and the velocity rows of the output
// plane they complete arrive by TMA through a PlaneRing; the centre values of
// the last 3 planes of p sit in registers, the x and y differences of a plane
// are taken on its arrival. (The plane-streaming form it replaces read the
// velocity with plain loads, which its warps then waited for: FP64 at 256^3 194
// us, now 155 = 6.1 TB/s at 56 B/cell; the FP32 adjoint's gradient at
// 256x128x128 50 us, now 19.)
// REDUCE: per-CTA FP64 partials of max |u + uinf| (the next calcMaxTimestep,
// source/operators/ProcessHelpers.h:74-99) over cells outside the obstacle box
// (the penalization kernel covers the box) and of the kinetic energy sum
// |u|^2/2 (ComputeDissipation.cpp:47-116 pattern).
#pragma once

#include "common.cuh"
#include "ops.cuh"
#include "stencil.cuh"

namespace cup {

struct GradMaps {
  RowMaps p;         // FP64, 1 halo row
  CUtensorMap f[3];  // velocity in, box {nx, TY, 1}
};

struct GradParams {
  DtArg dt;
  double h;
  double uinf[3];
  Box box;
  int has_box;
};

constexpr int kGradLoads = 4;  // loads of a plane: p, u, v, w

template <typename T, int TY>
constexpr size_t grad_slot_bytes(int nx) {
  return (size_t)(TY + 2) * nx * sizeof(double) + (size_t)3 * TY * nx * sizeof(T);
}
template <typename T, int TY, int NS>
constexpr size_t grad_smem_bytes(int nx) {
  return NS * grad_slot_bytes<T, TY>(nx) + PlaneRing<NS, 0, kGradLoads>::kBytes + 2 * 32 * sizeof(double);
}

// blockDim.x * CPT == TY * nx (<= 512 threads).
template <typename T, bool REDUCE, int TY, int NS, int CPT, int NXC = 0>
__global__ void __launch_bounds__(512) k_grad_zq(const __grid_constant__ GradMaps maps, const StreamGeom g, T* ou, T* ov,
                                                T* ow, double* partials, const GradParams prm, int* err) {
  pdl_entry();
  constexpr int G = 1, Q = 3;
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  const int nx = NXC ? NXC : g.nx, ny = g.ny, nz = g.nz, zc = g.zc;
  const int slot_bytes = (int)grad_slot_bytes<T, TY>(nx), f_off = (TY + 2) * nx * (int)sizeof(double);
  const int f_bytes = TY * nx * (int)sizeof(T);
  PlaneRing<NS, 0, kGradLoads> ring(smem_raw + NS * slot_bytes, err);
  double* scratch = reinterpret_cast<double*>(smem_raw + NS * slot_bytes + PlaneRing<NS, 0, kGradLoads>::kBytes);
  const int tid = threadIdx.x;
  const int PL = zc + 2 * G;
  auto issue = [&](int l, int s, int j, const ItemPos& p) {
    unsigned char* dst = smem_raw + s * slot_bytes;
    if (l == 0) {
      int z = p.z0 - G + j;
      z = z < 0 ? z + nz : (z >= nz ? z - nz : z);
      mbar_arrive_expect_tx(&ring.full[s], (uint32_t)f_off);
      tma_load_rows<G, TY>(reinterpret_cast<double*>(dst), maps.p, nx, ny, p.y0, z, &ring.full[s]);
    } else if (j >= 2 * G) {
      // the velocity of the output plane completed by this load (< nz)
      mbar_arrive_expect_tx(&ring.full[s], (uint32_t)f_bytes);
      tma_load_3d(dst + f_off + (l - 1) * f_bytes, &maps.f[l - 1], 0, p.y0, p.z0 + j - 2 * G, &ring.full[s]);
    } else {
      mbar_arrive(&ring.full[s]);
    }
  };
  ring.start(item_pos(g, blockIdx.x, TY, zc), issue);

  const int mask = nx - 1;
  int cx[CPT], cy[CPT];
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int c = tid + i * blockDim.x;
    cx[i] = c & mask;
    cy[i] = NXC ? c / NXC : c >> g.log2nx;
  }
  const double fac = -0.5 * prm.dt.get() / prm.h;
  double pq[Q][CPT];               // centre values of the last planes, plane j in slot j % Q
  double gx[CPT], gy[CPT];         // differences of the plane before
  double vmax = 0.0, ke = 0.0;
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    gx[i] = gy[i] = 0.0;
#pragma unroll
    for (int d = 0; d < Q; ++d) pq[d][i] = 0.0;
  }
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
          const unsigned char* sl = smem_raw + ring.slot * slot_bytes;
          const double* P = reinterpret_cast<const double*>(sl);
          const T* F = reinterpret_cast<const T*>(sl + f_off);
#pragma unroll
          for (int i = 0; i < CPT; ++i) {
            const double* Pc = P + (G + cy[i]) * nx;
            pq[jj][i] = Pc[cx[i]];
            if (j >= 2 * G) {  // output plane j - 2
              const int c = cy[i] * nx + cx[i];
              const T tu = (T)((double)F[c] + fac * gx[i]);
              const T tv = (T)((double)F[TY * nx + c] + fac * gy[i]);
              const T tw = (T)((double)F[2 * TY * nx + c] + fac * (pq[jj][i] - pq[(jj + 1) % Q][i]));
              ou[o[i]] = tu;
              ov[o[i]] = tv;
              ow[o[i]] = tw;
              o[i] += (size_t)nx * ny;
              if constexpr (REDUCE) {
                if (!(prm.has_box && prm.box.contains(cx[i], pos.y0 + cy[i], pos.z0 + j - 2 * G, nx, ny, nz)))
                  vmax = fmax(vmax, fmax(fmax(fabs((double)tu + prm.uinf[0]), fabs((double)tv + prm.uinf[1])),
                                         fabs((double)tw + prm.uinf[2])));
                ke += 0.5 * ((double)tu * tu + (double)tv * tv + (double)tw * tw);
              }
            }
            if (j >= G && j < G + zc) {
              gx[i] = Pc[(cx[i] + 1) & mask] - Pc[(cx[i] - 1) & mask];
              gy[i] = Pc[nx + cx[i]] - Pc[cx[i] - nx];
            }
          }
        }
        ring.step(ok, ring.n & 1, j, PL, pos, nextp, more, issue);
      }
    }
    pos = nextp;
  }
  ring.drain(ok);
  if constexpr (REDUCE) {
    __syncthreads();
    double mx[1] = {vmax}, sm[1] = {ke};
    block_reduce<1, true>(mx, scratch);
    block_reduce<1, false>(sm, scratch + 32);
    if (tid == 0) {
      partials[2 * blockIdx.x + 0] = mx[0];
      partials[2 * blockIdx.x + 1] = sm[0];
    }
  }
}

}  // namespace cup
