// Advection-diffusion kernels with register z-queues (KernelAdvectDiffuse,
// source/operators/AdvectionDiffusion.cpp:111-144, and the upwind3 + RK2
// stages), the device replacement of Operator::compute's block/lab loop
// (source/operators/Operator.h:112-170) for this operator.
//
// Each thread owns CPT fixed (x, y) columns of a TY x nx row tile and marches
// down z. Planes arrive by TMA into a ring of NS shared-memory slots (TY main
// rows plus G periodic halo rows per field; the x halo is the row's periodic
// wrap; PlaneRing). When plane j lands, a thread
//   1. pushes its columns' centre values into a register queue of the last
//      2G+1 planes (the z stencil),
//   2. finishes output plane j-2G: adds the z terms (from the queue) to that
//      plane's x/y partial, and stores it,
//   3. computes the x/y partial of output plane j-2G+1, plane j-G+1 of the
//      stream (x/y neighbours from its slot, advecting velocity from the
//      queue), and releases the slot of that plane,
// so one partial per column is alive and only G planes are held in shared
// memory. For RK2 stage 2 the point-wise base values u^n are loaded at the end
// of the plane before their use. Work items (TY rows x ZC planes) of a CTA form
// one flat load stream, so the pipeline never drains between items.
//
// The upwind3 stages were bound by the FP64 pipe (about 130 FP64 instructions
// per cell with both one-sided stencils evaluated) and by shared-memory reads.
// Their update is written with four taps per direction whose weights depend on
// the advecting velocity a only, with B = dt |a| / 6h and D = nu dt / h^2:
//   upwind neighbour 6 B + D, downwind neighbour D - 2 B, second upwind cell -B,
//   centre -3 B - 2 D,
// so the three components share them and a tap costs one FMA (about 50 FP64
// instructions per cell); the neighbours swap weights with the sign of a, the
// second upwind cell is one select (x: of its address). A thread's two columns
// are two rows of one x (six row loads serve both). SELECT: both one-sided
// stencils instead, for runs that amplify rounding (amplifies_rounding in
// cup_b200.cu has the rule); bound by the FP64 pipe again, stage 1 203 us instead
// of 169 at 256^3, stage 2 232 instead of 208.
#pragma once

#include "common.cuh"
#include "ops.cuh"
#include "stencil.cuh"

namespace cup {

struct AdvectMaps {
  RowMaps f[3];  // stencil fields
};

// SCHEME 0: central2 (reference) Euler; 1: upwind3 stage 1; 2: upwind3 stage 2.
template <int SCHEME>
struct AdvectTraits {
  static constexpr int G = SCHEME == 0 ? 1 : 2;
};

template <typename T, int SCHEME, int TY, int NS>
constexpr size_t advect_smem_bytes(int nx) {
  return (size_t)NS * 3 * (TY + 2 * AdvectTraits<SCHEME>::G) * nx * sizeof(T) +
         PlaneRing<NS, AdvectTraits<SCHEME>::G - 1, 3>::kBytes;
}

// The weights of one direction of an upwind3 update (see the head of the file):
// m1, p1 of the neighbours at -1 and +1, far = -B of the second upwind cell.
template <typename T>
struct UpW {
  T m1, p1, far;
  bool pos;
};
template <typename T>
__device__ __forceinline__ UpW<T> up_weights(T a, T absA, T facD) {
  const T B = absA * fabs(a);
  const T wu = (T)6 * B + facD, wd = facD - (T)2 * B;
  UpW<T> w;
  w.pos = a > (T)0;
  w.m1 = w.pos ? wu : wd;
  w.p1 = w.pos ? wd : wu;
  w.far = -B;
  return w;
}

// The pieces of the SELECT form, FP64, with every rounding spelled out: left to
// the compiler, which products are fused depends on the code around them.
// The one-sided difference of a's sign (up3).
__device__ __forceinline__ double up3_rn(double a, double fm2, double fm1, double f0, double fp1, double fp2) {
  const double p = __dadd_rn(__fma_rn(-6.0, fm1, __fma_rn(3.0, f0, __dmul_rn(2.0, fp1))), fm2);
  const double n = __fma_rn(-2.0, fm1, __fma_rn(-3.0, f0, __fma_rn(6.0, fp1, -fp2)));
  return a > 0.0 ? p : n;
}

// blockDim.x * CPT must equal TY * nx (<= 512 threads).
// NXC: nx fixed at compile time (0: read from g); fixed, the stencil's
// shared-memory offsets are immediates.
// Columns of a thread: SCHEME 0, tid + i blockDim.x; upwind3, rows CPT (tid / nx) + i of x = tid % nx.
// bu, bv, bw: u^n of stage 2 (else unused).
// SELECT (upwind3): the update from both one-sided stencils and a select (up3).
template <typename T, int SCHEME, int TY, int NS, int CPT, int NXC = 0, bool SELECT = false>
__global__ void __launch_bounds__(512) k_advect_zq(const __grid_constant__ AdvectMaps maps, const StreamGeom g,
                                                  const T* __restrict__ bu, const T* __restrict__ bv,
                                                  const T* __restrict__ bw, T* __restrict__ ou, T* __restrict__ ov,
                                                  T* __restrict__ ow, DtArg dt, double h, double nu, double ux,
                                                  double uy, double uz, int* err) {
  pdl_entry();
  constexpr int G = AdvectTraits<SCHEME>::G;
  constexpr bool UP = SCHEME != 0, BASE = SCHEME == 2, TAPS = UP && !SELECT;
  constexpr int ROWS = TY + 2 * G;
  constexpr int Q = 2 * G + 1;
  // a G-row halo box starting at y0 - G (wrapped) stays inside [0, ny) only if y0 is a multiple of TY >= G
  static_assert(TY >= G, "tile height must cover the halo depth");
  static_assert(NS > G, "the ring must hold the planes in use and one in flight");
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  const int nx = NXC ? NXC : g.nx, ny = g.ny, nz = g.nz, zc = g.zc;
  const int field_elems = ROWS * nx;
  const int slot_elems = 3 * field_elems;
  T* slots = reinterpret_cast<T*>(smem_raw);
  PlaneRing<NS, G - 1, 3> ring(smem_raw + (size_t)NS * slot_elems * sizeof(T), err);
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
    const int c = UP ? tid : tid + i * blockDim.x;
    cx[i] = c & mask;
    cy[i] = NXC ? c / NXC : c >> g.log2nx;
    if constexpr (UP) cy[i] = CPT * cy[i] + i;
  }
  const double dtv = dt.get();
  const T facA = (T)(SCHEME == 0 ? -dtv / (2 * h) : (TAPS ? dtv : -dtv) / (6 * h));  // TAPS: the B of the weights over |a|
  const T facD = (T)((nu / h) * (dtv / h));
  const T uinf[3] = {(T)ux, (T)uy, (T)uz};

  // qv: the centre values of the last Q planes (plane j in slot j % Q); the
  // plane loop is unrolled by Q, so the ring indices fold to constants.
  T qv[3][Q][CPT];
  T part[3][CPT];
  T base[BASE ? 3 : 1][CPT];  // u^n of the next output plane
  const T* bsrc[3] = {bu, bv, bw};
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      part[f][i] = (T)0;
#pragma unroll
      for (int d = 0; d < Q; ++d) qv[f][d][i] = (T)0;
    }

  // A thread whose wait timed out stops waiting and computing but keeps
  // releasing slots, so the block never deadlocks and the error word tells the host.
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
          const int QN = jj;  // queue slot of the newest plane
          // 1. centre values of plane j
#pragma unroll
          for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int i = 0; i < CPT; ++i) qv[f][QN][i] = sl[f * field_elems + (G + cy[i]) * nx + cx[i]];
          // 2. finish output plane k = j - 2G (queue slot of plane k + d - G: (jj - 2G + d) mod Q)
          if (j >= 2 * G) {
            const int QC = (jj + 3 * Q - G) % Q;       // centre (load j - G)
            const int QM1 = (jj + 3 * Q - G - 1) % Q;  // plane k - 1
            const int QP1 = (jj + 3 * Q - G + 1) % Q;  // plane k + 1
            const int QM2 = (jj + 3 * Q - G - 2) % Q;  // plane k - 2 (G = 2)
            const int QP2 = (jj + 3 * Q - G + 2) % Q;  // plane k + 2 (G = 2)
#pragma unroll
            for (int i = 0; i < CPT; ++i) {
              const T ww = qv[2][QC][i] + uinf[2];
              T outv[3];
              if constexpr (TAPS) {
                const UpW<T> wz = up_weights(ww, facA, facD);
                const T cz = (T)3 * wz.far - (T)2 * facD;
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                  const T f0 = qv[f][QC][i];
                  const T far = wz.pos ? qv[f][QM2][i] : qv[f][QP2][i];
                  T acc = part[f][i] + wz.far * far;
                  acc += wz.m1 * qv[f][QM1][i];
                  acc += wz.p1 * qv[f][QP1][i];
                  acc += cz * f0;
                  outv[f] = f0 + acc;
                }
              } else {
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                  const T f0 = qv[f][QC][i];
                  const T lz = qv[f][QM1][i] + qv[f][QP1][i];
                  if constexpr (UP) {
                    const T dz = up3_rn(ww, qv[f][QM2][i], qv[f][QM1][i], f0, qv[f][QP1][i], qv[f][QP2][i]);
                    const T s = __fma_rn(facA, __dmul_rn(ww, dz), __dadd_rn(f0, part[f][i]));
                    outv[f] = __fma_rn(facD, __fma_rn(f0, -6.0, lz), s);
                  } else {
                    const T dz = qv[f][QP1][i] - qv[f][QM1][i];
                    outv[f] = f0 + part[f][i] + facA * (ww * dz) + facD * (lz - f0 * 6);
                  }
                }
              }
              if constexpr (BASE) {
#pragma unroll
                for (int f = 0; f < 3; ++f) outv[f] = (T)0.5 * (base[f][i] + outv[f]);
              }
              ou[o[i]] = outv[0];
              ov[o[i]] = outv[1];
              ow[o[i]] = outv[2];
              o[i] += (size_t)nx * ny;
            }
          }
          // 3. x/y partial of plane j - G + 1 (output plane j - 2G + 1)
          if (j >= 2 * G - 1 && j < PL - 1) {
            const T* sp = slots + ring.slot_back(G - 1) * slot_elems;
            const int QX = (jj + 3 * Q - G + 1) % Q;
            if constexpr (UP) {
              const int x = cx[0], r = G + cy[0];
              const int xm1 = (x - 1) & mask, xp1 = (x + 1) & mask, xm2 = (x - 2) & mask, xp2 = (x + 2) & mask;
              [[maybe_unused]] UpW<T> wx[CPT], wy[CPT];
              [[maybe_unused]] T cxy[CPT];
              [[maybe_unused]] int xfar[CPT];
              if constexpr (TAPS) {
#pragma unroll
                for (int i = 0; i < CPT; ++i) {
                  wx[i] = up_weights(qv[0][QX][i] + uinf[0], facA, facD);
                  wy[i] = up_weights(qv[1][QX][i] + uinf[1], facA, facD);
                  cxy[i] = (T)3 * (wx[i].far + wy[i].far) - (T)4 * facD;
                  xfar[i] = wx[i].pos ? xm2 : xp2;
                }
              }
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                const T* F = sp + f * field_elems + r * nx;
                // rows r - 2 .. r + CPT + 1 of this x (the thread's own rows from the queue)
                T row[CPT + 2 * G];
#pragma unroll
                for (int d = 0; d < CPT + 2 * G; ++d)
                  row[d] = d >= G && d < G + CPT ? qv[f][QX][d - G] : F[(d - G) * nx + x];
#pragma unroll
                for (int i = 0; i < CPT; ++i) {
                  const T* Fx = F + i * nx;
                  if constexpr (TAPS) {
                    T acc = cxy[i] * row[G + i] + wx[i].far * Fx[xfar[i]];
                    acc += wx[i].m1 * Fx[xm1];
                    acc += wx[i].p1 * Fx[xp1];
                    acc += wy[i].far * (wy[i].pos ? row[i] : row[i + 4]);
                    acc += wy[i].m1 * row[i + 1];
                    acc += wy[i].p1 * row[i + 3];
                    part[f][i] = acc;
                  } else {
                    const T uu = qv[0][QX][i] + uinf[0], vv = qv[1][QX][i] + uinf[1];
                    const T fxm1 = Fx[xm1], fxp1 = Fx[xp1], fym1 = row[i + 1], fyp1 = row[i + 3];
                    const T dx = up3_rn(uu, Fx[xm2], fxm1, row[G + i], fxp1, Fx[xp2]);
                    const T dy = up3_rn(vv, row[i], fym1, row[G + i], fyp1, row[i + 4]);
                    const T adv = __fma_rn(uu, dx, __dmul_rn(vv, dy));
                    part[f][i] = __fma_rn(facD, fyp1 + fym1 + fxp1 + fxm1, __dmul_rn(facA, adv));
                  }
                }
              }
            } else {
#pragma unroll
              for (int i = 0; i < CPT; ++i) {
                const T uu = qv[0][QX][i] + uinf[0], vv = qv[1][QX][i] + uinf[1];
                const int x = cx[i], r = G + cy[i];
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                  const T* F = sp + f * field_elems;
                  const T xm1 = F[r * nx + ((x - 1) & mask)], xp1 = F[r * nx + ((x + 1) & mask)];
                  const T ym1 = F[(r - 1) * nx + x], yp1 = F[(r + 1) * nx + x];
                  part[f][i] = facA * (uu * (xp1 - xm1) + vv * (yp1 - ym1)) + facD * (yp1 + ym1 + xp1 + xm1);
                }
              }
            }
            if constexpr (BASE) {
              // u^n of output plane j - 2G + 1, finished by the next plane
#pragma unroll
              for (int i = 0; i < CPT; ++i)
#pragma unroll
                for (int f = 0; f < 3; ++f) base[f][i] = __ldg(bsrc[f] + o[i]);
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
