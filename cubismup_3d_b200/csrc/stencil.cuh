// Plane-streaming stencil kernels (the device replacement of Cubism's
// BlockLab + Operator::compute block loop, source/operators/Operator.h:112-170).
//
// A CTA owns work items of TY full x-rows by ZC z-planes. For every z plane
// it needs (ZC + 2G planes per item, wrapped periodically in z), one elected
// thread issues TMA tiled loads of NF fields into a ring of NS shared-memory
// plane slots: the TY main rows plus G halo rows below and above, one box
// unless the rows wrap in y (because y0 is a multiple of TY the halo rows are
// then contiguous G-row boxes of their own). The x halo is the periodic wrap of the full row in
// shared memory. Output plane k uses slots for planes k-G..k+G; loads run
// NS-(2G+1) planes ahead of compute. No load ever leaves the tensor bounds,
// so the zero fill of TMA is never used.
#pragma once

#include "common.cuh"

namespace cup {

constexpr int kStreamAcc = 20;

// Boxes of a field's tile rows with G halo rows on each side.
struct RowMaps {
  CUtensorMap all;   // {nx, TY + 2G, 1}
  CUtensorMap main;  // {nx, TY, 1}
  CUtensorMap halo;  // {nx, G, 1}
};

// Loads rows y0 - G .. y0 + TY + G - 1 (periodic) of plane z. One box unless
// they wrap (each load spared is time off the issuing warp's share of a plane).
template <int G, int TY, typename T>
__device__ __forceinline__ void tma_load_rows(T* dst, const RowMaps& m, int nx, int ny, int y0, int z, uint64_t* bar) {
  if (y0 >= G && y0 + TY + G <= ny) {
    tma_load_3d(dst, &m.all, 0, y0 - G, z, bar);
  } else {
    tma_load_3d(dst, &m.halo, 0, y0 < G ? y0 - G + ny : y0 - G, z, bar);
    tma_load_3d(dst + G * nx, &m.main, 0, y0, z, bar);
    tma_load_3d(dst + (G + TY) * nx, &m.halo, 0, y0 + TY >= ny ? y0 + TY - ny : y0 + TY, z, bar);
  }
}

template <int NF>
struct FieldMaps {
  RowMaps f[NF];
};

struct StreamGeom {
  int nx, ny, nz;
  int log2nx;
  int zc;       // z planes per work item
  int items_y;  // ny / TY
  int n_items;  // items_y * nz / zc
};

// First row and plane of a work item.
struct ItemPos {
  int y0, z0;
};
__device__ __forceinline__ ItemPos item_pos(const StreamGeom& g, int item, int TY, int zc) {
  const int zi = item / g.items_y;
  return ItemPos{(item - zi * g.items_y) * TY, zi * zc};
}

// Ring of NS plane slots of a z-queue kernel, fed by TMA; the plane index
// advances over the block's items as one stream. A plane's slot is free LAG
// planes after its own. Every two planes (every plane when the ring is shallow)
// a block barrier separates the last reads of the slots that came free from
// their refill. The NL loads of a plane are issued by NL different warps, one
// each: issued by one thread they held its warp back, and with it the whole
// block at the next barrier. At 256^3, with the halo rows' loads merged, the
// index divisions gone and a runtime item height in 5 or 10 unrolled planes (a
// fully unrolled item with its loads inlined missed the instruction cache):
// FP32 upwind stage 1 100 -> 93 us, stage 2 127 -> 99, residual 92 -> 79,
// gradient 160 -> 138; FP64 stage 1 220 -> 166, stage 2 299 -> 209 (with the
// upwind taps of advect.cuh). A ring without block barriers, its slots released
// by mbarrier arrivals of the warps and refilled by one thread, took 117, 188,
// 124, 196 for the FP32 passes.
template <int NS, int LAG, int NL>
struct PlaneRing {
  static constexpr size_t kBytes = (NS * sizeof(uint64_t) + 15) / 16 * 16;
  static constexpr bool PAIR = NS - LAG >= 4;
  uint64_t* full;
  int* err;
  int slot = 0;     // slot and phase of the current plane
  uint32_t ph = 0;
  int n = 0;        // planes done
  __device__ __forceinline__ PlaneRing(void* mem, int* e) : full((uint64_t*)mem), err(e) {
    if (threadIdx.x == 0) {
      for (int s = 0; s < NS; ++s) mbar_init(&full[s], NL);
      mbar_fence_init();
    }
    __syncthreads();
  }
  // slot of the plane d planes before the current one
  __device__ __forceinline__ int slot_back(int d) const { return slot < d ? slot - d + NS : slot - d; }
  // The first NS planes of the block's first item (NS <= planes per item).
  // issue(load, slot, plane, item) arrives once on full[slot].
  template <class Issue>
  __device__ __forceinline__ void start(const ItemPos& first, const Issue& issue) const {
    if ((threadIdx.x & 31) == 0)
#pragma unroll 1
      for (int q = threadIdx.x >> 5; q < NS * NL; q += (blockDim.x + 31) >> 5) issue(q % NL, q / NL, q / NL, first);
  }
  __device__ __forceinline__ bool wait() const { return mbar_wait(&full[slot], ph, err); }
  // After plane j of `cur` (PL planes per item, an even number): the barrier
  // and the loads of the planes NS - LAG ahead, of `cur` or of the block's next
  // item (more: there is one). odd: n is odd. A thread whose wait timed out
  // (ok false) takes the barriers but issues nothing more.
  template <class Issue>
  __device__ __forceinline__ void step(bool ok, bool odd, int j, int PL, const ItemPos& cur, const ItemPos& next,
                                       bool more, const Issue& issue) {
    if (!PAIR || odd) {
      __syncthreads();
      constexpr int NP = PAIR ? 2 : 1;
      if ((threadIdx.x & 31) == 0 && ok)
#pragma unroll 1
        for (int q = threadIdx.x >> 5; q < NP * NL; q += (blockDim.x + 31) >> 5) {
          const int r = PAIR && q < NL ? 1 : 0;     // the older plane first
          const int l = PAIR && q >= NL ? q - NL : q;
          const int jn = j - LAG - r + NS;
          const bool same = jn < PL;
          if ((LAG == 0 || n - LAG - r >= 0) && (same || more))
            issue(l, slot_back(LAG + r), same ? jn : jn - PL, same ? cur : next);
        }
    }
    ++n;
    if (++slot == NS) slot = 0, ph ^= 1;
  }
  // Thread 0, after a timed-out wait: bounded drain of the loads that may be in flight.
  __device__ __forceinline__ void drain(bool ok) const {
    if (!ok && threadIdx.x == 0)
      for (int s = 0; s < NS; ++s) {
        mbar_wait(&full[s], 0, nullptr);
        mbar_wait(&full[s], 1, nullptr);
      }
  }
};

// Read-only view of the resident planes for the output plane being computed.
template <typename T, int NF, int G, int TY>
struct PlaneCtx {
  static constexpr int ROWS = TY + 2 * G;
  const T* base[2 * G + 1];  // slot base for dz = -G..G
  int nx, mask;
  // value of field f at (x+dx, y+dy, z+dz), y a local row in [0, TY)
  __device__ __forceinline__ T v(int f, int x, int y, int dx, int dy, int dz) const {
    return base[dz + G][(f * ROWS + (G + y + dy)) * nx + ((x + dx) & mask)];
  }
};

template <typename T, int NF, int G, int TY, int NS>
constexpr size_t stream_smem_bytes(int nx) {
  return (size_t)NS * NF * (TY + 2 * G) * nx * sizeof(T) + NS * sizeof(uint64_t) + 32 * kStreamAcc * sizeof(double);
}

// Op must provide:
//   template <class Ctx> __device__ void cell(const Ctx&, int x, int y, int gy, int gz, double* acc) const;
//   __device__ void finish(double* acc, double* scratch) const;  // block epilogue (reductions)
// acc[kStreamAcc] is a per-thread accumulator array, zero-initialised.
template <typename T, int NF, int G, int TY, int NS, class Op>
__global__ void __launch_bounds__(256) k_stencil_stream(const __grid_constant__ FieldMaps<NF> maps,
                                                       const StreamGeom g, Op op, int* err, const int* skip) {
  pdl_entry();
  static_assert(NS >= 2 * G + 1, "ring must hold the stencil planes");
  // a G-row halo box starting at y0 - G (wrapped) stays inside [0, ny) only if y0 is a multiple of TY >= G
  static_assert(TY >= G, "tile height must cover the halo depth");
  if (skip && *skip) return;  // device-side early exit (converged defect correction)
  constexpr int ROWS = TY + 2 * G;
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const size_t slot_elems = (size_t)NF * ROWS * nx;
  T* slots = reinterpret_cast<T*>(smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + NS * slot_elems * sizeof(T));
  double* scratch = reinterpret_cast<double*>(full + NS);
  const int tid = threadIdx.x;
  const int PL = g.zc + 2 * G;
  const int my_items = blockIdx.x < g.n_items ? (g.n_items - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  const int L = my_items * PL;
  const uint32_t slot_bytes = (uint32_t)(slot_elems * sizeof(T));

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) mbar_init(&full[s], 1);
    mbar_fence_init();
  }
  __syncthreads();

  // the load stream's position: plane ij of the item at ipos
  ItemPos ipos = item_pos(g, blockIdx.x, TY, g.zc);
  int ij = 0, iitem = blockIdx.x, islot = 0;
  auto issue = [&]() {
    int z = ipos.z0 - G + ij;
    z = z < 0 ? z + nz : (z >= nz ? z - nz : z);
    T* dst = slots + islot * slot_elems;
    mbar_arrive_expect_tx(&full[islot], slot_bytes);
#pragma unroll
    for (int f = 0; f < NF; ++f)
      tma_load_rows<G, TY>(dst + f * ROWS * nx, maps.f[f], nx, ny, ipos.y0, z, &full[islot]);
    islot = islot + 1 == NS ? 0 : islot + 1;
    if (++ij == PL) {
      ij = 0;
      iitem += gridDim.x;
      ipos = item_pos(g, iitem, TY, g.zc);
    }
  };

  int q_issued = 0;
  if (tid == 0)
    for (; q_issued < min(L, NS); ++q_issued) issue();

  const int cells = nx * TY;
  double acc[kStreamAcc];
#pragma unroll
  for (int i = 0; i < kStreamAcc; ++i) acc[i] = 0.0;
  int a = 0;
  bool ok = true;
  for (int it = 0; it < my_items && ok; ++it) {
    const ItemPos pos = item_pos(g, blockIdx.x + it * gridDim.x, TY, g.zc);
    const int y0 = pos.y0, z0 = pos.z0;
    for (int k = 0; k < g.zc; ++k) {
      a = it * PL + k;
      bool mine = true;
#pragma unroll
      for (int d = 0; d <= 2 * G; ++d) mine = mine && mbar_wait(&full[(a + d) % NS], ((a + d) / NS) & 1, err);
      ok = __syncthreads_and(mine);
      if (!ok) break;
      PlaneCtx<T, NF, G, TY> ctx;
#pragma unroll
      for (int d = 0; d <= 2 * G; ++d) ctx.base[d] = slots + ((a + d) % NS) * slot_elems;
      ctx.nx = nx;
      ctx.mask = nx - 1;
      for (int c = tid; c < cells; c += blockDim.x) {
        const int x = c & (nx - 1), y = c >> g.log2nx;
        op.cell(ctx, x, y, y0 + y, z0 + k, acc);
      }
      __syncthreads();
      const int a_next = (k + 1 < g.zc) ? a + 1 : (it + 1) * PL;
      if (tid == 0)
        for (; q_issued < min(L, a_next + NS); ++q_issued) issue();
    }
  }
  if (!ok) {
    // Drain the loads this CTA still has in flight (bounded), then leave.
    for (int q = a; q < q_issued; ++q) mbar_wait(&full[q % NS], (q / NS) & 1, nullptr);
    __syncthreads();
    return;
  }
  op.finish(acc, scratch);
}

}  // namespace cup
