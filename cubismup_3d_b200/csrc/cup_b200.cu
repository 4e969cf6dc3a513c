// C-ABI implementation of the B200-native periodic fractional-step solver.
// Host orchestration: handle, device buffers, tensor maps, kernel launches
// and the operator pipeline of Simulation::timestep (source/Simulation.cpp:593-623).

#include "../../include/cup_b200.h"

#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <type_traits>
#include <utility>
#include <vector>

#include "adjoint.cuh"
#include "adjoint_f2.cuh"
#include "adjoint_obstacle.cuh"
#include "advect.cuh"
#include "advect_f2.cuh"
#include "common.cuh"
#include "dht.cuh"
#include "grad_zq.cuh"
#include "pfft.cuh"
#include "pressure_zq.cuh"
#include "ops.cuh"
#include "spectral.cuh"
#include "stencil.cuh"

using namespace cup;

namespace {

// Device-resident step state: the CFL dt chain, reductions and counters.
struct DevState {
  double dt, lambda, umax, ke;
  double corr, rhs_sums[3];
  double force[3], torque[3];
  double com[3], mass;
  double time;
  double res2, b2;
  double cmean[8];  // parity-class means of p (the 8 null-mode components)
  double rmean[8];  // parity-class means of the first residual (the RHS's null parts)
  double res_hist[16];  // relative residual at each check of the last solve
  double adj_sq;        // obstacle adjoint: sum over the corrected surface cells of b1 q
  int err_word;         // device error word (kDevErr* bits), read back with the state
  int step, n_solves, converged;
  int n_unconverged;  // steps whose defect correction missed the tolerance (cumulative)
  long long solves_total;  // correction solves of all decided defect corrections (cumulative)
};

enum PartialRegion { P_GRAD = 0, P_PEN, P_RHSOB, P_CHI, P_MAX, P_RES, P_DIAG, P_RIGID, P_COUNT };
constexpr int kPartialCap = 98304;  // doubles per region (>= 20 per CTA of a 4096-CTA pass)

constexpr int kBoxThreads = 256;
constexpr int kBoxBlocksMax = 296;

// ---------------------------------------------------------------------------
// small device kernels

template <typename T>
__global__ void k_convert_from_f64(T* dst, const double* src, size_t n) {
  pdl_entry();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = (T)src[i];
}
template <typename T>
__global__ void k_convert_to_f64(double* dst, const T* src, size_t n) {
  pdl_entry();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = (double)src[i];
}

// findMaxU (source/operators/ProcessHelpers.h:74-99): per-CTA partial maxima.
template <typename T>
__global__ void k_max_u(const T* u, const T* v, const T* w, size_t n, double ux, double uy, double uz,
                        double* partials) {
  pdl_entry();
  __shared__ double scratch[32];
  double m[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const double a = fabs((double)u[i] + ux), b = fabs((double)v[i] + uy), c = fabs((double)w[i] + uz);
    m[0] = fmax(m[0], fmax(fmax(a, b), c));
  }
  block_reduce<1, true>(m, scratch);
  if (threadIdx.x == 0) partials[blockIdx.x] = m[0];
}

// Simulation::calcMaxTimestep (source/Simulation.cpp:403-424) on the device,
// from st->umax and st->step.
struct CflParams {
  double h, nu, CFL;
  int rampup;
  double DLM;
};
__device__ __forceinline__ void calc_dt_device(DevState* st, const CflParams& c) {
  const double h = c.h, nu = c.nu, CFL = c.CFL, DLM = c.DLM;
  const int rampup = c.rampup;
  const double hMin = h;
  const double dtDif = hMin * hMin / nu;
  const double dtAdv = hMin / (st->umax + 1e-8);
  double dt = CFL * fmin(dtDif, dtAdv);
  if (st->step < rampup) {
    const double x = (st->step + 1.0) / rampup;
    const double rampCFL = exp(log(1e-3) * (1 - x) + log(CFL) * x);
    dt = rampCFL * fmin(dtDif, dtAdv);
  }
  st->dt = dt;
  if (DLM > 0) st->lambda = DLM / dt;
}

// The maximum of np partials, and with next_dt the CFL time step from it.
// step >= 0: the host's step counter, stored first (the ramp-up reads it).
__global__ void k_finalize_max(const double* partials, int np, DevState* st, int next_dt, CflParams cfl, int step) {
  pdl_entry();
  __shared__ double scratch[32];
  double m[1] = {0.0};
  for (int i = threadIdx.x; i < np; i += blockDim.x) m[0] = fmax(m[0], partials[i]);
  block_reduce<1, true>(m, scratch);
  if (threadIdx.x == 0) {
    st->umax = m[0];
    if (step >= 0) st->step = step;
    if (next_dt) calc_dt_device(st, cfl);
  }
}
__global__ void k_calc_dt(DevState* st, CflParams cfl, int step) {
  pdl_entry();
  if (step >= 0) st->step = step;
  calc_dt_device(st, cfl);
}

// Host-side scalars into the device state without a pageable copy (which
// would serialise the host with the stream): bit 1 dt (and lambda = DLM/dt
// when DLM > 0), bit 2 lambda (when DLM <= 0), bit 4 step and time; bit 8: then
// the CFL time step (what k_calc_dt computes).
enum { SET_DT = 1, SET_LAMBDA = 2, SET_CLOCK = 4, CALC_DT = 8 };
__global__ void k_set_state(DevState* st, int what, double dt, double lambda, int step, double time, CflParams cfl) {
  pdl_entry();
  if (what & SET_DT) {
    st->dt = dt;
    if (cfl.DLM > 0) st->lambda = cfl.DLM / dt;
  }
  if ((what & SET_LAMBDA) && !(cfl.DLM > 0)) st->lambda = lambda;
  if (what & SET_CLOCK) {
    st->step = step;
    st->time = time;
  }
  if (what & CALC_DT) calc_dt_device(st, cfl);
}

// Sum (or maximum) over np partials of one column by one warp; result in every
// lane. Columns side by side instead of one block reduction after another: bound
// by the latency of one block's loads and reduction; with the three merged
// launches above 172 -> 167 us per FP32_DC step on 128x64x256.
template <bool IS_MAX>
__device__ __forceinline__ double warp_column(const double* p, int np, int stride, int col) {
  double a = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x & 31; i < np; i += 32) {
    const double x = p[(size_t)stride * i + col];
    a = IS_MAX ? fmax(a, x) : a + x;
  }
  return IS_MAX ? warp_max(a) : warp_sum(a);
}

// End of step: umax (grid part outside the obstacle box, box part after
// penalization), kinetic energy, force/torque; advances step and time.
// next_dt: then the CFL time step of the next step (what k_calc_dt would
// compute before it), saving its launch in a run of steps. 256 threads.
__global__ void k_finalize_step(const double* pgrad, int ngrad, int gstride, int max_off, int ke_off,
                                const double* ppen, int npen, DevState* st, double h3, int advance, int next_dt,
                                CflParams cfl) {
  pdl_entry();
  // one warp per column: 0 the maximum, 1 the kinetic energy, 2-7 force and torque
  __shared__ double s[8];
  const int wid = threadIdx.x >> 5;
  double v;
  if (wid == 0) {
    v = warp_column<true>(pgrad, ngrad, gstride, max_off);
    if (npen > 0) v = fmax(v, warp_column<true>(ppen, npen, 8, 6));
  } else if (wid == 1) {
    v = warp_column<false>(pgrad, ngrad, gstride, ke_off);
  } else {
    v = warp_column<false>(ppen, npen, 8, wid - 2);
  }
  if ((threadIdx.x & 31) == 0) s[wid] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    st->umax = s[0];
    st->ke = s[1] * h3;
    if (npen > 0) {
      for (int k = 0; k < 3; ++k) {
        st->force[k] = s[2 + k];
        st->torque[k] = s[5 + k];
      }
    }
    if (advance) {
      st->step += 1;
      st->time += st->dt;
    }
    if (next_dt) calc_dt_device(st, cfl);
  }
}

// Penalization-only finalize (operator-by-operator path); lambda as SET_LAMBDA. 192 threads.
__global__ void k_finalize_pen(const double* ppen, int npen, DevState* st, double DLM, double lambda) {
  pdl_entry();
  const int wid = threadIdx.x >> 5;
  const double v = warp_column<false>(ppen, npen, 8, wid);
  if ((threadIdx.x & 31) == 0) (wid < 3 ? st->force[wid] : st->torque[wid - 3]) = v;
  if (threadIdx.x == 0 && !(DLM > 0)) st->lambda = lambda;
}

// PressureRHS correction factor (source/operators/PressureRHS.cpp:328-334).
__global__ void k_finalize_rhs_obstacle(const double* p, int np, DevState* st) {
  pdl_entry();
  __shared__ double scratch[3 * 32];
  double s[3] = {0, 0, 0};
  for (int i = threadIdx.x; i < np; i += blockDim.x)
    for (int k = 0; k < 3; ++k) s[k] += p[3 * i + k];
  block_reduce<3, false>(s, scratch);
  if (threadIdx.x == 0) {
    const double EPS = 2.220446049250313080847e-16;
    const double sumRHS = s[0], posRHS = s[1], negRHS = s[2];
    const double corrDenom = sumRHS > 0 ? posRHS : negRHS;
    st->corr = sumRHS / fmax(corrDenom, EPS);
    st->rhs_sums[0] = sumRHS;
    st->rhs_sums[1] = posRHS;
    st->rhs_sums[2] = negRHS;
  }
}

// Zeroes a field of es-byte elements (4: FP32, 8: FP64) on a box, and moves the
// sphere's position in the device parameters (stream-ordered).
__global__ void k_clear_box(void* f, size_t es, Box box, int nx, int ny, int nz, SphereParams* sp, double px, double py,
                            double pz) {
  pdl_entry();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sp->position[0] = px;
    sp->position[1] = py;
    sp->position[2] = pz;
  }
  const long long n = box.count();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int x = wrapi(box.lo[0] + (int)(i % box.n[0]), nx);
    const int y = wrapi(box.lo[1] + (int)((i / box.n[0]) % box.n[1]), ny);
    const int z = wrapi(box.lo[2] + (int)(i / ((long long)box.n[0] * box.n[1])), nz);
    const size_t o = gidx(x, y, z, nx, ny);
    if (es == 4)
      static_cast<float*>(f)[o] = 0.f;
    else
      static_cast<double*>(f)[o] = 0.0;
  }
}

// Grid centre of mass (source/operators/ObstaclesCreate.cpp:230-256) -> SphereParams.
__global__ void k_finalize_com(const double* p, int np, DevState* st, SphereParams* sp) {
  pdl_entry();
  __shared__ double scratch[4 * 32];
  double s[4] = {0, 0, 0, 0};
  for (int i = threadIdx.x; i < np; i += blockDim.x)
    for (int k = 0; k < 4; ++k) s[k] += p[4 * i + k];
  block_reduce<4, false>(s, scratch);
  if (threadIdx.x == 0) {
    st->mass = s[0];
    for (int k = 0; k < 3; ++k) {
      st->com[k] = s[1 + k] / s[0];
      sp->centerOfMass[k] = st->com[k];
    }
  }
}

// KernelFinalizeObstacleVel (source/operators/ObstaclesUpdate.cpp:136-200)
// and Obstacle::computeVelocities (source/obstacles/Obstacle.cpp:153-264) for
// the sphere: the 29 momentum sums, then the 6x6 momentum balance with the
// rows of forced translations and blocked rotations replaced by their imposed
// values, solved by LU with partial pivoting (the GSL routines the reference
// calls); the free dofs take the computed velocities. force / torque are the
// rigid-body ones of computeVelocities (Penalization overwrites them).
__global__ void k_rigid_update(const double* partials, int np, SphereParams* sp, DevState* st, DtArg dt,
                               int implicit_pen) {
  pdl_entry();
  __shared__ double scratch[kRigidQoI * 32];
  double M[kRigidQoI];
  for (int k = 0; k < kRigidQoI; ++k) M[k] = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x)
    for (int k = 0; k < kRigidQoI; ++k) M[k] += partials[(size_t)kRigidQoI * i + k];
  block_reduce<kRigidQoI, false>(M, scratch);
  if (threadIdx.x != 0) return;
  SphereParams& s = *sp;
  const double dtv = dt.get();
  s.mass = M[0];
  for (int k = 0; k < 6; ++k) s.J[k] = M[7 + k];
  double pM, pC[3], pJ[6], Lm[3], Am[3];
  if (implicit_pen) {
    pM = M[13];
    for (int d = 0; d < 3; ++d) pC[d] = M[14 + d], Lm[d] = M[23 + d], Am[d] = M[26 + d];
    for (int k = 0; k < 6; ++k) pJ[k] = M[17 + k];
  } else {
    pM = M[0];
    for (int d = 0; d < 3; ++d) pC[d] = 0, Lm[d] = M[1 + d], Am[d] = M[4 + d];
    for (int k = 0; k < 6; ++k) pJ[k] = M[7 + k];
  }
  double A[6][6] = {{pM, 0, 0, 0, +pC[2], -pC[1]},
                    {0, pM, 0, -pC[2], 0, +pC[0]},
                    {0, 0, pM, +pC[1], -pC[0], 0},
                    {0, -pC[2], +pC[1], pJ[0], pJ[3], pJ[4]},
                    {+pC[2], 0, -pC[0], pJ[3], pJ[1], pJ[5]},
                    {-pC[1], +pC[0], 0, pJ[4], pJ[5], pJ[2]}};
  double b[6] = {Lm[0], Lm[1], Lm[2], Am[0], Am[1], Am[2]};
  for (int d = 0; d < 3; ++d) {
    if (s.forced[d]) {
      for (int k = 0; k < 6; ++k)
        if (k != d) A[d][k] = 0;
      b[d] = pM * s.transVel_imposed[d];
    }
    if (s.block_rot[d]) {
      for (int k = 0; k < 6; ++k)
        if (k != 3 + d) A[3 + d][k] = 0;
      b[3 + d] = 0;
    }
  }
  // LU with partial pivoting, then forward and back substitution
  int perm[6] = {0, 1, 2, 3, 4, 5};
  for (int j = 0; j < 5; ++j) {
    int piv = j;
    double mx = fabs(A[j][j]);
    for (int i = j + 1; i < 6; ++i)
      if (fabs(A[i][j]) > mx) mx = fabs(A[i][j]), piv = i;
    if (piv != j) {
      for (int k = 0; k < 6; ++k) {
        const double t = A[j][k];
        A[j][k] = A[piv][k];
        A[piv][k] = t;
      }
      const int t = perm[j];
      perm[j] = perm[piv];
      perm[piv] = t;
    }
    if (A[j][j] == 0) continue;
    for (int i = j + 1; i < 6; ++i) {
      const double l = A[i][j] / A[j][j];
      A[i][j] = l;
      for (int k = j + 1; k < 6; ++k) A[i][k] -= l * A[j][k];
    }
  }
  double x[6];
  for (int i = 0; i < 6; ++i) x[i] = b[perm[i]];
  for (int i = 0; i < 6; ++i)
    for (int k = 0; k < i; ++k) x[i] -= A[i][k] * x[k];
  for (int i = 5; i >= 0; --i) {
    for (int k = i + 1; k < 6; ++k) x[i] -= A[i][k] * x[k];
    x[i] /= A[i][i];
  }
  double dAv[3];
  for (int d = 0; d < 3; ++d) {
    s.transVel_computed[d] = x[d];
    s.angVel_computed[d] = x[3 + d];
    st->force[d] = s.mass * (x[d] - s.transVel[d]) / dtv;
    dAv[d] = (x[3 + d] - s.angVel[d]) / dtv;
  }
  st->torque[0] = s.J[0] * dAv[0] + s.J[3] * dAv[1] + s.J[4] * dAv[2];
  st->torque[1] = s.J[3] * dAv[0] + s.J[1] * dAv[1] + s.J[5] * dAv[2];
  st->torque[2] = s.J[4] * dAv[0] + s.J[5] * dAv[1] + s.J[2] * dAv[2];
  for (int d = 0; d < 3; ++d) {
    s.transVel[d] = s.forced[d] ? s.transVel_imposed[d] : x[d];
    s.angVel[d] = s.block_rot[d] ? 0.0 : x[3 + d];
  }
}

// Defect-correction bookkeeping after a residual pass (check k, before solve k):
// FP64 norms with the null-mode components projected out (they are not
// reachable by any pressure: the spectral factor is zero there), the
// parity-class means of p, and the decision |r| <= tol |b| (from check
// min_iter on; check max_iter is final).
__global__ void k_finalize_residual(const double* p, int stride, int np, DevState* st, double tol, int k,
                                    int min_iter, int max_iter, double inv_class_cells) {
  pdl_entry();
  if (k > 0 && st->converged) return;
  // one warp per sum (576 threads)
  __shared__ double s[18];
  const double v = warp_column<false>(p, np, stride, threadIdx.x >> 5);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double res2, b2;
    if (k == 0) {
      // the null parts of r are those of b (L_2h p has none); keep them for later checks
      double null2 = 0.0;
      for (int j = 0; j < 8; ++j) {
        st->rmean[j] = s[10 + j] * inv_class_cells;
        null2 += s[10 + j] * s[10 + j] * inv_class_cells;
      }
      b2 = fmax(s[1] - null2, 0.0);
      res2 = fmax(s[0] - null2, 0.0);
    } else {
      b2 = st->b2;
      res2 = s[0];  // accumulated with the null parts removed per cell
    }
    st->res2 = res2;
    st->b2 = b2;
    if (k < 16) st->res_hist[k] = b2 > 0 ? sqrt(res2 / b2) : 0.0;
    for (int j = 0; j < 8; ++j) st->cmean[j] = s[2 + j] * inv_class_cells;
    const bool met = b2 == 0.0 || sqrt(res2) <= tol * sqrt(b2);
    st->n_solves = k;
    st->converged = (k >= min_iter && met) ? 1 : 0;
    if (k >= max_iter) {
      st->converged = met ? 1 : 2;  // 2: not converged after max_iter solves
      if (!met) st->n_unconverged += 1;
    }
    if (st->converged) st->solves_total += k;
  }
}

// Periodic shift through the plane-streaming path (TestBoundaries restatement).
struct OpShift {
  double* out;
  int dx, dy, dz;
  int nx, ny;
  template <class C>
  __device__ __forceinline__ void cell(const C& c, int x, int y, int gy, int gz, double*) const {
    out[gidx(x, gy, gz, nx, ny)] = c.v(0, x, y, -dx, -dy, -dz);
  }
  __device__ void finish(double*, double*) const {}
};

// ---------------------------------------------------------------------------
// Allocation-free max |u + uinf| (cup_max_velocity_noalloc). Its per-CTA
// partial maxima live in this fixed device array instead of handle-owned
// memory: every GPU that loads the library holds the array until exit, and all
// calls share it. A call splits the n cells into at most kNoAllocMaxCtas
// contiguous chunks (a multiple of 1024 cells each), one per CTA; the host
// caps n at kNoAllocMaxCtas * kNoAllocChunk cells. The maximum propagates NaN
// (fmax would drop it), so a non-finite field gives a NaN result.
constexpr int kNoAllocMaxCtas = 4096;
constexpr long long kNoAllocChunk = 65536;
static __device__ __align__(256) double g_noalloc_partials[kNoAllocMaxCtas];

__device__ __forceinline__ double nan_max(double a, double b) { return (a > b || a != a) ? a : b; }

__device__ __forceinline__ double noalloc_block_max(double m, double* scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) scratch[wid] = m;
  __syncthreads();
  if (wid == 0) {
    m = lane < nw ? scratch[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, o));
  }
  return m;
}

// One CTA of 256 threads per chunk of `chunk` cells; four independent loads in
// flight per thread and field.
__global__ void __launch_bounds__(256) k_noalloc_max_partial(const double* __restrict__ u,
                                                             const double* __restrict__ v,
                                                             const double* __restrict__ w, long long n,
                                                             long long chunk, double ux, double uy, double uz,
                                                             double* partials) {
  __shared__ double scratch[32];
  double m0 = 0.0, m1 = 0.0, m2 = 0.0, m3 = 0.0;
  const long long lo = blockIdx.x * chunk;
  const long long hi = lo + chunk < n ? lo + chunk : n;
  auto cell = [&](long long i) {
    return nan_max(nan_max(fabs(u[i] + ux), fabs(v[i] + uy)), fabs(w[i] + uz));
  };
  long long i = lo + threadIdx.x;
  for (; i + 768 < hi; i += 1024) {
    m0 = nan_max(m0, cell(i));
    m1 = nan_max(m1, cell(i + 256));
    m2 = nan_max(m2, cell(i + 512));
    m3 = nan_max(m3, cell(i + 768));
  }
  for (; i < hi; i += 256) m0 = nan_max(m0, cell(i));
  const double m = noalloc_block_max(nan_max(nan_max(m0, m1), nan_max(m2, m3)), scratch);
  if (threadIdx.x == 0) partials[blockIdx.x] = m;  // every used slot is written before it is read
}

__global__ void __launch_bounds__(256) k_noalloc_max_final(const double* partials, int np, double* out) {
  __shared__ double scratch[32];
  double m = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) m = nan_max(m, partials[i]);
  m = noalloc_block_max(m, scratch);
  if (threadIdx.x == 0) *out = m;
}

// ---------------------------------------------------------------------------
// host helpers

PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::mutex g_encode_mu;

bool get_encode() {
  std::lock_guard<std::mutex> lk(g_encode_mu);
  if (g_encode) return true;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !fn)
    return false;
  g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  return true;
}

template <typename T>
CUtensorMapDataType tma_dtype();
template <>
CUtensorMapDataType tma_dtype<double>() {
  return CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
}
template <>
CUtensorMapDataType tma_dtype<float>() {
  return CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
}

int ilog2(int n) {
  int l = 0;
  while ((1 << l) < n) ++l;
  return l;
}
bool is_pow2(int n) { return n > 0 && (n & (n - 1)) == 0; }

const long double kPi = 3.141592653589793238462643383279502884L;

template <int M>
void build_table_M(std::vector<double2>& t64) {
  using Pl = FFTPlan<M>;
  t64.assign(Pl::table_len(), double2{0, 0});
  auto put = [&](int i, long double ang) { t64[i] = double2{(double)cosl(ang), (double)sinl(ang)}; };
  for (int s = 1; s < Pl::nstages; ++s) {
    const int R = Pl::radix(s), Ns = Pl::ns(s), off = Pl::tw_off(s);
    for (int r = 0; r < R; ++r)
      for (int j = 0; j < Ns; ++j) put(off + r * Ns + j, -2.0L * kPi * r * j / ((long double)Ns * R));
  }
  for (int k = 0; k <= M / 2; ++k) put(Pl::post_off() + k, -2.0L * kPi * k / (2.0L * M));
  if (M == 128)
    for (int r = 0; r < 8; ++r)
      for (int j = 0; j < 16; ++j) put(Pl::r16_off() + 16 * r + j, -2.0L * kPi * r * j / (long double)M);
}

// Tables of the packed transforms (pfft.cuh): the twiddles W_M^(k1 t) and
// cos(2 pi k / M) of the bin at each position (rows: the swizzled order); c is
// the reference's cos(4 pi k / N), k < N.
template <int M>
void build_ptable_M(const std::vector<double>& c, bool rows, std::vector<double2>& t64, std::vector<float2>& t32,
                    std::vector<double>& pc) {
  using P = PPlan<M>;
  t64.resize(M), t32.resize(M), pc.resize(M);
  for (int k1 = 0; k1 < P::R1; ++k1)
    for (int t = 0; t < P::R2; ++t) {
      const long double a = -2.0L * kPi * k1 * t / (long double)M;
      t64[k1 * P::R2 + t] = double2{(double)cosl(a), (double)sinl(a)};
      t32[k1 * P::R2 + t] = float2{(float)cosl(a), (float)sinl(a)};
    }
  for (int i = 0; i < M; ++i) pc[i] = c[rows ? P::row_bin(i) : P::bin(i)];
}

void build_tables(int N, const std::vector<double>& c, bool rows, std::vector<double2>& t64, std::vector<double2>& p64,
                  std::vector<float2>& p32, std::vector<double>& pc) {
  switch (N / 2) {
    case 8: build_table_M<8>(t64), build_ptable_M<8>(c, rows, p64, p32, pc); break;
    case 16: build_table_M<16>(t64), build_ptable_M<16>(c, rows, p64, p32, pc); break;
    case 32: build_table_M<32>(t64), build_ptable_M<32>(c, rows, p64, p32, pc); break;
    case 64: build_table_M<64>(t64), build_ptable_M<64>(c, rows, p64, p32, pc); break;
    case 128: build_table_M<128>(t64), build_ptable_M<128>(c, rows, p64, p32, pc); break;
    default: break;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
struct cup_handle {
  cup_config cfg;
  int nx = 0, ny = 0, nz = 0;
  size_t n = 0;
  double h = 0;
  int dev = 0, num_sms = 148;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::string err;
  bool fp32 = false;
  // fields (T = double or float by precision)
  void *u = nullptr, *v = nullptr, *w = nullptr;
  void *tu = nullptr, *tv = nullptr, *tw = nullptr;
  void *u1 = nullptr, *v1 = nullptr, *w1 = nullptr;
  void* chi = nullptr;
  double* p = nullptr;    // pressure (FP64)
  // FP32_DC without obstacle: pressure of the previous step and the next
  // step's warm start (extrapolated by the gradient pass); p_valid counts the
  // valid levels among (p, p_old), pred_ready says p_pred holds a warm start
  double* p_old = nullptr;
  double* p_pred = nullptr;
  int p_valid = 0;
  bool pred_ready = false;
  double* rhs = nullptr;  // pressure RHS (FP64); FP64 mode: also the FFT work array
  float* work32 = nullptr;  // FP32_DC FFT work array (residual, forward x/y passes)
  double* work64 = nullptr;  // FP32_DC FFT work array (z pass onwards, FP64)
  double* partials = nullptr;
  DevState* dstate = nullptr;
  int* derr = nullptr;
  // FFT tables (per axis) and spectral cos tables
  double2* tw64[3] = {nullptr, nullptr, nullptr};
  // packed transforms of the pressure solve (pfft.cuh): twiddles and the
  // cosines in spectrum order, per axis
  double2* ptw64[3] = {nullptr, nullptr, nullptr};
  float2* ptw32[3] = {nullptr, nullptr, nullptr};
  double* pcos[3] = {nullptr, nullptr, nullptr};
  double *cosx = nullptr, *cosy = nullptr, *cosz = nullptr;
  double norm_factor = 0;
  double pnorm = 0;  // of the packed transforms: 4 / h / (Mx My Mz)
  void* tables = nullptr;       // the one allocation behind the tables above
  double* cosy_win = nullptr;   // cosy of cup_set_spectral_window
  // spectral window of a y-split pencil of a decomposed grid (cup_set_spectral_window):
  // the global y length of the cos table and of the null modes, and this handle's first y
  int spec_ny = 0, spec_y0 = 0;
  // obstacle
  bool has_sphere = false;
  cup_sphere sphere{};  // host mirror; sphere.position follows Obstacle::update
  double sphere_vel[3] = {0, 0, 0};  // transVel (the imposed velocity of the forced dofs)
  bool sphere_moves = false;         // transVel + uinf != 0: chi is rebuilt every step
  bool sphere_free = false;          // a translation is not forced: UpdateObstacles computes the velocities
  double sphere_angvel[3] = {0, 0, 0};       // angVel (host mirror, read back after each step when free)
  double sphere_quat[4] = {1, 0, 0, 0};      // Obstacle::quaternion
  SphereParams* sp_dev = nullptr;
  Box box{};
  // with the sphere: the RHS's obstacle terms on the box (b2 - b0, box order)
  // that the passes forming b from u* add to it, and the box array the obstacle
  // kernels work on; box_cap: their length
  double* box_delta = nullptr;
  double* box_b = nullptr;
  long long box_cap = 0;
  // host mirrors
  int step = 0;
  double time = 0, dt = 0, lambda = 0;
  double uinf[3] = {0, 0, 0};
  bool umax_fresh = false;
  int n_grad_partials = 0, n_pen_partials = 0;
  // layout of the gradient pass's partials: values per CTA, offsets of max |u| and the kinetic energy
  int grad_stride = 2, grad_max_off = 0, grad_ke_off = 1;
  DevState* hstate = nullptr;  // pinned host copy
  // per-step solve stats
  int last_n_solves = 0;
  // discrete adjoint scratch (allocated on the first adjoint call)
  void *au = nullptr, *av = nullptr, *aw = nullptr;
  double* p_adj = nullptr;
  // spectral analysis / forcing: FP64 Hartley coefficients of u, v, w (allocated on first use)
  // (one allocation), the forcing band's coefficients, sums on their way to the
  // host and the pinned buffer they land in
  double* spec[3] = {nullptr, nullptr, nullptr};
  double* band_coef = nullptr;
  double *dsum = nullptr, *hsum = nullptr;
  bool forcing = false;                 // SpectralForcing inside cup_step / cup_run
  double forcing_target = 0, forcing_rate = 0, forcing_prev_tke = 0;
  double forcing_stats[6] = {0, 0, 0, 0, 0, 0};
  // obstacle adjoint scratch: the velocity before penalization u** (T) and the
  // RHS before its obstacle terms b0 (FP64, on the box), recomputed per adjoint step
  void *aus = nullptr, *avs = nullptr, *aws = nullptr;
  double* ab0 = nullptr;
  // cup_run in steady state: kGraphSteps steps captured once as a CUDA graph
  // and replayed (the field pointers rotate with period 6: u/tmp swap every
  // step, the three FP32-DC pressure levels every step); the graph is tied to
  // the pointer tuple it was captured with
  bool use_graphs = true;
  // calcMaxTimestep right after timestep: cup_step's stats read-back brings
  // the next step's CFL dt (computed on the device at the end of the step) to
  // the host; dt_next_call is the API call count at that read, and the cached
  // dt is used only by the next API call (api_calls counts every entry point)
  unsigned long long api_calls = 0, dt_next_call = 0;
  double dt_next = 0, lambda_next = 0;
  // kernels launched as programmatic dependent launches: off by default (the
  // captured 6-step graphs measured 34 us per step slower at 256^3 with it);
  // CUP_PDL=1 in the environment at cup_create turns it on
  bool pdl = false;
  // host state a step reads and advances (the graph replays the device part)
  struct StepState {
    void* f[9];  // u, v, w, tu, tv, tw, p, p_old, p_pred
    int p_valid, n_grad_partials, grad_stride, grad_max_off, grad_ke_off;
    bool pred_ready;
  };
  struct StepGraph {
    StepState in, out;
    int nsteps, next_dt;
    cudaGraph_t graph;
    cudaGraphExec_t exec;
    long long launches;
  };
  std::vector<StepGraph> graphs;
  cudaStream_t cap_stream = nullptr;  // captures run here: the default streams cannot be captured
  long long steps_run = 0;            // steps since creation
  // launch accounting and optional per-kernel CUDA-event profiling
  long long launches = 0;
  bool prof_on = false;
  struct Pending {
    const char* name;
    cudaEvent_t a, b;
  };
  std::vector<Pending> pending;
  std::vector<cudaEvent_t> ev_pool;
  std::map<std::string, std::vector<float>> prof;  // name -> duration (ms) of each launch
};

namespace {

int fail(cup_handle* H, int code, const char* fmt, ...) {
  if (H) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    H->err = buf;
  }
  return code;
}

#define CK(call)                                                                                      \
  do {                                                                                                \
    cudaError_t e_ = (call);                                                                          \
    if (e_ != cudaSuccess) return fail(H, CUP_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

#define CKL()                                                                                          \
  do {                                                                                                 \
    cudaError_t e_ = cudaGetLastError();                                                               \
    if (e_ != cudaSuccess) return fail(H, CUP_ERR_CUDA, "kernel launch failed: %s", cudaGetErrorString(e_)); \
  } while (0)

double* partial(cup_handle* H, int region) { return H->partials + (size_t)region * kPartialCap; }

cudaEvent_t ev_get(cup_handle* H) {
  if (!H->ev_pool.empty()) {
    cudaEvent_t e = H->ev_pool.back();
    H->ev_pool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}

// Resolves recorded event pairs into the per-kernel totals (synchronises).
void prof_flush(cup_handle* H) {
  if (H->pending.empty()) return;
  cudaStreamSynchronize(H->stream);
  for (auto& p : H->pending) {
    float ms = 0;
    cudaEventElapsedTime(&ms, p.a, p.b);
    H->prof[p.name].push_back(ms);
    H->ev_pool.push_back(p.a);
    H->ev_pool.push_back(p.b);
  }
  H->pending.clear();
}

// Counts one kernel launch and, when profiling is on, brackets it with events.
template <class F>
int launch_named(cup_handle* H, const char* name, F&& f) {
  H->launches += 1;
  cudaEvent_t a = nullptr;
  if (H->prof_on) {
    a = ev_get(H);
    cudaEventRecord(a, H->stream);
  }
  const int rc = f();
  if (H->prof_on) {
    cudaEvent_t b = ev_get(H);
    cudaEventRecord(b, H->stream);
    H->pending.push_back({name, a, b});
    if (H->pending.size() > 4096) prof_flush(H);
  }
  return rc;
}

// nf: fields one after the other, as one of nf times the planes.
int make_map(cup_handle* H, CUtensorMap* m, const void* base, CUtensorMapDataType dt, size_t elem, int bx, int by,
             int bz, int nf = 1) {
  if (!get_encode()) return fail(H, CUP_ERR_CUDA, "cuTensorMapEncodeTiled entry point unavailable");
  cuuint64_t dims[3] = {(cuuint64_t)H->nx, (cuuint64_t)H->ny, (cuuint64_t)H->nz * nf};
  cuuint64_t strides[2] = {(cuuint64_t)H->nx * elem, (cuuint64_t)H->nx * H->ny * elem};
  cuuint32_t box[3] = {(cuuint32_t)bx, (cuuint32_t)by, (cuuint32_t)bz};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = g_encode(m, dt, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(H, CUP_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return CUP_OK;
}

// The boxes of a field's TY tile rows with G halo rows (RowMaps).
template <typename T>
int make_row_maps(cup_handle* H, RowMaps* m, const void* base, int TY, int G) {
  int rc = make_map(H, &m->all, base, tma_dtype<T>(), sizeof(T), H->nx, TY + 2 * G, 1);
  if (!rc) rc = make_map(H, &m->main, base, tma_dtype<T>(), sizeof(T), H->nx, TY, 1);
  if (!rc) rc = make_map(H, &m->halo, base, tma_dtype<T>(), sizeof(T), H->nx, G, 1);
  return rc;
}

template <class K>
int prepare_kernel(cup_handle* H, K kern, size_t smem, int threads, int* blocks_per_sm) {
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kern, threads, smem));
  if (*blocks_per_sm < 1) return fail(H, CUP_ERR_ARG, "kernel does not fit on an SM (smem %zu)", smem);
  return CUP_OK;
}

// Launches a kernel on the handle's stream; with H->pdl (off unless CUP_PDL=1) as
// a programmatic dependent launch: its CTAs may be scheduled while the previous
// kernel of the stream finishes, and wait in pdl_entry() for that kernel's
// completion before touching its data. A failure is left for CKL() to report.
template <typename... KArgs, typename... Args>
void klaunch(cup_handle* H, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = H->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // (the default streams keep plain stream order)
  const bool named = H->stream && H->stream != cudaStreamLegacy && H->stream != cudaStreamPerThread;
  cfg.numAttrs = H->pdl && named ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// Planes per work item (16, 8 or 4): the fewest plane loads on the busiest CTA,
// waves of items times the planes an item loads (its 2G halo planes too), so
// that a small grid spreads over the SMs. (At 64^3 the FP64 upwind3 stages had
// run 64 items of 20 planes on 148 SMs.)
int planes_per_item(const cup_handle* H, int TY, int G, int bpsm) {
  int zc = std::min(16, H->nz);
  long long best = -1;
  for (int c = std::min(16, H->nz); c >= 4; c /= 2) {
    const long long items = (long long)(H->ny / TY) * (H->nz / c);
    const long long resident = std::min<long long>(items, (long long)bpsm * H->num_sms);
    const long long cost = (items + resident - 1) / resident * (c + 2 * G);
    if (best < 0 || cost < best) best = cost, zc = c;
  }
  return zc;
}

// Launches k_stencil_stream over `fields` (device arrays of T). Returns the
// grid size through *grid_out (the number of per-CTA partials written).
template <typename T, int NF, int G, int TY, int NS, class Op>
int launch_stream(cup_handle* H, const char* name, const void* const* fields, const Op& op, int* grid_out = nullptr,
                  const int* skip = nullptr) {
  FieldMaps<NF> maps;
  for (int f = 0; f < NF; ++f) {
    int rc = make_row_maps<T>(H, &maps.f[f], fields[f], TY, G);
    if (rc) return rc;
  }
  const size_t smem = stream_smem_bytes<T, NF, G, TY, NS>(H->nx) + 128;
  auto kern = k_stencil_stream<T, NF, G, TY, NS, Op>;
  int bpsm = 0;
  int rc = prepare_kernel(H, kern, smem, 256, &bpsm);
  if (rc) return rc;
  const int zc = planes_per_item(H, TY, G, bpsm);
  StreamGeom g{H->nx, H->ny, H->nz, ilog2(H->nx), zc, H->ny / TY, (H->ny / TY) * (H->nz / zc)};
  const int grid = std::min(g.n_items, bpsm * H->num_sms);
  if (grid > kPartialCap / 16) return fail(H, CUP_ERR_ARG, "too many CTAs for the partial buffers");
  rc = launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, 256, smem, maps, g, op, H->derr, skip);
    CKL();
    return CUP_OK;
  });
  if (rc) return rc;
  if (grid_out) *grid_out = grid;
  return CUP_OK;
}

// Pipelined Hartley x pass (k_dht_rows_pipe): the rows of nf fields (FP64, or
// FP32 widened on the way) into out, one field after the other.
template <int M, typename RIN>
int launch_rows_pipe_M(cup_handle* H, const char* name, const RIN* const* f, int nf, double* out) {
  constexpr int N = 2 * M, TPL = M / 8;
  constexpr bool PAD = FFTPlan<M>::nstages > 1;
  constexpr int NB = 2;
  const int lpc = 256 / TPL;
  const RowsIn<RIN> in{{f[0], nf > 1 ? f[1] : nullptr, nf > 2 ? f[2] : nullptr}, H->ny * H->nz};
  const size_t smem = (size_t)NB * lpc * N * sizeof(double) + (PAD ? (size_t)lpc * 2 * (M + M / 8) * sizeof(double) : 0) +
                      FFTPlan<M>::rows_table_len() * sizeof(double2) + NB * sizeof(uint64_t) + 128;
  auto kern = k_dht_rows_pipe<M, RIN, NB>;
  const int threads = lpc * TPL;
  int bpsm = 0;
  int rc = prepare_kernel(H, kern, smem, threads, &bpsm);
  if (rc) return rc;
  const int ntiles = nf * in.rows / lpc;  // ny nz is a multiple of 256 >= lpc
  const int grid = std::min(ntiles, bpsm * H->num_sms);
  return launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, threads, smem, in, out, nf * in.rows, lpc, (const double2*)H->tw64[0], H->derr);
    CKL();
    return CUP_OK;
  });
}

template <typename RIN>
int launch_rows_pipe(cup_handle* H, const char* name, const RIN* const* f, int nf, double* out) {
  switch (H->nx / 2) {
    case 8: return launch_rows_pipe_M<8, RIN>(H, name, f, nf, out);
    case 16: return launch_rows_pipe_M<16, RIN>(H, name, f, nf, out);
    case 32: return launch_rows_pipe_M<32, RIN>(H, name, f, nf, out);
    case 64: return launch_rows_pipe_M<64, RIN>(H, name, f, nf, out);
    case 128: return launch_rows_pipe_M<128, RIN>(H, name, f, nf, out);
  }
  return fail(H, CUP_ERR_ARG, "unsupported nx %d", H->nx);
}
int launch_rows_pipe(cup_handle* H, const char* name, double* buf) {
  const double* f[1] = {buf};
  return launch_rows_pipe<double>(H, name, f, 1, buf);
}

// First Hartley x pass of the RHS formed from f (RHS never stored).
template <int M, typename T>
int launch_rows_rhs_M(cup_handle* H, const char* name, void* const* f, double* out, DtArg dt) {
  constexpr int N = 2 * M, TPL = M / 8, lpc = 256 / TPL;
  constexpr bool PAD = FFTPlan<M>::nstages > 1;
  const size_t smem = (size_t)lpc * N * sizeof(double) + (PAD ? (size_t)lpc * 2 * (M + M / 8) * sizeof(double) : 0) +
                      FFTPlan<M>::rows_table_len() * sizeof(double2) + 128;
  auto kern = k_dht_rows_rhs<M, T>;
  int bpsm = 0;
  int rc = prepare_kernel(H, kern, smem, 256, &bpsm);
  if (rc) return rc;
  return launch_named(H, name, [&]() -> int {
    klaunch(H, kern, H->ny * H->nz / lpc, 256, smem, (const T*)f[0], (const T*)f[1], (const T*)f[2], out, dt, H->h, H->ny,
            H->nz, (const double2*)H->tw64[0]);
    CKL();
    return CUP_OK;
  });
}

// Hartley y or z pass (z: with the spectral divide and the inverse when DIVIDE),
// in place on buf; y: of nf fields one after the other.
template <int M, int AXIS, bool DIVIDE>
int launch_cols_M(cup_handle* H, double* buf, int nf) {
  // 16 x-columns per tile (128-B rows), NB tile buffers; 256-long lines: the
  // 8-thread plan (radix 16, then radix 8 fused with the split)
  constexpr bool T8 = M == 128;
  constexpr int N = 2 * M, TPL = T8 ? 8 : M / 8, NB = T8 ? 2 : 3, W = 16;
  if (AXIS == 2 && H->cfg.z_halo)
    return fail(H, CUP_ERR_STATE, "a z-slab handle has no z transform (the Poisson solve runs over the ranks)");
  CUtensorMap map;
  int rc = make_map(H, &map, buf, tma_dtype<double>(), sizeof(double), W, AXIS == 1 ? N : 1, AXIS == 2 ? N : 1, nf);
  if (rc) return rc;
  const size_t smem = (size_t)NB * N * W * sizeof(double) + FFTPlan<M>::table_len() * sizeof(double2) +
                      NB * sizeof(uint64_t) + (DIVIDE ? (M / 2 + 1) * sizeof(double) : 0) + 128;
  auto kern = k_dht_cols_pipe<M, double, AXIS, DIVIDE, W, NB, T8>;
  const int threads = W * TPL;
  int bpsm = 0;
  rc = prepare_kernel(H, kern, smem, threads, &bpsm);
  if (rc) return rc;
  const int ntx = H->nx / W;
  const int ntiles = ntx * (AXIS == 1 ? nf * H->nz : H->ny);
  const int grid = std::min(ntiles, bpsm * H->num_sms);
  SpectralParams sp{H->cosx, H->cosy, H->cosz, H->norm_factor, H->nx, H->spec_ny, H->nz, H->spec_y0};
  return launch_named(H, AXIS == 1 ? "dht_y" : "dht_z_solve", [&]() -> int {
    klaunch(H, kern, grid, threads, smem, map, ntx, ntiles, (const double2*)H->tw64[AXIS], sp, H->derr);
    CKL();
    return CUP_OK;
  });
}

template <int AXIS, bool DIVIDE>
int launch_cols(cup_handle* H, double* buf, int nf = 1) {
  const int N = AXIS == 1 ? H->ny : H->nz;
  switch (N / 2) {
    case 8: return launch_cols_M<8, AXIS, DIVIDE>(H, buf, nf);
    case 16: return launch_cols_M<16, AXIS, DIVIDE>(H, buf, nf);
    case 32: return launch_cols_M<32, AXIS, DIVIDE>(H, buf, nf);
    case 64: return launch_cols_M<64, AXIS, DIVIDE>(H, buf, nf);
    case 128: return launch_cols_M<128, AXIS, DIVIDE>(H, buf, nf);
  }
  return fail(H, CUP_ERR_ARG, "unsupported line length %d", N);
}

// ---- the pressure solve's passes (pfft.cuh) --------------------------------
// Calls fn<M>() for the line length N = 2 M.
#define PFFT_DISPATCH(N, call)                                          \
  switch ((N) / 2) {                                                    \
    case 8: { constexpr int M = 8; return call; }                       \
    case 16: { constexpr int M = 16; return call; }                     \
    case 32: { constexpr int M = 32; return call; }                     \
    case 64: { constexpr int M = 64; return call; }                     \
    case 128: { constexpr int M = 128; return call; }                   \
  }                                                                     \
  return fail(H, CUP_ERR_ARG, "unsupported line length %d", (int)(N))

template <typename S>
const typename Cplx<S>::T* ptable(cup_handle* H, int axis) {
  if constexpr (sizeof(S) == 8) return H->ptw64[axis];
  else return H->ptw32[axis];
}

// x pass: MODE as k_pfft_x; rev walks the tiles backwards (a pass that starts
// where the pass before it ended finds that part of the array in L2: at 256^3
// FP64 the y pass took 43.0 against 47.1 us and the last x pass 45.2 against 51.1).
// Warps per CTA and buffers per warp as measured at 256^3: FP32 forward 27.4 us
// (2 to 8 warps and 2 to 4 buffers within 1 us), FP64 45 us, with p 65.5 us.
template <int M, typename S, int MODE>
int launch_pfft_x_M(cup_handle* H, const char* name, const S* in, S* out, S* out2, int rev, const int* skip) {
  constexpr bool ADDP = MODE == PROW_INV_ADDP;
  constexpr int NB = sizeof(S) == 4 ? 3 : 2, WARPS = ADDP ? 2 : 4;
  constexpr bool LATE = sizeof(S) == 4 || ADDP;
  using Rw = PRows<M>;
  const size_t smem = (size_t)WARPS * NB * Rw::ELEMS * (ADDP ? 2 : 1) * sizeof(S) + M * sizeof(typename Cplx<S>::T) +
                      WARPS * NB * sizeof(uint64_t) + 8 * sizeof(double) + 128;
  auto kern = k_pfft_x<M, S, MODE, NB, WARPS, LATE>;
  int bpsm = 0;
  int rc = prepare_kernel(H, kern, smem, 32 * WARPS, &bpsm);
  if (rc) return rc;
  const int ntiles = H->ny * H->nz / Rw::ROWS;
  const int grid = std::min((ntiles + WARPS - 1) / WARPS, bpsm * H->num_sms);
  return launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, 32 * WARPS, smem, in, out, out2, (const double*)H->dstate->cmean, ilog2(H->ny), ntiles, rev,
            ptable<S>(H, 0), H->derr, skip);
    CKL();
    return CUP_OK;
  });
}
template <typename S, int MODE>
int launch_pfft_x(cup_handle* H, const char* name, const S* in, S* out, S* out2, int rev, const int* skip) {
  PFFT_DISPATCH(H->nx, (launch_pfft_x_M<M, S, MODE>(H, name, in, out, out2, rev, skip)));
}

// y pass in place. L: double (16-column tiles) or F2 (FP32, 32 columns in pairs).
template <int M, typename L, bool INV>
int launch_pfft_y_M(cup_handle* H, const char* name, typename Lane<L>::S* buf, int rev, const int* skip) {
  using S = typename Lane<L>::S;
  constexpr int W = sizeof(S) == 8 ? 16 : 32, NB = 2, N = 2 * M;
  using Tile = PTile<M, L, W>;
  if (H->nx % W) return fail(H, CUP_ERR_ARG, "nx must be a multiple of %d for this precision", W);
  CUtensorMap map;
  int rc = make_map(H, &map, buf, tma_dtype<S>(), sizeof(S), W, N, Tile::P);
  if (rc) return rc;
  const size_t smem = (size_t)NB * N * W * Tile::P * sizeof(S) + M * sizeof(typename Cplx<S>::T) +
                      NB * sizeof(uint64_t) + 128;
  auto kern = k_pfft_y<M, L, INV, W, NB>;
  int bpsm = 0;
  if ((rc = prepare_kernel(H, kern, smem, Tile::THREADS, &bpsm))) return rc;
  const int ntx = H->nx / W, ntiles = ntx * (H->nz / Tile::P);
  const int grid = std::min(ntiles, bpsm * H->num_sms);
  return launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, Tile::THREADS, smem, map, ntx, ntiles, rev, ptable<S>(H, 1), H->derr, skip);
    CKL();
    return CUP_OK;
  });
}
template <typename L, bool INV>
int launch_pfft_y(cup_handle* H, const char* name, typename Lane<L>::S* buf, int rev, const int* skip) {
  PFFT_DISPATCH(H->ny, (launch_pfft_y_M<M, L, INV>(H, name, buf, rev, skip)));
}

// z pass with the spectral divide, from `in` to `out` (FP64: the same array).
template <int M, typename T>
int launch_pfft_z_M(cup_handle* H, const char* name, T* in, double* out, const int* skip) {
  constexpr bool MIXED = sizeof(T) == 4;
  constexpr int W = 16, NB = 2, N = 2 * M;
  using Tile = PTile<M, T, W>;
  constexpr size_t ELEMS = (size_t)N * W * Tile::P;
  CUtensorMap map_in, map_out;
  int rc = make_map(H, &map_in, in, tma_dtype<T>(), sizeof(T), W, Tile::P, N);
  if (!rc) rc = make_map(H, &map_out, out, tma_dtype<double>(), sizeof(double), W, Tile::P, N);
  if (rc) return rc;
  const size_t smem = NB * ELEMS * sizeof(T) + (MIXED ? ELEMS * sizeof(double) : 0) +
                      M * (sizeof(double2) + sizeof(double) + (MIXED ? sizeof(float2) : 0)) + NB * sizeof(uint64_t) + 128;
  auto kern = k_pfft_z<M, T, W, NB>;
  int bpsm = 0;
  if ((rc = prepare_kernel(H, kern, smem, Tile::THREADS, &bpsm))) return rc;
  const int ntx = H->nx / W, ntiles = ntx * (H->ny / Tile::P);
  const int grid = std::min(ntiles, bpsm * H->num_sms);
  const PSpectral sp{H->pcos[0], H->pcos[1], H->pcos[2], H->pnorm};
  return launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, Tile::THREADS, smem, map_in, map_out, ntx, ntiles, ptable<T>(H, 2),
            (const double2*)H->ptw64[2], sp, H->derr, skip);
    CKL();
    return CUP_OK;
  });
}
template <typename T>
int launch_pfft_z(cup_handle* H, const char* name, T* in, double* out, const int* skip) {
  PFFT_DISPATCH(H->nz, (launch_pfft_z_M<M, T>(H, name, in, out, skip)));
}

// First x pass of the FP64 solve on the RHS formed from f (RHS never stored).
// box: plus the obstacle's terms on its box (H->box_delta).
template <int M, typename T>
int launch_pfft_x_rhs_M(cup_handle* H, const char* name, void* const* f, double* out, DtArg dt, bool box) {
  constexpr int WARPS = 4;
  using Rw = PRows<M>;
  const size_t smem = (size_t)WARPS * Rw::ELEMS * sizeof(double) + M * sizeof(double2) + 128;
  auto kern = k_pfft_x_rhs<M, T, WARPS>;
  int bpsm = 0;
  int rc = prepare_kernel(H, kern, smem, 32 * WARPS, &bpsm);
  if (rc) return rc;
  const int ntiles = H->ny * H->nz / Rw::ROWS;
  return launch_named(H, name, [&]() -> int {
    klaunch(H, kern, (ntiles + WARPS - 1) / WARPS, 32 * WARPS, smem, (const T*)f[0], (const T*)f[1], (const T*)f[2], out,
            dt, H->h, H->ny, H->nz, ntiles, (const double2*)H->ptw64[0], H->box,
            box ? (const double*)H->box_delta : nullptr);
    CKL();
    return CUP_OK;
  });
}
template <typename T>
int launch_pfft_x_rhs(cup_handle* H, const char* name, void* const* f, double* out, DtArg dt, bool box) {
  PFFT_DISPATCH(H->nx, (launch_pfft_x_rhs_M<M, T>(H, name, f, out, dt, box)));
}

template <typename T>
int launch_rows_rhs(cup_handle* H, const char* name, void* const* f, double* out, DtArg dt) {
  PFFT_DISPATCH(H->nx, (launch_rows_rhs_M<M, T>(H, name, f, out, dt)));
}

// The passes of an FP64 solve after the first x pass, from `work` to `out`.
int pfft_finish(cup_handle* H, const char* name_x, double* work, double* out, double* out2 = nullptr) {
  int rc;
  if ((rc = launch_pfft_y<double, false>(H, "dht_y", work, 1, nullptr))) return rc;
  if ((rc = launch_pfft_z<double>(H, "dht_z_solve", work, work, nullptr))) return rc;
  if ((rc = launch_pfft_y<double, true>(H, "dht_y", work, 0, nullptr))) return rc;
  return launch_pfft_x<double, PROW_INV>(H, name_x, work, out, out2, 1, nullptr);
}

// The same with Hartley passes.
int hartley_finish(cup_handle* H, const char* name_x, double* work, double* out) {
  int rc;
  const double* f[1] = {work};
  if ((rc = launch_cols<1, false>(H, work))) return rc;
  if ((rc = launch_cols<2, true>(H, work))) return rc;
  if ((rc = launch_cols<1, false>(H, work))) return rc;
  return launch_rows_pipe<double>(H, name_x, f, 1, out);
}

// Whether a step of the handle's CFL number can be beyond its stability limit,
// in FP64. Explicit diffusion and upwind3 damp the shortest wave by 12 nu dt / h^2
// + 4 umax dt / h a step, which may not exceed 2, and dt = CFL min(h^2 / nu, h /
// umax): with CFL <= 1/8 the step is stable whatever the flow. Beyond, a run
// amplifies the rounding of its steps (at CFL 0.5 and nu = 0.01 on sides of 256
// cells up to 1e9 times in 38 steps), so that any other order of the same
// arithmetic shows in its FP64 results: the four taps of the upwind stages and
// the packed transforms of the pressure, either alone, moved u by 1e-9 to 5e-7.
// Such runs keep their arithmetic: the one-sided stencils of both signs
// (k_advect_zq, SELECT) and the Hartley passes of dht.cuh for the pressure. An
// upwind3 step takes 48 us then instead of 42 at 64^3, 136 instead of 117 at
// 128^3, 914 instead of 780 at 256^3. FP32 runs take the same passes either way:
// their order of arithmetic also depends on how their sums are split.
bool amplifies_rounding(const cup_handle* H) { return !H->fp32 && H->cfg.CFL > 0.125; }

// p = f . b over the three axes, FP64, the RHS in `work` (overwritten). Handles
// whose steps can amplify rounding (amplifies_rounding) run the Hartley passes.
int fft_poisson(cup_handle* H, double* work, double* out) {
  int rc;
  if (amplifies_rounding(H)) {
    if ((rc = launch_rows_pipe(H, "dht_x", work))) return rc;
    return hartley_finish(H, "dht_x", work, out);
  }
  if ((rc = launch_pfft_x<double, PROW_FWD>(H, "dht_x", work, work, nullptr, 0, nullptr))) return rc;
  return pfft_finish(H, "dht_x", work, out);
}

// Correction solve of the defect-correction loop, mixed precision: the x and y
// forward transforms of the FP32 residual in FP32; the z pass widens to FP64
// between the spectral factor and the inverse; the y and x inverse transforms
// in FP64, the last one adding the correction to p (minus the parity-class
// means of p measured by the preceding residual pass). An FP32 inverse would
// leave white rounding noise in the correction whose wide-Laplacian image is
// large next to a smooth residual; with the inverse in FP64 one solve contracts
// the residual by about 1e-7 whatever its spectrum.
int dc_correction_solve(cup_handle* H, double* p, const int* skip) {
  int rc;
  if ((rc = launch_pfft_x<float, PROW_FWD>(H, "dht_x", H->work32, H->work32, nullptr, 0, skip))) return rc;
  if ((rc = launch_pfft_y<F2, false>(H, "dht_y", H->work32, 0, skip))) return rc;
  if ((rc = launch_pfft_z<float>(H, "dht_z_solve_mixed", H->work32, H->work64, skip))) return rc;
  if ((rc = launch_pfft_y<double, true>(H, "dht_y_f64", H->work64, 0, skip))) return rc;
  return launch_pfft_x<double, PROW_INV_ADDP>(H, "dht_x_update_p", H->work64, p, nullptr, 1, skip);
}

int box_grid(const Box& b) {
  const long long n = (long long)b.n[0] * b.n[1] * b.n[2];
  return (int)std::max<long long>(1, std::min<long long>(kBoxBlocksMax, (n + kBoxThreads - 1) / kBoxThreads));
}

// The warm-start history of the FP32 pressure stage is only valid along one
// trajectory of cup_step/cup_run; anything else that sets the velocity or the
// pressure restarts it.
void reset_pressure_history(cup_handle* H) {
  H->p_valid = 0;
  H->pred_ready = false;
}

int dev_error_status(cup_handle* H, int e) {
  if (e & kDevErrMbarTimeout) return fail(H, CUP_ERR_TIMEOUT, "device wait timed out (mbarrier)");
  if (e & kDevErrBulkTimeout) return fail(H, CUP_ERR_TIMEOUT, "device wait timed out (bulk store)");
  return CUP_OK;
}

int check_dev_error(cup_handle* H) {
  int e = 0;
  CK(cudaMemcpy(&e, H->derr, sizeof(int), cudaMemcpyDeviceToHost));
  return dev_error_status(H, e);
}

// One stream-ordered read of the device state (the error word included).
int read_state(cup_handle* H) {
  CK(cudaMemcpyAsync(H->hstate, H->dstate, sizeof(DevState), cudaMemcpyDeviceToHost, H->stream));
  CK(cudaStreamSynchronize(H->stream));
  return dev_error_status(H, H->hstate->err_word);
}

// ---- typed pipeline pieces -------------------------------------------------
// Launches one k_advect_zq pass: fields `in` (stencil), `base` (stage-2
// point-wise u^n, else unused), output `out`. Grids of nx 64, 128 or 256 take
// the compile-time-nx kernels; other shapes the same kernel with runtime sizes.
// (The planes per item stay a runtime count: unrolling a whole 20-plane item
// measured slower for the FP64 stages than the 10-plane loop.)
template <typename T, int SCHEME, int TY, int NS, int CPT, int NXC, bool SELECT>
int launch_advect_sized(cup_handle* H, const char* name, void* const* in, void* const* base, void* const* out,
                        DtArg dt) {
  constexpr int G = AdvectTraits<SCHEME>::G;
  const int cells = TY * H->nx;
  if (cells % CPT || cells / CPT > 512 || H->ny % TY)
    return fail(H, CUP_ERR_ARG, "advection tile does not fit the grid");
  AdvectMaps maps;
  for (int f = 0; f < 3; ++f) {
    int rc = make_row_maps<T>(H, &maps.f[f], in[f], TY, G);
    if (rc) return rc;
  }
  if (NXC && NXC != H->nx) return fail(H, CUP_ERR_ARG, "advection specialisation mismatch");
  const size_t smem = advect_smem_bytes<T, SCHEME, TY, NS>(H->nx) + 128;
  auto kern = k_advect_zq<T, SCHEME, TY, NS, CPT, NXC, SELECT>;
  const int threads = cells / CPT;
  int bpsm = 0;
  int rc = prepare_kernel(H, kern, smem, threads, &bpsm);
  if (rc) return rc;
  const int zc = planes_per_item(H, TY, G, bpsm);
  StreamGeom g{H->nx, H->ny, H->nz, ilog2(H->nx), zc, H->ny / TY, (H->ny / TY) * (H->nz / zc)};
  const int grid = std::min(g.n_items, bpsm * H->num_sms);
  return launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, threads, smem, maps, g, (const T*)base[0], (const T*)base[1], (const T*)base[2], (T*)out[0],
            (T*)out[1], (T*)out[2], dt, H->h, H->cfg.nu, H->uinf[0], H->uinf[1], H->uinf[2], H->derr);
    CKL();
    return CUP_OK;
  });
}

template <typename T, int SCHEME, int TY, int NS, int CPT, bool SELECT = false>
int launch_advect(cup_handle* H, const char* name, void* const* in, void* const* base, void* const* out, DtArg dt) {
  switch (H->nx) {
    case 64: return launch_advect_sized<T, SCHEME, TY, NS, CPT, 64, SELECT>(H, name, in, base, out, dt);
    case 128: return launch_advect_sized<T, SCHEME, TY, NS, CPT, 128, SELECT>(H, name, in, base, out, dt);
    case 256: return launch_advect_sized<T, SCHEME, TY, NS, CPT, 256, SELECT>(H, name, in, base, out, dt);
    default: break;
  }
  return launch_advect_sized<T, SCHEME, TY, NS, CPT, 0, SELECT>(H, name, in, base, out, dt);
}

// Launches one packed-FP32 upwind3 stage (k_advect_zq_f2): `in` stencil
// fields, `base` the stage-2 point-wise u^n, `out` the result.
// NXC: compile-time nx (0: runtime).
template <bool STAGE2, int TY, int NS, int PPT, int NXC = 0>
int launch_advect_f2(cup_handle* H, const char* name, void* const* in, void* const* base, void* const* out, DtArg dt) {
  constexpr int G = 2;
  const int pairs = TY * H->nx / 2;
  if (pairs % PPT || pairs / PPT > 512 || H->ny % TY) return fail(H, CUP_ERR_ARG, "advection tile does not fit the grid");
  AdvectF2Maps maps;
  for (int f = 0; f < 3; ++f) {
    int rc = make_row_maps<float>(H, &maps.f[f], in[f], TY, G);
    if (!rc) rc = make_map(H, &maps.base[f], STAGE2 ? base[f] : in[f], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, sizeof(float),
                           H->nx, TY, 1);
    if (rc) return rc;
  }
  if (NXC && NXC != H->nx) return fail(H, CUP_ERR_ARG, "advection specialisation mismatch");
  const size_t smem = advect_f2_smem_bytes<STAGE2, TY, NS>(H->nx) + 128;
  auto kern = k_advect_zq_f2<STAGE2, TY, NS, PPT, NXC>;
  const int threads = pairs / PPT;
  int bpsm = 0;
  int rc = prepare_kernel(H, kern, smem, threads, &bpsm);
  if (rc) return rc;
  const int zc = planes_per_item(H, TY, G, bpsm);
  StreamGeom g{H->nx, H->ny, H->nz, ilog2(H->nx), zc, H->ny / TY, (H->ny / TY) * (H->nz / zc)};
  const int grid = std::min(g.n_items, bpsm * H->num_sms);
  return launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, threads, smem, maps, g, (float*)out[0], (float*)out[1], (float*)out[2], dt, H->h,
                                             H->cfg.nu, H->uinf[0], H->uinf[1], H->uinf[2], H->derr);
    CKL();
    return CUP_OK;
  });
}

// FP32 upwind3 stages: packed FP32x2 kernels (shared by the forward step and
// the adjoint's stage recompute, so both see the same u1). Grids of nx 64, 128
// or 256 take the compile-time-nx kernels; other shapes the same kernel with
// runtime sizes.
template <bool STAGE2, int TY, int NS, int PPT>
int launch_advect_f2_sized(cup_handle* H, const char* name, void* const* in, void* const* base, void* const* out,
                           DtArg dt) {
  switch (H->nx) {
    case 64: return launch_advect_f2<STAGE2, TY, NS, PPT, 64>(H, name, in, base, out, dt);
    case 128: return launch_advect_f2<STAGE2, TY, NS, PPT, 128>(H, name, in, base, out, dt);
    case 256: return launch_advect_f2<STAGE2, TY, NS, PPT, 256>(H, name, in, base, out, dt);
    default: break;
  }
  return launch_advect_f2<STAGE2, TY, NS, PPT>(H, name, in, base, out, dt);
}
int upwind_stage1_f32(cup_handle* H, const char* name, void* const* in, void* const* out, DtArg dt) {
  return launch_advect_f2_sized<false, 8, 6, 2>(H, name, in, in, out, dt);
}
int upwind_stage2_f32(cup_handle* H, const char* name, void* const* in, void* const* base, void* const* out,
                      DtArg dt) {
  return launch_advect_f2_sized<true, 4, 6, 1>(H, name, in, base, out, dt);
}

// FP64 upwind3 stage (shared like the FP32 ones): `base` the stage-2 point-wise u^n.
template <typename T, int STAGE>
int upwind_stage_f64(cup_handle* H, const char* name, void* const* in, void* const* base, void* const* out, DtArg dt) {
  if (amplifies_rounding(H)) return launch_advect<T, STAGE, 4, 4, 2, true>(H, name, in, base, out, dt);
  return launch_advect<T, STAGE, 4, 4, 2>(H, name, in, base, out, dt);
}

template <typename T>
int do_advect_diffuse(cup_handle* H, DtArg dt) {
  constexpr bool F32 = std::is_same<T, float>::value;
  int rc;
  void* uvw[3] = {H->u, H->v, H->w};
  void* tmp[3] = {H->tu, H->tv, H->tw};
  // tile height TY, ring depth NS, cells per thread CPT: the shapes measured
  // best at 256^3 for each scheme and precision (the FP32 upwind3 stages run
  // the packed FP32x2 kernels)
  if (H->cfg.scheme == CUP_SCHEME_REF) {
    if constexpr (F32) rc = launch_advect<T, 0, 8, 5, 4>(H, "advect_diffuse_ref", uvw, uvw, tmp, dt);
    else rc = launch_advect<T, 0, 4, 5, 2>(H, "advect_diffuse_ref", uvw, uvw, tmp, dt);
  } else {
    void* st1[3] = {H->u1, H->v1, H->w1};
    if constexpr (F32) {
      if ((rc = upwind_stage1_f32(H, "upwind3_stage1", uvw, st1, dt))) return rc;
      rc = upwind_stage2_f32(H, "upwind3_stage2", st1, uvw, tmp, dt);
    } else {
      if ((rc = upwind_stage_f64<T, 1>(H, "upwind3_stage1", uvw, uvw, st1, dt))) return rc;
      rc = upwind_stage_f64<T, 2>(H, "upwind3_stage2", st1, uvw, tmp, dt);
    }
  }
  if (rc) return rc;
  // UpdateAndCorrectInflow's tmp -> u copy (AdvectionDiffusion.cpp:315-328) is a pointer swap.
  std::swap(H->u, H->tu);
  std::swap(H->v, H->tv);
  std::swap(H->w, H->tw);
  return CUP_OK;
}

template <typename T>
int do_pressure_rhs(cup_handle* H, DtArg dt) {
  int rc;
  const void* uvw[3] = {H->u, H->v, H->w};
  OpPressureRHS<T> op{H->rhs, dt, H->h, H->nx, H->ny};
  rc = launch_stream<T, 3, 1, 4, 4>(H, "pressure_rhs", uvw, op);
  if (rc) return rc;
  if (H->has_sphere) {
    const int gb = box_grid(H->box);
    {
      int rc_ = launch_named(H, "rhs_obstacle", [&]() -> int {
        klaunch(H, k_rhs_obstacle<T>, gb, kBoxThreads, 0, H->rhs, (const T*)H->chi, H->box, H->nx, H->ny, H->nz,
                                                         partial(H, P_RHSOB));
        CKL();
        return CUP_OK;
      });
      if (rc_) return rc_;
    }
    {
      int rc_ = launch_named(H, "finalize_rhs_obstacle", [&]() -> int {
        klaunch(H, k_finalize_rhs_obstacle, 1, 256, 0, partial(H, P_RHSOB), gb, H->dstate);
        CKL();
        return CUP_OK;
      });
      if (rc_) return rc_;
    }
    {
      int rc_ = launch_named(H, "rhs_obstacle_correct", [&]() -> int {
        klaunch(H, k_rhs_obstacle_correct<T>, gb, kBoxThreads, 0, H->rhs, (const T*)H->chi, H->box, H->nx, H->ny,
                                                                 H->nz, &H->dstate->corr, (double*)nullptr);
        CKL();
        return CUP_OK;
      });
      if (rc_) return rc_;
    }
  }
  return CUP_OK;
}

// The sphere's RHS terms on its box, for the passes that form b from u*: b0 of u*
// on the box, the obstacle terms (bulk source, surface sums, correction) on
// that box array, and H->box_delta = b2 - b0.
// D: the type the velocity differences are formed in, as the pass that adds
// box_delta does; f: the fields (u* of the step), save_b0: a copy of b0 on the box.
// Against forming b as an array first (37 us at 256x128x128, then read again):
// an obstacle gradient of 4 steps there 3.92 -> 3.78 ms.
template <typename T, typename D>
int do_box_rhs_terms(cup_handle* H, DtArg dt, void* const* f, double* save_b0 = nullptr) {
  if (H->box.count() > H->box_cap) return fail(H, CUP_ERR_STATE, "obstacle box larger than its buffers");
  const int gb = box_grid(H->box);
  int rc = launch_named(H, "box_rhs_obstacle", [&]() -> int {
    klaunch(H, k_box_rhs_obstacle<T, D>, gb, kBoxThreads, 0, (const T*)f[0], (const T*)f[1], (const T*)f[2],
            (const T*)H->chi, H->box, H->nx, H->ny, H->nz, dt, H->h, H->box_b, H->box_delta, save_b0,
            partial(H, P_RHSOB));
    CKL();
    return CUP_OK;
  });
  if (!rc)
    rc = launch_named(H, "finalize_rhs_obstacle", [&]() -> int {
      klaunch(H, k_finalize_rhs_obstacle, 1, 256, 0, partial(H, P_RHSOB), gb, H->dstate);
      CKL();
      return CUP_OK;
    });
  if (!rc)
    rc = launch_named(H, "rhs_obstacle_correct", [&]() -> int {
      klaunch(H, k_rhs_obstacle_correct<T, true>, gb, kBoxThreads, 0, H->box_b, (const T*)H->chi, H->box, H->nx,
              H->ny, H->nz, &H->dstate->corr, H->box_delta);
      CKL();
      return CUP_OK;
    });
  return rc;
}

double dc_tol(const cup_handle* H) { return H->cfg.dc_tol > 0 ? H->cfg.dc_tol : 1e-10; }
int dc_max_iter(const cup_handle* H) { return H->cfg.dc_max_iter > 0 ? H->cfg.dc_max_iter : 2; }
int dc_min_iter(const cup_handle* H) {
  return std::min(dc_max_iter(H), H->cfg.dc_min_iter > 0 ? H->cfg.dc_min_iter : 1);
}

// Launches one k_pres_zq pass; returns the grid size (number of partials).
template <typename T, int MODE, int TY, int NS, int CPT, int NXC, bool BD>
int launch_pzq_sized(cup_handle* H, const char* name, double* pw, double* partials, const double* rmean, DtArg dt,
                     int* grid_out, const int* skip, int pred_order, double* pred_out, void* const* out) {
  const int cells = TY * H->nx;
  if (cells % CPT || cells / CPT > 512 || H->ny % TY)
    return fail(H, CUP_ERR_ARG, "pressure tile does not fit the grid");
  PzqMaps maps;
  int rc = make_row_maps<double>(H, &maps.p, pw, TY, 2);
  if (!rc) rc = make_map(H, &maps.h_main, pred_order >= 1 ? H->p : pw, CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                         sizeof(double), H->nx, TY, 1);
  const void* f[3] = {H->u, H->v, H->w};
  for (int q = 0; q < 3 && !rc; ++q) rc = make_map(H, &maps.f_main[q], f[q], tma_dtype<T>(), sizeof(T), H->nx, TY, 1);
  if (!rc) rc = make_row_maps<T>(H, &maps.v, H->v, TY, 1);
  if (rc) return rc;
  if (NXC && NXC != H->nx) return fail(H, CUP_ERR_ARG, "pressure specialisation mismatch");
  const size_t smem = pzq_smem_bytes_host<T, MODE, TY, NS>(H->nx) + 128;
  auto kern = k_pres_zq<T, MODE, TY, NS, CPT, NXC, BD>;
  const int threads = cells / CPT;
  int bpsm = 0;
  if ((rc = prepare_kernel(H, kern, smem, threads, &bpsm))) return rc;
  const int zc = planes_per_item(H, TY, 2, bpsm);
  StreamGeom geo{H->nx, H->ny, H->nz, ilog2(H->nx), zc, H->ny / TY, (H->ny / TY) * (H->nz / zc)};
  const int grid = std::min(geo.n_items, bpsm * H->num_sms);
  if (grid > kPartialCap / pzq_partials_per_cta<MODE>())
    return fail(H, CUP_ERR_ARG, "too many CTAs for the partial buffers");
  if (BD && !H->box_delta) return fail(H, CUP_ERR_STATE, "no obstacle RHS terms on the box");
  PzqParams prm{dt, H->h, {H->uinf[0], H->uinf[1], H->uinf[2]}, pred_order, pred_out, H->box, H->box_delta};
  T* o[3] = {nullptr, nullptr, nullptr};
  if (out)
    for (int q = 0; q < 3; ++q) o[q] = (T*)out[q];
  rc = launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, threads, smem, maps, geo, o[0], o[1], o[2], H->work32, partials, rmean, prm,
                                             H->derr, skip);
    CKL();
    return CUP_OK;
  });
  if (rc) return rc;
  if (grid_out) *grid_out = grid;
  return CUP_OK;
}

// Grids of nx 64, 128 or 256 take the compile-time-nx kernels; other shapes the
// same kernel with runtime sizes. BD: b carries the obstacle terms on the box
// (H->box_delta).
template <typename T, int MODE, int TY, int NS, int CPT, bool BD = false>
int launch_pzq(cup_handle* H, const char* name, double* pw, double* partials, const double* rmean, DtArg dt,
               int* grid_out, const int* skip, int pred_order = -1, double* pred_out = nullptr,
               void* const* out = nullptr) {
  switch (H->nx) {
    case 64:
      return launch_pzq_sized<T, MODE, TY, NS, CPT, 64, BD>(H, name, pw, partials, rmean, dt, grid_out, skip, pred_order,
                                                            pred_out, out);
    case 128:
      return launch_pzq_sized<T, MODE, TY, NS, CPT, 128, BD>(H, name, pw, partials, rmean, dt, grid_out, skip,
                                                             pred_order, pred_out, out);
    case 256:
      return launch_pzq_sized<T, MODE, TY, NS, CPT, 256, BD>(H, name, pw, partials, rmean, dt, grid_out, skip,
                                                             pred_order, pred_out, out);
    default: break;
  }
  return launch_pzq_sized<T, MODE, TY, NS, CPT, 0, BD>(H, name, pw, partials, rmean, dt, grid_out, skip, pred_order,
                                                       pred_out, out);
}

int launch_finalize_residual(cup_handle* H, const double* partials, int stride, int grid, int k) {
  const double inv_class = 8.0 / (double)H->n;
  return launch_named(H, "finalize_residual", [&]() -> int {
    klaunch(H, k_finalize_residual, 1, 18 * 32, 0, partials, stride, grid, H->dstate, dc_tol(H), k, dc_min_iter(H),
            dc_max_iter(H), inv_class);
    CKL();
    return CUP_OK;
  });
}

// FP32 defect-correction pressure stage without obstacle, in z-queue passes.
// Check k measures the FP64 residual of p after k correction solves; from
// k = 1 on the check is fused with the gradient correction, which writes
// u = u* - dt grad p to the spare velocity buffer, so the usual step (one
// solve meets the tolerance) is
//   RHS + check 0 (warm start p) -> FP32 solve -> gradient + check 1.
// When check k misses the tolerance, a residual pass writes the FP32 residual
// again, solve k + 1 refines p and the gradient pass runs again from u* (still
// intact). A check that meets the tolerance (after at least dc_min_iter
// solves) turns every later kernel of the loop into an exit at entry, so the
// loop needs no host round trip. Only the first gradient pass writes the next
// step's warm start.
// b is recomputed from u* in every pass (not stored); with the sphere the
// passes add its RHS terms on the box (H->box_delta, from do_box_rhs_terms).
template <typename T>
int do_pressure_dc_zq(cup_handle* H, DtArg dt) {
  const int max_iter = dc_max_iter(H);
  const int* conv = &H->dstate->converged;
  const bool box = H->has_sphere;
  double* W = H->p_pred;  // this step's pressure, starting from the warm start
  if (!H->pred_ready) CK(cudaMemcpyAsync(W, H->p, H->n * sizeof(double), cudaMemcpyDeviceToDevice, H->stream));
  int rc, grid = 0;
  if (box)
    rc = launch_pzq<T, PZQ_RHS_RES, 4, 6, 2, true>(H, "rhs_residual", W, partial(H, P_RES), nullptr, dt,
                                                             &grid, nullptr);
  else
    rc = launch_pzq<T, PZQ_RHS_RES, 4, 6, 2>(H, "rhs_residual", W, partial(H, P_RES), nullptr, dt, &grid,
                                                   nullptr);
  if (rc) return rc;
  if ((rc = launch_finalize_residual(H, partial(H, P_RES), 18, grid, 0))) return rc;
  const int order = std::min(H->p_valid, 1);  // valid levels among (p) before this step
  void* unew[3] = {H->tu, H->tv, H->tw};      // u^n is dead after the advection stages
  constexpr int kGradStride = pzq_partials_per_cta<PZQ_GRAD_CHECK>();
  for (int k = 1; k <= max_iter; ++k) {
    if (k > 1) {
      if (box)
        rc = launch_pzq<T, PZQ_RES, 4, 6, 2, true>(H, "dc_residual", W, partial(H, P_RES),
                                                             H->dstate->rmean, dt, &grid, conv);
      else
        rc = launch_pzq<T, PZQ_RES, 4, 6, 2>(H, "dc_residual", W, partial(H, P_RES), H->dstate->rmean, dt, &grid,
                                                   conv);
      if (rc) return rc;
    }
    if ((rc = dc_correction_solve(H, W, conv))) return rc;
    const int* skip = k > 1 ? conv : nullptr;
    const int pred = k == 1 ? order : -1;
    if (box)
      rc = launch_pzq<T, PZQ_GRAD_CHECK_BOX, 4, 4, 2, true>(H, "grad_p_check", W, partial(H, P_GRAD),
                                                                     H->dstate->rmean, dt, &H->n_grad_partials, skip,
                                                                     pred, H->p_old, unew);
    else
      rc = launch_pzq<T, PZQ_GRAD_CHECK, 4, 4, 2>(H, "grad_p_check", W, partial(H, P_GRAD), H->dstate->rmean, dt,
                                                        &H->n_grad_partials, skip, pred, H->p_old, unew);
    if (rc) return rc;
    if ((rc = launch_finalize_residual(H, partial(H, P_GRAD), kGradStride, H->n_grad_partials, k))) return rc;
  }
  H->grad_stride = kGradStride;
  H->grad_max_off = 18;
  H->grad_ke_off = 19;
  std::swap(H->u, H->tu);
  std::swap(H->v, H->tv);
  std::swap(H->w, H->tw);
  double* next_pred = H->p_old;
  H->p_old = H->p;
  H->p = W;
  H->p_pred = next_pred;
  H->p_valid = std::min(order + 1, 1);
  H->pred_ready = true;
  return CUP_OK;
}

// FP32 correction solve inside an FP64 defect-correction loop, warm-started
// from the current p, on the RHS array b. Check k: the FP64 residual
// r = b - h^3 L_2h p (TMA plane stream over p with a 2-ring halo), its norms
// and parity-class sums, FP32 r out; a one-block kernel decides convergence on
// the device. Solve k: the five FFT passes in FP32, the last x pass adding the
// correction to p in FP64. Kernels after convergence exit at entry.
int do_poisson_dc(cup_handle* H) {
  const double tol = dc_tol(H);
  const int max_iter = dc_max_iter(H);
  const int min_iter = dc_min_iter(H);
  const int* conv = &H->dstate->converged;
  const double inv_class = 8.0 / (double)H->n;
  int rc;
  for (int k = 0; k <= max_iter; ++k) {
    const void* pf[1] = {H->p};
    OpResidual op{H->rhs, H->work32, partial(H, P_RES), k > 0 ? H->dstate->rmean : nullptr, H->h / 4, H->nx, H->ny};
    int grid = 0;
    if ((rc = launch_stream<double, 1, 2, 4, 6>(H, "dc_residual", pf, op, &grid, k > 0 ? conv : nullptr))) return rc;
    {
      int rc_ = launch_named(H, "finalize_residual", [&]() -> int {
        klaunch(H, k_finalize_residual, 1, 18 * 32, 0, partial(H, P_RES), 18, grid, H->dstate, tol, k, min_iter, max_iter,
                inv_class);
        CKL();
        return CUP_OK;
      });
      if (rc_) return rc_;
    }
    if (k == max_iter) break;
    if ((rc = dc_correction_solve(H, H->p, conv))) return rc;
  }
  return CUP_OK;
}

// FP64 solve with the RHS of the fields f computed inside the first x pass (no
// RHS array). box: with the obstacle's terms (after do_box_rhs_terms of f).
template <typename T>
int do_solve_rhs_of(cup_handle* H, const char* name_rhs, const char* name_x, void* const* f, double* out, DtArg dt,
                    bool box = false) {
  if constexpr (std::is_same<T, double>::value)
    if (amplifies_rounding(H) && !box) {
      int rc = launch_rows_rhs<T>(H, name_rhs, f, H->rhs, dt);
      return rc ? rc : hartley_finish(H, name_x, H->rhs, out);
    }
  int rc = launch_pfft_x_rhs<T>(H, name_rhs, f, H->rhs, dt, box);
  return rc ? rc : pfft_finish(H, name_x, H->rhs, out);
}

// Poisson solve of the RHS array (operator-by-operator path, obstacles).
int do_poisson(cup_handle* H) {
  if (!H->fp32) return fft_poisson(H, H->rhs, H->p);
  return do_poisson_dc(H);
}

// Launches one k_grad_zq pass: out = in - dt/(2h) grad_c p; returns the grid
// size (number of partials). Grids of nx 64, 128 or 256 take the
// compile-time-nx kernels. Ring depth 4, measured: FP64 256^3 155 us (5: 162, 6:
// 164), FP32 256x128x128 18.6 us with two CTAs per SM (6: 22.7, one CTA).
template <typename T, bool REDUCE, int NXC>
int launch_grad_sized(cup_handle* H, const char* name, void* const* in, void* const* out, const double* p, DtArg dt,
                      int* grid_out) {
  constexpr int TY = 4, NS = 4, CPT = 2;
  GradMaps maps;
  int rc = make_row_maps<double>(H, &maps.p, p, TY, 1);
  for (int q = 0; q < 3 && !rc; ++q) rc = make_map(H, &maps.f[q], in[q], tma_dtype<T>(), sizeof(T), H->nx, TY, 1);
  if (rc) return rc;
  auto kern = k_grad_zq<T, REDUCE, TY, NS, CPT, NXC>;
  const size_t smem = grad_smem_bytes<T, TY, NS>(H->nx) + 128;
  const int threads = TY * H->nx / CPT;
  int bpsm = 0;
  if ((rc = prepare_kernel(H, kern, smem, threads, &bpsm))) return rc;
  const int zc = planes_per_item(H, TY, 1, bpsm);
  StreamGeom geo{H->nx, H->ny, H->nz, ilog2(H->nx), zc, H->ny / TY, (H->ny / TY) * (H->nz / zc)};
  const int grid = std::min(geo.n_items, bpsm * H->num_sms);
  if (grid > kPartialCap / 2) return fail(H, CUP_ERR_ARG, "too many CTAs for the partial buffers");
  const GradParams prm{dt, H->h, {H->uinf[0], H->uinf[1], H->uinf[2]}, H->box, H->has_sphere ? 1 : 0};
  rc = launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, threads, smem, maps, geo, (T*)out[0], (T*)out[1], (T*)out[2], partial(H, P_GRAD), prm,
            H->derr);
    CKL();
    return CUP_OK;
  });
  if (grid_out) *grid_out = grid;
  return rc;
}
template <typename T, bool REDUCE>
int launch_grad(cup_handle* H, const char* name, void* const* in, void* const* out, const double* p, DtArg dt,
                int* grid_out = nullptr) {
  switch (H->nx) {
    case 64: return launch_grad_sized<T, REDUCE, 64>(H, name, in, out, p, dt, grid_out);
    case 128: return launch_grad_sized<T, REDUCE, 128>(H, name, in, out, p, dt, grid_out);
    case 256: return launch_grad_sized<T, REDUCE, 256>(H, name, in, out, p, dt, grid_out);
    default: break;
  }
  return launch_grad_sized<T, REDUCE, 0>(H, name, in, out, p, dt, grid_out);
}

template <typename T>
int do_grad(cup_handle* H, DtArg dt) {
  void* u[3] = {H->u, H->v, H->w};
  H->grad_stride = 2;
  H->grad_max_off = 0;
  H->grad_ke_off = 1;
  return launch_grad<T, true>(H, "grad_p", u, u, H->p, dt, &H->n_grad_partials);
}

template <typename T>
int do_penalize(cup_handle* H, DtArg dt, const double* lambda_dev) {
  if (!H->has_sphere) {
    H->n_pen_partials = 0;
    return CUP_OK;
  }
  const int gb = box_grid(H->box);
  {
    int rc_ = launch_named(H, "penalize", [&]() -> int {
      klaunch(H, k_penalize<T>, gb, kBoxThreads, 0, (T*)H->u, (T*)H->v, (T*)H->w, (const T*)H->chi, H->sp_dev, H->box,
                                                   H->nx, H->ny, H->nz, H->h, dt, lambda_dev, H->lambda,
                                                   H->cfg.bImplicitPenalization, H->uinf[0], H->uinf[1], H->uinf[2],
                                                   partial(H, P_PEN));
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  H->n_pen_partials = gb;
  return CUP_OK;
}

template <typename T>
int do_surface_forces(cup_handle* H, double* part, int gb) {
  return launch_named(H, "surface_forces", [&]() -> int {
    klaunch(H, k_surface_forces<T>, gb, kBoxThreads, 0, (const T*)H->u, (const T*)H->v, (const T*)H->w,
            (const double*)H->p, (const SphereParams*)H->sp_dev, H->box, H->nx, H->ny, H->nz, H->h, H->cfg.nu, part);
    CKL();
    return CUP_OK;
  });
}

CflParams cfl_params(const cup_handle* H) {
  return CflParams{H->h, H->cfg.nu, H->cfg.CFL, H->cfg.rampup, H->cfg.DLM};
}

// next_dt: then the CFL time step, for the host's step counter.
template <typename T>
int do_max_u(cup_handle* H, int next_dt = 0) {
  const int grid = std::min<size_t>(H->num_sms * 4, (H->n + 255) / 256);
  {
    int rc_ = launch_named(H, "max_u", [&]() -> int {
      klaunch(H, k_max_u<T>, grid, 256, 0, (const T*)H->u, (const T*)H->v, (const T*)H->w, H->n, H->uinf[0], H->uinf[1],
                                          H->uinf[2], partial(H, P_MAX));
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  {
    int rc_ = launch_named(H, "finalize_max", [&]() -> int {
      klaunch(H, k_finalize_max, 1, 256, 0, partial(H, P_MAX), grid, H->dstate, next_dt, cfl_params(H),
              next_dt ? H->step : -1);
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  return CUP_OK;
}

// One full step of the hot-path pipeline (Simulation::timestep with the
// periodic pipeline of Simulation::setupOperators, source/Simulation.cpp:307-401):
// AdvectionDiffusion -> PressureRHS -> PressureProjection -> UpdateObstacles
// (forced sphere: no-op) -> Penalization, with grad-P and the reductions fused.
// Active box of the sphere at its current position: every cell within
// radius + (2 + SURFDH) h + 1 cell of the centre (SphereObstacle::FillBlocks
// safety margin, source/obstacles/Sphere.cpp:21-27, plus the surface-detection
// neighbour), wrapped periodically; the whole axis when it does not fit.
void sphere_box(cup_handle* H) {
  const int N[3] = {H->nx, H->ny, H->nz};
  for (int d = 0; d < 3; ++d) {
    const double r = H->sphere.radius + 3 * H->h;
    int lo = (int)std::floor((H->sphere.position[d] - r) / H->h - 0.5) - 1;
    int hi = (int)std::ceil((H->sphere.position[d] + r) / H->h - 0.5) + 1;
    int cnt = hi - lo + 1;
    if (cnt >= N[d]) {
      lo = 0;
      cnt = N[d];
    }
    lo = ((lo % N[d]) + N[d]) % N[d];
    H->box.lo[d] = lo;
    H->box.n[d] = cnt;
  }
}

// chi on the active box and the grid centre of mass (the chi and CoM parts
// of CreateObstacles, source/operators/ObstaclesCreate.cpp:51-136, 230-256).
int build_sphere_chi(cup_handle* H) {
  const int gb = box_grid(H->box);
  {
    int rc_ = launch_named(H, "sphere_chi", [&]() -> int {
      if (H->fp32)
        klaunch(H, k_sphere_chi<float>, gb, kBoxThreads, 0, (float*)H->chi, H->sp_dev, H->box, H->nx, H->ny, H->nz,
                                                                H->h, partial(H, P_CHI));
      else
        klaunch(H, k_sphere_chi<double>, gb, kBoxThreads, 0, (double*)H->chi, H->sp_dev, H->box, H->nx, H->ny,
                                                                 H->nz, H->h, partial(H, P_CHI));
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  return launch_named(H, "finalize_com", [&]() -> int {
    klaunch(H, k_finalize_com, 1, 256, 0, partial(H, P_CHI), gb, H->dstate, H->sp_dev);
    CKL();
    return CUP_OK;
  });
}

// CreateObstacles (source/operators/ObstaclesCreate.cpp:444-540) for a sphere
// that moves in the frame (transVel + uinf != 0): updateUinf, then
// Obstacle::update (source/obstacles/Obstacle.cpp:314-321) advances the
// position by dt (transVel + uinf) on the host mirror; chi is cleared on the
// old box and rebuilt with the centre of mass on the box of the new position.
// A sphere at rest in the frame keeps its chi (the rebuild would reproduce it).
int relocate_sphere(cup_handle* H);

int do_create_obstacles(cup_handle* H, double dt) {
  if (!H->has_sphere || !H->sphere_moves) return CUP_OK;
  if (H->sphere_free) {
    // updateUinf with the velocities of the last UpdateObstacles
    for (int d = 0; d < 3; ++d) H->uinf[d] = H->sphere.bFixFrameOfRef[d] ? -H->sphere_vel[d] : 0.0;
    // orientation (Obstacle::update, source/obstacles/Obstacle.cpp:323-346;
    // the sphere's chi does not depend on it)
    const double* w = H->sphere_angvel;
    const double* Q = H->sphere_quat;
    const double dqdt[4] = {.5 * (-w[0] * Q[1] - w[1] * Q[2] - w[2] * Q[3]), .5 * (+w[0] * Q[0] + w[1] * Q[3] - w[2] * Q[2]),
                            .5 * (-w[0] * Q[3] + w[1] * Q[0] + w[2] * Q[1]), .5 * (+w[0] * Q[2] - w[1] * Q[1] + w[2] * Q[0])};
    const double DQ[4] = {dqdt[0] * dt, dqdt[1] * dt, dqdt[2] * dt, dqdt[3] * dt};
    const double DQn = std::sqrt(DQ[0] * DQ[0] + DQ[1] * DQ[1] + DQ[2] * DQ[2] + DQ[3] * DQ[3]);
    if (DQn > 2.220446049250313080847e-16) {
      const double tanF = std::tan(DQn) / DQn;
      const double D[4] = {Q[0] + tanF * DQ[0], Q[1] + tanF * DQ[1], Q[2] + tanF * DQ[2], Q[3] + tanF * DQ[3]};
      const double invD = 1 / std::sqrt(D[0] * D[0] + D[1] * D[1] + D[2] * D[2] + D[3] * D[3]);
      for (int k = 0; k < 4; ++k) H->sphere_quat[k] = D[k] * invD;
    }
  }
  for (int d = 0; d < 3; ++d) H->sphere.position[d] += dt * (H->sphere_vel[d] + H->uinf[d]);
  return relocate_sphere(H);
}

// UpdateObstacles (source/operators/ObstaclesUpdate.cpp:202-236) for a sphere
// with free dofs: the momentum integrals over its box, then the 6x6 balance
// on the device (k_rigid_update), which sets the sphere's velocities for the
// penalization that follows.
template <typename T>
int do_rigid_update(cup_handle* H, DtArg dt, const double* lambda_dev) {
  const int gb = box_grid(H->box);
  int rc = launch_named(H, "integrate_momenta", [&]() -> int {
    klaunch(H, k_integrate_momenta<T>, gb, kBoxThreads, 0, (const T*)H->u, (const T*)H->v, (const T*)H->w,
            (const T*)H->chi, (const SphereParams*)H->sp_dev, H->box, H->nx, H->ny, H->nz, H->h, dt, lambda_dev,
            H->lambda, H->cfg.bImplicitPenalization, partial(H, P_RIGID));
    CKL();
    return CUP_OK;
  });
  if (rc) return rc;
  return launch_named(H, "rigid_update", [&]() -> int {
    klaunch(H, k_rigid_update, 1, 256, 0, (const double*)partial(H, P_RIGID), gb, H->sp_dev, H->dstate, dt,
            H->cfg.bImplicitPenalization);
    CKL();
    return CUP_OK;
  });
}

// The velocities UpdateObstacles computed, into the host mirror (the next
// CreateObstacles moves the sphere and the frame with them). Synchronises.
int read_sphere_motion(cup_handle* H) {
  SphereParams sp;
  CK(cudaMemcpyAsync(&sp, H->sp_dev, sizeof(sp), cudaMemcpyDeviceToHost, H->stream));
  CK(cudaStreamSynchronize(H->stream));
  for (int d = 0; d < 3; ++d) {
    H->sphere_vel[d] = sp.transVel[d];
    H->sphere_angvel[d] = sp.angVel[d];
  }
  return CUP_OK;
}

// chi of the sphere at H->sphere.position: cleared on the old box, rebuilt
// with the centre of mass on the box of the new position.
int relocate_sphere(cup_handle* H) {
  const size_t es = H->fp32 ? sizeof(float) : sizeof(double);
  {
    const Box old = H->box;
    const int gb = box_grid(old);
    const double* pos = H->sphere.position;
    int rc_ = launch_named(H, "sphere_clear", [&]() -> int {
      klaunch(H, k_clear_box, gb, kBoxThreads, 0, H->chi, es, old, H->nx, H->ny, H->nz, H->sp_dev, pos[0], pos[1],
              pos[2]);
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  sphere_box(H);
  return build_sphere_chi(H);
}

constexpr int kSumCap = 256;  // doubles of dsum / hsum (a spectrum has at most 127 bins)
int alloc_sums(cup_handle* H) {
  if (!H->dsum) CK(cudaMalloc(&H->dsum, kSumCap * sizeof(double)));
  if (!H->hsum) CK(cudaMallocHost(&H->hsum, kSumCap * sizeof(double)));
  return CUP_OK;
}
// Column sums of per-CTA partials (max_col: that column's maximum) to
// dsum[at..], stream-ordered.
int sum_columns(cup_handle* H, const double* part, int np, int ncol, int max_col, int at) {
  int rc = alloc_sums(H);
  if (rc) return rc;
  return launch_named(H, "sum_columns", [&]() -> int {
    klaunch(H, k_reduce_columns, ncol, 256, 0, part, np, ncol, max_col, H->dsum + at);
    CKL();
    return CUP_OK;
  });
}
// The first n sums in H->hsum, and the device error word: one synchronisation.
int read_sums(cup_handle* H, int n) {
  CK(cudaMemcpyAsync(H->hsum, H->dsum, n * sizeof(double), cudaMemcpyDeviceToHost, H->stream));
  CK(cudaMemcpyAsync(H->hsum + kSumCap - 1, H->derr, sizeof(int), cudaMemcpyDeviceToHost, H->stream));
  CK(cudaStreamSynchronize(H->stream));
  int e;
  memcpy(&e, H->hsum + kSumCap - 1, sizeof e);
  return dev_error_status(H, e);
}

// Blocks and planes per block of the diagnostics that march down z: 16 planes,
// or fewer until the grid fills the SMs a few times over.
void march_grid(const cup_handle* H, int* zc, int* grid) {
  const int per_plane = H->nx * H->ny / 256;
  *zc = 16;
  while (*zc > 4 && per_plane * (H->nz / *zc) < 4 * H->num_sms) *zc /= 2;
  *grid = per_plane * (H->nz / *zc);
}

// The z transform of the three components in spec[0] with the mode sums.
template <int M>
int launch_z_modes_M(cup_handle* H, const ModeParams& mp, double* part, int* np) {
  constexpr bool T8 = M == 128;
  constexpr int N = 2 * M, W = 16;
  CUtensorMap map;
  int rc = make_map(H, &map, H->spec[0], tma_dtype<double>(), sizeof(double), W, 1, N, 3);
  if (rc) return rc;
  const size_t smem = (size_t)3 * N * W * sizeof(double) + FFTPlan<M>::table_len() * sizeof(double2) +
                      mp.nbin * sizeof(double) + sizeof(uint64_t) + 128;
  auto kern = k_dht_z_modes<M, T8>;
  int bpsm = 0;
  if ((rc = prepare_kernel(H, kern, smem, 128, &bpsm))) return rc;
  const int ntiles = H->nx / W * H->ny;
  *np = std::min({ntiles, bpsm * H->num_sms, kPartialCap / (3 + mp.nbin)});
  return launch_named(H, "spectral_z_modes", [&]() -> int {
    klaunch(H, kern, *np, 128, smem, map, mp, (const double2*)H->tw64[2], ntiles, part, H->derr);
    CKL();
    return CUP_OK;
  });
}
int launch_z_modes(cup_handle* H, const ModeParams& mp, double* part, int* np) {
  PFFT_DISPATCH(H->nz, (launch_z_modes_M<M>(H, mp, part, np)));
}

// The spectral sums of the current velocity (see k_dht_z_modes): raw[0..2]
// = tke, lIntegral, tkeFiltered over the separable modes (unnormalised), raw[3]
// = sum of |curl_c u|^2 over the cells; bins = the unnormalised spectrum
// (nBin = max(N)/2 - 1 values, HITstatistics). mp: the modes' parameters; with
// mp.coef the coefficients of the forcing band are left there. spec[] then
// holds the x and y transforms.
int do_spectral(cup_handle* H, const ModeParams& mp, double raw[4], std::vector<double>& bins) {
  int rc;
  const char* nm = "spectral_dht_x";
  if (H->fp32) {
    const float* f[3] = {(const float*)H->u, (const float*)H->v, (const float*)H->w};
    rc = launch_rows_pipe<float>(H, nm, f, 3, H->spec[0]);
  } else {
    const double* f[3] = {(const double*)H->u, (const double*)H->v, (const double*)H->w};
    rc = launch_rows_pipe<double>(H, nm, f, 3, H->spec[0]);
  }
  int np = 0, zc, gv;
  double* part = partial(H, P_DIAG);
  double* pv = partial(H, P_RES);
  if (!rc) rc = launch_cols<1, false>(H, H->spec[0], 3);
  if (!rc) rc = launch_z_modes(H, mp, part, &np);
  if (rc) return rc;
  march_grid(H, &zc, &gv);
  rc = launch_named(H, "spectral_vorticity", [&]() -> int {
    if (H->fp32)
      klaunch(H, k_vorticity2<float>, gv, 256, 0, (const float*)H->u, (const float*)H->v, (const float*)H->w,
              ilog2(H->nx), ilog2(H->ny), H->nz, zc, 0.5 / H->h, pv);
    else
      klaunch(H, k_vorticity2<double>, gv, 256, 0, (const double*)H->u, (const double*)H->v, (const double*)H->w,
              ilog2(H->nx), ilog2(H->ny), H->nz, zc, 0.5 / H->h, pv);
    CKL();
    return CUP_OK;
  });
  if (!rc) rc = sum_columns(H, part, np, 3 + mp.nbin, -1, 0);
  if (!rc) rc = sum_columns(H, pv, gv, 1, -1, 3 + mp.nbin);
  if (!rc) rc = read_sums(H, 4 + mp.nbin);
  if (rc) return rc;
  for (int k = 0; k < 3; ++k) raw[k] = H->hsum[k];
  raw[3] = H->hsum[3 + mp.nbin];
  bins.assign(H->hsum + 3, H->hsum + 3 + mp.nbin);
  return CUP_OK;
}

// The modes of the handle's grid; allocates the coefficient arrays on first use.
int mode_params(cup_handle* H, ModeParams* mp) {
  if (!H->spec[0]) {
    CK(cudaMalloc(&H->spec[0], 3 * H->n * sizeof(double)));
    H->spec[1] = H->spec[0] + H->n;
    H->spec[2] = H->spec[1] + H->n;
    CK(cudaMalloc(&H->band_coef, (size_t)3 * kBandN * kBandN * kBandN * sizeof(double)));
  }
  const int n[3] = {H->nx, H->ny, H->nz};
  mp->nx = n[0], mp->ny = n[1], mp->nz = n[2];
  mp->nyquist = std::max(H->nx, std::max(H->ny, H->nz)) / 2;
  mp->nbin = mp->nyquist - 1;
  mp->nyq_scaling = (mp->nyquist - 1) / (double)mp->nyquist;
  for (int d = 0; d < 3; ++d) {
    mp->wf[d] = 2.0 * M_PI / (n[d] * H->h);
    // every mode with |i| wf <= 2 (one more index against rounding; its coefficients are zero)
    mp->band[d] = (int)std::min((double)(n[d] / 2 - 1), std::floor(2.0 / mp->wf[d]) + 1);
  }
  mp->coef = nullptr;
  return CUP_OK;
}

// SpectralForcing::operator() (source/spectralOperators/SpectralForcing.cpp:23-86):
// the energy of the band 0 < k^2 <= 4 is raised so that the total kinetic
// energy meets turbKinEn_target (or grows at enInjectionRate): u += fac/N H(H(u)
// restricted to the band), fac = dt rate / (2 tke_band). out: totalKinEn,
// largeModesKinEn, viscousDissip, dissipationRate, injectionRate, lIntegral.
// A band of up to kBandMax modes a side (a box of side 2 pi has 2, and one more
// index is carried) is summed mode by mode in one pass over the velocity (24
// B/cell FP32, against nine FP64 transform passes and three updates); a wider
// one (boxes of 4 pi and longer) goes through the inverse transforms.
template <typename T>
int do_spectral_forcing(cup_handle* H, DtArg step_dt) {
  double raw[4];
  std::vector<double> bins;
  ModeParams mp;
  int rc = mode_params(H, &mp);
  if (rc) return rc;
  const bool small = std::max({mp.band[0], mp.band[1], mp.band[2]}) <= kBandMax;
  if (small) mp.coef = H->band_coef;
  // a dt chained on the device comes to the host with the sums: one
  // synchronisation a step, where reading it before the step took a second one
  // (the injection needs it, the advection before it does not)
  if ((rc = alloc_sums(H))) return rc;
  double* dt_host = H->hsum + kSumCap - 2;
  if (step_dt.dev) CK(cudaMemcpyAsync(dt_host, step_dt.dev, sizeof(double), cudaMemcpyDeviceToHost, H->stream));
  if ((rc = do_spectral(H, mp, raw, bins))) return rc;
  if (step_dt.dev) {
    H->dt = *dt_host;
    if (!(H->dt > 0)) return fail(H, CUP_ERR_ARG, "dt must be > 0");
    if (H->cfg.DLM > 0) H->lambda = H->cfg.DLM / H->dt;
  }
  const double dt = step_dt.dev ? H->dt : step_dt.host;
  const double NF = (double)H->n;  // normalizeFFT
  const double tke = raw[0] / (NF * NF), tkeF = raw[2] / (NF * NF);
  const double eps = H->cfg.nu * raw[3] / NF;
  const double dissipationRate = (H->forcing_prev_tke - tke) / dt;
  double rate = 0;
  if (H->forcing_target > 0) rate = (H->forcing_target - tke) / dt;
  else if (H->forcing_rate > 0) rate = H->forcing_rate;
  const double fac = dt * rate / (2 * tkeF);
  H->forcing_stats[0] = tke;
  H->forcing_stats[1] = tkeF;
  H->forcing_stats[2] = eps;
  H->forcing_stats[3] = dissipationRate;
  H->forcing_stats[4] = rate;
  H->forcing_stats[5] = raw[0] > 0 ? raw[1] / raw[0] : 0.0;
  if (!(fac > 0)) {
    H->forcing_prev_tke = tke;
    return CUP_OK;
  }
  H->forcing_prev_tke = tke + dt * rate;
  if (small) {
    const int rpb = std::min(32, H->ny);
    return launch_named(H, "spectral_force", [&]() -> int {
      klaunch(H, k_force_band<T>, H->nz * (H->ny / rpb), 256, (size_t)rpb * 4 * kBandN * sizeof(double),
              (T*)H->u, (T*)H->v, (T*)H->w, mp, fac / NF, rpb);
      CKL();
      return CUP_OK;
    });
  }
  void* f[3] = {H->u, H->v, H->w};
  const int grid = std::min<size_t>(H->num_sms * 4, (H->n + 255) / 256);
  for (int c = 0; c < 3; ++c)
    if ((rc = launch_cols<2, false>(H, H->spec[c]))) return rc;
  rc = launch_named(H, "spectral_filter", [&]() -> int {
    klaunch(H, k_spectral_filter, grid, 256, 0, H->spec[0], H->spec[1], H->spec[2], ilog2(H->nx), ilog2(H->ny), H->nz,
            mp.wf[0], mp.wf[1], mp.wf[2]);
    CKL();
    return CUP_OK;
  });
  for (int c = 0; c < 3 && !rc; ++c) {
    rc = launch_rows_pipe(H, "spectral_dht_x", H->spec[c]);
    if (!rc) rc = launch_cols<1, false>(H, H->spec[c]);
    if (!rc) rc = launch_cols<2, false>(H, H->spec[c]);
    if (!rc)
      rc = launch_named(H, "spectral_force", [&]() -> int {
        klaunch(H, k_add_scaled<T>, grid, 256, 0, (T*)f[c], (const double*)H->spec[c], fac / NF, H->n);
        CKL();
        return CUP_OK;
      });
  }
  return rc;
}

// next_dt: finalize_step also computes the next step's CFL dt.
template <typename T>
int do_step(cup_handle* H, DtArg dt, const double* lambda_dev, int advance, int next_dt = 0) {
  int rc;
  // CreateObstacles first (source/Simulation.cpp:307-401 pipeline order); a
  // moving sphere needs this step's dt on the host for its new position
  if (H->has_sphere && H->sphere_moves) {
    if (dt.dev) return fail(H, CUP_ERR_STATE, "a moving obstacle needs the step's dt on the host");
    if ((rc = do_create_obstacles(H, dt.host))) return rc;
  }
  if ((rc = do_advect_diffuse<T>(H, dt))) return rc;
  // SpectralForcing follows AdvectionDiffusion (source/Simulation.cpp:330-340)
  if (H->forcing && (rc = do_spectral_forcing<T>(H, dt))) return rc;
  if constexpr (std::is_same<T, float>::value) {
    // RHS, defect correction and gradient correction in z-queue passes. The
    // sphere's RHS terms need global sums over the RHS first: they are formed on
    // its box and added back by the passes, which recompute the rest of b from u*
    void* us[3] = {H->u, H->v, H->w};
    if (H->has_sphere && (rc = do_box_rhs_terms<T, float>(H, dt, us))) return rc;
    if ((rc = do_pressure_dc_zq<T>(H, dt))) return rc;
  } else {
    void* us[3] = {H->u, H->v, H->w};
    if (H->has_sphere && amplifies_rounding(H)) {
      if ((rc = do_pressure_rhs<T>(H, dt))) return rc;
      if ((rc = do_poisson(H))) return rc;
    } else {
      if (H->has_sphere && (rc = do_box_rhs_terms<T, double>(H, dt, us))) return rc;
      if ((rc = do_solve_rhs_of<T>(H, "rhs_dht_x", "dht_x", us, H->p, dt, H->has_sphere))) return rc;
    }
    if ((rc = do_grad<T>(H, dt))) return rc;
  }
  // UpdateObstacles: the free dofs' velocities from the pre-penalization flow
  if (H->has_sphere && H->sphere_free && (rc = do_rigid_update<T>(H, dt, lambda_dev))) return rc;
  if ((rc = do_penalize<T>(H, dt, lambda_dev))) return rc;
  {
    int rc_ = launch_named(H, "finalize_step", [&]() -> int {
      klaunch(H, k_finalize_step, 1, 256, 0, partial(H, P_GRAD), H->n_grad_partials, H->grad_stride,
                                            H->grad_max_off, H->grad_ke_off, partial(H, P_PEN), H->n_pen_partials,
                                            H->dstate, H->h * H->h * H->h, advance,
                                            next_dt, cfl_params(H));
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  return CUP_OK;
}

// ---- discrete adjoint ------------------------------------------------------
// Launches one k_adjoint_zq pass: out = alpha lam + beta S'(f)^T g.
template <typename T, int SCHEME, bool LAM, int TY, int NS, int CPT>
int launch_adjoint(cup_handle* H, const char* name, const void* const* f, const void* const* g, const void* const* lam,
                   void* const* out, double alpha, double beta, DtArg dt) {
  constexpr int G = SCHEME == 0 ? 1 : 2;
  const int cells = TY * H->nx;
  if (cells % CPT || cells / CPT > 512 || H->ny % TY)
    return fail(H, CUP_ERR_ARG, "adjoint tile does not fit the grid");
  AdjointMaps maps;
  for (int q = 0; q < 3; ++q) {
    int rc = make_row_maps<T>(H, &maps.f[q], f[q], TY, G);
    if (!rc) rc = make_row_maps<T>(H, &maps.f[3 + q], g[q], TY, G);
    if (rc) return rc;
  }
  const size_t smem = adjoint_smem_bytes<T, SCHEME, TY, NS>(H->nx) + 128;
  auto kern = k_adjoint_zq<T, SCHEME, LAM, TY, NS, CPT>;
  const int threads = cells / CPT;
  int bpsm = 0;
  int rc = prepare_kernel(H, kern, smem, threads, &bpsm);
  if (rc) return rc;
  const int zc = planes_per_item(H, TY, G, bpsm);
  StreamGeom geo{H->nx, H->ny, H->nz, ilog2(H->nx), zc, H->ny / TY, (H->ny / TY) * (H->nz / zc)};
  const int grid = std::min(geo.n_items, bpsm * H->num_sms);
  const void* lm[3] = {LAM ? lam[0] : nullptr, LAM ? lam[1] : nullptr, LAM ? lam[2] : nullptr};
  return launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, threads, smem, maps, geo, (const T*)lm[0], (const T*)lm[1], (const T*)lm[2], (T*)out[0],
            (T*)out[1], (T*)out[2], (T)alpha, (T)beta, dt, H->h,
                                             H->cfg.nu, H->uinf[0], H->uinf[1], H->uinf[2], H->derr);
    CKL();
    return CUP_OK;
  });
}

// The projection P = I - G L^+ D of the pipeline (PressureRHS, the periodic
// FFT solve in FP64, the gradient correction) applied to the fields `in`,
// result in `out` (may equal `in`). D = -G^T on the periodic grid and L = D G
// is the wide-stencil Laplacian the spectral factor inverts, so P is
// symmetric: the adjoint of the projection is P itself.
template <typename T>
int do_project_fields(cup_handle* H, void* const* in, void* const* out, double* pbuf, DtArg dt) {
  int rc;
  if ((rc = do_solve_rhs_of<T>(H, "adjoint_rhs_dht_x", "adjoint_dht_x", in, pbuf, dt))) return rc;
  return launch_grad<T, false>(H, "adjoint_grad_p", in, out, pbuf, dt);
}

// Adjoint of one step u_{n+1} = P(H(u_n)) with the dt given, at the state un:
// lam (dJ/du_{n+1}) becomes dJ/du_n.
//   upwind3 + RK2:  lam* = P lam,  u1 = S(un),
//                   mu = 1/2 S'(u1)^T lam*,  lam = 1/2 lam* + S'(un)^T mu
//   central + Euler: lam = S'(un)^T (P lam)
// FP32 upwind3 stage transposes on x-pairs (k_adjoint_zq_f2); grids of nx 64,
// 128 or 256 take the compile-time-nx kernels.
template <bool LAM, int TY, int NS, int PPT, int NXC = 0>
int launch_adjoint_f2(cup_handle* H, const char* name, const void* const* f, const void* const* g,
                      const void* const* lam, void* const* out, double alpha, double beta, DtArg dt) {
  constexpr int G = 2;
  const int pairs = TY * H->nx / 2;
  if (pairs % PPT || pairs / PPT > 512 || H->ny % TY)
    return fail(H, CUP_ERR_ARG, "adjoint tile does not fit the grid");
  AdjointMaps maps;
  for (int q = 0; q < 3; ++q) {
    int rc = make_row_maps<float>(H, &maps.f[q], f[q], TY, G);
    if (!rc) rc = make_row_maps<float>(H, &maps.f[3 + q], g[q], TY, G);
    if (rc) return rc;
  }
  if (NXC && NXC != H->nx) return fail(H, CUP_ERR_ARG, "adjoint specialisation mismatch");
  const size_t smem = adjoint_f2_smem_bytes<TY, NS>(H->nx) + 128;
  auto kern = k_adjoint_zq_f2<LAM, TY, NS, PPT, NXC>;
  const int threads = pairs / PPT;
  int bpsm = 0;
  int rc = prepare_kernel(H, kern, smem, threads, &bpsm);
  if (rc) return rc;
  const int zc = planes_per_item(H, TY, G, bpsm);
  StreamGeom geo{H->nx, H->ny, H->nz, ilog2(H->nx), zc, H->ny / TY, (H->ny / TY) * (H->nz / zc)};
  const int grid = std::min(geo.n_items, bpsm * H->num_sms);
  const void* lm[3] = {LAM ? lam[0] : nullptr, LAM ? lam[1] : nullptr, LAM ? lam[2] : nullptr};
  return launch_named(H, name, [&]() -> int {
    klaunch(H, kern, grid, threads, smem, maps, geo, (const float*)lm[0], (const float*)lm[1], (const float*)lm[2],
            (float*)out[0], (float*)out[1], (float*)out[2], (float)alpha,
            (float)beta, dt, H->h, H->cfg.nu, H->uinf[0], H->uinf[1], H->uinf[2], H->derr);
    CKL();
    return CUP_OK;
  });
}

template <bool LAM, int TY, int NS, int PPT>
int launch_adjoint_f2_sized(cup_handle* H, const char* name, const void* const* f, const void* const* g,
                            const void* const* lam, void* const* out, double alpha, double beta, DtArg dt) {
  switch (H->nx) {
    case 64: return launch_adjoint_f2<LAM, TY, NS, PPT, 64>(H, name, f, g, lam, out, alpha, beta, dt);
    case 128: return launch_adjoint_f2<LAM, TY, NS, PPT, 128>(H, name, f, g, lam, out, alpha, beta, dt);
    case 256: return launch_adjoint_f2<LAM, TY, NS, PPT, 256>(H, name, f, g, lam, out, alpha, beta, dt);
    default: break;
  }
  return launch_adjoint_f2<LAM, TY, NS, PPT>(H, name, f, g, lam, out, alpha, beta, dt);
}

// The two transposed upwind3 stages of an FP32 adjoint step: mu = 1/2 S'(u1)^T
// lam*, then lam = 1/2 lam* + S'(u^n)^T mu (lam* = the projected adjoint, in
// lam on entry). 4-row tiles and one pair per thread measured best at
// 256^3: 1.235 ms per adjoint step against 1.52 ms with 2-row tiles, and 2.17
// ms for the scalar kernels (k_adjoint_zq). The ring is 4 deep: two planes in
// flight while a plane and the one before it are read.
int adjoint_upwind_f32(cup_handle* H, void* const* un, void* const* st1, void* const* lam, void* const* mu, DtArg dt) {
  int rc;
  if ((rc = launch_adjoint_f2_sized<false, 4, 4, 1>(H, "adjoint_stage2", st1, lam, nullptr, mu, 0.0, 0.5, dt)))
    return rc;
  return launch_adjoint_f2_sized<true, 4, 4, 1>(H, "adjoint_stage1", un, mu, lam, lam, 0.5, 1.0, dt);
}

// The projection reads its fields in 16-byte pieces: *in = f, or `copy` with the
// fields copied there when one of them lies between such boundaries.
template <typename T>
int aligned_fields(cup_handle* H, void* const* f, void* const* copy, void* const** in) {
  *in = f;
  if (((uintptr_t)f[0] | (uintptr_t)f[1] | (uintptr_t)f[2]) % 16 == 0) return CUP_OK;
  for (int q = 0; q < 3; ++q)
    CK(cudaMemcpyAsync(copy[q], f[q], H->n * sizeof(T), cudaMemcpyDeviceToDevice, H->stream));
  *in = copy;
  return CUP_OK;
}

template <typename T>
int do_adjoint_step(cup_handle* H, void* const* un, void* const* lam, DtArg dt) {
  constexpr bool F32 = std::is_same<T, float>::value;
  int rc;
  void* mu[3] = {H->au, H->av, H->aw};
  if (H->cfg.scheme == CUP_SCHEME_REF) {
    void* const* in;
    if ((rc = aligned_fields<T>(H, lam, mu, &in))) return rc;
    if ((rc = do_project_fields<T>(H, in, mu, H->p_adj, dt))) return rc;
    if constexpr (F32) return launch_adjoint<T, 0, false, 4, 3, 2>(H, "adjoint_ref", un, mu, nullptr, lam, 0.0, 1.0, dt);
    else return launch_adjoint<T, 0, false, 2, 3, 1>(H, "adjoint_ref", un, mu, nullptr, lam, 0.0, 1.0, dt);
  }
  void* st1[3] = {H->u1, H->v1, H->w1};
  if ((rc = do_project_fields<T>(H, lam, lam, H->p_adj, dt))) return rc;
  if constexpr (F32) {
    if ((rc = upwind_stage1_f32(H, "adjoint_recompute_stage1", un, st1, dt))) return rc;
    return adjoint_upwind_f32(H, un, st1, lam, mu, dt);
  } else {
    if ((rc = upwind_stage_f64<T, 1>(H, "adjoint_recompute_stage1", un, un, st1, dt))) return rc;
    if ((rc = launch_adjoint<T, 1, false, 2, 3, 1>(H, "adjoint_stage2", st1, lam, nullptr, mu, 0.0, 0.5, dt))) return rc;
    return launch_adjoint<T, 1, true, 2, 3, 1>(H, "adjoint_stage1", un, mu, lam, lam, 0.5, 1.0, dt);
  }
}

// Adjoint of one step with the sphere (penalization, its force and the
// obstacle terms of the RHS; adjoint_obstacle.cuh): lam (dJ/du_{n+1}) becomes
// dJ/du_n for J = <g, u_T> + sum_n wF . F_n, and dJ/dchi, dJ/dU (the sphere's
// penalization target velocity) are added to g_chi, g_vel. The step is
// recomputed from un up to the velocity before penalization (projection by
// the FP64 FFT solve), then
//   lam** = Pen^T lam (- force term),  q = L^+ RHS(lam**),  q' = M^T q,
//   lam* = lam** - dt/(2h) grad_c q',  then the advection transposes.
template <typename T>
int do_adjoint_step_obstacle(cup_handle* H, void* const* un, void* const* lam, DtArg dt, const double* wF,
                             double* g_chi, double* g_vel) {
  constexpr bool F32 = std::is_same<T, float>::value;
  int rc;
  void* mu[3] = {H->au, H->av, H->aw};
  void* us[3] = {H->aus, H->avs, H->aws};
  void* st1[3] = {H->u1, H->v1, H->w1};
  const double dtv = dt.host;
  // 1. forward recompute: advection, RHS with its obstacle terms, solve, gradient
  if (H->cfg.scheme == CUP_SCHEME_REF) {
    if constexpr (F32) rc = launch_advect<T, 0, 8, 5, 4>(H, "adjoint_recompute_ref", un, un, us, dt);
    else rc = launch_advect<T, 0, 4, 5, 2>(H, "adjoint_recompute_ref", un, un, us, dt);
    if (rc) return rc;
  } else if constexpr (F32) {
    if ((rc = upwind_stage1_f32(H, "adjoint_recompute_stage1", un, st1, dt))) return rc;
    if ((rc = upwind_stage2_f32(H, "adjoint_recompute_stage2", st1, un, us, dt))) return rc;
  } else {
    if ((rc = upwind_stage_f64<T, 1>(H, "adjoint_recompute_stage1", un, un, st1, dt))) return rc;
    if ((rc = upwind_stage_f64<T, 2>(H, "adjoint_recompute_stage2", st1, un, us, dt))) return rc;
  }
  if ((rc = do_box_rhs_terms<T, double>(H, dt, us, H->ab0))) return rc;
  if ((rc = do_solve_rhs_of<T>(H, "adjoint_rhs_dht_x", "adjoint_dht_x", us, H->p_adj, dt, true))) return rc;
  if ((rc = launch_grad<T, false>(H, "adjoint_recompute_grad_p", us, us, H->p_adj, dt))) return rc;
  // 2. penalization and force
  const int gb = box_grid(H->box);
  const double lambda = H->cfg.DLM > 0 ? H->cfg.DLM / dtv : H->lambda;
  {
    int rc_ = launch_named(H, "adjoint_penalize", [&]() -> int {
      klaunch(H, k_adj_penalize<T>, gb, kBoxThreads, 0, 
          (T*)lam[0], (T*)lam[1], (T*)lam[2], (const T*)us[0], (const T*)us[1], (const T*)us[2], (const T*)H->chi,
          H->sp_dev, H->box, H->nx, H->ny, H->nz, H->h, dtv, lambda, H->cfg.bImplicitPenalization, wF[0], wF[1],
          wF[2], g_chi, partial(H, P_PEN));
      CKL();
      klaunch(H, k_adj_accumulate, 1, 256, 0, partial(H, P_PEN), gb, 3, 3, g_vel);
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  // 3. projection with the transposed obstacle RHS terms
  void* const* in;
  if ((rc = aligned_fields<T>(H, lam, mu, &in))) return rc;
  if ((rc = do_solve_rhs_of<T>(H, "adjoint_rhs_dht_x", "adjoint_dht_x", in, H->p_adj, dt))) return rc;
  const double kappa = dtv * dtv / (H->h * H->h * H->h);  // dJ/db2 = kappa q
  {
    int rc_ = launch_named(H, "adjoint_rhs_obstacle", [&]() -> int {
      CK(cudaMemsetAsync(&H->dstate->adj_sq, 0, sizeof(double), H->stream));
      klaunch(H, k_adj_rhs_sum<T>, gb, kBoxThreads, 0, H->p_adj, H->ab0, (const T*)H->chi, H->box, H->nx, H->ny,
                                                         H->nz, H->dstate->rhs_sums, &H->dstate->corr,
                                                         partial(H, P_RHSOB));
      CKL();
      klaunch(H, k_adj_accumulate, 1, 256, 0, partial(H, P_RHSOB), gb, 1, 1, &H->dstate->adj_sq);
      CKL();
      klaunch(H, k_adj_rhs_apply<T>, gb, kBoxThreads, 0, H->p_adj, H->ab0, (const T*)H->chi, H->box, H->nx,
                                                           H->ny, H->nz, H->dstate->rhs_sums, &H->dstate->corr,
                                                           &H->dstate->adj_sq, kappa, g_chi);
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  // 4. gradient correction, then the advection transposes
  if (H->cfg.scheme == CUP_SCHEME_REF) {
    if ((rc = launch_grad<T, false>(H, "adjoint_grad_p", in, mu, H->p_adj, dt))) return rc;
    if constexpr (F32) return launch_adjoint<T, 0, false, 4, 3, 2>(H, "adjoint_ref", un, mu, nullptr, lam, 0.0, 1.0, dt);
    else return launch_adjoint<T, 0, false, 2, 3, 1>(H, "adjoint_ref", un, mu, nullptr, lam, 0.0, 1.0, dt);
  }
  if ((rc = launch_grad<T, false>(H, "adjoint_grad_p", lam, lam, H->p_adj, dt))) return rc;
  if constexpr (F32) {
    return adjoint_upwind_f32(H, un, st1, lam, mu, dt);
  } else {
    if ((rc = launch_adjoint<T, 1, false, 2, 3, 1>(H, "adjoint_stage2", st1, lam, nullptr, mu, 0.0, 0.5, dt))) return rc;
    return launch_adjoint<T, 1, true, 2, 3, 1>(H, "adjoint_stage1", un, mu, lam, lam, 0.5, 1.0, dt);
  }
}

template <typename T>
int set_field(cup_handle* H, void* dst, const double* src, int where) {
  if (!H->fp32) {
    CK(cudaMemcpyAsync(dst, src, H->n * sizeof(double),
                       where == CUP_WHERE_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, H->stream));
    return CUP_OK;
  }
  const double* s = src;
  if (where == CUP_WHERE_HOST) {
    CK(cudaMemcpyAsync(H->rhs, src, H->n * sizeof(double), cudaMemcpyHostToDevice, H->stream));
    s = H->rhs;
  }
  {
    int rc_ = launch_named(H, "convert_from_f64", [&]() -> int {
      klaunch(H, k_convert_from_f64<T>, H->num_sms * 4, 256, 0, (T*)dst, s, H->n);
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  return CUP_OK;
}

template <typename T>
int get_field(cup_handle* H, const void* src, double* dst, int where) {
  if (!H->fp32) {
    CK(cudaMemcpyAsync(dst, src, H->n * sizeof(double),
                       where == CUP_WHERE_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, H->stream));
    return CUP_OK;
  }
  double* d = where == CUP_WHERE_HOST ? H->rhs : dst;
  {
    int rc_ = launch_named(H, "convert_to_f64", [&]() -> int {
      klaunch(H, k_convert_to_f64<T>, H->num_sms * 4, 256, 0, d, (const T*)src, H->n);
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  if (where == CUP_WHERE_HOST)
    CK(cudaMemcpyAsync(dst, H->rhs, H->n * sizeof(double), cudaMemcpyDeviceToHost, H->stream));
  return CUP_OK;
}

int valid_where(int where) { return where == CUP_WHERE_HOST || where == CUP_WHERE_DEVICE; }

#define DISPATCH_T(H, fn, ...) ((H)->fp32 ? fn<float>(H, ##__VA_ARGS__) : fn<double>(H, ##__VA_ARGS__))

constexpr int kGraphSteps = 6;

cup_handle::StepState step_state(const cup_handle* H) {
  cup_handle::StepState s{{H->u, H->v, H->w, H->tu, H->tv, H->tw, H->p, H->p_old, H->p_pred},
                          H->p_valid, H->n_grad_partials, H->grad_stride, H->grad_max_off, H->grad_ke_off,
                          H->pred_ready};
  return s;
}

void set_step_state(cup_handle* H, const cup_handle::StepState& s) {
  H->u = s.f[0], H->v = s.f[1], H->w = s.f[2], H->tu = s.f[3], H->tv = s.f[4], H->tw = s.f[5];
  H->p = (double*)s.f[6], H->p_old = (double*)s.f[7], H->p_pred = (double*)s.f[8];
  H->p_valid = s.p_valid, H->n_grad_partials = s.n_grad_partials, H->grad_stride = s.grad_stride;
  H->grad_max_off = s.grad_max_off, H->grad_ke_off = s.grad_ke_off, H->pred_ready = s.pred_ready;
}

bool same_state(const cup_handle::StepState& a, const cup_handle::StepState& b) {
  for (size_t i = 0; i < sizeof(a.f) / sizeof(a.f[0]); ++i)
    if (a.f[i] != b.f[i]) return false;
  return a.p_valid == b.p_valid && a.n_grad_partials == b.n_grad_partials && a.grad_stride == b.grad_stride &&
         a.grad_max_off == b.grad_max_off && a.grad_ke_off == b.grad_ke_off && a.pred_ready == b.pred_ready;
}

void drop_graph(cup_handle* H) {
  for (auto& g : H->graphs) {
    if (g.exec) cudaGraphExecDestroy(g.exec);
    if (g.graph) cudaGraphDestroy(g.graph);
  }
  H->graphs.clear();
}

// Steps may replay a captured graph: no per-kernel profiling, a stream that is
// not itself being captured by the caller, nothing that needs the host between
// steps (a moving obstacle, spectral forcing), and the FP32-DC pressure history
// in its steady state (warm start ready), so that every step issues the same
// launches.
bool graph_ok(const cup_handle* H) {
  if (!H->use_graphs || H->prof_on || !H->stream || H->forcing) return false;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(H->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return false;
  }
  if (H->has_sphere && H->sphere_moves) return false;
  if (H->fp32 && !(H->pred_ready && H->p_valid >= 1)) return false;
  return true;
}

// Captures (without running) the nsteps-step graph of the current host state
// (dt from the device state; next_dt: each step computes the next step's dt)
// unless it is cached; *out = the cached graph, or nullptr when the capture
// failed (graphs are then off for the handle). The host state is left as it
// was: the captured steps only move it forward when the graph is replayed. The
// capture runs on a stream of its own, so that a handle bound to a default
// stream (torch's, unless its caller opened another) replays graphs too.
int capture_graph(cup_handle* H, int nsteps, int next_dt, cup_handle::StepGraph** out) {
  *out = nullptr;
  const cup_handle::StepState in = step_state(H);
  for (auto& g : H->graphs)
    if (g.nsteps == nsteps && g.next_dt == next_dt && same_state(g.in, in)) {
      *out = &g;
      return CUP_OK;
    }
  if (H->graphs.size() >= 32) drop_graph(H);
  const long long l0 = H->launches;
  if ((!H->cap_stream && cudaStreamCreateWithFlags(&H->cap_stream, cudaStreamNonBlocking) != cudaSuccess) ||
      cudaStreamBeginCapture(H->cap_stream, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
    cudaGetLastError();
    H->use_graphs = false;
    return CUP_OK;
  }
  const cudaStream_t run_stream = H->stream;
  H->stream = H->cap_stream;
  int rc = CUP_OK;
  for (int s = 0; s < nsteps && rc == CUP_OK; ++s)
    rc = DISPATCH_T(H, do_step, DtArg{0.0, &H->dstate->dt}, (const double*)&H->dstate->lambda, 1, next_dt);
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(H->cap_stream, &g);
  H->stream = run_stream;
  cudaGraphExec_t ex = nullptr;
  const cup_handle::StepState after = step_state(H);
  set_step_state(H, in);
  const long long nl = H->launches - l0;
  H->launches = l0;
  if (rc == CUP_OK && e == cudaSuccess && g && cudaGraphInstantiate(&ex, g, 0) == cudaSuccess) {
    cudaGraphUpload(ex, H->stream);  // the first replay then starts at once
    H->graphs.push_back({in, after, nsteps, next_dt, g, ex, nl});
    *out = &H->graphs.back();
    return CUP_OK;
  }
  if (g) cudaGraphDestroy(g);
  cudaGetLastError();
  H->use_graphs = false;
  return CUP_OK;
}

// Runs nsteps steps from the CUDA graph of the current host state, captured
// once per host state (the field pointers rotate with period 6: the u/tmp
// swap and the three FP32-DC pressure levels) and replayed with the host
// state set to what the captured steps left. *ran = false: the capture
// failed, nothing ran, the host state is as before and graphs are off for
// the handle, or the handle has not run long enough to capture.
// A handle captures for itself once it has run kGraphAfter steps: a 6-step
// graph and the one-step graphs of a tail take about 1.5 ms of host time with
// the GPU idle, and replaying saves 20-60 us a step, so a run that ends earlier
// would not win it back. cup_prepare_run captures at any time.
constexpr int kGraphAfter = 24;
int run_graph(cup_handle* H, int nsteps, int next_dt, bool* ran) {
  *ran = false;
  cup_handle::StepGraph* hit = nullptr;
  if (H->steps_run < kGraphAfter) {
    const cup_handle::StepState in = step_state(H);
    bool cached = false;
    for (const auto& g : H->graphs) cached = cached || (g.nsteps == nsteps && g.next_dt == next_dt && same_state(g.in, in));
    if (!cached) return CUP_OK;
  }
  int rc = capture_graph(H, nsteps, next_dt, &hit);
  if (rc || !hit) return rc;
  CK(cudaGraphLaunch(hit->exec, H->stream));
  H->launches += hit->launches;
  H->steps_run += nsteps;
  set_step_state(H, hit->out);
  *ran = true;
  return CUP_OK;
}

}  // namespace


#define REQUIRE_H(H)                        \
  do {                                      \
    if (!(H)) return CUP_ERR_ARG;           \
    ++(H)->api_calls;                       \
    cudaError_t e0_ = cudaSetDevice((H)->dev); \
    if (e0_ != cudaSuccess) return fail(H, CUP_ERR_CUDA, "cudaSetDevice: %s", cudaGetErrorString(e0_)); \
  } while (0)

// Entry points that need the whole grid (its z transform, obstacle or global
// sums) refuse a z-slab handle (cup_config.z_halo) before they change anything.
#define REQUIRE_WHOLE_GRID(H)                                                                          \
  do {                                                                                                 \
    if ((H)->cfg.z_halo)                                                                               \
      return fail(H, CUP_ERR_STATE, "%s needs a whole grid (this handle holds a z-slab)", __func__); \
  } while (0)

// Entry points that solve on the handle's own grid refuse a handle whose z pass
// is that of a pencil of a larger grid (cup_set_spectral_window).
#define REQUIRE_OWN_SPECTRUM(H)                                                                               \
  do {                                                                                                        \
    if ((H)->spec_ny != (H)->ny)                                                                              \
      return fail(H, CUP_ERR_STATE, "%s needs the handle's own spectrum (it has a spectral window)", __func__); \
  } while (0)

extern "C" {

int cup_create(const cup_config* cfg, cup_handle** out) {
  if (!cfg || !out) return CUP_ERR_ARG;
  *out = nullptr;
  cup_handle* H = new cup_handle();
  H->cfg = *cfg;
  H->nx = cfg->bpdx * 16;
  H->ny = cfg->bpdy * 16;
  H->nz = cfg->bpdz * 16;
  const int N[3] = {H->nx, H->ny, H->nz};
  auto reject = [&](int code) {
    // keep the handle so that the caller can read the message, then free it
    fprintf(stderr, "cup_create: %s\n", H->err.c_str());
    delete H;
    return code;
  };
  const bool slab = cfg->z_halo != 0;
  for (int d = 0; d < 3; ++d) {
    if (slab && d == 2) {
      // a z-slab with ghost planes: no z transform on this handle
      if (cfg->z_halo < 4 || N[2] < 2 * cfg->z_halo + 16 || N[2] > 512) {
        fail(H, CUP_ERR_ARG, "a z-slab handle needs z_halo >= 4 and 16 to %d interior planes (got z_halo %d, nz %d)",
             512 - 2 * cfg->z_halo, cfg->z_halo, N[2]);
        return reject(CUP_ERR_ARG);
      }
      continue;
    }
    if (N[d] < 16 || N[d] > 256 || !is_pow2(N[d])) {
      fail(H, CUP_ERR_ARG, "cells per dimension must be a power of two in [16, 256] (got %d)", N[d]);
      return reject(CUP_ERR_ARG);
    }
  }
  if (slab && cfg->precision != CUP_PREC_FP64) {
    fail(H, CUP_ERR_ARG, "a z-slab handle is FP64 (its defect correction would need sums over the ranks)");
    return reject(CUP_ERR_ARG);
  }
  if (!(cfg->maxextent > 0)) {
    fail(H, CUP_ERR_ARG, "maxextent must be > 0");
    return reject(CUP_ERR_ARG);
  }
  if (cfg->precision != CUP_PREC_FP64 && cfg->precision != CUP_PREC_FP32_DC) {
    fail(H, CUP_ERR_ARG, "unknown precision %d", cfg->precision);
    return reject(CUP_ERR_ARG);
  }
  if (cfg->scheme != CUP_SCHEME_REF && cfg->scheme != CUP_SCHEME_UPWIND3_RK2) {
    fail(H, CUP_ERR_ARG, "unknown scheme %d", cfg->scheme);
    return reject(CUP_ERR_ARG);
  }
  if (cfg->nu < 0 || !(cfg->CFL > 0)) {
    fail(H, CUP_ERR_ARG, "need nu >= 0 and CFL > 0");
    return reject(CUP_ERR_ARG);
  }
  H->fp32 = cfg->precision == CUP_PREC_FP32_DC;
  if (H->fp32 && H->nx < 32) {
    fail(H, CUP_ERR_ARG, "FP32 storage needs nx >= 32 (128-byte TMA rows)");
    return reject(CUP_ERR_ARG);
  }
  H->n = (size_t)H->nx * H->ny * H->nz;
  const double maxbpd = std::max({(double)N[0], (double)N[1], (double)N[2]});
  H->h = cfg->maxextent / maxbpd;
  H->lambda = cfg->lambda;
  for (int d = 0; d < 3; ++d) H->uinf[d] = cfg->uinf[d];
  H->dev = cfg->device;
  if (const char* pdl = getenv("CUP_PDL")) H->pdl = atoi(pdl) != 0;
  cudaError_t e = cudaSetDevice(H->dev);
  if (e != cudaSuccess) {
    fail(H, CUP_ERR_CUDA, "cudaSetDevice(%d): %s", H->dev, cudaGetErrorString(e));
    return reject(CUP_ERR_CUDA);
  }
  int rc = [&]() -> int {
    CK(cudaDeviceGetAttribute(&H->num_sms, cudaDevAttrMultiProcessorCount, H->dev));
    CK(cudaStreamCreateWithFlags(&H->stream, cudaStreamNonBlocking));
    H->own_stream = true;
    const size_t es = H->fp32 ? sizeof(float) : sizeof(double);
    for (void** f : {&H->u, &H->v, &H->w, &H->tu, &H->tv, &H->tw}) CK(cudaMalloc(f, H->n * es));
    if (cfg->scheme == CUP_SCHEME_UPWIND3_RK2)
      for (void** f : {&H->u1, &H->v1, &H->w1}) CK(cudaMalloc(f, H->n * es));
    CK(cudaMalloc(&H->p, H->n * sizeof(double)));
    CK(cudaMalloc(&H->rhs, H->n * sizeof(double)));
    if (H->fp32) CK(cudaMalloc(&H->work32, H->n * sizeof(float)));
    if (H->fp32) CK(cudaMalloc(&H->work64, H->n * sizeof(double)));
    if (H->fp32) {
      CK(cudaMalloc(&H->p_old, H->n * sizeof(double)));
      CK(cudaMalloc(&H->p_pred, H->n * sizeof(double)));
    }
    for (void* f : {H->u, H->v, H->w, H->tu, H->tv, H->tw, (void*)H->p, (void*)H->rhs})
      CK(cudaMemsetAsync(f, 0, H->n * (f == (void*)H->p || f == (void*)H->rhs ? sizeof(double) : es), H->stream));
    CK(cudaMalloc(&H->partials, sizeof(double) * kPartialCap * P_COUNT));
    CK(cudaMalloc(&H->dstate, sizeof(DevState)));
    CK(cudaMemsetAsync(H->dstate, 0, sizeof(DevState), H->stream));
    H->derr = &H->dstate->err_word;  // zeroed with the state
    CK(cudaMallocHost(&H->hstate, sizeof(DevState)));
    // FFT tables per axis, spectral cosines exactly as PoissonSolverPeriodic::_solve
    // computes them (source/poisson/PoissonSolverPeriodic.cpp:23-33).
    // (one allocation and one copy for all of them)
    double** cs[3] = {&H->cosx, &H->cosy, &H->cosz};
    std::vector<unsigned char> blob;
    std::vector<std::pair<void**, size_t>> at;
    auto add = [&](auto** dst, const auto& v) {
      const size_t bytes = v.size() * sizeof(v[0]), o = blob.size();
      blob.resize(o + (bytes + 255) / 256 * 256);
      memcpy(blob.data() + o, v.data(), bytes);
      at.push_back({reinterpret_cast<void**>(dst), o});
    };
    for (int d = 0; d < 3; ++d) {
      if (slab && d == 2) continue;  // no z transform on a z-slab handle
      const long nK = N[d];
      const double wFac = 4 * M_PI / nK;
      std::vector<double> c(nK), pc;
      for (long i = 0; i < nK; ++i) c[i] = std::cos(wFac * i);
      std::vector<double2> t64, p64;
      std::vector<float2> p32;
      build_tables(N[d], c, d == 0, t64, p64, p32, pc);
      add(cs[d], c);
      add(&H->tw64[d], t64);
      add(&H->ptw64[d], p64);
      add(&H->ptw32[d], p32);
      add(&H->pcos[d], pc);
    }
    CK(cudaMalloc(&H->tables, blob.size()));
    CK(cudaMemcpy(H->tables, blob.data(), blob.size(), cudaMemcpyHostToDevice));
    for (auto& a : at) *a.first = static_cast<unsigned char*>(H->tables) + a.second;
    H->norm_factor = 4 / ((size_t)N[0] * H->h * (size_t)N[1] * (size_t)N[2]);
    H->pnorm = 8 * H->norm_factor;
    H->spec_ny = H->ny;
    H->spec_y0 = 0;
    H->hstate->lambda = H->lambda;
    CK(cudaMemcpyAsync(&H->dstate->lambda, &H->lambda, sizeof(double), cudaMemcpyHostToDevice, H->stream));
    CK(cudaStreamSynchronize(H->stream));
    if (!get_encode()) return fail(H, CUP_ERR_CUDA, "cuTensorMapEncodeTiled entry point unavailable");
    return CUP_OK;
  }();
  if (rc) {
    fprintf(stderr, "cup_create: %s\n", H->err.c_str());
    cup_destroy(H);
    return rc;
  }
  *out = H;
  return CUP_OK;
}

int cup_destroy(cup_handle* H) {
  if (!H) return CUP_OK;
  cudaSetDevice(H->dev);
  if (H->stream) cudaStreamSynchronize(H->stream);
  drop_graph(H);
  for (void* f : {H->aus, H->avs, H->aws, (void*)H->ab0, (void*)H->spec[0], (void*)H->band_coef, (void*)H->dsum})
    if (f) cudaFree(f);
  for (void* f : {H->u, H->v, H->w, H->tu, H->tv, H->tw, H->u1, H->v1, H->w1, H->au, H->av, H->aw, (void*)H->p_adj,
                  H->chi, (void*)H->p, (void*)H->p_old, (void*)H->p_pred, (void*)H->rhs,
                  (void*)H->work32, (void*)H->work64, (void*)H->partials, (void*)H->dstate, H->tables,
                  (void*)H->cosy_win, (void*)H->sp_dev, (void*)H->box_b, (void*)H->box_delta})
    if (f) cudaFree(f);
  prof_flush(H);
  for (cudaEvent_t e : H->ev_pool) cudaEventDestroy(e);
  if (H->hstate) cudaFreeHost(H->hstate);
  if (H->hsum) cudaFreeHost(H->hsum);
  if (H->cap_stream) cudaStreamDestroy(H->cap_stream);
  if (H->own_stream && H->stream) cudaStreamDestroy(H->stream);
  delete H;
  return CUP_OK;
}

const char* cup_last_error(const cup_handle* H) { return H ? H->err.c_str() : "null handle"; }

int cup_set_stream(cup_handle* H, void* stream) {
  REQUIRE_H(H);
  CK(cudaStreamSynchronize(H->stream));
  if (stream) {
    if (H->own_stream) CK(cudaStreamDestroy(H->stream));
    H->own_stream = false;
    H->stream = (cudaStream_t)stream;
  } else if (!H->own_stream) {
    CK(cudaStreamCreateWithFlags(&H->stream, cudaStreamNonBlocking));
    H->own_stream = true;
  }
  return CUP_OK;
}

int cup_sync(cup_handle* H) {
  REQUIRE_H(H);
  CK(cudaStreamSynchronize(H->stream));
  return check_dev_error(H);
}

int cup_get_dims(const cup_handle* H, int cells[3], double* hgrid) {
  if (!H || !cells) return CUP_ERR_ARG;
  cells[0] = H->nx;
  cells[1] = H->ny;
  cells[2] = H->nz;
  if (hgrid) *hgrid = H->h;
  return CUP_OK;
}

int cup_set_velocity(cup_handle* H, const double* u, const double* v, const double* w, int where) {
  REQUIRE_H(H);
  reset_pressure_history(H);
  if (!u || !v || !w || !valid_where(where)) return fail(H, CUP_ERR_ARG, "bad velocity arguments");
  int rc;
  if ((rc = DISPATCH_T(H, set_field, H->u, u, where))) return rc;
  if ((rc = DISPATCH_T(H, set_field, H->v, v, where))) return rc;
  if ((rc = DISPATCH_T(H, set_field, H->w, w, where))) return rc;
  H->umax_fresh = false;
  if (where == CUP_WHERE_HOST) CK(cudaStreamSynchronize(H->stream));
  return CUP_OK;
}

int cup_get_velocity(cup_handle* H, double* u, double* v, double* w, int where) {
  REQUIRE_H(H);
  if (!u || !v || !w || !valid_where(where)) return fail(H, CUP_ERR_ARG, "bad velocity arguments");
  int rc;
  for (auto pr : {std::make_pair(H->u, u), std::make_pair(H->v, v), std::make_pair(H->w, w)}) {
    if ((rc = DISPATCH_T(H, get_field, pr.first, pr.second, where))) return rc;
    if (where == CUP_WHERE_HOST) CK(cudaStreamSynchronize(H->stream));
  }
  return check_dev_error(H);
}

int cup_get_pressure(cup_handle* H, double* p, int where) {
  REQUIRE_H(H);
  if (!p || !valid_where(where)) return fail(H, CUP_ERR_ARG, "bad pressure arguments");
  CK(cudaMemcpyAsync(p, H->p, H->n * sizeof(double),
                     where == CUP_WHERE_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, H->stream));
  CK(cudaStreamSynchronize(H->stream));
  return check_dev_error(H);
}

int cup_get_rhs(cup_handle* H, double* r, int where) {
  REQUIRE_H(H);
  if (!r || !valid_where(where)) return fail(H, CUP_ERR_ARG, "bad rhs arguments");
  CK(cudaMemcpyAsync(r, H->rhs, H->n * sizeof(double),
                     where == CUP_WHERE_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, H->stream));
  CK(cudaStreamSynchronize(H->stream));
  return check_dev_error(H);
}

int cup_field_ptr(cup_handle* H, int field, void** ptr) {
  REQUIRE_H(H);
  if (!ptr) return fail(H, CUP_ERR_ARG, "cup_field_ptr: null output");
  switch (field) {
    case CUP_FIELD_U: *ptr = H->u; break;
    case CUP_FIELD_V: *ptr = H->v; break;
    case CUP_FIELD_W: *ptr = H->w; break;
    case CUP_FIELD_P: *ptr = H->p; break;
    case CUP_FIELD_RHS: *ptr = H->rhs; break;
    default: return fail(H, CUP_ERR_ARG, "cup_field_ptr: unknown field %d", field);
  }
  return CUP_OK;
}

int cup_get_chi(cup_handle* H, double* chi, int where) {
  REQUIRE_H(H);
  if (!chi || !valid_where(where)) return fail(H, CUP_ERR_ARG, "bad chi arguments");
  if (!H->chi) {
    if (where == CUP_WHERE_HOST) std::fill(chi, chi + H->n, 0.0);
    else CK(cudaMemsetAsync(chi, 0, H->n * sizeof(double), H->stream));
  } else {
    int rc = DISPATCH_T(H, get_field, H->chi, chi, where);
    if (rc) return rc;
  }
  CK(cudaStreamSynchronize(H->stream));
  return CUP_OK;
}

int cup_blocks_to_global(const double* blocks, double* global, int nx, int ny, int nz) {
  if (!blocks || !global || nx % 16 || ny % 16 || nz % 16 || nx <= 0 || ny <= 0 || nz <= 0) return CUP_ERR_ARG;
  const int bx = nx / 16, by = ny / 16;
  size_t i = 0;
  for (int bz = 0; bz < nz / 16; ++bz)
    for (int byy = 0; byy < by; ++byy)
      for (int bxx = 0; bxx < bx; ++bxx)
        for (int iz = 0; iz < 16; ++iz)
          for (int iy = 0; iy < 16; ++iy)
            for (int ix = 0; ix < 16; ++ix)
              global[((size_t)(bz * 16 + iz) * ny + (byy * 16 + iy)) * nx + (bxx * 16 + ix)] = blocks[i++];
  return CUP_OK;
}

int cup_global_to_blocks(const double* global, double* blocks, int nx, int ny, int nz) {
  if (!blocks || !global || nx % 16 || ny % 16 || nz % 16 || nx <= 0 || ny <= 0 || nz <= 0) return CUP_ERR_ARG;
  const int bx = nx / 16, by = ny / 16;
  size_t i = 0;
  for (int bz = 0; bz < nz / 16; ++bz)
    for (int byy = 0; byy < by; ++byy)
      for (int bxx = 0; bxx < bx; ++bxx)
        for (int iz = 0; iz < 16; ++iz)
          for (int iy = 0; iy < 16; ++iy)
            for (int ix = 0; ix < 16; ++ix)
              blocks[i++] = global[((size_t)(bz * 16 + iz) * ny + (byy * 16 + iy)) * nx + (bxx * 16 + ix)];
  return CUP_OK;
}

int cup_add_sphere(cup_handle* H, const cup_sphere* s) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  reset_pressure_history(H);
  if (!s || !(s->radius > 0)) return fail(H, CUP_ERR_ARG, "sphere radius must be > 0");
  if (H->has_sphere) return fail(H, CUP_ERR_STATE, "only one obstacle is supported");
  bool anyForced = false;
  for (int d = 0; d < 3; ++d) anyForced = anyForced || s->bForcedInSimFrame[d];
  H->has_sphere = true;
  H->sphere = *s;
  drop_graph(H);  // captured steps hold no obstacle
  const size_t es = H->fp32 ? sizeof(float) : sizeof(double);
  CK(cudaMalloc(&H->chi, H->n * es));
  CK(cudaMemsetAsync(H->chi, 0, H->n * es, H->stream));
  CK(cudaMalloc(&H->sp_dev, sizeof(SphereParams)));
  // updateUinf (source/obstacles/ObstacleVector.h:60-76) for one obstacle: the
  // frame follows the obstacle on its fixed dofs and is at rest on the others
  for (int d = 0; d < 3; ++d) {
    H->sphere_vel[d] = s->bForcedInSimFrame[d] ? s->enforcedVelocity[d] : 0.0;
    H->uinf[d] = s->bFixFrameOfRef[d] ? -H->sphere_vel[d] : 0.0;
  }
  H->sphere_free = !(s->bForcedInSimFrame[0] && s->bForcedInSimFrame[1] && s->bForcedInSimFrame[2]);
  H->sphere_moves = H->sphere_free;
  for (int d = 0; d < 3; ++d) H->sphere_moves = H->sphere_moves || (H->sphere_vel[d] + H->uinf[d] != 0.0);
  for (int d = 0; d < 3; ++d) H->sphere_angvel[d] = 0.0;
  H->sphere_quat[0] = 1, H->sphere_quat[1] = H->sphere_quat[2] = H->sphere_quat[3] = 0;
  SphereParams sp{};
  sp.radius = s->radius;
  for (int d = 0; d < 3; ++d) {
    sp.position[d] = s->position[d];
    sp.transVel[d] = s->bForcedInSimFrame[d] ? s->enforcedVelocity[d] : 0.0;
    sp.angVel[d] = 0.0;
    sp.transVel_imposed[d] = sp.transVel[d];
    sp.forced[d] = s->bForcedInSimFrame[d] ? 1 : 0;
    sp.block_rot[d] = anyForced ? 1 : 0;  // any forced dof blocks rotation (Obstacle.cpp:131-137)
  }
  sp.lambda_factor = 1.0;
  sphere_box(H);
  {
    // the box spans at most 2 (R + 3h) / h + 5 cells per axis wherever the sphere moves
    const int N[3] = {H->nx, H->ny, H->nz};
    long long cap = 1;
    for (int d = 0; d < 3; ++d)
      cap *= std::min<long long>(N[d], (long long)std::ceil(2 * (s->radius + 3 * H->h) / H->h) + 6);
    H->box_cap = cap;
    CK(cudaMalloc(&H->box_b, cap * sizeof(double)));
    CK(cudaMalloc(&H->box_delta, cap * sizeof(double)));
  }
  CK(cudaMemcpyAsync(H->sp_dev, &sp, sizeof(sp), cudaMemcpyHostToDevice, H->stream));
  int rc = build_sphere_chi(H);
  if (rc) return rc;
  H->umax_fresh = false;
  CK(cudaStreamSynchronize(H->stream));
  return check_dev_error(H);
}

int cup_set_sphere_position(cup_handle* H, const double position[3]) {
  REQUIRE_H(H);
  if (!H->has_sphere) return fail(H, CUP_ERR_ARG, "cup_set_sphere_position: the handle has no obstacle");
  if (!position) return fail(H, CUP_ERR_ARG, "null position");
  for (int d = 0; d < 3; ++d) H->sphere.position[d] = position[d];
  drop_graph(H);  // captured steps hold the obstacle's box
  int rc = relocate_sphere(H);
  if (rc) return rc;
  H->umax_fresh = false;
  CK(cudaStreamSynchronize(H->stream));
  return check_dev_error(H);
}

int cup_get_sphere_position(cup_handle* H, double position[3]) {
  REQUIRE_H(H);
  if (!H->has_sphere) return fail(H, CUP_ERR_ARG, "cup_get_sphere_position: the handle has no obstacle");
  if (!position) return fail(H, CUP_ERR_ARG, "null position");
  for (int d = 0; d < 3; ++d) position[d] = H->sphere.position[d];
  return CUP_OK;
}

int cup_set_uinf(cup_handle* H, const double uinf[3]) {
  REQUIRE_H(H);
  if (!uinf) return fail(H, CUP_ERR_ARG, "null uinf");
  if (H->has_sphere) return fail(H, CUP_ERR_STATE, "cup_set_uinf: with an obstacle the frame velocity follows it");
  for (int d = 0; d < 3; ++d) H->uinf[d] = uinf[d];
  drop_graph(H);  // captured steps hold uinf
  H->umax_fresh = false;
  return CUP_OK;
}

int cup_set_graphs(cup_handle* H, int on) {
  REQUIRE_H(H);
  H->use_graphs = on != 0;
  if (!H->use_graphs) drop_graph(H);
  return CUP_OK;
}

int cup_prepare_run(cup_handle* H, int nsteps, int* captured) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  REQUIRE_OWN_SPECTRUM(H);
  if (captured) *captured = 0;
  if (nsteps < 0) return fail(H, CUP_ERR_ARG, "nsteps must be >= 0");
  if (!graph_ok(H)) return CUP_OK;
  // walk the graphs cup_run(nsteps) would replay from here, capturing the
  // missing ones; the host state is put back afterwards
  const cup_handle::StepState start = step_state(H);
  int n = 0, rc = CUP_OK;
  for (int i = 0; i < nsteps && rc == CUP_OK;) {
    const bool whole = nsteps - i > kGraphSteps;
    cup_handle::StepGraph* g = nullptr;
    rc = capture_graph(H, whole ? kGraphSteps : 1, whole || i + 1 < nsteps ? 1 : 0, &g);
    if (rc || !g) break;
    set_step_state(H, g->out);
    ++n;
    i += whole ? kGraphSteps : 1;
    if (whole && nsteps - i > kGraphSteps) i += (nsteps - i - 1) / kGraphSteps * kGraphSteps;  // same state again
  }
  set_step_state(H, start);
  if (captured) *captured = n;
  return rc;
}

int cup_create_obstacles(cup_handle* H, double dt) {
  REQUIRE_H(H);
  if (!(dt >= 0)) return fail(H, CUP_ERR_ARG, "dt must be >= 0");
  int rc = do_create_obstacles(H, dt);
  if (rc) return rc;
  return CUP_OK;
}

int cup_update_obstacles(cup_handle* H, double dt) {
  REQUIRE_H(H);
  if (!(dt > 0)) return fail(H, CUP_ERR_ARG, "dt must be > 0");
  if (!H->has_sphere || !H->sphere_free) return CUP_OK;  // forced dofs keep their imposed velocity
  // lambda from the host, as cup_penalize takes it
  int rc = H->fp32 ? do_rigid_update<float>(H, DtArg{dt, nullptr}, nullptr)
                   : do_rigid_update<double>(H, DtArg{dt, nullptr}, nullptr);
  if (rc) return rc;
  return read_sphere_motion(H);
}

int cup_get_sphere_motion(cup_handle* H, double transVel[3], double angVel[3], double quaternion[4]) {
  REQUIRE_H(H);
  if (!H->has_sphere) return fail(H, CUP_ERR_ARG, "the handle has no obstacle");
  if (!transVel || !angVel || !quaternion) return fail(H, CUP_ERR_ARG, "null output");
  for (int d = 0; d < 3; ++d) {
    transVel[d] = H->sphere_vel[d];
    angVel[d] = H->sphere_angvel[d];
  }
  for (int k = 0; k < 4; ++k) quaternion[k] = H->sphere_quat[k];
  return CUP_OK;
}

int cup_set_sphere_motion(cup_handle* H, const double transVel[3], const double angVel[3], const double quaternion[4]) {
  REQUIRE_H(H);
  if (!H->has_sphere) return fail(H, CUP_ERR_ARG, "the handle has no obstacle");
  if (!transVel || !angVel || !quaternion) return fail(H, CUP_ERR_ARG, "null input");
  for (int d = 0; d < 3; ++d) {
    H->sphere_vel[d] = transVel[d];
    H->sphere_angvel[d] = angVel[d];
  }
  for (int k = 0; k < 4; ++k) H->sphere_quat[k] = quaternion[k];
  CK(cudaMemcpyAsync(reinterpret_cast<char*>(H->sp_dev) + offsetof(SphereParams, transVel), transVel,
                     3 * sizeof(double), cudaMemcpyHostToDevice, H->stream));
  CK(cudaMemcpyAsync(reinterpret_cast<char*>(H->sp_dev) + offsetof(SphereParams, angVel), angVel, 3 * sizeof(double),
                     cudaMemcpyHostToDevice, H->stream));
  CK(cudaStreamSynchronize(H->stream));
  if (H->sphere_free)
    for (int d = 0; d < 3; ++d) H->uinf[d] = H->sphere.bFixFrameOfRef[d] ? -H->sphere_vel[d] : 0.0;
  drop_graph(H);
  H->umax_fresh = false;
  return CUP_OK;
}

int cup_get_obstacle_state(cup_handle* H, double force[3], double torque[3], double com[3], double uinf[3]) {
  REQUIRE_H(H);
  int rc = read_state(H);
  if (rc) return rc;
  for (int d = 0; d < 3; ++d) {
    if (force) force[d] = H->hstate->force[d];
    if (torque) torque[d] = H->hstate->torque[d];
    if (com) com[d] = H->hstate->com[d];
    if (uinf) uinf[d] = H->uinf[d];
  }
  return CUP_OK;
}

int cup_set_clock(cup_handle* H, int step, double time) {
  REQUIRE_H(H);
  if (step < 0) return fail(H, CUP_ERR_ARG, "step must be >= 0");
  H->step = step;
  H->time = time;
  return CUP_OK;
}

int cup_max_velocity(cup_handle* H, double* umax) {
  REQUIRE_H(H);
  int rc = DISPATCH_T(H, do_max_u);
  if (rc) return rc;
  if ((rc = read_state(H))) return rc;
  if (umax) *umax = H->hstate->umax;
  H->umax_fresh = true;
  return CUP_OK;
}

int cup_calc_max_timestep(cup_handle* H, double* dt) {
  REQUIRE_H(H);
  int rc;
  if (H->dt_next_call && H->api_calls == H->dt_next_call + 1 && H->umax_fresh) {
    // nothing happened since timestep read back the dt its step computed
    // (the same calc_dt_device on the same max |u| and step counter)
    H->dt = H->dt_next;
    if (H->cfg.DLM > 0) H->lambda = H->lambda_next;
    if (dt) *dt = H->dt;
    return CUP_OK;
  }
  // (the device keeps its own step counter in sync with the host mirror)
  if (!H->umax_fresh) {
    if ((rc = DISPATCH_T(H, do_max_u, 1))) return rc;
    H->umax_fresh = true;
  } else {
    rc = launch_named(H, "calc_dt", [&]() -> int {
      klaunch(H, k_calc_dt, 1, 1, 0, H->dstate, cfl_params(H), H->step);
      CKL();
      return CUP_OK;
    });
    if (rc) return rc;
  }
  if ((rc = read_state(H))) return rc;
  H->dt = H->hstate->dt;
  if (H->cfg.DLM > 0) H->lambda = H->hstate->lambda;
  if (dt) *dt = H->dt;
  return CUP_OK;
}

int cup_advect_diffuse(cup_handle* H, double dt) {
  REQUIRE_H(H);
  reset_pressure_history(H);
  H->umax_fresh = false;
  return DISPATCH_T(H, do_advect_diffuse, DtArg{dt, nullptr});
}

int cup_pressure_rhs(cup_handle* H, double dt) {
  REQUIRE_H(H);
  reset_pressure_history(H);
  return DISPATCH_T(H, do_pressure_rhs, DtArg{dt, nullptr});
}

int cup_set_rhs(cup_handle* H, const double* r, int where) {
  REQUIRE_H(H);
  if (!r || !valid_where(where)) return fail(H, CUP_ERR_ARG, "bad rhs arguments");
  CK(cudaMemcpyAsync(H->rhs, r, H->n * sizeof(double),
                     where == CUP_WHERE_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, H->stream));
  CK(cudaStreamSynchronize(H->stream));
  return check_dev_error(H);
}

int cup_poisson_buffer(cup_handle* H, double** data, size_t strides[3], size_t* data_size) {
  REQUIRE_H(H);
  if (!data || !strides || !data_size) return fail(H, CUP_ERR_ARG, "null output");
  *data = H->rhs;
  strides[0] = 1;
  strides[1] = (size_t)H->nx;
  strides[2] = (size_t)H->nx * H->ny;
  *data_size = H->n;
  return CUP_OK;
}

int cup_poisson_reset(cup_handle* H) {
  REQUIRE_H(H);
  CK(cudaMemsetAsync(H->rhs, 0, H->n * sizeof(double), H->stream));
  return CUP_OK;
}

int cup_set_spectral_window(cup_handle* H, int y0, int ny_global) {
  REQUIRE_H(H);
  if (ny_global < H->ny || !is_pow2(ny_global) || y0 < 0 || y0 + H->ny > ny_global || y0 % H->ny)
    return fail(H, CUP_ERR_ARG, "spectral window: need 0 <= y0, y0 + ny <= ny_global (a power of two), y0 a multiple of ny");
  std::vector<double> c(ny_global);
  const double wFac = 4 * M_PI / (long)ny_global;
  for (long i = 0; i < ny_global; ++i) c[i] = std::cos(wFac * i);
  double* d = nullptr;
  CK(cudaMalloc(&d, ny_global * sizeof(double)));
  CK(cudaMemcpy(d, c.data(), ny_global * sizeof(double), cudaMemcpyHostToDevice));
  cudaFree(H->cosy_win);
  H->cosy = H->cosy_win = d;
  H->spec_ny = ny_global;
  H->spec_y0 = y0;
  H->norm_factor = 4 / ((double)H->nx * H->h * (double)ny_global * (double)H->nz);
  drop_graph(H);
  return CUP_OK;
}

int cup_poisson_pass(cup_handle* H, double* buf, int pass) {
  REQUIRE_H(H);
  if (!buf) return fail(H, CUP_ERR_ARG, "null buffer");
  switch (pass) {
    case 0: return launch_rows_pipe(H, "dht_x", buf);
    case 1: return launch_cols<1, false>(H, buf);
    case 2: return launch_cols<2, true>(H, buf);
    default: return fail(H, CUP_ERR_ARG, "pass must be 0 (x), 1 (y) or 2 (z with the spectral divide)");
  }
}

int cup_poisson_solve(cup_handle* H, cup_solve_stats* stats) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  REQUIRE_OWN_SPECTRUM(H);
  reset_pressure_history(H);
  int rc = do_poisson(H);
  if (rc) return rc;
  if (stats) {
    stats->n_solves = 1;
    stats->rel_residual = 0;
    if (H->fp32) {
      if ((rc = read_state(H))) return rc;
      stats->n_solves = H->hstate->n_solves;
      stats->rel_residual = H->hstate->b2 > 0 ? std::sqrt(H->hstate->res2 / H->hstate->b2) : 0.0;
      if (H->hstate->converged == 2)
        return fail(H, CUP_ERR_NOT_CONVERGED, "defect correction: relative residual %.3e after %d solves",
                    stats->rel_residual, stats->n_solves);
    }
  }
  return CUP_OK;
}

int cup_grad_correct(cup_handle* H, double dt) {
  REQUIRE_H(H);
  reset_pressure_history(H);
  H->umax_fresh = false;
  return DISPATCH_T(H, do_grad, DtArg{dt, nullptr});
}

int cup_pressure_projection(cup_handle* H, double dt, cup_solve_stats* stats) {
  int rc = cup_poisson_solve(H, stats);
  if (rc) return rc;
  return cup_grad_correct(H, dt);
}

int cup_penalize(cup_handle* H, double dt, double force_torque[6]) {
  REQUIRE_H(H);
  reset_pressure_history(H);
  H->umax_fresh = false;
  if (!H->has_sphere) {
    if (force_torque) std::fill(force_torque, force_torque + 6, 0.0);
    return CUP_OK;
  }
  int rc = DISPATCH_T(H, do_penalize, DtArg{dt, nullptr}, (const double*)nullptr);
  if (rc) return rc;
  {
    int rc_ = launch_named(H, "finalize_pen", [&]() -> int {
      klaunch(H, k_finalize_pen, 1, 192, 0, partial(H, P_PEN), H->n_pen_partials, H->dstate, H->cfg.DLM, H->lambda);
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  if (force_torque) {
    if ((rc = read_state(H))) return rc;
    for (int d = 0; d < 3; ++d) {
      force_torque[d] = H->hstate->force[d];
      force_torque[3 + d] = H->hstate->torque[d];
    }
  }
  return CUP_OK;
}

static int fill_stats(cup_handle* H, cup_step_stats* st) {
  int rc = read_state(H);
  if (rc) return rc;
  const DevState& s = *H->hstate;
  st->dt = s.dt;
  st->time = H->time;
  st->step = H->step;
  st->umax = s.umax;
  st->kinetic_energy = s.ke;
  for (int d = 0; d < 3; ++d) {
    st->force[d] = s.force[d];
    st->torque[d] = s.torque[d];
  }
  st->n_solves = H->fp32 ? s.n_solves : 1;
  st->n_unconverged = s.n_unconverged;
  st->n_solves_total = H->fp32 ? s.solves_total : 0;
  st->rel_residual = H->fp32 && s.b2 > 0 ? std::sqrt(s.res2 / s.b2) : 0.0;
  if (H->fp32 && s.converged == 2)
    return fail(H, CUP_ERR_NOT_CONVERGED, "defect correction: relative residual %.3e after %d solves",
                st->rel_residual, s.n_solves);
  if (!std::isfinite(s.umax) || !std::isfinite(s.ke)) return fail(H, CUP_ERR_NONFINITE, "non-finite velocity");
  return CUP_OK;
}

int cup_step(cup_handle* H, double dt, cup_step_stats* stats) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  REQUIRE_OWN_SPECTRUM(H);
  if (!(dt > 0)) return fail(H, CUP_ERR_ARG, "dt must be > 0");
  H->dt = dt;
  if (H->cfg.DLM > 0) H->lambda = H->cfg.DLM / dt;
  // device dt/lambda follow the host values for this step
  {
    int rc_ = launch_named(H, "set_dt", [&]() -> int {
      klaunch(H, k_set_state, 1, 1, 0, H->dstate, SET_DT | SET_LAMBDA, dt, H->lambda, 0, 0.0, cfl_params(H));
      CKL();
      return CUP_OK;
    });
    if (rc_) return rc_;
  }
  // one step from a captured graph in the steady state (it reads dt from the
  // device state set above), else launched; either way the step ends by
  // computing the next step's CFL dt on the device, which the stats read-back
  // brings to the host for a following calcMaxTimestep
  bool ran = false;
  int rc = graph_ok(H) ? run_graph(H, 1, 1, &ran) : CUP_OK;
  if (rc) return rc;
  if (!ran) {
    rc = DISPATCH_T(H, do_step, DtArg{dt, nullptr}, (const double*)&H->dstate->lambda, 1, 1);
    H->steps_run += 1;
  }
  if (rc) return rc;
  if (H->has_sphere && H->sphere_free && (rc = read_sphere_motion(H))) return rc;
  H->step += 1;
  H->time += dt;
  H->umax_fresh = true;
  H->dt_next_call = 0;
  if (!stats) return CUP_OK;
  rc = fill_stats(H, stats);
  stats->dt = dt;  // this step's dt (the device state now holds the next one)
  if (rc == CUP_OK && H->hstate->step == H->step) {
    H->dt_next = H->hstate->dt;
    H->lambda_next = H->hstate->lambda;
    H->dt_next_call = H->api_calls;
  }
  return rc;
}

static int alloc_adjoint(cup_handle* H) {
  if (H->p_adj) return CUP_OK;
  const size_t es = H->fp32 ? sizeof(float) : sizeof(double);
  for (void** f : {&H->au, &H->av, &H->aw}) CK(cudaMalloc(f, H->n * es));
  CK(cudaMalloc(&H->p_adj, H->n * sizeof(double)));
  return CUP_OK;
}

static int check_adjoint_fields(cup_handle* H, const void* un, const void* vn, const void* wn, void* lu, void* lv,
                                void* lw) {
  if (!un || !vn || !wn || !lu || !lv || !lw) return fail(H, CUP_ERR_ARG, "null field pointer");
  const void* st[3] = {un, vn, wn};
  const void* lm[3] = {lu, lv, lw};
  for (int a = 0; a < 3; ++a)
    for (int b = 0; b < 3; ++b) {
      if (st[a] == lm[b]) return fail(H, CUP_ERR_ARG, "the state and the adjoint fields must not alias");
      if (a < b && (lm[a] == lm[b] || st[a] == st[b])) return fail(H, CUP_ERR_ARG, "field pointers must be distinct");
    }
  // TMA reads the state, and the upwind3 transposes read and write the adjoint
  // fields in pieces of up to 16 bytes (the central scheme stores single values)
  const uintptr_t es = H->fp32 ? sizeof(float) : sizeof(double);
  const uintptr_t al = H->cfg.scheme == CUP_SCHEME_REF ? es : 16;
  for (int a = 0; a < 3; ++a) {
    if ((uintptr_t)st[a] % 16) return fail(H, CUP_ERR_ARG, "the state's fields must be aligned to 16 bytes");
    if ((uintptr_t)lm[a] % al) return fail(H, CUP_ERR_ARG, "the adjoint fields must be aligned to %d bytes", (int)al);
  }
  return CUP_OK;
}

int cup_adjoint_step(cup_handle* H, const void* un, const void* vn, const void* wn, double dt, void* lu, void* lv,
                     void* lw) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  REQUIRE_OWN_SPECTRUM(H);
  if (!(dt > 0)) return fail(H, CUP_ERR_ARG, "dt must be > 0");
  if (H->has_sphere) return fail(H, CUP_ERR_ARG, "cup_adjoint_step: the handle has an obstacle (use cup_adjoint_step_obstacle)");
  if (H->forcing)
    return fail(H, CUP_ERR_STATE, "cup_adjoint_step: spectral forcing is on and has no adjoint (turn it off first)");
  int rc = check_adjoint_fields(H, un, vn, wn, lu, lv, lw);
  if (!rc) rc = alloc_adjoint(H);
  if (rc) return rc;
  void* s3[3] = {const_cast<void*>(un), const_cast<void*>(vn), const_cast<void*>(wn)};
  void* l3[3] = {lu, lv, lw};
  return DISPATCH_T(H, do_adjoint_step, s3, l3, DtArg{dt, nullptr});
}

int cup_adjoint_step_obstacle(cup_handle* H, const void* un, const void* vn, const void* wn, double dt, void* lu,
                              void* lv, void* lw, const double w_force[3], double* g_chi, double* g_vel) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  REQUIRE_OWN_SPECTRUM(H);
  if (!(dt > 0)) return fail(H, CUP_ERR_ARG, "dt must be > 0");
  if (!H->has_sphere) return fail(H, CUP_ERR_ARG, "cup_adjoint_step_obstacle: the handle has no obstacle");
  if (H->sphere_moves)
    return fail(H, CUP_ERR_STATE, "cup_adjoint_step_obstacle: the adjoint of a moving obstacle is not supported");
  if (H->forcing)
    return fail(H, CUP_ERR_STATE,
                "cup_adjoint_step_obstacle: spectral forcing is on and has no adjoint (turn it off first)");
  if (!w_force || !g_chi || !g_vel) return fail(H, CUP_ERR_ARG, "null w_force / g_chi / g_vel");
  int rc = check_adjoint_fields(H, un, vn, wn, lu, lv, lw);
  if (!rc) rc = alloc_adjoint(H);
  if (rc) return rc;
  if (!H->ab0) {
    const size_t es = H->fp32 ? sizeof(float) : sizeof(double);
    for (void** f : {&H->aus, &H->avs, &H->aws}) CK(cudaMalloc(f, H->n * es));
    CK(cudaMalloc(&H->ab0, H->box_cap * sizeof(double)));
  }
  void* s3[3] = {const_cast<void*>(un), const_cast<void*>(vn), const_cast<void*>(wn)};
  void* l3[3] = {lu, lv, lw};
  const double wF[3] = {w_force[0], w_force[1], w_force[2]};
  return DISPATCH_T(H, do_adjoint_step_obstacle, s3, l3, DtArg{dt, nullptr}, wF, g_chi, g_vel);
}

int cup_set_chi(cup_handle* H, const double* chi, int where) {
  REQUIRE_H(H);
  if (!H->has_sphere || !H->chi) return fail(H, CUP_ERR_ARG, "cup_set_chi: the handle has no obstacle");
  if (!chi || !valid_where(where)) return fail(H, CUP_ERR_ARG, "bad chi arguments");
  return DISPATCH_T(H, set_field, H->chi, chi, where);
}

int cup_set_sphere_velocity(cup_handle* H, const double vel[3]) {
  REQUIRE_H(H);
  if (!H->has_sphere) return fail(H, CUP_ERR_ARG, "cup_set_sphere_velocity: the handle has no obstacle");
  if (!vel) return fail(H, CUP_ERR_ARG, "null velocity");
  // SphereParams::transVel only (the device copy is read by every penalization)
  CK(cudaMemcpyAsync(reinterpret_cast<char*>(H->sp_dev) + offsetof(SphereParams, transVel), vel, 3 * sizeof(double),
                     cudaMemcpyHostToDevice, H->stream));
  CK(cudaStreamSynchronize(H->stream));
  return CUP_OK;
}

int cup_get_velocity_raw(cup_handle* H, void* u, void* v, void* w) {
  REQUIRE_H(H);
  if (!u || !v || !w) return fail(H, CUP_ERR_ARG, "null field pointer");
  const size_t bytes = H->n * (H->fp32 ? sizeof(float) : sizeof(double));
  CK(cudaMemcpyAsync(u, H->u, bytes, cudaMemcpyDeviceToDevice, H->stream));
  CK(cudaMemcpyAsync(v, H->v, bytes, cudaMemcpyDeviceToDevice, H->stream));
  CK(cudaMemcpyAsync(w, H->w, bytes, cudaMemcpyDeviceToDevice, H->stream));
  return CUP_OK;
}

int cup_set_velocity_raw(cup_handle* H, const void* u, const void* v, const void* w) {
  REQUIRE_H(H);
  reset_pressure_history(H);
  if (!u || !v || !w) return fail(H, CUP_ERR_ARG, "null field pointer");
  const size_t bytes = H->n * (H->fp32 ? sizeof(float) : sizeof(double));
  CK(cudaMemcpyAsync(H->u, u, bytes, cudaMemcpyDeviceToDevice, H->stream));
  CK(cudaMemcpyAsync(H->v, v, bytes, cudaMemcpyDeviceToDevice, H->stream));
  CK(cudaMemcpyAsync(H->w, w, bytes, cudaMemcpyDeviceToDevice, H->stream));
  H->umax_fresh = false;
  return CUP_OK;
}

int cup_run(cup_handle* H, int nsteps, cup_step_stats* stats) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  REQUIRE_OWN_SPECTRUM(H);
  if (nsteps < 0) return fail(H, CUP_ERR_ARG, "nsteps must be >= 0");
  int rc;
  if (!H->umax_fresh) {
    if ((rc = DISPATCH_T(H, do_max_u))) return rc;
    H->umax_fresh = true;
  }
  // the clock, and the dt of the first step; each step then ends with the next one's
  rc = launch_named(H, "set_state", [&]() -> int {
    klaunch(H, k_set_state, 1, 1, 0, H->dstate, SET_LAMBDA | SET_CLOCK | (nsteps ? CALC_DT : 0), 0.0, H->lambda, H->step,
            H->time, cfl_params(H));
    CKL();
    return CUP_OK;
  });
  if (rc) return rc;
  if (H->has_sphere && H->sphere_moves) {
    // a moving sphere's box follows its position on the host: dt is read back
    // every step (calcMaxTimestep + timestep, as the reference runs them)
    for (int i = 0; i < nsteps; ++i) {
      if ((rc = read_state(H))) return rc;
      if ((rc = cup_step(H, H->hstate->dt, nullptr))) return rc;
    }
    if (!stats) return CUP_OK;
    rc = fill_stats(H, stats);
    if (nsteps) stats->dt = H->dt;  // the last step's (the device state holds the next one's)
    return rc;
  }
  for (int i = 0; i < nsteps;) {
    // (the dt of step i > 0 comes from the end of step i - 1)
    // steady state: whole graphs of kGraphSteps steps, each computing the
    // next step's dt; the steps of the run's tail from one-step graphs (the
    // last one computes no next dt)
    if (graph_ok(H)) {
      const bool whole = nsteps - i > kGraphSteps;
      bool ran = false;
      if ((rc = run_graph(H, whole ? kGraphSteps : 1, whole || i + 1 < nsteps ? 1 : 0, &ran))) return rc;
      if (ran) {
        i += whole ? kGraphSteps : 1;
        continue;
      }
    }
    rc = DISPATCH_T(H, do_step, DtArg{0.0, &H->dstate->dt}, (const double*)&H->dstate->lambda, 1,
                    i + 1 < nsteps ? 1 : 0);
    if (rc) return rc;
    H->steps_run += 1;
    if (H->forcing) {  // the host has this step's dt
      H->step += 1;
      H->time += H->dt;
    }
    ++i;
  }
  if ((rc = read_state(H))) return rc;
  H->step = H->hstate->step;
  H->time = H->hstate->time;
  H->dt = H->hstate->dt;
  if (H->cfg.DLM > 0) H->lambda = H->hstate->lambda;
  if (stats) return fill_stats(H, stats);
  return CUP_OK;
}

int cup_poisson_solve_field(cup_handle* H, const double* rhs, double* p, int where) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  REQUIRE_OWN_SPECTRUM(H);
  reset_pressure_history(H);
  if (!rhs || !p || !valid_where(where)) return fail(H, CUP_ERR_ARG, "bad poisson arguments");
  const cudaMemcpyKind in = where == CUP_WHERE_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  const cudaMemcpyKind out = where == CUP_WHERE_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  // Device arrays of the direct solve: the first pass reads rhs and the last
  // writes p beside the handle's pressure (two copies of the field less; 337 ->
  // 275 us at 256^3). The passes move 16-byte pieces, and p must not overlap the
  // arrays the last pass reads and writes; anything else is copied.
  const size_t bytes = H->n * sizeof(double);
  auto apart = [&](const void* a, const void* b) {
    const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
    return x + bytes <= y || y + bytes <= x;
  };
  int rc;
  if (where == CUP_WHERE_DEVICE && !H->fp32 && (uintptr_t)rhs % 16 == 0 &&
      (uintptr_t)p % 16 == 0 && apart(p, H->rhs) && apart(p, H->p) && (rhs == H->rhs || apart(rhs, H->rhs))) {
    if ((rc = launch_pfft_x<double, PROW_FWD>(H, "dht_x", rhs, H->rhs, nullptr, 0, nullptr))) return rc;
    if ((rc = pfft_finish(H, "dht_x", H->rhs, H->p, p))) return rc;
  } else {
    CK(cudaMemcpyAsync(H->rhs, rhs, bytes, in, H->stream));
    if (H->fp32) CK(cudaMemsetAsync(H->p, 0, bytes, H->stream));
    if ((rc = do_poisson(H))) return rc;
    CK(cudaMemcpyAsync(p, H->p, bytes, out, H->stream));
  }
  CK(cudaStreamSynchronize(H->stream));
  return check_dev_error(H);
}

int cup_diagnostics(cup_handle* H, double out[3]) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  if (!out) return fail(H, CUP_ERR_ARG, "null output");
  int zc, grid;
  march_grid(H, &zc, &grid);
  double* part = partial(H, P_DIAG);
  int rc = launch_named(H, "diag", [&]() -> int {
    if (H->fp32)
      klaunch(H, k_diag<float>, grid, 256, 0, (const float*)H->u, (const float*)H->v, (const float*)H->w, ilog2(H->nx),
              ilog2(H->ny), H->nz, zc, 0.5 / H->h, part);
    else
      klaunch(H, k_diag<double>, grid, 256, 0, (const double*)H->u, (const double*)H->v, (const double*)H->w,
              ilog2(H->nx), ilog2(H->ny), H->nz, zc, 0.5 / H->h, part);
    CKL();
    return CUP_OK;
  });
  if (!rc) rc = sum_columns(H, part, grid, 3, 2, 0);
  if (!rc) rc = read_sums(H, 3);
  if (rc) return rc;
  const double ke = H->hsum[0], d2 = H->hsum[1], dm = H->hsum[2];
  const double h3 = H->h * H->h * H->h;
  out[0] = ke * h3;
  out[1] = std::sqrt(d2 * h3);
  out[2] = dm;
  return CUP_OK;
}

int cup_spectral_analysis(cup_handle* H, double stats[7], double* spectrum, int nbin) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  if (!stats) return fail(H, CUP_ERR_ARG, "null stats");
  const int N = std::max(H->nx, std::max(H->ny, H->nz));
  if (spectrum && nbin != N / 2 - 1) return fail(H, CUP_ERR_ARG, "spectrum needs max(N)/2 - 1 = %d bins", N / 2 - 1);
  double raw[4];
  std::vector<double> bins;
  ModeParams mp;
  int rc = mode_params(H, &mp);
  if (!rc) rc = do_spectral(H, mp, raw, bins);
  if (rc) return rc;
  const double NF = (double)H->n, nu = H->cfg.nu;
  const double tke = raw[0] / (NF * NF), eps = nu * raw[3] / NF;
  const double uprime = std::sqrt(2 * tke / 3);
  const double lambda = std::sqrt(15 * nu / eps) * uprime;
  const double l_integral = raw[0] > 0 ? raw[1] / raw[0] : 0.0;
  stats[0] = tke;
  stats[1] = eps;
  stats[2] = uprime;
  stats[3] = lambda;
  stats[4] = uprime * lambda / nu;
  stats[5] = l_integral;
  stats[6] = l_integral / uprime;
  if (spectrum)
    for (int b = 0; b < nbin; ++b) spectrum[b] = bins[b] / (NF * NF);
  return CUP_OK;
}

int cup_set_spectral_forcing(cup_handle* H, double turbKinEn_target, double enInjectionRate) {
  REQUIRE_H(H);
  if (turbKinEn_target > 0 && enInjectionRate > 0)
    return fail(H, CUP_ERR_ARG, "give either turbKinEn_target or energyInjectionRate, not both");
  H->forcing = turbKinEn_target > 0 || enInjectionRate > 0;
  H->forcing_target = turbKinEn_target > 0 ? turbKinEn_target : 0.0;
  H->forcing_rate = enInjectionRate > 0 ? enInjectionRate : 0.0;
  return CUP_OK;
}

int cup_spectral_forcing(cup_handle* H, double dt, double stats[6]) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  if (!(dt > 0)) return fail(H, CUP_ERR_ARG, "dt must be > 0");
  reset_pressure_history(H);
  H->umax_fresh = false;
  int rc = DISPATCH_T(H, do_spectral_forcing, DtArg{dt, nullptr});
  if (rc) return rc;
  if (stats)
    for (int k = 0; k < 6; ++k) stats[k] = H->forcing_stats[k];
  CK(cudaStreamSynchronize(H->stream));
  return check_dev_error(H);
}

int cup_get_forcing_stats(cup_handle* H, double stats[6]) {
  REQUIRE_H(H);
  if (!stats) return fail(H, CUP_ERR_ARG, "null stats");
  for (int k = 0; k < 6; ++k) stats[k] = H->forcing_stats[k];
  return CUP_OK;
}

int cup_compute_forces(cup_handle* H, double out[27]) {
  REQUIRE_H(H);
  if (!out) return fail(H, CUP_ERR_ARG, "null output");
  for (int k = 0; k < 27; ++k) out[k] = 0.0;
  if (!H->has_sphere) return CUP_OK;  // ComputeForces: nothing without obstacles
  const int gb = box_grid(H->box);
  double* part = partial(H, P_DIAG);
  int rc = H->fp32 ? do_surface_forces<float>(H, part, gb) : do_surface_forces<double>(H, part, gb);
  if (rc) return rc;
  std::vector<double> hp((size_t)kSurfQoI * gb);
  SphereParams sp;
  CK(cudaMemcpyAsync(hp.data(), part, hp.size() * sizeof(double), cudaMemcpyDeviceToHost, H->stream));
  CK(cudaMemcpyAsync(&sp, H->sp_dev, sizeof(SphereParams), cudaMemcpyDeviceToHost, H->stream));
  CK(cudaStreamSynchronize(H->stream));
  for (int b = 0; b < gb; ++b)
    for (int k = 0; k < kSurfQoI; ++k) out[k] += hp[(size_t)kSurfQoI * b + k];
  // derived quantities of Obstacle::computeForces (source/obstacles/Obstacle.cpp:283-294)
  const double EPS = 2.220446049250313080847e-16;
  const double vel_norm = std::sqrt(sp.transVel[0] * sp.transVel[0] + sp.transVel[1] * sp.transVel[1] +
                                    sp.transVel[2] * sp.transVel[2]);
  const double drag = out[15], thrust = out[16], defPower = out[19], defPowerBnd = out[20];
  out[22] = thrust * vel_norm;                                            // Pthrust
  out[23] = drag * vel_norm;                                              // Pdrag
  out[24] = out[22] / (out[22] - std::min(defPower, 0.0) + EPS);          // EffPDef
  out[25] = out[22] / (out[22] - defPowerBnd + EPS);                      // EffPDefBnd
  if ((rc = read_state(H))) return rc;
  out[26] = H->hstate->mass;  // the grid mass of chi (ObstaclesCreate.cpp:230-256)
  return check_dev_error(H);
}

int cup_compute_dissipation(cup_handle* H, double out[20]) {
  REQUIRE_H(H);
  REQUIRE_WHOLE_GRID(H);
  if (!out) return fail(H, CUP_ERR_ARG, "null output");
  int zc, grid;
  march_grid(H, &zc, &grid);
  double* part = partial(H, P_DIAG);
  const double h = H->h;
  const double hCube = std::pow(h, 3), inv2h = .5 / h, invHh = 1 / (h * h);
  const double cx = H->nx * h / 2, cy = H->ny * h / 2, cz = H->nz * h / 2;  // extent / 2
  int rc = launch_named(H, "dissipation", [&]() -> int {
    if (H->fp32)
      klaunch(H, k_dissipation<float>, grid, 256, 0, (const float*)H->u, (const float*)H->v, (const float*)H->w, H->p,
              H->has_sphere ? (const float*)H->chi : nullptr, ilog2(H->nx), ilog2(H->ny), H->nz, zc, h, H->cfg.nu,
              hCube, inv2h, invHh, cx, cy, cz, part);
    else
      klaunch(H, k_dissipation<double>, grid, 256, 0, (const double*)H->u, (const double*)H->v, (const double*)H->w,
              H->p, H->has_sphere ? (const double*)H->chi : nullptr, ilog2(H->nx), ilog2(H->ny), H->nz, zc, h,
              H->cfg.nu, hCube, inv2h, invHh, cx, cy, cz, part);
    CKL();
    return CUP_OK;
  });
  if (!rc) rc = sum_columns(H, part, grid, 20, -1, 0);
  if (!rc) rc = read_sums(H, 20);
  if (rc) return rc;
  for (int k = 0; k < 20; ++k) out[k] = H->hsum[k];
  return CUP_OK;
}

int cup_debug_shift(cup_handle* H, const double* f, double* out, int g, int dx, int dy, int dz, int where) {
  REQUIRE_H(H);
  if (!f || !out || !valid_where(where) || (g != 1 && g != 2) || std::abs(dx) > g || std::abs(dy) > g ||
      std::abs(dz) > g)
    return fail(H, CUP_ERR_ARG, "bad shift arguments");
  // stage through the (FP64) rhs and p buffers
  const cudaMemcpyKind in = where == CUP_WHERE_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  const cudaMemcpyKind outk = where == CUP_WHERE_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  CK(cudaMemcpyAsync(H->rhs, f, H->n * sizeof(double), in, H->stream));
  const void* fl[1] = {H->rhs};
  OpShift op{H->p, dx, dy, dz, H->nx, H->ny};
  int rc = g == 1 ? launch_stream<double, 1, 1, 4, 4>(H, "debug_shift", fl, op)
                  : launch_stream<double, 1, 2, 4, 6>(H, "debug_shift", fl, op);
  if (rc) return rc;
  CK(cudaMemcpyAsync(out, H->p, H->n * sizeof(double), outk, H->stream));
  CK(cudaStreamSynchronize(H->stream));
  return check_dev_error(H);
}

// Device address of g_noalloc_partials in the current context, looked up once
// per (device, context) with that device current: host code must not use the
// symbol itself as an address. Keying on the context as well as the ordinal
// makes a new primary context (after cudaDeviceReset) or a context the caller
// made current look the address up again.
using PFN_ctxGetCurrent = CUresult (*)(CUcontext*);
static void* current_context() {
  static PFN_ctxGetCurrent fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_ctxGetCurrent>(f);
  });
  CUcontext c = nullptr;
  if (fn && fn(&c) != CUDA_SUCCESS) c = nullptr;
  return c;
}

static double* noalloc_partials_ptr(int dev, int* err_out) {
  struct Entry {
    int dev;
    void* ctx;
    double* ptr;
  };
  static std::mutex mu;
  static std::vector<Entry> cache;
  void* ctx = current_context();
  std::lock_guard<std::mutex> lk(mu);
  for (const Entry& e : cache)
    if (e.dev == dev && e.ctx == ctx) return e.ptr;
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);
  if (e != cudaSuccess || !p) {
    fprintf(stderr, "cup_max_velocity_noalloc: cudaGetSymbolAddress failed on device %d: %s\n", dev,
            cudaGetErrorString(e));
    *err_out = CUP_ERR_CUDA;
    return nullptr;
  }
  ctx = current_context();  // the lookup may have created the primary context
  for (Entry& en : cache)
    if (en.dev == dev) {
      en.ctx = ctx;
      en.ptr = static_cast<double*>(p);
      return en.ptr;
    }
  cache.push_back({dev, ctx, static_cast<double*>(p)});
  return cache.back().ptr;
}

int cup_max_velocity_noalloc(const double* u, const double* v, const double* w, long long n, const double uinf[3],
                             double* umax_dev, void* stream) {
  if (!u || !v || !w || !uinf || !umax_dev || n <= 0) {
    fprintf(stderr, "cup_max_velocity_noalloc: null pointer or n <= 0\n");
    return CUP_ERR_ARG;
  }
  const long long max_cells = (long long)kNoAllocMaxCtas * kNoAllocChunk;
  if (n > max_cells) {
    fprintf(stderr,
            "cup_max_velocity_noalloc: %lld cells exceed the fixed scratch limit of %lld cells per call "
            "(%d partials of at most %lld cells); split the field or use cup_max_velocity\n",
            n, max_cells, kNoAllocMaxCtas, kNoAllocChunk);
    return CUP_ERR_ARG;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    fprintf(stderr, "cup_max_velocity_noalloc: cudaGetDevice: %s\n", cudaGetErrorString(e));
    return CUP_ERR_CUDA;
  }
  int rc = CUP_OK;
  double* partials = noalloc_partials_ptr(dev, &rc);
  if (!partials) return rc;
  // chunks of a multiple of 1024 cells, at most kNoAllocMaxCtas of them
  long long chunk = (n + kNoAllocMaxCtas - 1) / kNoAllocMaxCtas;
  chunk = std::max(4096LL, (chunk + 1023) / 1024 * 1024);
  const int nblocks = (int)((n + chunk - 1) / chunk);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaGetLastError();  // an earlier launch's error is not this call's
  k_noalloc_max_partial<<<nblocks, 256, 0, st>>>(u, v, w, n, chunk, uinf[0], uinf[1], uinf[2], partials);
  e = cudaGetLastError();
  if (e == cudaSuccess) {
    k_noalloc_max_final<<<1, 256, 0, st>>>(partials, nblocks, umax_dev);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    fprintf(stderr, "cup_max_velocity_noalloc: kernel launch failed: %s\n", cudaGetErrorString(e));
    return CUP_ERR_CUDA;
  }
  return CUP_OK;
}

int cup_dc_history(cup_handle* H, double* out, int n, int* n_checks) {
  REQUIRE_H(H);
  if (!out || n <= 0) return fail(H, CUP_ERR_ARG, "bad history buffer");
  int rc = read_state(H);
  if (rc) return rc;
  const int m = H->fp32 ? std::min(std::min(n, 16), H->hstate->n_solves + 1) : 0;
  for (int i = 0; i < m; ++i) out[i] = H->hstate->res_hist[i];
  if (n_checks) *n_checks = m;
  return CUP_OK;
}

int cup_profile_enable(cup_handle* H, int on) {
  REQUIRE_H(H);
  prof_flush(H);
  H->prof_on = on != 0;
  return CUP_OK;
}

int cup_profile_report(cup_handle* H, char* buf, size_t len, int reset) {
  REQUIRE_H(H);
  prof_flush(H);
  std::string js = "{";
  bool first = true;
  for (const auto& kv : H->prof) {
    // launches that did the pass's work: longer than a quarter of the longest
    // (the later kernels of a converged defect-correction loop exit at entry)
    double total = 0, tmax = 0, work = 0;
    long long nwork = 0;
    for (float d : kv.second) {
      total += d;
      tmax = std::max(tmax, (double)d);
    }
    for (float d : kv.second)
      if (d >= 0.25 * tmax) {
        work += d;
        nwork += 1;
      }
    char item[320];
    snprintf(item, sizeof item,
             "%s\"%s\": {\"count\": %lld, \"ms\": %.6f, \"work_count\": %lld, \"work_ms\": %.6f}",
             first ? "" : ", ", kv.first.c_str(), (long long)kv.second.size(), total, nwork, work);
    js += item;
    first = false;
  }
  js += "}";
  if (reset) H->prof.clear();
  if (!buf || len == 0) return fail(H, CUP_ERR_ARG, "null buffer");
  if (js.size() + 1 > len) return fail(H, CUP_ERR_ARG, "buffer too small (%zu needed)", js.size() + 1);
  memcpy(buf, js.c_str(), js.size() + 1);
  return CUP_OK;
}

int cup_launch_count(const cup_handle* H, long long* n) {
  if (!H || !n) return CUP_ERR_ARG;
  *n = H->launches;
  return CUP_OK;
}

}  // extern "C"
