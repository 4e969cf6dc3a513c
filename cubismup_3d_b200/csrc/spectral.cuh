// Spectral analysis and forcing (source/spectralOperators/SpectralManipFFTW.cpp:25-193,
// SpectralForcing.cpp:23-86) on the separable Hartley coefficients (dht.cuh)
// instead of FFTW's r2c spectrum. The separable transform mixes the DFT
// coefficients of the 8 modes (+-kx, +-ky, +-kz) orthogonally, and every
// quantity the reference takes per mode is a function of |k| (the shell of the
// spectrum, 1/|k|, the 0 < k^2 <= 4 forcing band), so sums over modes are the
// same: E = 1/2 (Hu^2 + Hv^2 + Hw^2) per separable mode is the reference's
// mult/2 |U|^2 summed over the conjugate-symmetric full spectrum. The vorticity
// sum is taken in physical space, where Parseval puts it: the reference's eps
// is nu times the mean of |curl_c u|^2 (central differences).
//
// The z pass holds all coefficients of its columns, so it also takes the mode
// sums there and writes nothing back but the few coefficients of the forcing
// band; the force of a small band is then summed mode by mode in one pass over
// the velocity instead of nine inverse passes.
#pragma once

#include "common.cuh"
#include "dht.cuh"
#include "ops.cuh"

namespace cup {

// Wavenumbers of a mode index i of n (negative in the upper half).
__device__ __forceinline__ int mode_of(int i, int n) { return i <= n / 2 ? i : i - n; }

struct ModeParams {
  int nx, ny, nz;
  double wf[3];        // 2 pi / L per axis
  int nyquist, nbin;   // of the longest axis
  double nyq_scaling;  // (nyquist - 1) / nyquist
  // forcing band 0 < k^2 <= 4: modes |i| <= band[d] per axis, their coefficients
  // to coef[c][kz][ky][kx] (2 band[d] + 1 each, zero outside the band); nullptr: none
  int band[3];
  double* coef;
};

// z transform of the three components with the mode sums. A CTA of 128 threads
// walks tiles of 16 x-columns at one y; per-CTA partials: [tke, lIntegral,
// tkeFiltered, nbin spectrum values] (bin floor(sqrt(kind) nyq_scaling) for kind
// = ii^2 + jj^2 + kk^2 < nyquist^2, summed with shared-memory atomics; z and
// nz - z share a bin and go in together).
template <int M, bool T8>
__global__ void __launch_bounds__(128) k_dht_z_modes(const __grid_constant__ CUtensorMap map /* dims nx, ny, 3 nz */,
                                                    const ModeParams mp, const double2* tw_g, int ntiles,
                                                    double* partials, int* err) {
  pdl_entry();
  constexpr int N = 2 * M, W = 16, TPL = T8 ? 8 : M / 8, TL = FFTPlan<M>::table_len();
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char* smem_raw = smem_align128(smem_dyn);
  double* tile = reinterpret_cast<double*>(smem_raw);  // [3][N][W]
  double2* tw = reinterpret_cast<double2*>(tile + 3 * N * W);
  double* bins = reinterpret_cast<double*>(tw + TL);
  uint64_t* bar = reinterpret_cast<uint64_t*>(bins + mp.nbin);
  __shared__ double scratch[3 * 32];
  const int tid = threadIdx.x;
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
  }
  load_table(tw, tw_g, TL);
  for (int b = tid; b < mp.nbin; b += blockDim.x) bins[b] = 0.0;
  __syncthreads();
  const int l = tid % W, t = tid / W;
  const bool active = t < TPL;
  const int ntx = mp.nx / W;
  const long long nyq2 = (long long)mp.nyquist * mp.nyquist;
  double acc[3] = {0, 0, 0};
  uint32_t ph = 0;
  bool ok = true;
  for (int i = blockIdx.x; i < ntiles; i += gridDim.x, ph ^= 1) {
    const int x0 = (i % ntx) * W, y = i / ntx;
    if (tid == 0) {
      mbar_arrive_expect_tx(bar, (uint32_t)(3 * N * W * sizeof(double)));
      for (int c = 0; c < 3; ++c) tma_load_3d(tile + c * N * W, &map, x0, y, c * N, bar);
    }
    ok = __syncthreads_and(mbar_wait(bar, ph, err));
    if (!ok) break;
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      ColLines<double> A{tile + c * N * W, W};
      if constexpr (T8) dht128_t8<double>(A, tw, l, t, active, NoScale());
      else dht_lines<M, false, double>(A, A, tw, l, t, active);
    }
    // Mode sums: a thread takes 8 of the 16 columns of one k (and of N - k; with
    // k = 0 the mode N/2). Along x the shell changes slowly, so a thread sums a run
    // of equal shells before it adds to the block's (a shared-memory FP64 atomic
    // is a retry loop, and with one column per lane most lanes of a warp wanted
    // the same shell). Lanes start at different columns, on different banks. 6
    // forced FP32 steps on 128^3 2523 -> 2356 us, the FP64 diagnostics of a
    // 256x128x128 flow 401 -> 396 us.
    const int jj = mode_of(y, mp.ny);
    const double ky = jj * mp.wf[1];
    for (int q = tid; q < N; q += blockDim.x) {
      const int k = q >> 1, l0 = (q & 1) * 8, k1 = k ? N - k : N / 2;
      int run = -1;
      double sum = 0.0;
      auto mode = [&](double E, int ii, int kk) {
        const double kx = ii * mp.wf[0], kz = kk * mp.wf[2];
        const double k2 = kx * kx + ky * ky + kz * kz;
        acc[0] += E;
        acc[1] += k2 > 0 ? E / sqrt(k2) : 0.0;
        const bool in = k2 > 0 && k2 <= 4;
        if (in) acc[2] += E;
        const long long kind = (long long)ii * ii + (long long)jj * jj + (long long)kk * kk;
        if (kind < nyq2) {
          const int bin = (int)floor(sqrt((double)kind) * mp.nyq_scaling);
          if (bin != run) {
            if (run >= 0) atomicAdd(&bins[run], sum);
            run = bin < mp.nbin ? bin : -1;
            sum = 0.0;
          }
          sum += E;
        }
        return in;
      };
#pragma unroll 1
      for (int e = 0; e < 8; ++e) {
        const int c0 = l0 + ((e + k) & 7), ii = mode_of(x0 + c0, mp.nx);
        const double* a = tile + k * W + c0;
        const double* b = tile + k1 * W + c0;
        const double Ea = 0.5 * (a[0] * a[0] + a[N * W] * a[N * W] + a[2 * N * W] * a[2 * N * W]);
        const double Eb = 0.5 * (b[0] * b[0] + b[N * W] * b[N * W] + b[2 * N * W] * b[2 * N * W]);
        const bool in = mode(k ? Ea + Eb : Ea, ii, k);
        if (!k) mode(Eb, ii, N / 2);
        if (mp.coef && abs(ii) <= mp.band[0] && abs(jj) <= mp.band[1]) {
          const int n0 = 2 * mp.band[0] + 1, n1 = 2 * mp.band[1] + 1, n2 = 2 * mp.band[2] + 1;
          for (int c = 0; c < 3; ++c) {
            double* o = mp.coef + ((size_t)c * n2 * n1 + jj + mp.band[1]) * n0 + ii + mp.band[0];
            if (k <= mp.band[2]) o[(size_t)(mp.band[2] + k) * n1 * n0] = in ? a[c * N * W] : 0.0;
            if (k && k <= mp.band[2]) o[(size_t)(mp.band[2] - k) * n1 * n0] = in ? b[c * N * W] : 0.0;
          }
        }
      }
      if (run >= 0) atomicAdd(&bins[run], sum);
    }
    fence_proxy_async_smem();
    __syncthreads();
  }
  // after a timed-out wait: bounded drain of the tile's loads, which write to this block's shared memory
  if (!ok && tid == 0) mbar_wait(bar, ph, nullptr);
  block_reduce<3, false>(acc, scratch);
  const int stride = 3 + mp.nbin;
  if (tid == 0)
    for (int k = 0; k < 3; ++k) partials[(size_t)stride * blockIdx.x + k] = acc[k];
  for (int b = tid; b < mp.nbin; b += blockDim.x) partials[(size_t)stride * blockIdx.x + 3 + b] = bins[b];
}

// Every mode outside the forcing band zeroed in place, for a band too wide to
// force mode by mode.
__global__ void k_spectral_filter(double* hu, double* hv, double* hw, int lnx, int lny, int nz, double wfx, double wfy,
                                  double wfz) {
  pdl_entry();
  const int nx = 1 << lnx, ny = 1 << lny, n = nx * ny * nz;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int x = i & (nx - 1), y = (i >> lnx) & (ny - 1), z = i >> (lnx + lny);
    const double kx = mode_of(x, nx) * wfx, ky = mode_of(y, ny) * wfy, kz = mode_of(z, nz) * wfz;
    const double k2 = kx * kx + ky * ky + kz * kz;
    if (!(k2 > 0 && k2 <= 4)) hu[i] = hv[i] = hw[i] = 0.0;
  }
}

// f += factor * g (g FP64), rounded once to the storage type.
template <typename T>
__global__ void k_add_scaled(T* f, const double* g, double factor, size_t n) {
  pdl_entry();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    f[i] = (T)((double)f[i] + factor * g[i]);
}

// cas(2 pi k i / n) = cos + sin, the Hartley kernel.
__device__ __forceinline__ double cas(int k, int i, int n) {
  int m = (k * i) % n;
  if (m < 0) m += n;
  double s, c;
  sincospi(2.0 * m / n, &s, &c);
  return c + s;
}

constexpr int kBandMax = 4;                   // modes per axis and side that are forced one by one
constexpr int kBandN = 2 * kBandMax + 1;

// u += factor * (inverse Hartley transform of the band coefficients), mode by
// mode: block (z, part of the rows) sums over kz once, every row over ky, every
// cell over kx. Dynamic shared memory: rows_per_block * 4 * (most modes per axis) doubles.
template <typename T>
__global__ void __launch_bounds__(256) k_force_band(T* u, T* v, T* w, const ModeParams mp, double factor, int rows_per_block) {
  pdl_entry();
  __shared__ double A[3][kBandN * kBandN];  // [c][ky][kx] at this z
  __shared__ double cz[kBandN];
  extern __shared__ double B[];             // [row][3][kx], then cas of (row, ky)
  const int n0 = 2 * mp.band[0] + 1, n1 = 2 * mp.band[1] + 1, n2 = 2 * mp.band[2] + 1;
  double* cy = B + rows_per_block * 3 * n0;
  const int parts = mp.ny / rows_per_block;
  const int z = blockIdx.x / parts, y0 = (blockIdx.x % parts) * rows_per_block;
  const int tid = threadIdx.x;
  const int x = tid & (mp.nx - 1);
  double cx[kBandN];
#pragma unroll
  for (int k = 0; k < kBandN; ++k) cx[k] = k < n0 ? cas(k - mp.band[0], x, mp.nx) : 0.0;
  for (int i = tid; i < n2; i += blockDim.x) cz[i] = cas(i - mp.band[2], z, mp.nz);
  for (int i = tid; i < rows_per_block * n1; i += blockDim.x) cy[i] = cas(i % n1 - mp.band[1], y0 + i / n1, mp.ny);
  __syncthreads();
  for (int i = tid; i < 3 * n1 * n0; i += blockDim.x) {
    const int c = i / (n1 * n0), r = i - c * n1 * n0;
    double s = 0.0;
    for (int k = 0; k < n2; ++k) s += mp.coef[((size_t)c * n2 + k) * n1 * n0 + r] * cz[k];
    A[c][r] = s;
  }
  __syncthreads();
  for (int i = tid; i < rows_per_block * 3 * n0; i += blockDim.x) {
    const int row = i / (3 * n0), r = i - row * 3 * n0, c = r / n0, kx = r - c * n0;
    double s = 0.0;
    for (int k = 0; k < n1; ++k) s += A[c][k * n0 + kx] * cy[row * n1 + k];
    B[i] = s;
  }
  __syncthreads();
  T* f[3] = {u, v, w};
  for (int row = tid / mp.nx; row < rows_per_block; row += blockDim.x / mp.nx) {
    const size_t o = gidx(x, y0 + row, z, mp.nx, mp.ny);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double g = 0.0;
#pragma unroll
      for (int k = 0; k < kBandN; ++k)
        if (k < n0) g += B[(row * 3 + c) * n0 + k] * cx[k];
      f[c][o] = (T)((double)f[c][o] + factor * g);
    }
  }
}

// ---- diagnostics in physical space -----------------------------------------
// A thread marches down z with the values of the planes below, at and above its
// cell in registers (one load per field and plane instead of three), x and y
// neighbours by load. Blocks of 256 threads over (x, y), zc planes each. (With
// one cell per grid-stride step and 64-bit index divisions ComputeDissipation
// took 145 us, the vorticity sum 57 and the divergence norms 56 at 256x128x128
// FP64.)
struct MarchPos {
  int x, y, z0;
  size_t row, rN, rS;  // offset of the row in its plane, and of the rows y +- 1
  int xE, xW;
};
__device__ __forceinline__ MarchPos march_pos(int lnx, int lny, int zc) {
  MarchPos p;
  const int nx = 1 << lnx, ny = 1 << lny;
  const int per_plane = (nx * ny) >> 8;  // blocks over (x, y); nx ny is a multiple of 256
  const int i = (blockIdx.x % per_plane) * 256 + threadIdx.x;
  p.z0 = (blockIdx.x / per_plane) * zc;
  p.x = i & (nx - 1);
  p.y = i >> lnx;
  p.row = (size_t)p.y * nx;
  p.rN = (size_t)((p.y + 1) & (ny - 1)) * nx;
  p.rS = (size_t)((p.y - 1) & (ny - 1)) * nx;
  p.xE = (p.x + 1) & (nx - 1);
  p.xW = (p.x - 1) & (nx - 1);
  return p;
}

// ComputeDissipation (source/operators/ComputeDissipation.cpp:38-116): per
// cell, vorticity, pressure power -(1-chi) h^3 grad p . u, viscous power
// (1-chi) h^3 nu (u . lap u + 2 D:D), and the linear / angular invariants
// about the domain centre; per-CTA FP64 partials of the 20 sums in the order
// of the reference's reduction (:132-152). hCube = pow(h, 3), inv2h = 1/(2h),
// invHh = 1/h^2 and the centre come from the host as the reference computes
// them.
template <typename T>
__global__ void __launch_bounds__(256) k_dissipation(const T* __restrict__ u, const T* __restrict__ v,
                                                    const T* __restrict__ w, const double* __restrict__ p,
                                                    const T* __restrict__ chi, int lnx, int lny, int nz, int zc,
                                                    double h, double nu, double hCube, double inv2h, double invHh,
                                                    double cx, double cy, double cz,
                                                    double* partials /* [gridDim.x][20] */) {
  pdl_entry();
  __shared__ double scratch[20 * 32];
  double R[20];
#pragma unroll
  for (int k = 0; k < 20; ++k) R[k] = 0.0;
  const size_t plane = (size_t)1 << (lnx + lny);
  const MarchPos m = march_pos(lnx, lny, zc);
  const size_t at = m.row + m.x;
  auto pl = [&](int z) { return (size_t)(z < 0 ? z + nz : (z >= nz ? z - nz : z)) * plane; };
  size_t o = pl(m.z0 - 1) + at;
  double uF = u[o], vF = v[o], wF = w[o], pF = p[o];
  o = pl(m.z0) + at;
  double uc = u[o], vc = v[o], wc = w[o], pc = p[o];
  const double PX = (m.x + 0.5) * h - cx, PY = (m.y + 0.5) * h - cy;
#pragma unroll 1
  for (int z = m.z0; z < m.z0 + zc; ++z) {
    const size_t b = pl(z), on = pl(z + 1) + at;
    const double uB = u[on], vB = v[on], wB = w[on], pB = p[on];
    const size_t oE = b + m.row + m.xE, oW = b + m.row + m.xW, oN = b + m.rN + m.x, oS = b + m.rS + m.x;
    const double X = chi ? (double)chi[b + at] : 0.0;
    const double PZ = (z + 0.5) * h - cz;
    const double uE = u[oE], uW = u[oW], uN = u[oN], uS = u[oS];
    const double vE = v[oE], vW = v[oW], vN = v[oN], vS = v[oS];
    const double wE = w[oE], wW = w[oW], wN = w[oN], wS = w[oS];
    const double WX = inv2h * ((wN - wS) - (vB - vF));
    const double WY = inv2h * ((uB - uF) - (wE - wW));
    const double WZ = inv2h * ((vE - vW) - (uN - uS));
    const double dPdx = inv2h * (p[oE] - p[oW]);
    const double dPdy = inv2h * (p[oN] - p[oS]);
    const double dPdz = inv2h * (pB - pF);
    R[15] -= (1 - X) * hCube * (dPdx * uc + dPdy * vc + dPdz * wc);
    const double lapU = invHh * (uE + uW + uN + uS + uB + uF - 6 * uc);
    const double lapV = invHh * (vE + vW + vN + vS + vB + vF - 6 * vc);
    const double lapW = invHh * (wE + wW + wN + wS + wB + wF - 6 * wc);
    const double V1 = lapU * uc + lapV * vc + lapW * wc;
    const double D11 = inv2h * (uE - uW);
    const double D22 = inv2h * (vN - vS);
    const double D33 = inv2h * (wB - wF);
    const double D12 = inv2h * (uN - uS + vE - vW) / 2;
    const double D13 = inv2h * (uB - uF + wE - wW) / 2;
    const double D23 = inv2h * (wN - wS + vB - vF) / 2;
    const double V2 = D11 * D11 + D22 * D22 + D33 * D33 + 2 * (D12 * D12 + D13 * D13 + D23 * D23);
    R[16] += (1 - X) * hCube * nu * (V1 + 2 * V2);
    R[0] += hCube * WX;
    R[1] += hCube * WY;
    R[2] += hCube * WZ;
    R[3] += hCube / 2 * (PY * WZ - PZ * WY);
    R[4] += hCube / 2 * (PZ * WX - PX * WZ);
    R[5] += hCube / 2 * (PX * WY - PY * WX);
    R[6] += hCube * uc;
    R[7] += hCube * vc;
    R[8] += hCube * wc;
    R[9] += hCube / 3 * (PX * (PY * WY + PZ * WZ) - WX * (PY * PY + PZ * PZ));
    R[10] += hCube / 3 * (PY * (PX * WX + PZ * WZ) - WY * (PX * PX + PZ * PZ));
    R[11] += hCube / 3 * (PZ * (PX * WX + PY * WY) - WZ * (PX * PX + PY * PY));
    R[12] += hCube * (PY * wc - PZ * vc);
    R[13] += hCube * (PZ * uc - PX * wc);
    R[14] += hCube * (PX * vc - PY * uc);
    R[17] += hCube * (WX * uc + WY * vc + WZ * wc);
    R[18] += hCube * (uc * uc + vc * vc + wc * wc) / 2;
    R[19] += sqrt(WX * WX + WY * WY + WZ * WZ);
    uF = uc, vF = vc, wF = wc, pF = pc;
    uc = uB, vc = vB, wc = wB, pc = pB;
  }
  block_reduce<20, false>(R, scratch);
  if (threadIdx.x == 0)
    for (int k = 0; k < 20; ++k) partials[20 * blockIdx.x + k] = R[k];
}

// Per-CTA partial sums of |curl_c u|^2 (central differences / 2h).
template <typename T>
__global__ void __launch_bounds__(256) k_vorticity2(const T* __restrict__ u, const T* __restrict__ v,
                                                   const T* __restrict__ w, int lnx, int lny, int nz, int zc,
                                                   double inv2h, double* partials) {
  pdl_entry();
  __shared__ double scratch[32];
  double acc[1] = {0.0};
  const size_t plane = (size_t)1 << (lnx + lny);
  const MarchPos m = march_pos(lnx, lny, zc);
  const size_t at = m.row + m.x;
  auto pl = [&](int z) { return (size_t)(z < 0 ? z + nz : (z >= nz ? z - nz : z)) * plane; };
  size_t o = pl(m.z0 - 1) + at;
  double uF = u[o], vF = v[o];
  o = pl(m.z0) + at;
  double uc = u[o], vc = v[o];
#pragma unroll 2
  for (int z = m.z0; z < m.z0 + zc; ++z) {
    const size_t b = pl(z), on = pl(z + 1) + at;
    const double uB = u[on], vB = v[on];
    const size_t oE = b + m.row + m.xE, oW = b + m.row + m.xW, oN = b + m.rN + m.x, oS = b + m.rS + m.x;
    const double WX = inv2h * (((double)w[oN] - (double)w[oS]) - (vB - vF));
    const double WY = inv2h * ((uB - uF) - ((double)w[oE] - (double)w[oW]));
    const double WZ = inv2h * (((double)v[oE] - (double)v[oW]) - ((double)u[oN] - (double)u[oS]));
    acc[0] += WX * WX + WY * WY + WZ * WZ;
    uF = uc, vF = vc;
    uc = uB, vc = vB;
  }
  block_reduce<1, false>(acc, scratch);
  if (threadIdx.x == 0) partials[blockIdx.x] = acc[0];
}

// Per-CTA partials of the kinetic energy and the central-divergence norms (FP64): sum |u|^2/2, sum div^2, max |div|.
template <typename T>
__global__ void __launch_bounds__(256) k_diag(const T* __restrict__ u, const T* __restrict__ v, const T* __restrict__ w,
                                             int lnx, int lny, int nz, int zc, double inv2h, double* partials) {
  pdl_entry();
  __shared__ double scratch[3 * 32];
  double s[2] = {0, 0};
  double mx[1] = {0};
  const size_t plane = (size_t)1 << (lnx + lny);
  const MarchPos m = march_pos(lnx, lny, zc);
  const size_t at = m.row + m.x;
  auto pl = [&](int z) { return (size_t)(z < 0 ? z + nz : (z >= nz ? z - nz : z)) * plane; };
  double wF = w[pl(m.z0 - 1) + at], wc = w[pl(m.z0) + at];
#pragma unroll 2
  for (int z = m.z0; z < m.z0 + zc; ++z) {
    const size_t b = pl(z);
    const double wB = w[pl(z + 1) + at];
    const double uu = u[b + at], vv = v[b + at];
    s[0] += 0.5 * (uu * uu + vv * vv + wc * wc);
    const double div = inv2h * ((double)u[b + m.row + m.xE] - (double)u[b + m.row + m.xW] + (double)v[b + m.rN + m.x] -
                                (double)v[b + m.rS + m.x] + wB - wF);
    s[1] += div * div;
    mx[0] = fmax(mx[0], fabs(div));
    wF = wc;
    wc = wB;
  }
  block_reduce<2, false>(s, scratch);
  block_reduce<1, true>(mx, scratch + 2 * 32);
  if (threadIdx.x == 0) {
    partials[3 * blockIdx.x + 0] = s[0];
    partials[3 * blockIdx.x + 1] = s[1];
    partials[3 * blockIdx.x + 2] = mx[0];
  }
}

// out[j] = the sum (j != max_col) or maximum over np partials of column j; one block per column.
__global__ void __launch_bounds__(256) k_reduce_columns(const double* p, int np, int stride, int max_col, double* out) {
  pdl_entry();
  __shared__ double scratch[32];
  const int j = blockIdx.x;
  double a[1] = {0.0};
  if (j == max_col) {
    for (int i = threadIdx.x; i < np; i += blockDim.x) a[0] = fmax(a[0], p[(size_t)stride * i + j]);
    block_reduce<1, true>(a, scratch);
  } else {
    for (int i = threadIdx.x; i < np; i += blockDim.x) a[0] += p[(size_t)stride * i + j];
    block_reduce<1, false>(a, scratch);
  }
  if (threadIdx.x == 0) out[j] = a[0];
}

}  // namespace cup
