/*
 * kernels_epilogue.cu -- per-(column, wavelength) quantities derived from a solved block, on
 * the device where the block's arrays already are:
 *   k_intensities     I+ = U + V and I- = U - V on the interior z (auxiliary.f90:80-94,
 *                     calc_intensity: upward and downward intensities);
 *   k_optical_depth   tau(z) = cumulative sum over z from index 1 of kappa rho dz, and the
 *                     first z index where tau reaches a target (tools/ocoutils/ReadOcotillo.py:
 *                     248-293, calculate_optical_depth and find_photosphere), -1 if never.
 *   k_integrated_flux the wavelength-integrated emergent flux per column, the trapezoid rule
 *                     over the wavelength grid as a weighted sum (weights in cm) in increasing
 *                     wavelength index; one thread per column, so a warp reads 32 adjacent
 *                     columns of a [lambda][column] flux plane (coalesced) and the sum order is
 *                     fixed.  No reference counterpart (the reference writes per-lambda planes
 *                     only); the bolometric emergent flux of each column.
 * All are bound by HBM (each array once): lanes run along the fastest index of the layout.
 * Compiled without FMA contraction so that the products and the running sum round as the
 * reference tools' array arithmetic does.
 */
#include <cuda_runtime.h>

#include <algorithm>

#include <cstdint>

#include "oco_internal.h"

namespace oco {

/* I+- element by element in memory order: element i of V meets U's element i + 6 item + 3 (item =
 * i / nz, z fastest) or i + 3 items ([z][col][lambda]).  Tiles of EPI_TILE consecutive elements per
 * block, four per thread in flight; the item index advances with the tile instead of a division
 * per element.  Reference layout, 840 columns x 500 x 200: 3.2 ms with one thread per item (lanes
 * nz elements apart), 0.45 ms so (6.0 TB/s). */
constexpr int EPI_THREADS = 256, EPI_PER = 4, EPI_TILE = EPI_THREADS * EPI_PER;
__global__ void __launch_bounds__(EPI_THREADS) k_intensities(const EpilogueArgs a) {
  const int64_t items = a.ncol * a.nw, n = items * a.nz;
  const int q = EPI_THREADS / a.nz, r = EPI_THREADS % a.nz;
  for (int64_t base = blockIdx.x * (int64_t)EPI_TILE; base < n; base += (int64_t)gridDim.x * EPI_TILE) {
    const int64_t i0 = base + threadIdx.x;
    int64_t item = 0;
    int z = 0;
    if (a.layout == 0) {
      item = i0 / a.nz;
      z = (int)(i0 - item * a.nz);
    }
    double u[EPI_PER], v[EPI_PER];
#pragma unroll
    for (int k = 0; k < EPI_PER; k++) {
      const int64_t i = i0 + k * EPI_THREADS;
      if (i < n) {
        u[k] = __ldcs(&a.U[i + (a.layout == 0 ? 6 * item + 3 : 3 * items)]);
        v[k] = __ldcs(&a.V[i]);
      }
      item += q;
      z += r;
      if (z >= a.nz) {
        z -= a.nz;
        item++;
      }
    }
#pragma unroll
    for (int k = 0; k < EPI_PER; k++) {
      const int64_t i = i0 + k * EPI_THREADS;
      if (i >= n) break;
      if (a.Ip) __stcs(&a.Ip[i], u[k] + v[k]);
      if (a.Im) __stcs(&a.Im[i], u[k] - v[k]);
    }
  }
}

/* tau, [z][col][lambda]: one thread per item in memory order, the terms of TAU_Z levels loaded
 * ahead of the running sum. */
constexpr int TAU_Z = 16;
__global__ void __launch_bounds__(128) k_optical_depth_lambda(const EpilogueArgs a) {
  const int64_t items = a.ncol * a.nw;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= items) return;
  const int64_t col = t / a.nw, iw = t - col * a.nw;
  const double *rho = a.rho + col * a.nz, *K = a.K + t;
  double tau = 0.0;
  int photo = -1;
  auto level = [&](int z, double term) {
    tau = tau + term;
    if (a.tau) __stcs(&a.tau[t + z * items], tau);
    if (photo < 0 && tau >= a.target) photo = z;
  };
  int z = 0;
  for (; z + TAU_Z <= a.nz; z += TAU_Z) {
    double x[TAU_Z];
#pragma unroll
    for (int k = 0; k < TAU_Z; k++) x[k] = (__ldcs(&K[(z + k) * items]) * __ldg(&rho[z + k])) * a.dz;
#pragma unroll
    for (int k = 0; k < TAU_Z; k++) level(z + k, x[k]);
  }
  for (; z < a.nz; z++) level(z, (K[z * items] * rho[z]) * a.dz);
  if (a.photo) a.photo[iw * a.ncol + col] = photo;
}

/* tau, z fastest: a warp takes 32 items in tiles of 32 levels.  The terms kappa rho dz are formed
 * with lanes along z (256-byte rows) and pass through shared memory to the lane that sums the
 * item (in order, as the definition's running sum), whose sums go back the same way.  1.4 ms with
 * one thread per item walking its row, 0.31 ms so (840 columns x 500 x 200; 4.3 TB/s, the second
 * wave of warps three quarters full).  Tiles of 16 levels, which hold every warp at once at 56
 * registers, spill and take 0.46 ms. */
constexpr int TAU_WARPS = 4;
__global__ void __launch_bounds__(32 * TAU_WARPS) k_optical_depth_z(const EpilogueArgs a) {
  __shared__ double s_tile[TAU_WARPS][32][33];
  const int lane = threadIdx.x & 31;
  double(*tile)[33] = s_tile[threadIdx.x >> 5];
  const int64_t items = a.ncol * a.nw;
  const int64_t item0 = (blockIdx.x * (int64_t)TAU_WARPS + (threadIdx.x >> 5)) * 32;
  if (item0 >= items) return;
  const int rows = (int)min((int64_t)32, items - item0);
  const int64_t col0 = item0 % a.ncol;
  double tau = 0.0;
  int photo = -1;
  for (int z0 = 0; z0 < a.nz; z0 += 32) {
    const int z = z0 + lane, nzt = min(32, a.nz - z0);
    const bool in = z < a.nz;
    for (int r0 = 0; r0 < rows; r0 += 16) {
      double k[16], d[16];
#pragma unroll
      for (int r = 0; r < 16; r++) {
        int64_t col = col0 + r0 + r; /* past the last column: the next wavelength's first */
        if (col >= a.ncol) col = a.ncol >= 32 ? col - a.ncol : (int)col % (int)a.ncol;
        const bool on = in && r0 + r < rows;
        k[r] = on ? __ldcs(&a.K[(item0 + r0 + r) * a.nz + z]) : 0.0;
        d[r] = on ? __ldg(&a.rho[col * a.nz + z]) : 0.0;
      }
#pragma unroll
      for (int r = 0; r < 16; r++) tile[r0 + r][lane] = (k[r] * d[r]) * a.dz;
    }
    __syncwarp();
    if (nzt == 32) {
#pragma unroll
      for (int j = 0; j < 32; j++) {
        tau = tau + tile[lane][j];
        tile[lane][j] = tau;
        if (photo < 0 && tau >= a.target) photo = z0 + j;
      }
    } else {
      for (int j = 0; j < nzt; j++) {
        tau = tau + tile[lane][j];
        tile[lane][j] = tau;
        if (photo < 0 && tau >= a.target) photo = z0 + j;
      }
    }
    __syncwarp();
    if (a.tau && in)
      for (int r = 0; r < rows; r++) __stcs(&a.tau[(item0 + r) * a.nz + z], tile[r][lane]);
    __syncwarp();
  }
  if (a.photo && lane < rows) a.photo[item0 + lane] = photo;
}

/* One warp-wide block per 32 columns, FLUX_W products loaded ahead of the running sum (840 columns
 * x 200 wavelengths: 56 us with 256-thread blocks and one load at a time, 14 us so). */
constexpr int FLUX_W = 32;
__global__ void __launch_bounds__(32) k_integrated_flux(const double *__restrict__ V, const double *__restrict__ w,
                                                        int64_t ncol, int nw, int64_t ld_col, double *__restrict__ F) {
  for (int64_t col = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; col < ncol;
       col += (int64_t)gridDim.x * blockDim.x) {
    double f = 0.0;
    int iw = 0;
    for (; iw + FLUX_W <= nw; iw += FLUX_W) {
      double x[FLUX_W];
#pragma unroll
      for (int k = 0; k < FLUX_W; k++) x[k] = __ldg(&w[iw + k]) * V[(int64_t)(iw + k) * ld_col + col];
#pragma unroll
      for (int k = 0; k < FLUX_W; k++) f = f + x[k];
    }
    for (; iw < nw; iw++) f = f + __ldg(&w[iw]) * V[(int64_t)iw * ld_col + col];
    F[col] = f;
  }
}

cudaError_t launch_integrated_flux(const double *V, const double *w, int64_t ncol, int nw, int64_t ld_col, double *F,
                                   int num_sms, cudaStream_t s) {
  const int64_t blocks = std::min<int64_t>((ncol + 31) / 32, (int64_t)num_sms * 32);
  k_integrated_flux<<<(unsigned)blocks, 32, 0, s>>>(V, w, ncol, nw, ld_col, F);
  return cudaGetLastError();
}

cudaError_t launch_intensities(const EpilogueArgs &a, int num_sms, cudaStream_t s) {
  const int64_t tiles = (a.ncol * a.nw * a.nz + EPI_TILE - 1) / EPI_TILE;
  k_intensities<<<(unsigned)std::min<int64_t>(tiles, (int64_t)num_sms * 8), EPI_THREADS, 0, s>>>(a);
  return cudaGetLastError();
}

/* The grid covers the items (not a fixed number of blocks walking them): at 2^31 blocks' limit
 * that is 2^38 items, beyond any array that fits the device. */
cudaError_t launch_optical_depth(const EpilogueArgs &a, cudaStream_t s) {
  const int64_t items = a.ncol * a.nw;
  const int64_t blocks = (items + 127) / 128; /* both kernels take 128 items per block */
  if (blocks > INT32_MAX) return cudaErrorInvalidValue;
  if (a.layout == 0)
    k_optical_depth_z<<<(unsigned)blocks, 32 * TAU_WARPS, 0, s>>>(a);
  else
    k_optical_depth_lambda<<<(unsigned)blocks, 128, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace oco
