// PR_MU spectral function (src/hawaii.c:3148-3978): the spectrum of each trajectory's
// dipole, weighted by its initial radial velocity.
//
// The reference integrates a trajectory from R0 inward, keeps the lab dipole at
// t = (k+1) dt for k = 0..N-1 (zero after it leaves the R0 sphere), apodizes each
// component with Connes' window, takes its real FFT (gsl_fft_real_radix2_transform)
// and adds SF_COEFF pR/mu sum_c |F_c(i)|^2 into the spectrum for the first L
// frequencies (hawaii.c:3812-3825).
//
// GPU mapping, per chunk of trajectories whose dipole series are in HBM:
//   1. prmu_weight: w = SF_COEFF pR/mu x spin weight of an included trajectory, else 0;
//   2. the spectra.  For a real series the FFT magnitudes are even, so of the complex series
//      X + iY, (|S_k|^2 + |S_{N-k}|^2) / 2 is |X_k|^2 + |Y_k|^2: two trajectories are three
//      complex series (x0 + i y0, x1 + i y1, z0 + i z1), each sqrt(w) times the Connes window.
//      256 <= N <= 4096: prmu_spectrum, a persistent block that takes pairs of trajectories
//      from the series through the transform in its shared memory to its own sums of the
//      first L terms; the series are read once and nothing else but the sums is written.
//      Other N (a series below one warp's tile, or above a block's): the transform by passes
//      (hh_fft.cuh) and prmu_accum over its output;
//   3. prmu_reduce: the blocks' sums in a fixed order.
// 4,096 CO2-Ar trajectories, N = 4096, 238 frequencies: pack 0.17, twelve radix-2 passes 2.1
// and one thread per frequency over all series 2.6 ms before -> 0.37 ms together.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "hh_consts.h"
#include "hh_fft.cuh"
#include "hh_traj.cuh"

namespace hh {

struct PrmuPackArgs {
  const void *series;         // [traj][slot][4] in the surface precision; slot k = sample at k dt
  const int *len;             // [item]: samples stored (forward items 2 t)
  const int *status;          // [item]: end status | 16 when the branch left the R0 sphere
  const double *qp;           // [traj][QP]: the drawn phase points of the chunk (pR at 5)
  int QP;
  long long n_traj;
  int N, stride;              // samples per trajectory; series slots per trajectory
  int allow_trunc;
  double coeff;               // SF_COEFF / mu
  double *w;                  // [traj]: sqrt of the trajectory's weight
  unsigned long long *counted;
  // spin weights of a LINEAR_MOLECULE_REQ_HALFINTEGER monomer (src/hawaii.c:3575-3594):
  // req_mode 2 and a positive weight select even_w / odd_w by the parity of
  // round(j_ini - 1.5), j_ini the requantized initial |j|; otherwise weight 1
  int req_mode;
  double even_w, odd_w;
};

// the trajectory weight of PR_MU from the drawn linear-monomer phase point
// (phi, p_phi, theta, p_theta at qp[6..9]): j_monomer (src/hawaii.c:398-431), then
// the requantized length
__device__ __forceinline__ double prmu_spin_weight(const PrmuPackArgs &a, const double *qp) {
  if (a.req_mode != 2 || !(a.even_w > 0.0 || a.odd_w > 0.0)) return 1.0;
  const double phi = qp[6], pphi = qp[7], th = qp[8], pth = qp[9];
  const double ct = cos(th) / sin(th);
  const double j0 = -pth * sin(phi) - pphi * cos(phi) * ct, j1 = pth * cos(phi) - pphi * sin(phi) * ct;
  const double jl = sqrt(j0 * j0 + j1 * j1 + pphi * pphi);
  const double jini = req_closest(2, jl);
  const long long j_int = llround(jini - 1.5);
  return (j_int % 2 == 0) ? a.even_w : a.odd_w;
}

__global__ void __launch_bounds__(256) prmu_weight_kernel(PrmuPackArgs a) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= a.n_traj) return;
  const int st = a.status[2 * t];
  const bool include = (st & 15) == HH_ST_OK && ((st & 16) || a.allow_trunc);
  const double pr_mu = -a.qp[t * a.QP + 5];
  a.w[t] = include ? sqrt(a.coeff * pr_mu * prmu_spin_weight(a, a.qp + t * a.QP)) : 0.0;
  if (include) atomicAdd(a.counted, 1ull);
}

// element j of the pair's series: part 0 and 1 the x + iy of its first and second trajectory,
// part 2 their z; connes_apodization (src/hawaii.c:5401-5410) with tmax = N dt
template <typename PHYS> struct PrmuPack {
  PrmuPackArgs a;
  __device__ double2 operator()(long long sr, long long j) const {
    const long long u = sr / 3;
    return load(u, int(sr - 3 * u), int(j));
  }
  __device__ __forceinline__ double2 load(long long u, int part, int j) const {
    double2 d = make_double2(0.0, 0.0);
    const long long t0 = 2 * u + (part == 1), t1 = 2 * u + 1;
    const double f = connes(double(j), 1.0 / double(a.N));
    if (has(t0, j)) {
      const PHYS *v = at(t0, j);
      const double s = a.w[t0] * f;
      d.x = s * double(v[part == 2 ? 2 : 0]);
      if (part < 2) d.y = s * double(v[1]);
    }
    if (part == 2 && has(t1, j)) d.y = a.w[t1] * f * double(at(t1, j)[2]);
    return d;
  }
  __device__ __forceinline__ bool has(long long t, int j) const {
    return t < a.n_traj && a.w[t] != 0.0 && j + 1 <= a.len[2 * t];
  }
  __device__ __forceinline__ const PHYS *at(long long t, int j) const {
    return static_cast<const PHYS *>(a.series) + ((size_t)t * a.stride + j + 1) * 4;
  }
};

__device__ __forceinline__ double prmu_term(double2 u, double2 v) {
  return 0.5 * (u.x * u.x + u.y * u.y + v.x * v.x + v.y * v.y);
}

// N = 2^logN in [256, 4096], N / 8 threads; partial[block][L]
template <typename PHYS>
__global__ void __launch_bounds__(1 << (FFT_MAX_LOG_TILE - 3)) prmu_spectrum_kernel(PrmuPack<PHYS> in, int logN, int L,
                                                                                    double *partial) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2 *sm = reinterpret_cast<double2 *>(smem_raw);
  double *acc = reinterpret_cast<double *>(sm + fft_pad(1 << logN));
  const int tid = threadIdx.x, threads = 1 << (logN - 3), N = 1 << logN;
  for (int k = tid; k < L; k += threads) acc[k] = 0.0;
  for (long long u = blockIdx.x; 2 * u < in.a.n_traj; u += gridDim.x) {
    const bool on0 = in.a.w[2 * u] != 0.0, on1 = 2 * u + 1 < in.a.n_traj && in.a.w[2 * u + 1] != 0.0;
    for (int part = 0; part < 3; ++part) {
      if (!(part == 0 ? on0 : part == 1 ? on1 : on0 || on1)) continue;
      double2 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = in.load(u, part, tid + i * threads);
      __syncthreads();  // the last series' terms are read
      block_fft(v, sm, logN, logN);
      for (int k = tid; k < L; k += threads) acc[k] += prmu_term(sm[fft_pad(k)], sm[fft_pad((N - k) & (N - 1))]);
    }
  }
  for (int k = tid; k < L; k += threads) partial[(size_t)blockIdx.x * L + k] = acc[k];
}

// partial[y][k], k < L: the terms of the block row's share of the B transformed series
__global__ void __launch_bounds__(256) prmu_accum_kernel(const double2 *z, long long B, long long N, int L,
                                                         double *partial) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= L) return;
  const long long kr = (N - k) & (N - 1), lo = B * blockIdx.y / gridDim.y, hi = B * (blockIdx.y + 1) / gridDim.y;
  double acc = 0.0;
  for (long long b = lo; b < hi; ++b) acc += prmu_term(z[b * N + k], z[b * N + kr]);
  partial[(size_t)blockIdx.y * L + k] = acc;
}

// sf[k] += sum over rows of partial[row][k]: lane = frequency, each warp every eighth row,
// then the warps in order
__global__ void __launch_bounds__(256) prmu_reduce_kernel(const double *partial, int rows, int L, double *sf) {
  __shared__ double red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
  double v = 0.0;
  if (k < L) {
#pragma unroll 4
    for (int b = w; b < rows; b += 8) v += partial[(size_t)b * L + k];
  }
  red[w][lane] = v;
  __syncthreads();
  if (w == 0 && k < L) {
    for (int i = 1; i < 8; ++i) v += red[i][lane];
    sf[k] += v;
  }
}

}  // namespace hh
