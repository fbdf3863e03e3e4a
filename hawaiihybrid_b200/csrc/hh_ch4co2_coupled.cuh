// FP64 CH4-CO2 dipole of the record path in coupled form (hh_ch4co2_coupled.h): one record
// per lane, the records sorted by radial piece as for ch4_dipole_kernel (hh_ch4co2_dip.cuh),
// whose entry stream it replaces on the FP64 path.
//
// Per record: the frame (e1, e2, n1), the 62 rotated-invariant coefficients p_K by
// polynomial products (about 330 complex products), and for m = 0..12 the Legendre values
// P_l^m (even l <= 12) against the piece's groups, each one sum of up to seven cubics in R
// and one product with a p_K: 591 cubics in all, about 4,200 FP64 instructions per record
// where the body-frame stream takes 41,000.  A warp's p_K lie in shared memory (31.7 KB:
// six warps per SM beside the piece's 20 KB of coefficients, which every lane reads as
// broadcasts), everything else in registers.  FP64 throughput bounds it.  4 x 25,013
// trajectories, 4.07e6 records: 2.98 ms, 11 TFLOP/s, against 70.3 ms of the stream.
#pragma once

#include <cuda_runtime.h>

#include "hh_ch4co2_coupled.h"
#include "hh_ch4co2_dip.cuh"

namespace hh {

constexpr int CH4C_WARPS = 6;
struct Ch4CoupledArgs {
  const double2 *coef;        // [NSEG][n_coef][2]: (c0, c1), (c2, c3)
  const unsigned short *desc; // [n_group]
  int n_coef, n_group;
  unsigned char count[13][8]; // groups of (m, n)
  double centre[CH4_NSEG];
  const void *records;
  const int *sorted;
  const long long *warp0;     // [NSEG + 1] first task (32 records) of each piece
  void *mu;                   // [record][4]
};
// shared memory: the piece's coefficients and the descriptors, then p_K of every warp
constexpr size_t ch4c_smem() {
  return CH4C_MAXCOEF * 2 * sizeof(double2) + CH4C_MAXGROUP * sizeof(int) +
         (size_t)CH4C_WARPS * CH4C_NTAU * 32 * sizeof(double2);
}

// coefficient K of a polynomial of degree (spin) J kept for K >= 0: p_{-K} = (-1)^K conj p_K
template <int N> __device__ __forceinline__ double2 ch4c_at(const double2 (&f)[N], int K) {
  if (K >= 0) return f[K];
  const double2 v = f[-K];
  return (K & 1) ? make_double2(-v.x, v.y) : make_double2(v.x, -v.y);
}
__device__ __forceinline__ void ch4c_madd(double2 &s, double2 a, double2 b) {
  s.x += a.x * b.x;
  s.x -= a.y * b.y;
  s.y += a.x * b.y;
  s.y += a.y * b.x;
}
// coefficient K of the product of f (spin A) and g (spin B)
template <int A, int B>
__device__ __forceinline__ double2 ch4c_mul_at(const double2 (&f)[A + 1], const double2 (&g)[B + 1], int K) {
  double2 s = make_double2(0.0, 0.0);
#pragma unroll
  for (int i = -A; i <= A; ++i)
    if (K - i >= -B && K - i <= B) ch4c_madd(s, ch4c_at(f, i), ch4c_at(g, K - i));
  return s;
}
template <int A, int B>
__device__ __forceinline__ void ch4c_mul(const double2 (&f)[A + 1], const double2 (&g)[B + 1], double2 (&o)[A + B + 1]) {
#pragma unroll
  for (int K = 0; K <= A + B; ++K) o[K] = ch4c_mul_at<A, B>(f, g, K);
}
// f^2: the cross terms once, doubled
template <int A> __device__ __forceinline__ double2 ch4c_sqr_at(const double2 (&f)[A + 1], int K) {
  double2 s = make_double2(0.0, 0.0);
#pragma unroll
  for (int i = -A; i <= A; ++i) {
    const int j = K - i;
    if (j >= -A && j <= A && i < j) ch4c_madd(s, ch4c_at(f, i), ch4c_at(f, j));
  }
  s.x *= 2.0;
  s.y *= 2.0;
  if ((K & 1) == 0) ch4c_madd(s, ch4c_at(f, K / 2), ch4c_at(f, K / 2));
  return s;
}
template <int A> __device__ __forceinline__ void ch4c_sqr(const double2 (&f)[A + 1], double2 (&o)[2 * A + 1]) {
#pragma unroll
  for (int K = 0; K <= 2 * A; ++K) o[K] = ch4c_sqr_at<A>(f, K);
}

// the p_K of all invariants into t[32 k] (this lane's column)
__device__ __forceinline__ void ch4c_tau(const double (&e1)[3], const double (&e2)[3], const double (&n1)[3],
                                         double2 *t) {
  double2 u[3][2];  // K = 0, 1
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    u[c][0] = make_double2(2.0 * n1[c], 0.0);
    u[c][1] = make_double2(-e1[c], e2[c]);
  }
  double2 xy[3], zz[3], I3[4], I4[5], I6[7];
  ch4c_mul<1, 1>(u[0], u[1], xy);
  ch4c_sqr<1>(u[2], zz);
  ch4c_mul<2, 1>(xy, u[2], I3);
  {
    double2 a[3], b[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      a[k] = make_double2(zz[k].x - xy[k].x, zz[k].y - xy[k].y);
      b[k] = make_double2(zz[k].x + xy[k].x, zz[k].y + xy[k].y);
    }
    ch4c_mul<2, 2>(a, b, I4);
  }
  ch4c_sqr<3>(I3, I6);
  t[0] = make_double2(1.0, 0.0);
#pragma unroll
  for (int K = 0; K <= 3; ++K) t[32 * (CH4C_TAU[1] + K)] = I3[K];
#pragma unroll
  for (int K = 0; K <= 4; ++K) t[32 * (CH4C_TAU[2] + K)] = I4[K];
#pragma unroll
  for (int K = 0; K <= 6; ++K) t[32 * (CH4C_TAU[3] + K)] = I6[K];
  {
    // i (ux^2 - uy^2) (2 uz^4 + (ux uy)^2)
    double2 d[3], s[5], q[3];
    ch4c_sqr<1>(u[0], d);
    ch4c_sqr<1>(u[1], q);
#pragma unroll
    for (int k = 0; k < 3; ++k) d[k] = make_double2(d[k].x - q[k].x, d[k].y - q[k].y);
#pragma unroll
    for (int K = 0; K <= 4; ++K) {
      const double2 a = ch4c_sqr_at<2>(zz, K), b = ch4c_sqr_at<2>(xy, K);
      s[K] = make_double2(2.0 * a.x + b.x, 2.0 * a.y + b.y);
    }
#pragma unroll
    for (int K = 0; K <= 6; ++K) {
      const double2 v = ch4c_mul_at<2, 4>(d, s, K);
      t[32 * (CH4C_TAU[4] + K)] = make_double2(-v.y, v.x);
    }
  }
#pragma unroll
  for (int K = 0; K <= 7; ++K) t[32 * (CH4C_TAU[5] + K)] = ch4c_mul_at<3, 4>(I3, I4, K);
#pragma unroll
  for (int K = 0; K <= 8; ++K) t[32 * (CH4C_TAU[6] + K)] = ch4c_sqr_at<4>(I4, K);
#pragma unroll
  for (int K = 0; K <= 9; ++K) t[32 * (CH4C_TAU[7] + K)] = ch4c_mul_at<3, 6>(I3, I6, K);
#pragma unroll
  for (int K = 0; K <= 10; ++K) t[32 * (CH4C_TAU[8] + K)] = ch4c_mul_at<4, 6>(I4, I6, K);
}

struct Ch4CAcc {
  double z, re, im;  // mu'_0 and the complex mu'_{+1}
};

// the groups of (m, n) = the n first even l >= m: p[] the Legendre values
template <int NL, int N>
__device__ __forceinline__ void ch4c_run(int count, const double (&p)[NL], double x, const double2 *&c, const int *&d,
                                         const double2 *t, Ch4CAcc &acc) {
  if constexpr (N >= 1) {
#pragma unroll 1
    for (int g = 0; g < count; ++g) {
      double H = 0.0;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const double2 lo = c[2 * i], hi = c[2 * i + 1];
        H += p[i] * (lo.x + x * (lo.y + x * (hi.x + x * hi.y)));
      }
      c += 2 * N;
      const int de = *d++;
      const double2 tk = t[32 * (de & 0xff)];
      if (de & 0x100) {
        acc.re += H * tk.x;
        acc.im += ((de & 0x200) ? -H : H) * tk.y;
      } else {
        acc.z += H * tk.x;
      }
    }
  }
}

// Legendre functions P_l^m(c) with the normalisation sqrt((l - m)! / (l + m)!), s = sin:
// pmm = P_m^m on entry; the even l of order M in p, then all runs of this m, then m + 1
template <int M>
__device__ __forceinline__ void ch4c_orders(const Ch4CoupledArgs &a, double cth, double sth, double pmm, double x,
                                            const double2 *c, const int *d, const double2 *t, Ch4CAcc &acc) {
  if constexpr (M <= CH4C_LMAX) {
    constexpr int NL = ch4c_nl(M);
    double p[NL];
    double qb = 0.0, q = pmm;
#pragma unroll
    for (int l = M; l <= CH4C_LMAX; ++l) {
      if (l > M) {
        const double n = l == M + 1
                             ? sqrt(double(2 * M + 1)) * cth * q
                             : (double(2 * l - 1) * cth * q - sqrt(double((l - 1) * (l - 1) - M * M)) * qb) *
                                   (1.0 / sqrt(double(l * l - M * M)));
        qb = q;
        q = n;
      }
      if ((l & 1) == 0) p[(l - ch4c_l0(M)) / 2] = q;
    }
    ch4c_run<NL, NL>(a.count[M][NL], p, x, c, d, t, acc);
    ch4c_run<NL, NL - 1>(a.count[M][NL - 1], p, x, c, d, t, acc);
    if constexpr (NL >= 3) ch4c_run<NL, NL - 2>(a.count[M][NL - 2], p, x, c, d, t, acc);
    if constexpr (NL >= 4) ch4c_run<NL, NL - 3>(a.count[M][NL - 3], p, x, c, d, t, acc);
    if constexpr (NL >= 5) ch4c_run<NL, NL - 4>(a.count[M][NL - 4], p, x, c, d, t, acc);
    if constexpr (NL >= 6) ch4c_run<NL, NL - 5>(a.count[M][NL - 5], p, x, c, d, t, acc);
    if constexpr (NL >= 7) ch4c_run<NL, NL - 6>(a.count[M][NL - 6], p, x, c, d, t, acc);
    ch4c_orders<M + 1>(a, cth, sth, -pmm * sth * sqrt(double(2 * M + 1) / double(2 * M + 2)), x, c, d, t, acc);
  }
}

__global__ void __launch_bounds__(32 * CH4C_WARPS, 1) ch4_dipole_coupled_kernel(Ch4CoupledArgs a) {
  extern __shared__ __align__(16) unsigned char cc_smem[];
  double2 *coef = reinterpret_cast<double2 *>(cc_smem);
  int *desc = reinterpret_cast<int *>(coef + 2 * CH4C_MAXCOEF);
  double2 *tau = reinterpret_cast<double2 *>(desc + CH4C_MAXGROUP);
  __shared__ long long w0[CH4_NSEG + 1];
  for (int i = threadIdx.x; i <= CH4_NSEG; i += blockDim.x) w0[i] = a.warp0[i];
  for (int i = threadIdx.x; i < a.n_group; i += blockDim.x) desc[i] = a.desc[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double2 *t = tau + (size_t)warp * CH4C_NTAU * 32 + lane;
  // each block takes one run of consecutive tasks, piece by piece
  const long long total = w0[CH4_NSEG];
  const long long per = (total + gridDim.x - 1) / gridDim.x;
  const long long lo = blockIdx.x * per, hi = min(total, lo + per);
  for (int seg = 0; seg < CH4_NSEG; ++seg) {
    const long long b0 = max(lo, w0[seg]), b1 = min(hi, w0[seg + 1]);
    if (b0 >= b1) continue;  // the whole block
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * a.n_coef; i += blockDim.x) coef[i] = a.coef[(size_t)seg * 2 * a.n_coef + i];
    __syncthreads();
    for (long long w = b0 + warp; w < b1; w += CH4C_WARPS) {
      // padding slots evaluate the task's first record (always valid) and store nothing
      const int mine = a.sorted[w * 32 + lane];
      const int first = __shfl_sync(0xffffffffu, mine, 0);
      const int src = mine >= 0 ? mine : first;
      const double *rec = static_cast<const double *>(a.records) + (size_t)src * HH_REC_WORDS;
      const double r[3] = {rec[0], rec[1], rec[2]};
      const double qt[4] = {rec[3], rec[4], rec[5], rec[6]};
      const double ua[3] = {rec[7], rec[8], rec[9]};
      double M[3][3];
      quat_matrix<double>(qt, M);
      const double R = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
      const double iR = 1.0 / R, iu = 1.0 / sqrt(ua[0] * ua[0] + ua[1] * ua[1] + ua[2] * ua[2]);
      double n1[3], n2[3], e1[3], e2[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        n1[k] = (M[0][k] * r[0] + M[1][k] * r[1] + M[2][k] * r[2]) * iR;
        n2[k] = (M[0][k] * ua[0] + M[1][k] * ua[1] + M[2][k] * ua[2]) * iu;
      }
      // e1: the part of n2 normal to n1 (any normal where there is none), made exactly
      // normal to n1 once more: for small angles its rounding would not be
      const double cth = n1[0] * n2[0] + n1[1] * n2[1] + n1[2] * n2[2];
#pragma unroll
      for (int k = 0; k < 3; ++k) e1[k] = n2[k] - cth * n1[k];
      const double sth = sqrt(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
      if (!(sth > 1e-12)) {
        const bool x0 = fabs(n1[0]) < 0.6;
        e1[0] = x0 ? 1.0 : 0.0;
        e1[1] = x0 ? 0.0 : 1.0;
        e1[2] = 0.0;
      } else {
        const double is = 1.0 / sth;
#pragma unroll
        for (int k = 0; k < 3; ++k) e1[k] *= is;
      }
      const double dt = e1[0] * n1[0] + e1[1] * n1[1] + e1[2] * n1[2];
#pragma unroll
      for (int k = 0; k < 3; ++k) e1[k] -= dt * n1[k];
      const double ie = 1.0 / sqrt(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
#pragma unroll
      for (int k = 0; k < 3; ++k) e1[k] *= ie;
      e2[0] = n1[1] * e1[2] - n1[2] * e1[1];
      e2[1] = n1[2] * e1[0] - n1[0] * e1[2];
      e2[2] = n1[0] * e1[1] - n1[1] * e1[0];
      ch4c_tau(e1, e2, n1, t);
      Ch4CAcc acc = {0.0, 0.0, 0.0};
      ch4c_orders<0>(a, cth, sth, 1.0, R - a.centre[seg], coef, desc, t, acc);
      // mu = -sqrt(2) Re(mu'_1) e1 + sqrt(2) Im(mu'_1) e2 + mu'_0 n1, then to the lab
      double f = 1.0;
      if (seg == CH4_NSEG - 1) {
        const double i2 = iR * iR;
        f = i2 * i2 * i2;
      }
      const double s2 = 1.41421356237309504880 * f;
      double m[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) m[k] = (acc.im * e2[k] - acc.re * e1[k]) * s2 + acc.z * f * n1[k];
      if (mine >= 0) {
        double *o = static_cast<double *>(a.mu) + (size_t)mine * 4;
#pragma unroll
        for (int i = 0; i < 3; ++i) o[i] = M[i][0] * m[0] + M[i][1] * m[1] + M[i][2] * m[2];
      }
    }
  }
}

}  // namespace hh
