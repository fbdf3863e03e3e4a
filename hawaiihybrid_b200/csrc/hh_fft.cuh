// Batched FP64 transform  Y[k] = sum_j x[j] e^{+2 pi i jk/L}  (L a power of two), and the
// CF -> SF transform on it.
//
// A pass takes R points of stride L / R of every column through shared memory (Stockham's
// step of radix R: with s the product of the radices before it and n = L / s, element
// q + s (p + (n/R) j) goes to q + s (R p + k) with the twiddle e^{2 pi i pk/n}), in steps of
// radix 8 held in registers, so L <= 4096 is one pass over memory and L <= 2^18 two, where
// radix-2 steps of one kernel each made log2 L of them.  A block holds C = 2^logT / R
// neighbouring columns (4 or 8: runs of 64 or 128 bytes); columns run on over the series of
// the batch.  The first pass reads through a functor and the last one writes through one, so
// that packing and scaling are not passes of their own.
//
// Bound by the FP64 unit (about 27 operations per point and step) at batch sizes, by latency
// for one series: L = 131,072 takes two launches of 11 and 8 us, 17 radix-2 ones took 60.
//
// Shared memory is indexed i + i / 8: the radix-8 step's stores (stride 8 elements of 16
// bytes) and the store loop's reads (stride C) then meet different banks.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "hh_consts.h"

namespace hh {

constexpr int FFT_MAX_LOG_TILE = 12;  // 4,096 points: 72 KB of shared memory, 512 threads
constexpr int FFT_MIN_LOG_TILE = 8;   // one warp

struct FftPass {
  int logL, logR, logS, logT;
  long long cols;  // (L / R) x series
};

__host__ __device__ __forceinline__ int fft_pad(int i) { return i + (i >> 3); }
inline size_t fft_smem(int logT) { return (size_t)fft_pad(1 << logT) * sizeof(double2); }

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmul_i(double2 a) { return make_double2(-a.y, a.x); }
__device__ __forceinline__ double2 cis_pi(double t) {  // e^{i pi t}
  double2 w;
  sincospi(t, &w.y, &w.x);
  return w;
}

__device__ __forceinline__ void fft4(double2 &a, double2 &b, double2 &c, double2 &d) {
  const double2 e = cadd(a, c), f = cadd(b, d), g = csub(a, c), h = cmul_i(csub(b, d));
  a = cadd(e, f);
  b = cadd(g, h);
  c = csub(e, f);
  d = csub(g, h);
}

__device__ __forceinline__ void fft8(double2 (&v)[8]) {
  const double r = 0.70710678118654752440;
  double2 a[4], b[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    a[j] = cadd(v[j], v[j + 4]);
    b[j] = csub(v[j], v[j + 4]);
  }
  b[1] = make_double2(r * (b[1].x - b[1].y), r * (b[1].x + b[1].y));
  b[2] = cmul_i(b[2]);
  b[3] = make_double2(-r * (b[3].x + b[3].y), r * (b[3].x - b[3].y));
  fft4(a[0], a[1], a[2], a[3]);
  fft4(b[0], b[1], b[2], b[3]);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[2 * j] = a[j];
    v[2 * j + 1] = b[j];
  }
}

// the 2^logR-point transforms of the 2^(logT - logR) columns of a tile, by 2^(logT - 3)
// threads.  Element e = column + C * j is v[i] of thread tid, e = tid + i * threads; output k
// of a column is left at sm[fft_pad(column + C * k)].  The caller synchronises before the
// first store to sm when something still reads it.
__device__ __forceinline__ void block_fft(double2 (&v)[8], double2 *sm, int logT, int logR) {
  const int tid = threadIdx.x, step = 1 << (logT - 3);
  int ls = logT - logR;
  if (logR == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) sm[fft_pad(tid + i * step)] = v[i];
    __syncthreads();
  }
  for (int left = logR; left > 0;) {
    if (left != logR) {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = sm[fft_pad(tid + i * step)];
      __syncthreads();
    }
    if (left >= 3) {
      fft8(v);
      const int p = tid >> ls, q = tid & ((1 << ls) - 1);
      if (left > 3) {
        // three of the seven twiddles by sincospi, the others as their products
        const double t = double(p) * (2.0 / double(1 << left));
        const double2 w1 = cis_pi(t), w2 = cis_pi(2.0 * t), w4 = cis_pi(4.0 * t), w3 = cmul(w1, w2);
        v[1] = cmul(v[1], w1);
        v[2] = cmul(v[2], w2);
        v[3] = cmul(v[3], w3);
        v[4] = cmul(v[4], w4);
        v[5] = cmul(v[5], cmul(w1, w4));
        v[6] = cmul(v[6], cmul(w2, w4));
        v[7] = cmul(v[7], cmul(w3, w4));
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) sm[fft_pad(q + ((8 * p + k) << ls))] = v[k];
      ls += 3;
      left -= 3;
    } else if (left == 2) {  // last step: p = 0
      fft4(v[0], v[2], v[4], v[6]);
      fft4(v[1], v[3], v[5], v[7]);
#pragma unroll
      for (int i = 0; i < 8; ++i) sm[fft_pad(tid + i * step)] = v[i];
      left = 0;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double2 a = v[i], b = v[i + 4];
        sm[fft_pad(tid + i * step)] = cadd(a, b);
        sm[fft_pad(tid + (i + 4) * step)] = csub(a, b);
      }
      left = 0;
    }
    __syncthreads();
  }
}

// element idx of series b of a batch in memory
struct FftFrom {
  const double2 *x;
  int logL;
  __device__ double2 operator()(long long b, long long idx) const { return x[(b << logL) + idx]; }
};
struct FftTo {
  double2 *y;
  int logL;
  __device__ void operator()(long long b, long long idx, double2 v) const { y[(b << logL) + idx] = v; }
};

template <class Load, class Store>
__global__ void __launch_bounds__(1 << (FFT_MAX_LOG_TILE - 3)) fft_pass_kernel(Load ld, Store st, FftPass P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2 *sm = reinterpret_cast<double2 *>(smem_raw);
  const int tid = threadIdx.x, threads = 1 << (P.logT - 3), logC = P.logT - P.logR;
  const int logB = P.logL - P.logR;  // columns per series
  const long long col0 = (long long)blockIdx.x << logC;
  double2 v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int e = tid + i * threads;
    const long long col = col0 + (e & ((1 << logC) - 1));
    v[i] = make_double2(0.0, 0.0);
    if (col < P.cols) {
      const long long b = col >> logB, t = col - (b << logB);
      v[i] = ld(b, t + ((long long)(e >> logC) << logB));
    }
  }
  block_fft(v, sm, P.logT, P.logR);
  const double rn = 2.0 / double(1ll << (P.logL - P.logS));
#pragma unroll 1
  for (int e = tid; e < 1 << P.logT; e += threads) {
    // first pass: a column's outputs lie together; later ones: the neighbouring columns' do
    const int c = P.logS == 0 ? e >> P.logR : e & ((1 << logC) - 1);
    const int k = P.logS == 0 ? e & ((1 << P.logR) - 1) : e >> logC;
    const long long col = col0 + c;
    if (col >= P.cols) continue;
    const long long b = col >> logB, t = col - (b << logB), p = t >> P.logS, q = t - (p << P.logS);
    double2 u = sm[fft_pad(c + (k << logC))];
    if (p) u = cmul(u, cis_pi(double(p * k) * rn));
    st(b, q + (((p << P.logR) + k) << P.logS), u);
  }
}

template <class Load, class Store>
cudaError_t fft_launch_pass(const Load &ld, const Store &st, const FftPass &P, cudaStream_t stream) {
  const size_t smem = fft_smem(P.logT);
  auto k = fft_pass_kernel<Load, Store>;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const int logC = P.logT - P.logR;
  k<<<(unsigned)((P.cols + (1ll << logC) - 1) >> logC), 1 << (P.logT - 3), smem, stream>>>(ld, st, P);
  return cudaGetLastError();
}

inline int fft_passes(int logL) { return logL <= FFT_MAX_LOG_TILE ? 1 : (logL + 8) / 9; }

// B transforms of length 2^logL from `ld` to `st`; w0 (two passes or more) and w1 (three or
// more) hold B << logL elements and may be what `ld` reads (w1) or `st` writes (w0 for an odd
// number of passes, w1 for an even one)
template <class Load, class Store>
cudaError_t fft_run(const Load &ld, const Store &st, int logL, long long B, double2 *w0, double2 *w1,
                    cudaStream_t stream) {
  const int np = fft_passes(logL);
  FftPass P;
  P.logL = logL;
  P.logS = 0;
  double2 *w[2] = {w0, w1};
  for (int i = 0; i < np; ++i) {
    P.logR = (logL - P.logS + np - i - 1) / (np - i);
    P.cols = B << (logL - P.logR);
    // eight columns where that leaves two blocks per SM or more, else four
    P.logT = np == 1 ? logL : P.logR + ((P.cols >> 3) >= 296 ? 3 : 2);
    if (P.logT < FFT_MIN_LOG_TILE) P.logT = FFT_MIN_LOG_TILE;
    if (P.logT > FFT_MAX_LOG_TILE) P.logT = FFT_MAX_LOG_TILE;
    cudaError_t e;
    if (np == 1) e = fft_launch_pass(ld, st, P, stream);
    else if (i == 0) e = fft_launch_pass(ld, FftTo{w[0], logL}, P, stream);
    else if (i == np - 1) e = fft_launch_pass(FftFrom{w[(i - 1) & 1], logL}, st, P, stream);
    else e = fft_launch_pass(FftFrom{w[(i - 1) & 1], logL}, FftTo{w[i & 1], logL}, P, stream);
    if (e != cudaSuccess) return e;
    P.logS += P.logR;
  }
  return cudaSuccess;
}

// CF -> SF transform (src/hawaii.c:5401-5410, 5478-5553, 5569-5601) in FP64.
//
// The reference apodizes C(t) with (1 - (t/tmax)^2)^2, packs the N samples into
// a 2N-point complex vector (Makhoul's half-sample shift, 1/(2N) scaling), runs
// a backward (exp(+i)) radix-2 FFT of length 2N and keeps the real part of the
// first N outputs, then scales to nu (cm^-1) and SF (J m^6 s).

// Connes' window at t / tmax = k / N, N a power of two (rN = 1 / N and the quotient are exact)
__host__ __device__ __forceinline__ double connes(double k, double rN) {
  const double r = k * rN, f = (1.0 - r) * (1.0 + r);
  return f * f;
}

struct IdctPack {
  const double *cf;
  long long N;
  __device__ double2 operator()(long long, long long i) const {
    if (i == N) return make_double2(0.0, 0.0);
    const double rN = 1.0 / double(N);
    const long long k = i < N ? i : 2 * N - i;
    const double v = cf[k] * connes(double(k), rN) * (0.5 * rN);
    const double2 w = cis_pi(0.5 * rN * double(i));
    return i < N ? make_double2(v * w.x, v * w.y) : make_double2(-v * w.x, -v * w.y);
  }
};

struct IdctFinish {
  double *sf;
  long long N;
  double scale;
  __device__ void operator()(long long, long long i, double2 v) const {
    if (i < N) sf[i] = v.x * scale;
  }
};

}  // namespace hh
