// Initial-condition sampler on the GPU.
//
// The reference draws every candidate phase point from one MT19937 stream
// (thirdparty/mtwist.c, seeded by mt_seed32 in init_ms, src/hawaii.c:157-163)
// and consumes a fixed number of words per candidate (src/hawaii.c:1206-1421):
//   q_generator: R, Phi, Theta (+ phi1, theta1 for a linear monomer; + phi1,
//                theta1, psi1 of a rotor and phi2, theta2 of a second, linear monomer)
//   p_generator: 3 (+2, or +3+2) Box-Muller normals, 2 words each
//   reject:      1 word
// i.e. D = 10 (atom-atom), 16 (linear-atom) or 25 (rotor-linear) words.  A Box-Muller draw only
// retries when its first word is exactly 0 (log(0) = -inf).
//
// GPU mapping:
//  1. mt_generate: one CTA advances the stream 227 words at a time in a ring in shared
//     memory and writes the tempered words to HBM;
//  2. candidates: one thread per candidate c reads the words [c*D, (c+1)*D),
//     restates q_generator/p_generator/Hamiltonian/reject/pair-state filter in
//     FP64 with the reference's operation order, and flags acceptance;
//  3. count/scan/scatter: accepted candidates are compacted in candidate order,
//     which is the order the reference's while-loop accepts them.
// A zero word at a Box-Muller position shifts every later candidate's window:
// the candidate kernel reports the first such candidate and the host restarts
// the following round right after it.
//
// Long requests of the stream (the 100 K rejection step of CH4-CO2 takes about
// 1.5e9 words per call) are generated in segments of HH_MT_SEG_BLOCKS blocks, one
// CTA each, from segment start states found by jumping ahead (hh_mt_jump.h):
// a chain of coarse jumps (HH_MT_COARSE segments each), then the fine jumps of every
// coarse interval in parallel.  The words are the same as those of the sequential
// generator.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "hh_consts.h"
#include "hh_internal.h"
#include "hh_mt_jump.h"
#include "hh_phase.cuh"
#include "hh_physics.cuh"
#include "hh_traj.cuh"

namespace hh {

__device__ __forceinline__ uint32_t mt_twist(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t y = (a & 0x80000000u) | (b & 0x7fffffffu);
  return c ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
}

__device__ __forceinline__ uint32_t mt_temper(uint32_t y) {
  y ^= y >> 11;
  y ^= (y << 7) & 0x9d2c5680u;
  y ^= (y << 15) & 0xefc60000u;
  y ^= y >> 18;
  return y;
}

// state[0..623] <- Knuth-69069 seeding (mts_seed32, thirdparty/mtwist.c:372-400):
// mt[0] = seed, mt[i] = 69069 * mt[i-1] (mod 2^32), i.e. 69069^i * seed
__global__ void mt_seed_kernel(uint32_t seed, uint32_t *state) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= MT_N) return;
  if (seed == 0) seed = 4357u;
  uint32_t p = 1u, b = 69069u;
  for (int e = i; e; e >>= 1) {
    if (e & 1) p *= b;
    b *= b;
  }
  state[i] = p * seed;
}

// The stream word after word, 227 at a time: x_{n+624} depends on x_n, x_{n+1} and x_{n+397},
// and x_{n+397} is the word that the same thread formed one step earlier, so it stays in a
// register and only x_n and x_{n+1} are read, from words formed two or three steps earlier.
// One barrier per two steps therefore orders the reads behind the writes; the ring of 2,048
// words is long enough that a step overwrites only words last read six steps before.
// 0.26 us per block of 624; a block-wise refresh in place (six barriers) took 0.51.
//
// mt_words: the words x_624 .. x_{n_words + 623} after the state x_0 .. x_623 in buf, where
// x_n is at buf[n & mask]; every new word goes to emit(n - 624, x_n).  256 threads, all
// calling; the caller's barrier follows the filling of buf, and one ends the call.
constexpr int MT_RING = 2048;
template <typename Emit>
__device__ __forceinline__ void mt_words(uint32_t *buf, unsigned mask, long long n_words, const Emit &emit) {
  constexpr unsigned W = MT_N - MT_M;
  const unsigned tid = threadIdx.x;
  const bool on = tid < W;
  unsigned n = tid;
  uint32_t prev = on ? buf[(n + MT_M) & mask] : 0u;
  const long long turns = (n_words + 2 * W - 1) / (2 * W);
  long long j = tid;
  for (long long t = 0; t < turns; ++t) {
    if (on) {
      // both steps' words first: they were formed before the last barrier
      const uint32_t a0 = buf[n & mask], b0 = buf[(n + 1) & mask];
      const uint32_t a1 = buf[(n + W) & mask], b1 = buf[(n + W + 1) & mask];
      const uint32_t x0 = mt_twist(a0, b0, prev), x1 = mt_twist(a1, b1, x0);
      if (j < n_words) {
        buf[(n + MT_N) & mask] = x0;
        emit(j, x0);
      }
      if (j + W < n_words) {
        buf[(n + W + MT_N) & mask] = x1;
        emit(j + W, x1);
      }
      prev = x1;
      n += 2 * W;
      j += 2 * W;
    }
    __syncthreads();
  }
}

// n_words of the stream after the block state `from` (global memory), tempered, to out, by
// one CTA; the 624 words that end the stream to `to` unless null.
__device__ __forceinline__ void mt_stream(const uint32_t *from, uint32_t *out, long long n_words, uint32_t *to,
                                          uint32_t *ring) {
  const int tid = threadIdx.x;
  for (int i = tid; i < MT_N; i += blockDim.x) ring[i] = from[i];
  __syncthreads();
  mt_words(ring, MT_RING - 1, n_words, [&](long long j, uint32_t x) { out[j] = mt_temper(x); });
  if (to) {
    for (int i = tid; i < MT_N; i += blockDim.x) to[i] = ring[(unsigned)(n_words + i) & (MT_RING - 1)];
  }
}

// Advance the generator by n_blocks refreshes, writing 624 tempered words per refresh to out.
__global__ void __launch_bounds__(256) mt_generate_kernel(uint32_t *state, uint32_t *out, long long n_blocks) {
  __shared__ uint32_t ring[MT_RING];
  mt_stream(state, out, n_blocks * MT_N, state, ring);
}

// One jump of J words: the state J words after `src` is the XOR of the windows, at the
// set-bit positions of x^J mod phi, of the 19,937 + 623 stream words after src, which each
// CTA generates in shared memory.  MT_JUMP_SPLIT CTAs share the positions and XOR their
// parts into dst (zero before): the windows' reads, about 9,950 x 624 words, bound a jump
// (0.24 ms in one CTA, 0.03 so).
constexpr int MT_JUMP_WIN = 33 * MT_N;  // the state and the 32 blocks after it
constexpr int MT_JUMP_THREADS = 640;
constexpr int MT_JUMP_SPLIT = 8;
constexpr int MT_JUMP_PART = (10240 + MT_JUMP_SPLIT - 1) / MT_JUMP_SPLIT;
__device__ __forceinline__ void mt_jump(const uint32_t *src, uint32_t *dst, const unsigned short *bits, int n_bits,
                                        int part, uint32_t *win, unsigned short *bs) {
  const int lo = part * MT_JUMP_PART, hi = min(n_bits, lo + MT_JUMP_PART);
  if (lo >= hi) return;  // the whole block
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) bs[i - lo] = bits[i];
  for (int i = threadIdx.x; i < MT_N; i += blockDim.x) win[i] = src[i];
  __syncthreads();
  mt_words(win, 0xffffffffu, MT_JUMP_WIN - MT_N, [](long long, uint32_t) {});
  if (threadIdx.x < MT_N) {
    const int j = threadIdx.x;
    uint32_t acc = 0;
#pragma unroll 8
    for (int t = 0; t < hi - lo; ++t) acc ^= win[bs[t] + j];
    atomicXor(&dst[j], acc);
  }
}

// The jump from states[base] to states[dst]: grid MT_JUMP_SPLIT.
__global__ void __launch_bounds__(MT_JUMP_THREADS) mt_jump_coarse_kernel(uint32_t *states, int base, int dst,
                                                                        const unsigned short *bits, int n_bits) {
  extern __shared__ uint32_t jsm[];
  mt_jump(states + (size_t)base * MT_N, states + (size_t)dst * MT_N, bits, n_bits, blockIdx.x, jsm,
          reinterpret_cast<unsigned short *>(jsm + MT_JUMP_WIN));
}

// Fine jumps: CTA (b, part) adds its part of segment s = (b / 31) * 32 + b % 31 + 1 (skipping
// the coarse states, which the chain made), one jump of k = s % 32 segments from
// states[s - k] with the table of x^(k J) mod phi, so every segment state of a round is one
// jump deep instead of a chain of up to 31.
constexpr size_t MT_FINE_OFFSET = 10240;  // the fine tables' offset in the segment-table buffer
static_assert(HH_MT_JUMP_FINE_MAX <= 10240, "fine jump table exceeds the buffer");
__global__ void __launch_bounds__(MT_JUMP_THREADS) mt_jump_fine_kernel(uint32_t *states, int n_seg,
                                                                      const unsigned short *fine,
                                                                      const unsigned short *fine_n) {
  extern __shared__ uint32_t jsm[];
  constexpr int PER = HH_MT_COARSE - 1;
  const long long s = (long long)(blockIdx.x / PER) * HH_MT_COARSE + (blockIdx.x % PER) + 1;
  if (s >= n_seg) return;  // the whole block
  const int k = (int)(s % HH_MT_COARSE);
  mt_jump(states + (s - k) * MT_N, states + s * MT_N, fine + (size_t)(k - 1) * HH_MT_JUMP_FINE_MAX, fine_n[k - 1],
          blockIdx.y, jsm, reinterpret_cast<unsigned short *>(jsm + MT_JUMP_WIN));
}

// Segment s: HH_MT_SEG_BLOCKS blocks from states[s], tempered words to
// out + s * HH_MT_SEG_BLOCKS * 624; the last segment's final block becomes the
// generator state.
__global__ void __launch_bounds__(256) mt_generate_segments_kernel(const uint32_t *states, uint32_t *out,
                                                                   int n_seg, uint32_t *final_state) {
  __shared__ uint32_t ring[MT_RING];
  const int s = blockIdx.x;
  mt_stream(states + (size_t)s * MT_N, out + (size_t)s * HH_MT_SEG_BLOCKS * MT_N, (long long)HH_MT_SEG_BLOCKS * MT_N,
            s == n_seg - 1 ? final_state : nullptr, ring);
}

// reference operation order is kept; FP contraction is disabled for this code
// by building with -fmad=false on the sampler translation unit
__device__ __forceinline__ double mt_d(const uint32_t *w, long long &pos) {
  return double(w[pos++]) * (1.0 / 4294967296.0);
}

__device__ __forceinline__ double bm_normal(const uint32_t *w, long long &pos, long long limit,
                                            int &retries, bool &overrun) {
  for (;;) {
    if (pos + 2 > limit) { overrun = true; return 0.0; }
    double U = mt_d(w, pos);
    double V = mt_d(w, pos);
    double logU = log(U);
    if (isnan(logU) || isinf(logU)) { ++retries; continue; }
    return 1.0 * sqrt(-2 * logU) * cos(2.0 * HH_PI * V);
  }
}

// Rejection ahead of the momenta (CH4-CO2, whose 100 K step accepts one candidate in 200).
// reject() compares exp(-V / kT) / M with the candidate's last uniform u; V depends on the
// positions alone, which are the first eight words.  One thread per candidate evaluates V
// in FP32 and rejects at once where the comparison is decided by more than a bound on its
// error, in the exponent 0.01 + (1e-4 |V| + 1e-6 |pesmin| + 1e-7 Hartree) / kT.  The others,
// and candidates with a zero word at a Box-Muller position (whose draw is retried), go on the
// list for candidate_kernel, which decides them as it would have decided all.
//
// The bound, e = 2^-24: with 1 + c = 2 u and 1 - c = 2 (1 - u) of a polar angle both from the
// integer word (c - 1 formed in FP32 would lose the angle beside a pole), sines, cosines and
// the quaternion are good to 15 e, the phases to 2 pi e and R to 5 e, so a site-site distance
// d is off by at most (20 R + 70) e, 1.1e-5 bohr at R = 6, and V by (12 P + 6 Q) / d times
// that (P, Q the sums of its repulsive and attractive terms).  Where the comparison is open
// at all, V - pesmin < 22 kT: P = 0.017 and Q = 0.01 Hartree at 100 K, an error of 6e-7
// against a bound of 4e-6; P = 0.003, Q = 0.0045 towards 0 K, 1.4e-7 against 2.5e-7; on the
// wall, where P is V, 6e-5 V against 1e-4 V.  The closest decisions of a million candidates,
// most of them beside a pole, agree with FP64 with an eighth of the bound too.
// 14.8e6 candidates: 6.6 ms with all in FP64, so 1.1 ms (bound by reading the words) and
// 0.8 ms for those left.
__global__ void __launch_bounds__(256) ch4_prefilter_kernel(SamplerArgs a, const uint32_t *words, long long word_base,
                                                            long long n_cand, unsigned char *accept,
                                                            unsigned char *consumed, unsigned *list,
                                                            unsigned long long *n_list) {
  constexpr int D = 25;
  __shared__ uint32_t w_s[256 * D];
  const long long c0 = blockIdx.x * 256ll;
  const int m = (int)min(256ll, n_cand - c0);
  const uint32_t *src = words + word_base + c0 * D;
  for (int i = threadIdx.x; i < m * D; i += 256) w_s[i] = src[i];
  __syncthreads();
  bool keep = false;
  if (threadIdx.x < m) {
    const uint32_t *w = w_s + threadIdx.x * D;
    constexpr float k = 1.f / 4294967296.f;
#pragma unroll
    for (int j = 8; j < 24; j += 2) keep = keep || w[j] == 0u;
    const float rmin3 = float(a.Rmin) * float(a.Rmin) * float(a.Rmin), rmax3 = float(a.Rmax) * float(a.Rmax) * float(a.Rmax);
    const float R = cbrtf(float(w[0]) * k * (rmax3 - rmin3) + rmin3);
    // r, the CH4 quaternion and the CO2 axis of ch4co2_qp_to_state
    float sP, cP, s1, c1, s3, c3, s2, c2;
    sincospif(2.f * float(w[1]) * k, &sP, &cP);
    sincospif(float(w[3]) * k, &s1, &c1);   // phi / 2
    sincospif(float(w[5]) * k, &s3, &c3);   // psi / 2
    sincospif(2.f * float(w[6]) * k, &s2, &c2);
    // u and 1 - u of the three polar angles: cos = u - (1 - u), sin = 2 sqrt(u (1 - u))
    const float uT = float(w[2]) * k, vT = (float(~w[2]) + 1.f) * k, ut = float(w[4]) * k, vt = (float(~w[4]) + 1.f) * k,
                uu = float(w[7]) * k, vu = (float(~w[7]) + 1.f) * k;
    const float cT = uT - vT, sT = 2.f * sqrtf(uT * vT), cu = uu - vu, su = 2.f * sqrtf(uu * vu);
    const float cb = sqrtf(ut), sb = sqrtf(vt);  // theta / 2
    const float r[3] = {-R * sT * cP, -R * sT * sP, R * cT}, u[3] = {-su * c2, -su * s2, cu};
    const float t0 = c1 * cb, t1 = c1 * sb, t2 = s1 * sb, t3 = s1 * cb;
    const float q[4] = {t0 * c3 - t3 * s3, t1 * c3 + t2 * s3, t2 * c3 - t1 * s3, t0 * s3 + t3 * c3};
    float M[3][3];
    quat_matrix<float>(q, M);
    const float V = ch4co2_lj<float>(a.x.lj, M, r, u).V;
    const float ikT = float(HH_HKT / a.T);
    // ln(exp(-V / kT) / M) against ln u, M = 1.5 exp(-pesmin / kT); a NaN keeps the candidate
    const float lw = (float(a.pesmin) - V) * ikT - 0.405465f;
    const float err = 0.01f + (1e-4f * fabsf(V) + 1e-6f * fabsf(float(a.pesmin)) + 1e-7f) * ikT;
    keep = keep || !(lw + err < logf(float(w[24]) * k));
    if (!keep) {
      accept[c0 + threadIdx.x] = 0;
      consumed[c0 + threadIdx.x] = D;
    }
  }
  const unsigned bal = __ballot_sync(0xffffffffu, keep);
  const int lane = threadIdx.x & 31;
  unsigned base = 0;
  if (bal && lane == 0) base = (unsigned)atomicAdd(n_list, (unsigned long long)__popc(bal));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (keep) list[base + __popc(bal & ((1u << lane) - 1u))] = (unsigned)(c0 + threadIdx.x);
}

// one thread per candidate (of the list, when there is one: *n_list candidates); words of
// candidate c start at word_base + c*D
__device__ __forceinline__ void candidate_at(
    const SamplerArgs &a, const Co2arTables<double> *tb, const uint32_t *words, long long n_words,
    long long word_base, int D, long long c, unsigned char *accept, unsigned char *consumed,
    double *qp_out, double *energy_out, unsigned long long *first_irregular);
__global__ void __launch_bounds__(256) candidate_kernel(
    SamplerArgs a, const Co2arTablesGlobal *gtab, const uint32_t *words, long long n_words,
    long long word_base, int D, long long n_cand, unsigned char *accept, unsigned char *consumed,
    double *qp_out, double *energy_out, unsigned long long *first_irregular, const unsigned *list,
    const unsigned long long *n_list) {
  extern __shared__ unsigned char smem_raw[];
  Co2arTables<double> *tb = reinterpret_cast<Co2arTables<double> *>(smem_raw);
  if (a.sys == SYS_CO2AR) load_tables<double>(tb, gtab);
  __syncthreads();
  const long long n = list ? (long long)*n_list : n_cand;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    candidate_at(a, tb, words, n_words, word_base, D, list ? (long long)list[i] : i, accept, consumed, qp_out,
                 energy_out, first_irregular);
}
__device__ __forceinline__ void candidate_at(
    const SamplerArgs &a, const Co2arTables<double> *tb, const uint32_t *words, long long n_words,
    long long word_base, int D, long long c, unsigned char *accept, unsigned char *consumed,
    double *qp_out, double *energy_out, unsigned long long *first_irregular) {
  long long pos = word_base + c * D;
  const long long limit = n_words;
  int retries = 0;
  bool overrun = false;
  const int QP = (a.sys == SYS_HEAR) ? 6 : (a.sys == SYS_CH4CO2 ? 16 : 10);
  double qp[16];
  double RMIN = a.Rmin, RMAX = a.Rmax, T = a.T;
  // q_generator (src/hawaii.c:1232-1290)
  double R3 = mt_d(words, pos) * (RMAX * RMAX * RMAX - RMIN * RMIN * RMIN) + RMIN * RMIN * RMIN;
  qp[4] = pow(R3, 1.0 / 3.0);
  qp[0] = mt_d(words, pos) * 2.0 * HH_PI;
  qp[2] = acos(2.0 * mt_d(words, pos) - 1.0);
  if (a.sys == SYS_CH4CO2) {
    qp[6] = mt_d(words, pos) * 2.0 * HH_PI;
    qp[8] = acos(2.0 * mt_d(words, pos) - 1.0);
    qp[10] = mt_d(words, pos) * 2.0 * HH_PI;
    qp[12] = mt_d(words, pos) * 2.0 * HH_PI;
    qp[14] = acos(2.0 * mt_d(words, pos) - 1.0);
  } else if (a.sys != SYS_HEAR) {
    qp[6] = mt_d(words, pos) * 2.0 * HH_PI;
    qp[8] = acos(2.0 * mt_d(words, pos) - 1.0);
  }
  const bool prmu = a.x.prmu_R0 > 0.0;
  if (prmu) qp[4] = a.x.prmu_R0;
  // p_generator (src/hawaii.c:1292-1380)
  double sqrt_MUKT = sqrt(a.mu / HH_HKT * T);
  double sinTheta = sin(qp[2]);
  double x0 = bm_normal(words, pos, limit, retries, overrun);
  double x1 = bm_normal(words, pos, limit, retries, overrun);
  double x2 = bm_normal(words, pos, limit, retries, overrun);
  qp[1] = sqrt_MUKT * qp[4] * sinTheta * x0;
  qp[3] = sqrt_MUKT * qp[4] * x1;
  qp[5] = sqrt_MUKT * x2;
  if (a.sys == SYS_CH4CO2) {
    // p_generator_rotor (src/hawaii.c:1305-1327)
    double sqrt_IIx = sqrt(a.x.II1[0] / HH_HKT * T);
    double sqrt_IIy = sqrt(a.x.II1[1] / HH_HKT * T);
    double sqrt_IIz = sqrt(a.x.II1[2] / HH_HKT * T);
    double sin_theta = sin(qp[8]), cos_theta = cos(qp[8]);
    double sin_psi = sin(qp[10]), cos_psi = cos(qp[10]);
    double r0 = bm_normal(words, pos, limit, retries, overrun);
    double r1 = bm_normal(words, pos, limit, retries, overrun);
    double r2 = bm_normal(words, pos, limit, retries, overrun);
    qp[7] = sqrt_IIx * sin_theta * sin_psi * r0 + sqrt_IIy * sin_theta * cos_psi * r1 + sqrt_IIz * cos_theta * r2;
    qp[9] = sqrt_IIx * cos_psi * r0 - sqrt_IIy * sin_psi * r1;
    qp[11] = sqrt_IIz * r2;
    // p_generator_linear_molecule of the second monomer (src/hawaii.c:1292-1303)
    double sqrt_IIKT = sqrt(a.II / HH_HKT * T);
    double sin_t2 = sin(qp[14]);
    double m0 = bm_normal(words, pos, limit, retries, overrun);
    double m1 = bm_normal(words, pos, limit, retries, overrun);
    qp[13] = sqrt_IIKT * sin_t2 * m1;
    qp[15] = sqrt_IIKT * m0;
  } else if (a.sys != SYS_HEAR) {
    double sqrt_IIKT = sqrt(a.II / HH_HKT * T);
    double sin_theta = sin(qp[8]);
    double m0 = bm_normal(words, pos, limit, retries, overrun);
    double m1 = bm_normal(words, pos, limit, retries, overrun);
    qp[7] = sqrt_IIKT * sin_theta * m1;
    qp[9] = sqrt_IIKT * m0;
  }
  if (!prmu && pos + 1 > limit) overrun = true;
  bool acc = false;
  double E = 0.0;
  if (prmu) {
    if (qp[5] > 0.0) qp[5] = -qp[5];
    acc = !overrun;
  } else if (!overrun) {
    // Hamiltonian, then reject() (src/hawaii.c:1382-1421), then the filter (2981-2994)
    double kin = kinetic(a, qp);
    double pot = potential(a, tb, qp);
    E = kin + pot;
    double u = mt_d(words, pos);
    double Mval = exp(-a.pesmin * HH_HKT / T);
    double M = 1.5 * Mval;
    double proposal = exp(-kin * HH_HKT / T);
    double desired = exp(-(kin + pot) * HH_HKT / T);
    double weight = desired / proposal / M;
    acc = !(weight < u);
    if (a.pair_state == 1 && E < 0.0) acc = false;
    if (a.pair_state == 2 && E > 0.0) acc = false;
  }
  if (retries || overrun) atomicMin(first_irregular, (unsigned long long)c);
  accept[c] = acc ? 1 : 0;
  consumed[c] = overrun ? 0 : (unsigned char)(pos - (word_base + c * D));
  for (int i = 0; i < QP; ++i) qp_out[c * QP + i] = qp[i];
  energy_out[c] = E;
}

// ---- CORRELATION_ARRAY reweighting (src/hawaii.c:2640-2676) ----
// One thread per trajectory: its energy at the base temperature T0 (the same
// Hamiltonian the sampler's filter used) and, per satellite temperature Ts,
//   weight = exp(-E HkT / T0 / Ts (T0 - Ts)) / WTT,
// with WTT = exp(-pesmin HkT / T0 / Ts (T0 - Ts)) for bound pairs below T0 and 1
// otherwise, and weight = 0 for free pairs above T0.  w[i][s] = weight * ratio_s
// feeds C(t); wraw[i][s] = weight feeds nstar.
struct SatArgs {
  int n_sat;
  double T0;
  double Ts[SAT_MAX];
  double ratio[SAT_MAX];
};

__global__ void __launch_bounds__(256) sat_weight_kernel(SamplerArgs a, SatArgs s,
                                                         const Co2arTablesGlobal *gtab,
                                                         const double *qp, long long n, double *w,
                                                         double *wraw) {
  extern __shared__ unsigned char smem_raw[];
  Co2arTables<double> *tb = reinterpret_cast<Co2arTables<double> *>(smem_raw);
  if (a.sys == SYS_CO2AR) load_tables<double>(tb, gtab);
  __syncthreads();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int QP = (a.sys == SYS_HEAR) ? 6 : (a.sys == SYS_CH4CO2 ? 16 : 10);
  double q[16];
  for (int c = 0; c < QP; ++c) q[c] = qp[i * QP + c];
  const double E = kinetic(a, q) + potential(a, tb, q);
  const double T0 = s.T0;
  for (int k = 0; k < s.n_sat; ++k) {
    const double T = s.Ts[k];
    double WTT = 1.0;
    if (a.pair_state == 2 && T < T0) WTT = exp(-a.pesmin * HH_HKT / T0 / T * (T0 - T));
    double weight = exp(-E * HH_HKT / T0 / T * (T0 - T)) / WTT;
    if (a.pair_state == 1 && T > T0) weight = 0.0;
    w[i * s.n_sat + k] = weight * s.ratio[k];
    wraw[i * s.n_sat + k] = weight;
  }
}

// ---- ordered compaction of accepted candidates ----
__global__ void __launch_bounds__(1024) count_kernel(const unsigned char *accept, long long n,
                                                     long long limit, unsigned int *block_counts) {
  long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int v = (c < n && c <= limit) ? accept[c] : 0;
  int cnt = __syncthreads_count(v);
  if (threadIdx.x == 0) block_counts[blockIdx.x] = cnt;
}

// exclusive scan of block counts in one CTA (n_blocks is small)
__global__ void __launch_bounds__(1024) scan_kernel(unsigned int *counts, int n_blocks,
                                                    unsigned long long *total) {
  __shared__ unsigned int partial[1024];
  __shared__ unsigned long long carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n_blocks; base += 1024) {
    int i = base + threadIdx.x;
    unsigned int v = (i < n_blocks) ? counts[i] : 0u;
    partial[threadIdx.x] = v;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
      unsigned int t = (threadIdx.x >= off) ? partial[threadIdx.x - off] : 0u;
      __syncthreads();
      partial[threadIdx.x] += t;
      __syncthreads();
    }
    if (i < n_blocks) counts[i] = (unsigned int)(carry + partial[threadIdx.x] - v);
    __syncthreads();
    if (threadIdx.x == 1023) carry += partial[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void __launch_bounds__(1024) scatter_kernel(const unsigned char *accept,
                                                       const double *qp_cand, long long n,
                                                       long long limit, const unsigned int *offsets,
                                                       int QP, long long out_base, long long out_cap,
                                                       double *qp_out, long long *cand_index_out,
                                                       long long cand_base) {
  __shared__ unsigned int warp_tot[32];
  long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int v = (c < n && c <= limit) ? accept[c] : 0;
  unsigned int ballot = __ballot_sync(0xffffffffu, v);
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned int before = __popc(ballot & ((1u << lane) - 1u));
  if (lane == 0) warp_tot[warp] = __popc(ballot);
  __syncthreads();
  unsigned int woff = 0;
  for (int w = 0; w < warp; ++w) woff += warp_tot[w];
  if (v) {
    long long dst = out_base + offsets[blockIdx.x] + woff + before;
    if (dst < out_cap) {
      for (int i = 0; i < QP; ++i) qp_out[dst * QP + i] = qp_cand[c * QP + i];
      if (cand_index_out) cand_index_out[dst] = cand_base + c;
    }
  }
}

}  // namespace hh
