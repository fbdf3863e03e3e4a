// Host builder of the folded CH4-CO2 dipole table (hh_ch4co2_fold.h) from the
// expanded reference tables of hh_ch4co2_tables.h, in FP64.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdint>
#include <cstring>
#include <map>
#include <tuple>

#include "hh_ch4co2_coupled.h"
#include "hh_ch4co2_fold.h"
#include "hh_ch4co2_tables.h"
#include "hh_ch4co2_tc_layout.h"

namespace {
void lm_of(int code, int *l, int *m, int *cs) {
  const int i = code >> 1;
  int L = 0;
  while ((L + 1) * (L + 2) / 2 <= i) ++L;
  *l = L;
  *m = i - L * (L + 1) / 2;
  *cs = code & 1;
}
// nearest TF32 value (10 explicit mantissa bits, ties away from zero) of a float
float tf32_rna(float v) {
  uint32_t b;
  memcpy(&b, &v, 4);
  b = (b + 0x1000u) & ~0x1FFFu;
  float r;
  memcpy(&r, &b, 4);
  return r;
}
double norm_lm(int l, int m) {  // sqrt((l+m)! / (l-m)!)
  double p = 1.0;
  for (int k = l - m + 1; k <= l + m; ++k) p *= k;
  return std::sqrt(p);
}
}  // namespace

int ch4co2_build_fold(Ch4Co2FoldHost *out) {
  // Y2 index in the kernel's generation order
  std::map<std::tuple<int, int, int>, int> y2idx;
  int n2 = 0;
  for (int m = 0; m <= HH_CH4CO2_L2MAX; ++m)
    for (int l = m; l <= HH_CH4CO2_L2MAX; ++l)
      if ((l & 1) == 0) {
        y2idx[{l, m, 0}] = n2++;
        if (m > 0) y2idx[{l, m, 1}] = n2++;
      }
  // entries keyed in the kernel's loop order: m1, l1, cs1, component, Y2
  using Key = std::tuple<int, int, int, int, int>;
  std::map<Key, std::vector<double>> acc;
  for (int t = 0; t < HH_CH4CO2_NTERM; ++t) {
    const short *ix = hh_ch4co2_tidx[t];
    int l1, m1, c1, l2, m2, c2;
    lm_of(ix[2], &l1, &m1, &c1);
    lm_of(ix[3], &l2, &m2, &c2);
    if (l1 > HH_CH4CO2_L1MAX) return -1;
    auto it = y2idx.find({l2, m2, c2});
    if (it == y2idx.end()) return -1;
    std::vector<double> &k = acc[Key(m1, l1, c1, ix[1], it->second)];
    if (k.empty()) k.assign(HH_CH4CO2_NSEG * 4, 0.0);
    const double w = hh_ch4co2_tcoef[t] * norm_lm(l1, m1) * norm_lm(l2, m2);
    for (int s = 0; s < HH_CH4CO2_NSEG; ++s)
      for (int j = 0; j < 4; ++j) k[s * 4 + j] += w * hh_ch4co2_rad[ix[0]][s][j];
  }
  const int E = (int)acc.size();
  out->n_entry = E;
  out->coef.assign((size_t)HH_CH4CO2_NSEG * E * 4, 0.0);
  out->y2.assign(E, 0);
  out->grp.clear();
  out->gcount.assign((HH_CH4CO2_L1MAX + 1) * (HH_CH4CO2_L1MAX + 2) / 2, 0);
  // (l1, m1) -> position in the m1-major order of the kernel
  auto lm_pos = [](int l, int m) {
    int p = 0;
    for (int mm = 0; mm < m; ++mm) p += HH_CH4CO2_L1MAX + 1 - mm;
    return p + (l - m);
  };
  int e = 0;
  Key prev(-1, -1, -1, -1, -1);
  for (auto &kv : acc) {
    const Key &k = kv.first;
    const bool same = std::get<0>(k) == std::get<0>(prev) && std::get<1>(k) == std::get<1>(prev) &&
                      std::get<2>(k) == std::get<2>(prev) && std::get<3>(k) == std::get<3>(prev);
    if (!same) {
      out->grp.push_back((unsigned)std::get<2>(k) | ((unsigned)std::get<3>(k) << 1));
      out->gcount[lm_pos(std::get<1>(k), std::get<0>(k))]++;
    }
    out->grp.back() += 1u << 3;
    out->y2[e] = (unsigned char)std::get<4>(k);
    for (int s = 0; s < HH_CH4CO2_NSEG; ++s)
      for (int j = 0; j < 4; ++j) out->coef[((size_t)s * E + e) * 4 + j] = kv.second[s * 4 + j];
    prev = k;
    ++e;
  }
  out->n_group = (int)out->grp.size();
  // padded batches: each group's entries followed by zero entries up to a multiple of 4
  out->bcoef.clear();
  out->by2.clear();
  out->bmeta.clear();
  std::vector<int> order;  // entry index or -1 (padding), in batch order
  {
    int g = 0, lm = 0, e0 = 0;
    for (int m = 0; m <= HH_CH4CO2_L1MAX; ++m)
      for (int l = m; l <= HH_CH4CO2_L1MAX; ++l, ++lm)
        for (int k = 0; k < out->gcount[lm]; ++k, ++g) {
          const unsigned d = out->grp[g];
          const int cnt = int(d >> 3);
          const int nb = (cnt + 3) / 4;
          for (int b = 0; b < nb; ++b) {
            for (int j = 0; j < 4; ++j) order.push_back(4 * b + j < cnt ? e0 + 4 * b + j : -1);
            out->bmeta.push_back((d & 7u) | (b == nb - 1 ? 8u : 0u) | ((unsigned)lm << 8));
          }
          e0 += cnt;
        }
  }
  out->n_batch = (int)out->bmeta.size();
  const size_t EP = order.size();
  out->bcoef.assign((size_t)HH_CH4CO2_NSEG * EP * 4, 0.0);
  out->by2.assign(EP, 0);
  for (size_t i = 0; i < EP; ++i) {
    if (order[i] < 0) continue;
    out->by2[i] = out->y2[order[i]];
    for (int s = 0; s < HH_CH4CO2_NSEG; ++s)
      for (int j = 0; j < 4; ++j)
        out->bcoef[((size_t)s * EP + i) * 4 + j] = out->coef[((size_t)s * E + order[i]) * 4 + j];
  }
  return 0;
}

int ch4co2_build_tc_blob(const Ch4Co2FoldHost &f, std::vector<float> *blob) {
  using namespace hh;
  const int E = f.n_entry;
  // B[piece][component][column][K] in FP64 from the entry stream (groups in (m1, l1, cs,
  // component) order, gcount groups per (l1, m1) in m-major order)
  const size_t per_comp = (size_t)CH4TC_N * CH4TC_K;
  std::vector<double> B((size_t)HH_CH4CO2_NSEG * 3 * per_comp, 0.0);
  int g = 0, e = 0, lm = 0;
  for (int m = 0; m <= HH_CH4CO2_L1MAX; ++m)
    for (int l = m; l <= HH_CH4CO2_L1MAX; ++l, ++lm)
      for (int k = 0; k < f.gcount[lm]; ++k, ++g) {
        const unsigned d = f.grp[g];
        const int cs = int(d & 1u), comp = int((d >> 1) & 3u), cnt = int(d >> 3);
        if (comp > 2 || (m == 0 && cs == 1)) return -1;
        const int col = ch4tc_y1_col(l, m, cs, HH_CH4CO2_L1MAX);
        if (col >= CH4TC_NY1) return -1;
        for (int i = 0; i < cnt; ++i, ++e) {
          const int y2 = f.y2[e];
          for (int s = 0; s < HH_CH4CO2_NSEG; ++s)
            for (int j = 0; j < 4; ++j)
              B[((size_t)s * 3 + comp) * per_comp + (size_t)col * CH4TC_K + 4 * y2 + j] =
                  f.coef[((size_t)s * E + e) * 4 + j];
        }
      }
  if (e != E) return -1;
  blob->assign((size_t)HH_CH4CO2_NSEG * CH4TC_PIECE_BYTES / 4, 0.0f);
  for (int s = 0; s < HH_CH4CO2_NSEG; ++s)
    for (int q = 0; q < 2; ++q) {
      const int ncomp = q == 0 ? 2 : 1, img = (q == 0 ? CH4TC_IMG0 : CH4TC_IMG1) / 4;
      for (int c = 0; c < CH4TC_NCHUNK; ++c) {
        float *hi = blob->data() + ch4tc_blob_off(s, q, c) / 4, *lo = hi + img;
        for (int cc = 0; cc < ncomp; ++cc) {
          const int comp = q == 0 ? cc : 2;
          for (int n = 0; n < CH4TC_N; ++n)
            for (int kk = 0; kk < CH4TC_KC; ++kk) {
              // the chunk's column kk: power kk % 4 of the Y2 its group holds
              const int k = ch4tc_k_of(c, kk / 4);
              const double v = k < 0 ? 0.0 : B[((size_t)s * 3 + comp) * per_comp + (size_t)n * CH4TC_K + 4 * k + kk % 4];
              const float h = tf32_rna((float)v);
              const int off = ch4tc_img_off(cc * CH4TC_N + n, kk);
              hi[off] = h;
              lo[off] = tf32_rna((float)(v - (double)h));
            }
        }
      }
    }
  return 0;
}

// ---------------------------------------------------------------------------
// coupled form (hh_ch4co2_coupled.h)
// ---------------------------------------------------------------------------
namespace {
using cplx = std::complex<double>;

// a tensor of l1 x l2 x vector over (m1, m2, q), spherical components
struct Tensor {
  int l1, l2;
  std::vector<cplx> v;
  Tensor(int a, int b) : l1(a), l2(b), v((size_t)(2 * a + 1) * (2 * b + 1) * 3, 0.0) {}
  cplx &at(int m1, int m2, int q) { return v[((size_t)(m1 + l1) * (2 * l2 + 1) + (m2 + l2)) * 3 + (q + 1)]; }
  cplx get(int m1, int m2, int q) const {
    if (std::abs(m1) > l1 || std::abs(m2) > l2 || std::abs(q) > 1) return 0.0;
    return v[((size_t)(m1 + l1) * (2 * l2 + 1) + (m2 + l2)) * 3 + (q + 1)];
  }
};
template <class F> void each(const Tensor &t, F f) {
  for (int a = -t.l1; a <= t.l1; ++a)
    for (int b = -t.l2; b <= t.l2; ++b)
      for (int q = -1; q <= 1; ++q) f(a, b, q);
}
double ladder(int l, int m, int s) { return std::sqrt(double(l * (l + 1) - m * (m + s))); }  // m -> m + s
// the elements of a tensor with a + b + q = K, one b for each (a, q)
struct Slice {
  int l1, l2, K;
  std::vector<cplx> v;
  Slice(int a, int b, int k) : l1(a), l2(b), K(k), v((size_t)(2 * a + 1) * 3, 0.0) {}
  cplx &at(int a, int q) { return v[(size_t)(a + l1) * 3 + (q + 1)]; }
  cplx get(int a, int b, int q) const {
    if (a + b + q != K || std::abs(a) > l1 || std::abs(b) > l2 || std::abs(q) > 1) return 0.0;
    return v[(size_t)(a + l1) * 3 + (q + 1)];
  }
};
template <class F> void each(const Slice &t, F f) {
  for (int a = -t.l1; a <= t.l1; ++a)
    for (int q = -1; q <= 1; ++q)
      if (std::abs(t.K - a - q) <= t.l2) f(a, t.K - a - q, q);
}
// element (a, b, q) of J_s T, s = +1 or -1: the sum of the three ladder operators
template <class T> cplx shifted(const T &t, int s, int a, int b, int q) {
  cplx x = 0.0;
  if (std::abs(a - s) <= t.l1) x += ladder(t.l1, a - s, s) * t.get(a - s, b, q);
  if (std::abs(b - s) <= t.l2) x += ladder(t.l2, b - s, s) * t.get(a, b - s, q);
  if (std::abs(q - s) <= 1) x += ladder(1, q - s, s) * t.get(a, b, q - s);
  return x;
}
// |J_s T|^2
double shift_norm2(const Tensor &t, int s) {
  double n = 0.0;
  each(t, [&](int a, int b, int q) { n += std::norm(shifted(t, s, a, b, q)); });
  return n;
}
// J_s T / c of a slice, which is the slice K + s.  (As whole tensors the ladder of slices took
// 25 ms of every process that binds the system, so a tenth of it.)
Slice shift(const Slice &t, int s, double c) {
  Slice o(t.l1, t.l2, t.K + s);
  each(o, [&](int a, int b, int q) { o.at(a, q) = shifted(t, s, a, b, q) / c; });
  return o;
}
Slice slice(const Tensor &t, int K) {
  Slice o(t.l1, t.l2, K);
  each(o, [&](int a, int b, int q) { o.at(a, q) = t.get(a, b, q); });
  return o;
}
double norm2(const Tensor &t) {
  double n = 0.0;
  for (const cplx &x : t.v) n += std::norm(x);
  return n;
}
// P_l^m(cos theta) cos or sin (m phi) (Condon-Shortley) over the complex harmonics: the
// coefficients of -m and m (m = 0: the first one)
struct RealHarmonic {
  cplx lo, hi;
};
RealHarmonic real_harmonic(int l, int m, int cs) {
  double r = 1.0;  // (l + m)! / (l - m)!
  for (int k = l - m + 1; k <= l + m; ++k) r *= k;
  const double n = std::sqrt((2 * l + 1) / (4.0 * M_PI) / r), sg = (m & 1) ? -1.0 : 1.0;
  if (m == 0) return {1.0 / n, 0.0};
  if (cs == 0) return {0.5 * sg / n, 0.5 / n};
  return {cplx(0.0, 0.5) * sg / n, cplx(0.0, -0.5) / n};
}
using Poly = std::vector<cplx>;  // coefficients K = -J..J
Poly mul(const Poly &a, const Poly &b) {
  Poly o(a.size() + b.size() - 1, 0.0);
  for (size_t i = 0; i < a.size(); ++i)
    for (size_t j = 0; j < b.size(); ++j) o[i + j] += a[i] * b[j];
  return o;
}
Poly comb(const Poly &a, double x, const Poly &b) {
  Poly o(a);
  for (size_t i = 0; i < o.size(); ++i) o[i] += x * b[i];
  return o;
}
// the invariants' coefficients in the body frame itself (e1 = x, e2 = y, n1 = z)
void invariants(Poly (&I)[hh::CH4C_NJ]) {
  const cplx i1(0.0, 1.0);
  const Poly ux = {1.0, 0.0, -1.0}, uy = {i1, 0.0, i1}, uz = {0.0, 2.0, 0.0};
  const Poly xy = mul(ux, uy), zz = mul(uz, uz);
  I[0] = {1.0};
  I[1] = mul(xy, uz);
  I[2] = mul(comb(zz, -1.0, xy), comb(zz, 1.0, xy));
  I[3] = mul(I[1], I[1]);
  Poly d = mul(comb(mul(ux, ux), -1.0, mul(uy, uy)), comb(mul(xy, xy), 2.0, mul(zz, zz)));
  for (cplx &x : d) x *= i1;
  I[4] = d;
  I[5] = mul(I[1], I[2]);
  I[6] = mul(I[2], I[2]);
  I[7] = mul(I[1], I[3]);
  I[8] = mul(I[2], I[3]);
}
double sqrt_binom(int J, int K) {  // sqrt((2J)! / ((J+K)! (J-K)!))
  double b = 1.0;
  for (int k = 1; k <= J - K; ++k) b = b * (J + K + k) / k;
  return std::sqrt(b);
}
}  // namespace

int ch4co2_build_coupled(Ch4Co2CoupledHost *out) {
  using namespace hh;
  Poly I[CH4C_NJ];
  invariants(I);
  // basis functions from the term list
  std::map<int, std::vector<int>> terms;
  for (int t = 0; t < HH_CH4CO2_NTERM; ++t) terms[hh_ch4co2_tidx[t][0]].push_back(t);
  const double s2 = std::sqrt(0.5);
  const cplx cart[3][3] = {{s2, 0.0, -s2}, {cplx(0.0, s2), 0.0, cplx(0.0, s2)}, {0.0, 1.0, 0.0}};  // e_x, e_y, e_z over q
  // g[(jx, m2, q)][l2][b]: the real coefficient of rad_b p_K P_l2^|m2|
  std::map<std::tuple<int, int, int>, std::map<int, std::vector<std::pair<int, double>>>> G;
  for (const auto &kv : terms) {
    const int b = kv.first;
    int l1, m1, c1, l2, m2, c2;
    lm_of(hh_ch4co2_tidx[kv.second[0]][2], &l1, &m1, &c1);
    lm_of(hh_ch4co2_tidx[kv.second[0]][3], &l2, &m2, &c2);
    if (l2 > CH4C_LMAX || (l2 & 1)) return -1;
    Tensor T(l1, l2);
    for (int t : kv.second) {
      const short *ix = hh_ch4co2_tidx[t];
      int a, am, ac, e, em, ec;
      lm_of(ix[2], &a, &am, &ac);
      lm_of(ix[3], &e, &em, &ec);
      if (a != l1 || e != l2) return -1;
      const RealHarmonic y1 = real_harmonic(a, am, ac), y2 = real_harmonic(e, em, ec);
      for (int p = -am; p <= am; p += std::max(1, 2 * am))
        for (int r = -em; r <= em; r += std::max(1, 2 * em)) {
          const cplx yy = hh_ch4co2_tcoef[t] * (p == -am ? y1.lo : y1.hi) * (r == -em ? y2.lo : y2.hi);
          for (int q = -1; q <= 1; ++q) T.at(p, r, q) += yy * cart[ix[1]][q + 1];
        }
    }
    const double n2 = norm2(T);
    if (!(n2 > 0.0)) continue;
    // J from <J^2> = |J_- T|^2 + <Jz^2 - Jz>
    double jj = shift_norm2(T, -1) / n2, kz = 0.0;
    each(T, [&](int a, int e, int q) {
      const int K = a + e + q;
      kz += double(K) * (K - 1) * std::norm(T.get(a, e, q));
    });
    jj += kz / n2;
    const double Jr = 0.5 * (std::sqrt(1.0 + 4.0 * jj) - 1.0);
    const int J = (int)std::lround(Jr);
    int jx = -1;
    for (int k = 0; k < CH4C_NJ; ++k)
      if (CH4C_J[k] == J && (k == 4) == (((l1 + l2 + 1 + J) & 1) != 0)) jx = k;
    if (jx < 0 || std::abs(Jr - J) > 1e-6) return -1;
    // the strongest K of the invariant, its slice, and the ladder from there to every K
    int K0 = 0;
    for (int K = 1; K <= J; ++K)
      if (std::abs(I[jx][K + J]) / sqrt_binom(J, K) > 1.0001 * std::abs(I[jx][K0 + J]) / sqrt_binom(J, K0)) K0 = K;
    const cplx alpha = sqrt_binom(J, K0) / I[jx][K0 + J];
    std::vector<Slice> sl(2 * J + 1, Slice(l1, l2, 0));  // K = -J..J
    sl[K0 + J] = slice(T, K0);
    for (int K = K0; K < J; ++K) sl[K + 1 + J] = shift(sl[K + J], 1, ladder(J, K, 1));
    for (int K = K0; K > -J; --K) sl[K - 1 + J] = shift(sl[K + J], -1, ladder(J, K, -1));
    // T = sum_K a_K |J K> with a_K = p_K / sqrt_binom(K) / alpha'
    std::vector<cplx> aK(2 * J + 1);
    for (int K = -J; K <= J; ++K) aK[K + J] = alpha * I[jx][K + J] / sqrt_binom(J, K);
    double off = 0.0;
    each(T, [&](int a, int e, int q) {
      const int K = a + e + q;
      cplx x = T.get(a, e, q);
      if (std::abs(K) <= J) x -= aK[K + J] * sl[K + J].get(a, e, q);
      off += std::norm(x);
    });
    if (!(off < 1e-18 * n2)) return -1;
    const double yy = std::sqrt(double(2 * l1 + 1) * (2 * l2 + 1)) / (4.0 * M_PI);
    for (int K = -J; K <= J; ++K)
      for (int q = 0; q <= 1; ++q) {
        const int mm = K - q;
        if (std::abs(mm) > l2 || (q == 0 && mm < 0)) continue;
        cplx gv = alpha * sl[K + J].get(0, mm, q) * yy / sqrt_binom(J, K);
        if (mm < 0 && (mm & 1)) gv = -gv;       // P^{-m} = (-1)^m P^m in this normalisation
        if (std::abs(gv.imag()) > 1e-10 * std::abs(gv) + 1e-14) return -1;
        double gr = gv.real();
        if (q == 0 && mm > 0) gr *= 2.0;        // m and -m add conjugate terms
        // p_K of K < 0 from p_|K|
        if (K < 0 && ((K & 1) != 0) != (jx == 4)) gr = -gr;
        if (gr != 0.0) G[{jx, mm, q}][l2].push_back({b, gr});
      }
  }
  // groups in the kernel's order
  struct Grp {
    int jx, mm, q, n;
  };
  std::vector<Grp> order;
  for (int m = 0; m <= CH4C_LMAX; ++m) {
    std::vector<Grp> at;
    for (const auto &kv : G) {
      int jx, mm, q;
      std::tie(jx, mm, q) = kv.first;
      if (std::abs(mm) != m) continue;
      const int lmax = kv.second.rbegin()->first;
      at.push_back({jx, mm, q, (lmax - ch4c_l0(m)) / 2 + 1});
    }
    std::stable_sort(at.begin(), at.end(), [](const Grp &x, const Grp &y) { return x.n > y.n; });
    for (const Grp &x : at) {
      if (x.n < 1 || x.n > ch4c_nl(m)) return -1;
      out->count[m][x.n]++;
      order.push_back(x);
    }
  }
  out->n_group = (int)order.size();
  out->n_coef = 0;
  for (const Grp &x : order) out->n_coef += x.n;
  if (out->n_coef > CH4C_MAXCOEF || out->n_group > CH4C_MAXGROUP) return -1;
  out->desc.clear();
  out->coef.assign((size_t)HH_CH4CO2_NSEG * out->n_coef * 4, 0.0);
  int c = 0;
  for (const Grp &x : order) {
    const int K = x.mm + x.q;
    out->desc.push_back((unsigned short)((CH4C_TAU[x.jx] + std::abs(K)) | (x.q << 8) | ((K < 0 ? 1 : 0) << 9)));
    const auto &by_l = G[{x.jx, x.mm, x.q}];
    for (int i = 0; i < x.n; ++i, ++c) {
      const auto it = by_l.find(ch4c_l0(std::abs(x.mm)) + 2 * i);
      if (it == by_l.end()) continue;
      for (const auto &br : it->second)
        for (int s = 0; s < HH_CH4CO2_NSEG; ++s)
          for (int j = 0; j < 4; ++j)
            out->coef[((size_t)s * out->n_coef + c) * 4 + j] += br.second * hh_ch4co2_rad[br.first][s][j];
    }
  }
  return 0;
}
