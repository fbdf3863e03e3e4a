// The CH4-CO2 dipole in coupled form, shared by the host builder (hh_ch4co2_host.cpp) and
// the FP64 kernel (hh_ch4co2_coupled.cuh).
//
// Each of the 320 basis functions of PES-IDS/ai_ids_ch4_co2.cpp:672-1067 couples a harmonic
// l1 of the intermolecular axis, a harmonic l2 of the CO2 axis and the vector (l = 1) to
// one total order J of the CH4 orientation, J in {0, 3, 4, 6, 7, 8, 9, 10}, contracted with
// the one tetrahedral invariant of that order (J = 6 also with the pseudoscalar one).  In
// the frame whose z axis is the intermolecular axis and whose xz plane holds the CO2 axis,
// the first harmonic is a constant and the second a real associated Legendre function:
//   mu'_q = sum_{J, m} tau^J_{m+q} sum_{l2} G_{J, l2, m, q}(R) P_l2^|m|(cos theta),
// theta the angle between the two axes, tau^J the invariant rotated into that frame.  The
// tetrahedral invariants are products of two polynomials I3 and I4 (below), so tau^J are
// polynomial products.  That leaves about 600 piecewise cubics G in place of the 9,528
// padded entries (l1, m1, l2, m2, component) of the body-frame expansion.
//
// tau^J: with e1, e2, n1 the frame's axes in CH4 body coordinates, w = e1 + i e2 and
// u_c(K) = (w_c, 2 n1_c, -conj w_c) for K = -1, 0, 1, the coefficients of the quadratic
// u_c in two spinor variables (the null vector of the complex sphere, rotated), an
// invariant's rotated components are the coefficients p_K, K = -J..J, of the same
// polynomial in u_x, u_y, u_z:  I3 = ux uy uz, I4 = (uz^2 - ux uy)(uz^2 + ux uy),
// I6 = I3^2, I7 = I3 I4, I8 = I4^2, I9 = I3 I6, I10 = I4 I6, and the pseudoscalar
// I6' = i (ux^2 - uy^2)(2 uz^4 + ux^2 uy^2).  p_{-K} = (-1)^K conj(p_K) (with a further
// minus sign for I6'), so K >= 0 is kept: 62 complex values in the order below.
#pragma once
#include <vector>

#if defined(__CUDACC__)
#define HH_CH4C_FN __host__ __device__ constexpr
#define HH_CH4C_TAB static __device__ constexpr
#else
#define HH_CH4C_FN constexpr
#define HH_CH4C_TAB constexpr
#endif

namespace hh {
constexpr int CH4C_NJ = 9;                                             // I0, I3, I4, I6, I6', I7, I8, I9, I10
constexpr int CH4C_J[CH4C_NJ] = {0, 3, 4, 6, 6, 7, 8, 9, 10};
HH_CH4C_TAB int CH4C_TAU[CH4C_NJ + 1] = {0, 1, 5, 10, 17, 24, 32, 41, 51, 62};  // first p_K of each
constexpr int CH4C_NTAU = CH4C_TAU[CH4C_NJ];
constexpr int CH4C_LMAX = 12;
// even l2 >= m: how many, and the first
HH_CH4C_FN int ch4c_nl(int m) { return (CH4C_LMAX - m) / 2 + 1; }
HH_CH4C_FN int ch4c_l0(int m) { return m + (m & 1); }
static_assert(ch4c_nl(0) == 7 && ch4c_nl(1) == 6 && ch4c_nl(2) == 6 && ch4c_nl(11) == 1 && ch4c_nl(12) == 1, "even l2");
constexpr int CH4C_MAXCOEF = 700, CH4C_MAXGROUP = 192;
}  // namespace hh

// The groups (J, m, q) in the kernel's order: m = 0..12, within it by n = how many l2 (from
// the first even l2 >= m) the group sums, descending.  desc: p_K index | (q == 1) << 8 |
// (K < 0) << 9.
struct Ch4Co2CoupledHost {
  int n_coef = 0, n_group = 0;
  unsigned char count[13][8] = {};        // groups of (m, n)
  std::vector<unsigned short> desc;       // [n_group]
  std::vector<double> coef;               // [NSEG][n_coef][4]: cubic in R - centre of each piece
};
// returns 0, or -1 on a basis that is not of the form above
int ch4co2_build_coupled(Ch4Co2CoupledHost *out);
