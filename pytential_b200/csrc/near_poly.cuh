// The target-specific near field of the 3D Laplace kernels as polynomials, float64.
//
// sum_{n <= Q} |a|^n / |b|^{n+1} P_n(cos g), cos g = a.b / (|a||b|), is rho F(x, y) with
// rho = 1 / |b|, x = (a.b) rho^2, y = |a|^2 rho^2 and F = sum_n sum_k p_nk x^{n-2k} y^k
// (P_n(t) = sum_k p_nk t^{n-2k}); its derivative in b along nu is
// rho^3 ((a.nu) dF/dx - (b.nu) H), H = F + 2 x dF/dx + 2 y dF/dy.  No square root of
// |a|, no division, no recurrence: Q + sum_j (Q - j) / 2 multiply-adds for F.
#pragma once

#include "common.cuh"

namespace qbx {

// p_nk (1 + s (n - 2k) + u k) laid out by the power j = n - 2k of x: coefficient of
// x^j y^k; kind 0: F, 1: H (factor 1 + 2n - 2k), 2: dF/dx (factor n - 2k, power j - 1)
template <int Q>
struct NearCoef {
  double f[Q + 1][Q / 2 + 1], h[Q + 1][Q / 2 + 1], d[Q + 1][Q / 2 + 1];
};

template <int Q>
constexpr NearCoef<Q> near_coef()
{
  NearCoef<Q> t{};
  for (int j = 0; j <= Q; ++j)
    for (int k = 0; j + 2 * k <= Q; ++k) {
      const int n = j + 2 * k;
      // (-1)^k (2n - 2k)! / (2^n k! (n - k)! (n - 2k)!)
      double v = (k & 1) ? -1.0 : 1.0;
      for (int i = n - k + 1; i <= 2 * n - 2 * k; ++i) v *= i;   // (2n-2k)! / (n-k)!
      for (int i = 2; i <= k; ++i) v /= i;
      for (int i = 2; i <= j; ++i) v /= i;
      for (int i = 0; i < n; ++i) v *= 0.5;
      t.f[j][k] = v;
      t.h[j][k] = v * (1 + 2 * n - 2 * k);
      if (j > 0) t.d[j - 1][k] = v * j;
    }
  return t;
}

template <int Q>
QBX_D double near_f(double x, double y)
{
  constexpr NearCoef<Q> C = near_coef<Q>();
  double r = 0.0;
#pragma unroll
  for (int j = Q; j >= 0; --j) {
    double p = C.f[j][(Q - j) / 2];
#pragma unroll
    for (int k = (Q - j) / 2 - 1; k >= 0; --k) p = fma(p, y, C.f[j][k]);
    r = j == Q ? p : fma(r, x, p);
  }
  return r;
}

template <int Q>
QBX_D double near_h(double x, double y)
{
  constexpr NearCoef<Q> C = near_coef<Q>();
  double r = 0.0;
#pragma unroll
  for (int j = Q; j >= 0; --j) {
    double p = C.h[j][(Q - j) / 2];
#pragma unroll
    for (int k = (Q - j) / 2 - 1; k >= 0; --k) p = fma(p, y, C.h[j][k]);
    r = j == Q ? p : fma(r, x, p);
  }
  return r;
}

// dF/dx: power j of x comes from the terms x^{j+1} y^k, k <= (Q - j - 1) / 2
template <int Q>
QBX_D double near_dx(double x, double y)
{
  constexpr NearCoef<Q> C = near_coef<Q>();
  double r = 0.0;
#pragma unroll
  for (int j = Q - 1; j >= 0; --j) {
    double p = C.d[j][(Q - j - 1) / 2];
#pragma unroll
    for (int k = (Q - j - 1) / 2 - 1; k >= 0; --k) p = fma(p, y, C.d[j][k]);
    r = j == Q - 1 ? p : fma(r, x, p);
  }
  return r;
}

}  // namespace qbx
