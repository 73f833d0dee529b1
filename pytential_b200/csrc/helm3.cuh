// 3D Helmholtz device helpers shared by the spherical-wave kernels: coefficient
// indexing, normalized Legendre recurrences, spherical Bessel and Hankel functions, the
// FP64 tensor-core product.
#pragma once

#include "laplace.cuh"

namespace qbx {

namespace {

constexpr int H3_LMAX = 44;        // largest order of a radial / harmonic table
constexpr int H3_MAXP = 17;        // largest FMM order
constexpr double FOUR_PI = 12.566370614359172953850573533118;

QBX_HD int hq(int n, int m) { return n * n + n + m; }

QBX_HD void hq_decode(int c, int& n, int& m)
{
  n = (int)sqrt((double)c);
  while ((n + 1) * (n + 1) <= c) ++n;
  while (n * n > c) --n;
  m = c - n * n - n;
}

// Recurrence table for the normalized associated Legendre polynomial parts, n <= N:
// rec[idx3(n, m)] = (p_m^m, 0) at n = m, (sqrt(2m + 3), 0) at n = m + 1, else
// (a_nm, b_nm) with p_n^m = a_nm (t p_{n-1}^m - b_nm p_{n-2}^m).
QBX_D void h3_rec_table(int N, double2* rec, int tid, int nt)
{
  int tot = (N + 1) * (N + 2) / 2;
  for (int e = tid; e < tot; e += nt) {
    int n, m;
    decode3(e, n, m);
    double a, b = 0.0;
    if (n == m) {
      a = 0.28209479177387814347;   // 1 / sqrt(4 pi)
      for (int i = 1; i <= m; ++i) a *= sqrt((2.0 * i + 1.0) / (2.0 * i));
    } else if (n == m + 1) {
      a = sqrt(2.0 * m + 3.0);
    } else {
      a = sqrt((4.0 * n * n - 1.0) / ((double)n * n - (double)m * m));
      b = sqrt(((n - 1.0) * (n - 1.0) - (double)m * m) / (4.0 * (n - 1.0) * (n - 1.0) - 1.0));
    }
    rec[e] = c2(a, b);
  }
}

// t = cos(theta), w = sin(theta) e^{i phi} of v (v = 0: t = 1, w = 0)
QBX_D double h3_dir(const double* v, double2& w, double& r)
{
  r = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
  if (r == 0.0) {
    w = c2(0.0);
    return 1.0;
  }
  double ri = 1.0 / r;
  w = c2(v[0] * ri, v[1] * ri);
  return v[2] * ri;
}

// j_n(x), n <= N, by Miller's backward recurrence normalized with j_0 or j_1
QBX_D void h3_sph_j(int N, double x, double* jv)
{
  for (int n = 0; n <= N; ++n) jv[n] = 0.0;
  if (x == 0.0) {
    jv[0] = 1.0;
    return;
  }
  int nmax = max(N, (int)x);
  int start = nmax + 16 + (int)sqrt(40.0 * (nmax + 1));
  double xi = 1.0 / x;
  double fp1 = 0.0, f = 1e-200, f1 = 0.0;
  for (int n = start; n >= 1; --n) {
    double fm1 = (2.0 * n + 1.0) * xi * f - fp1;
    fp1 = f;
    f = fm1;
    if (n - 1 <= N) jv[n - 1] = f;
    if (n - 1 == 1) f1 = f;
    if (fabs(f) > 1e200) {
      f *= 1e-200;
      fp1 *= 1e-200;
      f1 *= 1e-200;
      for (int j = n - 1; j <= N; ++j) jv[j] *= 1e-200;
    }
  }
  double s, c;
  sincos(x, &s, &c);
  double scale = (x < 1.0 || fabs(s) >= 0.5) ? (s * xi) / f : ((s * xi - c) * xi) / f1;
  for (int n = 0; n <= N; ++n) jv[n] *= scale;
}

// j_n^[T](x) = sum_{j: n + 2j <= T} (-x^2/2)^j x^n / (j! (2n+2j+1)!!), n <= N: the
// power series of j_n cut at total degree T (zero for n > T); T < 0: j_n itself.  The
// degree-T Taylor polynomial of sum L_nm j_n(k|v|) Y_n^m(v) is sum L_nm j_n^[T] Y_n^m.
QBX_D void h3_sph_j_cut(int N, double x, int T, double* jv)
{
  if (T < 0) {
    h3_sph_j(N, x, jv);
    return;
  }
  double xn = 1.0, dfac = 1.0, mx2 = -0.5 * x * x;
  for (int n = 0; n <= N; ++n) {
    if (n > 0) {
      xn *= x;
      dfac *= 2.0 * n + 1.0;
    }
    double term = xn / dfac, acc = 0.0;
    for (int j = 0; n + 2 * j <= T; ++j) {
      acc += term;
      term *= mx2 * rcp(j + 1) * rcp(2 * n + 2 * j + 3);
    }
    jv[n] = acc;
  }
}

// h_n(x) = j_n(x) + i y_n(x), n <= N, by the upward recurrence
QBX_D void h3_sph_h(int N, double x, double2* hv)
{
  double s, c;
  sincos(x, &s, &c);
  double xi = 1.0 / x;
  hv[0] = c2(s * xi, -c * xi);
  if (N >= 1) hv[1] = c2((s - c * x) * xi * xi, -(s * x + c) * xi * xi);
  for (int n = 1; n < N; ++n) {
    double f = (2.0 * n + 1.0) * xi;
    hv[n + 1] = c2(f * hv[n].x - hv[n - 1].x, f * hv[n].y - hv[n - 1].y);
  }
}

QBX_D double h3_scale(double k, double rho) { return fmin(1.0, k * rho); }

// i^e for integer e
QBX_D double2 ipow(int e)
{
  switch (e & 3) {
    case 0: return c2(1.0, 0.0);
    case 1: return c2(0.0, 1.0);
    case 2: return c2(-1.0, 0.0);
    default: return c2(0.0, -1.0);
  }
}

// D (8x8, two per lane: row lane/4, columns 2 (lane%4) + {0,1}) += A (8x4, row major,
// element (lane/4, lane%4)) B (4x8, column major, element (lane%4, lane/4)), FP64
QBX_D void h3_dmma(double& d0, double& d1, double a, double b)
{
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

}  // namespace

}  // namespace qbx
