// 2D Helmholtz (H2D) expansion arithmetic, float64.
//
// G = (i/4) H_0^(1)(k|x - y|).  With Z_m(u) = Z_m(k|u|) e^{i m arg u} (Z = J or
// H = J + iY), Graf's addition theorem gives the translations
//   M2M: M'_m = sum_n M_n J_{n-m}(c' - c)      L2L: L'_m = sum_n L_n J_{n-m}(c' - c)
//   M2L: L_m  = sum_n M_n H_{n-m}(c' - c)
// and the expansions M_m = sum q conj(J_m(y - c)), L_m = sum q Hb_m(y - c) with
// Hb_m(u) = H_m(k|u|) e^{-i m arg u} = (-1)^m H_{-m}(u).  Source-normal
// derivatives use (d_x + i d_y) Z_m = -k Z_{m+1}, (d_x - i d_y) Z_m = k Z_{m-1}.
// Coefficients are scaled by rscale^|m| (multipoles divided, locals multiplied).
//
// Bessel functions: J_0..J_N by Miller's backward recurrence normalized with
// J_0 + 2 sum_k J_2k = 1; Y_0, Y_1 from the CUDA math library (y0, y1) below x = 8 and
// Hankel's form above, where the library's error is absolute (5e-12);
// Y_{n+1} = (2n/x) Y_n - Y_{n-1} (stable upward).
#pragma once

#include "common.cuh"

namespace qbx {

// first index of Miller's recurrence for orders up to nmax and arguments up to nmax
QBX_D int miller_start(int nmax) { return 2 * ((nmax + 16 + (int)sqrt(40.0 * nmax)) / 2); }

// P_0, Q_0 x / 8, P_1, Q_1 x / 8 of Hankel's form of H_0 and H_1 (Abramowitz & Stegun
// 9.2.5-9.2.6) in powers of z = (8/x)^2, x >= 8: Chebyshev expansions computed from the
// integrals that define them, cut at degree 12 (tests/golden/make_hankel_pq.py)
static __constant__ double c_hankel_pq[4][13] = {
    {  // P0
     1, -0.0010986328124988106, 2.7380883622028302e-05, -2.183917912860027e-06,
     3.6202014961341726e-07, -1.0230381069471657e-07, 4.3424496202719202e-08, -2.4257416747728671e-08,
     1.4955669741118411e-08, -8.4244019168030117e-09, 3.6616327747651667e-09, -1.029775376082398e-09,
     1.3657578771623472e-10,
    },
    {  // Q0
     -0.015624999999999997, 0.00014305114745956593, -6.9307861041698743e-06, 8.2384278024370908e-07,
     -1.8162568982031541e-07, 6.4007335210559721e-08, -3.2323578736828035e-08, 2.0507328469913932e-08,
     -1.3732461399427442e-08, 8.1281000911352184e-09, -3.6388968690144927e-09, 1.0424810644356815e-09,
     -1.3997455046895388e-10,
    },
    {  // P1
     1, 0.0018310546874986088, -3.5203993240441122e-05, 2.5809940497456218e-06,
     -4.1029067171084456e-07, 1.1307836608916155e-07, -4.7219294565271443e-08, 2.6096037687254697e-08,
     -1.5984079019861392e-08, 8.9706334212754281e-09, -3.8918385551293495e-09, 1.0937431701070939e-09,
     -1.4506440493278205e-10,
    },
    {  // Q1
     0.046874999999999993, -0.00020027160644386617, 8.4709608075089276e-06, -9.5058801055065598e-07,
     2.0299488931624851e-07, -7.0110464104389147e-08, 3.4932506905851458e-08, -2.1971335618931054e-08,
     1.4637445489481168e-08, -8.6385753180392068e-09, 3.8609338134006537e-09, -1.1049507975258166e-09,
     1.482618472437025e-10,
    },
};

QBX_D double hankel_pq(int f, double z)
{
  double r = c_hankel_pq[f][12];
#pragma unroll
  for (int i = 11; i >= 0; --i) r = fma(r, z, c_hankel_pq[f][i]);
  return r;
}

// Y_0 and Y_1 at x > 0; from x = 8 on, where the library's error is absolute,
//   Y_0 = sqrt(2 / (pi x)) (P_0 sin(x - pi/4) + Q_0 cos(x - pi/4)), Y_1 alike from x - 3 pi/4,
// with the phases' sines and cosines as sums of sin x and cos x: 50 multiply-adds beside one
// sincos, no more than the library's.  (Their Neumann series over the J_k of a recurrence of
// its own took M2P from 110 to 207 us, M2QBXL from 401 to 681 and P2QBXL from 573 to 1572 of a
// 1024-node boundary with 100 points, k 20; with this form 109, 384
// and 510.)
QBX_D void bessel_y01(double x, double& Y0, double& Y1)
{
  if (x < 8.0) {
    Y0 = y0(x);
    Y1 = y1(x);
    return;
  }
  double s, c;
  sincos(x, &s, &c);
  const double w = 8.0 / x, z = w * w, a = 0.56418958354775628695 * sqrt(0.125 * w);   // 1 / sqrt(pi x)
  const double d = s - c, e = s + c;
  Y0 = a * (hankel_pq(0, z) * d + w * hankel_pq(1, z) * e);
  Y1 = a * (w * hankel_pq(3, z) * d - hankel_pq(2, z) * e);
}

// J[0..N], Y[0..N] (Y only if want_y) at x > 0.
QBX_D void bessel_jy(int N, double x, double* J, double* Y, bool want_y)
{
  double xinv = 1.0 / x;
  int nmax = N > (int)x ? N : (int)x;
  int start = miller_start(nmax);
  double fp1 = 0.0, f = 1e-200, sum = 0.0;
  for (int j = 0; j <= N; ++j) J[j] = 0.0;
  for (int k = start; k > 0; --k) {
    // f = f_k, fp1 = f_{k+1}; f_{k-1} = (2k/x) f_k - f_{k+1}
    double fm1 = 2.0 * k * xinv * f - fp1;
    fp1 = f;
    f = fm1;
    if (k - 1 <= N) J[k - 1] = f;
    if (((k - 1) & 1) == 0 && k - 1 > 0) sum += 2.0 * f;
    if (fabs(f) > 1e200) {
      f *= 1e-200;
      fp1 *= 1e-200;
      sum *= 1e-200;
      for (int j = k - 1; j <= N; ++j) J[j] *= 1e-200;
    }
  }
  sum += f;   // f = f_0
  double norm = 1.0 / sum;
  for (int j = 0; j <= N; ++j) J[j] *= norm;
  if (want_y) {
    double b;
    bessel_y01(x, Y[0], b);
    if (N >= 1) Y[1] = b;
    for (int j = 1; j < N; ++j) Y[j + 1] = 2.0 * j * xinv * Y[j] - Y[j - 1];
  }
}

// Z[N + m] = Z_m(u) for m in [-N, N]; Z = J (want_h false) or H (want_h true).
QBX_D void h2_zfun(int N, double k, double ux, double uy, double* Jb, double* Yb, double2* Z,
                   bool want_h)
{
  double r = sqrt(ux * ux + uy * uy);
  if (r == 0.0) {
    // J_0(0) = 1, J_m(0) = 0; the Hankel functions are singular there
    for (int m = -N; m <= N; ++m) Z[N + m] = c2(m == 0 && !want_h ? 1.0 : 0.0);
    return;
  }
  bessel_jy(N, k * r, Jb, Yb, want_h);
  double2 e1 = c2(ux / r, uy / r);
  double2 e = c2(1.0);
  for (int m = 0; m <= N; ++m) {
    double2 z = want_h ? c2(Jb[m], Yb[m]) : c2(Jb[m]);
    double2 v = cmul(z, e);
    Z[N + m] = v;
    double2 w = cmul(z, cconj(e));     // Z_m(kr) e^{-i m th}
    Z[N - m] = (m & 1) ? c2(-w.x, -w.y) : w;
    e = cmul(e, e1);
  }
}

}  // namespace qbx
