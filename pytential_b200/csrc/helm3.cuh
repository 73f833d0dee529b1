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

// list helpers (as in the Laplace kernels)
constexpr int MAXB = 128;       // list boxes staged per pass

QBX_D void h3_list_prefix(const qbxfmm_geometry& g, const int32_t* __restrict__ lists, int gb,
                          int nb, int* s_pref, int* s_start, int32_t* err)
{
  if (threadIdx.x >= 32) return;
  int lane = threadIdx.x;
  int cnt[4], loc = 0;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    int k = lane * 4 + u;
    cnt[u] = 0;
    if (k < nb) {
      int sb = lists[gb + k];
      int s0 = 0;
      if ((unsigned)sb < (unsigned)g.nboxes) {
        s0 = g.box_source_starts[sb];
        cnt[u] = g.box_source_counts_nonchild[sb];
      } else {
        report(err, QBX_DEVERR_BAD_BOX);
      }
      s_start[k] = s0;
    }
    loc += cnt[u];
  }
  int incl = loc;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    int v = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += v;
  }
  int run = incl - loc;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    int k = lane * 4 + u;
    if (k < nb) s_pref[k] = run;
    run += cnt[u];
  }
  if (lane == 31) s_pref[nb] = incl;
}

QBX_D int h3_stream_source(int v, int nb, const int* s_pref, const int* s_start)
{
  int lo = 0, hi = nb - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (s_pref[mid] <= v) lo = mid;
    else hi = mid - 1;
  }
  return s_start[lo] + (v - s_pref[lo]);
}

// Weights g_t of the Taylor coefficients b_t along a line of length |a| (x = k|a|) that
// give the order-Q expansion's value: 1 where j_n is cut to its power series (cut), else
// sum_n j_n Lambda_n with b_t = sum_{n + 2j = t} alpha_nj x^t Lambda_n, from the highest
// order down
template <int Q>
QBX_D void m2t_taylor_weights(bool cut, double x, double* gw)
{
#pragma unroll
  for (int n = 0; n <= Q; ++n) gw[n] = 1.0;
  if (cut) return;
  // jh_n = j_n(x) (2n+1)!! / x^n: by its series for small x, else from j_n
  double jh[Q + 1];
  const double mx2 = -0.5 * x * x;
  if (x < 2.0) {
#pragma unroll
    for (int n = 0; n <= Q; ++n) {
      double t = 1.0, acc = 0.0;
      for (int j = 0; j < 16; ++j) {
        acc += t;
        t *= mx2 * rcp(j + 1) * rcp(2 * n + 2 * j + 3);
      }
      jh[n] = acc;
    }
  } else {
    double jv[H3_LMAX + 2];
    h3_sph_j(Q, x, jv);
    double f = 1.0;
#pragma unroll
    for (int n = 0; n <= Q; ++n) {
      jh[n] = jv[n] * f;
      f *= (2.0 * n + 3.0) / x;
    }
  }
#pragma unroll
  for (int n = Q; n >= 0; --n) {
    double t = 1.0, v = jh[n];
#pragma unroll
    for (int j = 1; n + 2 * j <= Q; ++j) {
      t *= mx2 * rcp(j) * rcp(2 * n + 2 * j + 1);
      v -= gw[n + 2 * j] * t;
    }
    gw[n] = v;
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
