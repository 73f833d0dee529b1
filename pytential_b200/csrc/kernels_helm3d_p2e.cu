// 3D Helmholtz P2M (form_multipoles) and P2L (form_locals, list 4), complex128, sm_100a.
//
// M_nm += 4 pi i k sigma s^-n (cq + cd nu.grad) j_n Y_n^-m,  L_nm with h_n and s^n: per box
// a (coefficient x source) matrix of waves times the sources' densities.  With v(s) = v0 +
// s eta along the source normal and F_n = f_n(k|u|) / |v|^n, R_nm = |v|^n Y_nm,
//   (cq + cd d/ds) F_n R_nm = Phi0_n R_nm + Phi1_n R'_nm,
//   Phi0 = cq F_n + cd F'_n, Phi1 = cd F_n,
// R and R' = dR/ds by the recurrence along n and its derivative: about 28 FP64
// instructions per (n, +-m) pair, where the ladder formula read seven table entries.
//   P2L: v = u / |u|, F_n = h_n, F'_n = -(k|u| / 2) h_{n+1} d|v|^2/ds
//   P2M: v = u / w (w the box width), F_n the power series of j_n(k w |v|) / |v|^n, cut at
//        total degree p in the reference's default truncation (its multipole moments),
//        F'_n its derivative
// Tiles of 16 sources, three steps: (0) a thread per source forms its direction and radial
// factors, serial recurrences; (1) thread (source, column m) runs its column into the wave
// table in shared memory; (2) the table times the densities on the FP64 tensor cores, 8
// coefficients x 4 sources x (4 densities, re / im), the warps splitting the coefficients.
// PIPE: eight warps do (2) of tile t and eight (1) of t + 1, the last of them, whose columns
// are the shortest, also (0) of t + 2, one barrier a tile; two wave tables fit up to order 15
// (198 KB).  Above, eight warps do (1) and
// (2) in turn, (0) of the next tile by one of them, another for each tile, at the start of
// (2).  In both every thread of (2) has the load of one strength of the next tile in flight.
// Bound by the FP64 pipe, which the products and the recurrences share: about 4100 + 2200
// cycles an SM and tile at 16 densities, of about 9900 taken.  P2L: 50 ms term by term ->
// 34.7 ms (307 200 nodes, 16 densities, order 15).
#include <algorithm>

#include "../../include/qbxfmm_api.h"
#include "helm3.cuh"
#include "kernels.h"

namespace qbx {

namespace {

constexpr int P2E_SUB = 16;                 // sources per tile
constexpr int P2E_NTHR = 256;
constexpr int P2E_NPIPE = 2 * P2E_NTHR;
constexpr int P2E_WS = P2E_SUB + 4;         // row stride of the wave table (complex)

// shared memory in double2: nw wave tables, recurrence table, two staged tiles
__host__ __device__ constexpr int p2e_stage(int p, int nt)
{
  return 2 * (p + 1) * P2E_SUB + P2E_SUB * (4 * nt + 2) + 4 * P2E_SUB;
}

__host__ __device__ constexpr int p2e_smem(int p, int nt, int nw)
{
  return nw * ((p + 1) * (p + 1) + 7) * P2E_WS + (p + 1) * (p + 2) / 2 + 2 * p2e_stage(p, nt);
}

template <bool LOCAL, int NT, int MT, bool PIPE>
__global__ void __launch_bounds__(PIPE ? P2E_NPIPE : P2E_NTHR, PIPE || MT > 4 ? 1 : 2)
k_h3_p2e_mma(qbxfmm_geometry g, HelmCoeffs hc, int p, int nrhs,
             const double2* __restrict__ strengths, double2* __restrict__ exps, int32_t* err)
{
  constexpr int NR = 4 * NT, SS = 8 * NT + 4;
  extern __shared__ double2 smem2[];
  __shared__ int s_pref[MAXB + 1], s_start[MAXB];
  const int ncf = (p + 1) * (p + 1), nrec = (p + 1) * (p + 2) / 2;
  const int nW = (ncf + 7) * P2E_WS;
  double2* W0 = smem2;                                  // [PIPE ? 2 : 1][ncf + 7][P2E_WS]
  double2* rec = W0 + (size_t)(PIPE ? 2 : 1) * nW;      // [nrec]
  double2* stage = rec + nrec;                          // [2]{Phi [p+1][2][SUB], sigma, dir}
  const int nst = p2e_stage(p, NT);

  int b, l0 = 0, l1 = 1;
  if (LOCAL) {
    b = g.target_or_target_parent_boxes[blockIdx.x];
    l0 = g.list4_starts[blockIdx.x];
    l1 = g.list4_starts[blockIdx.x + 1];
    if (l1 <= l0) return;
  } else {
    b = g.source_boxes[blockIdx.x];
  }
  const int r0 = blockIdx.y * NR;
  const double rho = level_width(g, g.box_levels[b]);
  double c[3];
  load_point<3>(g.box_centers, g.nboxes, b, c);
  const bool dip = hc.cd.x != 0.0 || hc.cd.y != 0.0;
  // PIPE: warps 0..7 step (2), 8..15 step (1), the last of them (with the shortest columns)
  // also step (0); tid and warp count within a role
  const int lane = threadIdx.x & 31;
  const int role = PIPE ? threadIdx.x / P2E_NTHR : 0;
  const int tid = threadIdx.x - role * P2E_NTHR, warp = tid >> 5;
  h3_rec_table(p, rec, threadIdx.x, blockDim.x);

  // this thread's strength of the tile [base, base + 16): source tid % 16, density tid / 16
  auto load_strength = [&](int base, int total, int nb, int s0) {
    const int j = tid & 15, r = tid >> 4;
    double2 v = c2(0.0);
    if (r < NR && base + j < total && r0 + r < nrhs) {
      const int s = LOCAL ? h3_stream_source(base + j, nb, s_pref, s_start) : s0 + base + j;
      v = __ldg(strengths + (size_t)(r0 + r) * g.nsources + s);
    }
    return v;
  };
  auto store_strength = [&](double2* st, double2 v) {
    const int j = tid & 15, r = tid >> 4;
    double* sig = reinterpret_cast<double*>(st + 2 * (p + 1) * P2E_SUB);   // [SUB][SS]
    if (r < NR) *reinterpret_cast<double2*>(sig + j * SS + 2 * r) = v;
  };
  // the radial factors and directions of tile [base, base + 16), by one warp
  auto prepare = [&](double2* st, int base, int total, int nb, int s0) {
    double2* Phi = st;                                             // [n][2][SUB]
    double* dir = reinterpret_cast<double*>(Phi + 2 * (p + 1) * P2E_SUB) + P2E_SUB * SS;  // [8][SUB]
    const int j = lane & 15;
    const bool on = base + j < total;
    int s = 0;
    if (on) s = LOCAL ? h3_stream_source(base + j, nb, s_pref, s_start) : s0 + base + j;
    if (lane >= 16) return;
    double u[3] = {0.0, 0.0, 1.0}, nv[3] = {0.0, 0.0, 0.0};
    if (on) {
      load_point<3>(g.sources, g.nsources, s, u);
#pragma unroll
      for (int d = 0; d < 3; ++d) u[d] -= c[d];
      if (dip) load_point<3>(g.source_normals, g.nsources, s, nv);
    }
    const double d2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
    const double li = LOCAL ? rsqrt_h(d2) : 1.0 / rho;             // 1 / length unit
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      u[d] *= li;
      nv[d] *= li;
      dir[d * P2E_SUB + j] = u[d];
      dir[(3 + d) * P2E_SUB + j] = nv[d];
    }
    const double c1 = 2.0 * (u[0] * nv[0] + u[1] * nv[1] + u[2] * nv[2]);
    const double r2 = LOCAL ? 1.0 : u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
    dir[6 * P2E_SUB + j] = r2;
    dir[7 * P2E_SUB + j] = c1;
    auto put = [&](int n, double2 f, double2 fp) {
      if (!on) f = fp = c2(0.0);
      Phi[(2 * n) * P2E_SUB + j] = dip ? cfma(hc.cd, fp, cmul(hc.cq, f)) : cmul(hc.cq, f);
      Phi[(2 * n + 1) * P2E_SUB + j] = dip ? cmul(hc.cd, f) : c2(0.0);
    };
    if (LOCAL) {
      const double x0 = hc.k * d2 * li, xi = 1.0 / x0;
      double sn, cs;
      sincos(x0, &sn, &cs);
      double2 h = c2(sn * xi, -cs * xi);
      double2 hn = c2((sn - cs * x0) * xi * xi, -(sn * x0 + cs) * xi * xi);
      const double fs = -0.5 * x0 * c1;
      for (int n = 0; n <= p; ++n) {
        put(n, h, cscale(fs, hn));
        const double f = (2.0 * n + 3.0) * xi;
        const double2 nx = c2(f * hn.x - h.x, f * hn.y - h.y);
        h = hn;
        hn = nx;
      }
    } else {
      const double kap = hc.k * rho, x2 = kap * kap * r2, mh = -0.5 * kap * kap * c1;
      if (hc.taylor || x2 < 0.25) {
        double lead = 1.0;                                          // kap^n / (2n+1)!!
        for (int n = 0; n <= p; ++n) {
          // sum_j t_j, and its derivative in r2: -(kap^2 / 2) sum_j t_j / (2n + 2j + 3)
          const int jm = hc.taylor ? (p - n) / 2 : 12;
          double t = lead, f = 0.0, fd = 0.0;
          for (int i = 0; i <= jm; ++i) {
            f += t;
            const double q = t * rcp(2 * n + 2 * i + 3);
            if (i < jm) fd += q;
            t = -0.5 * x2 * q * rcp(i + 1);
          }
          put(n, c2(f), c2(mh * fd));
          lead *= kap * rcp(2 * n + 3);
        }
      } else {
        double jv[H3_LMAX + 2];
        const double v = sqrt(r2), vi = 1.0 / v;
        h3_sph_j(p + 1, kap * v, jv);
        double f = 1.0;
        for (int n = 0; n <= p; ++n, f *= vi)
          put(n, c2(f * jv[n]), c2(-0.5 * kap * c1 * f * vi * jv[n + 1]));
      }
    }
  };

  double acc[MT][NT][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[i][n][0] = acc[i][n][1] = 0.0;
  const int row = lane >> 2, kq = lane & 3;
  const int ntile = (ncf + 7) >> 3;

  // step (1): the wave table of a staged tile
  auto waves = [&](const double2* st, double2* W) {
    const double2* Phi = st;
    const double* dir = reinterpret_cast<const double*>(Phi + 2 * (p + 1) * P2E_SUB) + P2E_SUB * SS;
    const int j = tid & 15;
    const double z = dir[2 * P2E_SUB + j], z1 = dir[5 * P2E_SUB + j];
    const double r2 = dir[6 * P2E_SUB + j], c1 = dir[7 * P2E_SUB + j];
    const double2 X = c2(dir[j], dir[P2E_SUB + j]);
    const double2 X1 = c2(dir[3 * P2E_SUB + j], dir[4 * P2E_SUB + j]);
    for (int m = tid >> 4; m <= p; m += P2E_NTHR / P2E_SUB) {
      // start c X^m and its derivative c m X^{m-1} X', the power by squaring
      double2 a = c2(rec[idx3(m, m)].x), a1 = c2(0.0);
      if (m > 0) {
        double2 b = X;
        for (int e = m - 1; e > 0; e >>= 1, b = cmul(b, b))
          if (e & 1) a = cmul(a, b);
        a1 = cscale((double)m, cmul(a, X1));
        a = cmul(a, X);
      }
      double2 pa = c2(0.0), pa1 = c2(0.0);
      for (int n = m; n <= p; ++n) {
        const double2 f0 = Phi[(2 * n) * P2E_SUB + j], f1 = Phi[(2 * n + 1) * P2E_SUB + j];
        const double2 P = caxpy(a1.x, f1, cscale(a.x, f0));
        const double2 Qv = caxpy(a1.y, f1, cscale(a.y, f0));
        const int o = n * n + n;
        W[(o + m) * P2E_WS + j] = c2(P.x + Qv.y, P.y - Qv.x);         // wave -m
        if (m > 0) W[(o - m) * P2E_WS + j] = c2(P.x - Qv.y, P.y + Qv.x);
        if (n == p) break;
        const double2 ab = rec[idx3(n + 1, m)];
        const double az = ab.x * z, bb = -ab.x * ab.y, br = bb * r2;
        const double2 na = caxpy(br, pa, cscale(az, a));
        double2 n1 = caxpy(br, pa1, cscale(az, a1));
        n1 = caxpy(ab.x * z1, a, caxpy(bb * c1, pa, n1));
        pa = a;
        pa1 = a1;
        a = na;
        a1 = n1;
      }
    }
  };
  // step (2): its product with the densities
  auto product = [&](const double2* st, const double2* W) {
    const double* sig = reinterpret_cast<const double*>(st + 2 * (p + 1) * P2E_SUB);
#pragma unroll
    for (int ks = 0; ks < P2E_SUB / 4; ++ks) {
      const double* B = sig + (4 * ks + kq) * SS;
      double bv[NT], bx[NT];
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        bv[n] = B[8 * n + row];
        const double x = B[8 * n + (row ^ 1)];
        bx[n] = (row & 1) ? x : -x;
      }
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const int tl = warp + 8 * i;
        if (tl >= ntile) break;
        const double2 w = W[(8 * tl + row) * P2E_WS + 4 * ks + kq];
#pragma unroll
        for (int n = 0; n < NT; ++n) h3_dmma(acc[i][n][0], acc[i][n][1], w.x, bv[n]);
#pragma unroll
        for (int n = 0; n < NT; ++n) h3_dmma(acc[i][n][0], acc[i][n][1], w.y, bx[n]);
      }
    }
  };

  for (int gb = l0; gb < l1; gb += LOCAL ? MAXB : 1) {
    int nb = 0, total, s0 = 0;
    __syncthreads();
    if (LOCAL) {
      nb = min(MAXB, l1 - gb);
      h3_list_prefix(g, g.list4_lists, gb, nb, s_pref, s_start, err);
      __syncthreads();
      total = s_pref[nb];
    } else {
      total = g.box_source_counts_nonchild[b];
      s0 = g.box_source_starts[b];
    }
    if constexpr (PIPE) {
      const int nt = (total + P2E_SUB - 1) / P2E_SUB;
      if (role == 0 && nt > 0) store_strength(stage, load_strength(0, total, nb, s0));
      // tile t: (0) at t - 2, (1) at t - 1, (2) at t; buffers by the parity of the tile
      for (int t = -2; t < nt; ++t) {
        if (role == 1) {
          if (warp == 7 && t + 2 < nt)
            prepare(stage + (t & 1) * nst, (t + 2) * P2E_SUB, total, nb, s0);
          if (t + 1 >= 0 && t + 1 < nt)
            waves(stage + ((t + 1) & 1) * nst, W0 + (size_t)((t + 1) & 1) * nW);
        }
        if (role == 0 && t >= 0) {
          const bool more = t + 1 < nt;
          double2 nxt = c2(0.0);
          if (more) nxt = load_strength((t + 1) * P2E_SUB, total, nb, s0);
          product(stage + (t & 1) * nst, W0 + (size_t)(t & 1) * nW);
          if (more) store_strength(stage + ((t + 1) & 1) * nst, nxt);
        }
        __syncthreads();
      }
    } else {
      if (total > 0) {
        store_strength(stage, load_strength(0, total, nb, s0));
        if (warp == 0) prepare(stage, 0, total, nb, s0);
      }
      int buf = 0, turn = 0;
      for (int base = 0; base < total; base += P2E_SUB, buf ^= 1) {
        __syncthreads();       // this tile is staged; the table and the other buffer are free
        waves(stage + buf * nst, W0);
        __syncthreads();       // the table is complete
        const bool more = base + P2E_SUB < total;
        double2 nxt = c2(0.0);
        if (more) {
          nxt = load_strength(base + P2E_SUB, total, nb, s0);
          if (warp == turn) prepare(stage + (buf ^ 1) * nst, base + P2E_SUB, total, nb, s0);
        }
        turn = (turn + 1) & 7;
        product(stage + buf * nst, W0);
        if (more) store_strength(stage + (buf ^ 1) * nst, nxt);
      }
    }
  }
  if (role != 0) return;
  const double sc = h3_scale(hc.k, rho);
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int ci = 8 * (warp + 8 * i) + row;
    if (ci >= ncf) continue;
    int n, m;
    hq_decode(ci, n, m);
    const double f = FOUR_PI * hc.k * (LOCAL ? pow(sc, (double)n) : pow(sc, -(double)n));
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int r = r0 + 4 * nt + kq;
      if (r >= nrhs) continue;
      // 4 pi i k f acc
      double2* E = exps + ((size_t)b * nrhs + r) * ncf + ci;
      *E = cadd(*E, c2(-f * acc[i][nt][1], f * acc[i][nt][0]));
    }
  }
}

template <bool LOCAL, int NT, int MT, bool PIPE>
cudaError_t p2e_launch(int nbox, const qbxfmm_geometry& g, HelmCoeffs hc, int p, int nrhs,
                       const double2* s, double2* exps, int32_t* err, cudaStream_t st)
{
  const size_t sh = (size_t)p2e_smem(p, NT, PIPE ? 2 : 1) * sizeof(double2);
  auto k = k_h3_p2e_mma<LOCAL, NT, MT, PIPE>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  if (e != cudaSuccess) return e;
  k<<<dim3(nbox, (nrhs + 4 * NT - 1) / (4 * NT)), PIPE ? P2E_NPIPE : P2E_NTHR, sh, st>>>(
      g, hc, p, nrhs, s, exps, err);
  return cudaGetLastError();
}

template <bool LOCAL>
cudaError_t p2e(int nbox, const qbxfmm_geometry& g, HelmCoeffs hc, int p, int nrhs,
                const double2* s, double2* exps, int32_t* err, cudaStream_t st)
{
  if (nbox == 0) return cudaSuccess;
  if (p > H3_MAXP) return cudaErrorInvalidValue;
  if (hc.rb_p2e == 16 && p > 15) return cudaErrorInvalidValue;
  const int want = hc.rb_p2e > 0 ? hc.rb_p2e : nrhs;    // the plan's tuning, else by nrhs
  // Order 15 and below (32 tiles of 8 coefficients).  PIPE up to 8 densities, where (1) is the
  // longer step (P2L of 1 density 2.58 -> 2.20 ms, of 6 1.34 -> 1.17 ms, 24 300 and 19 200
  // nodes); above, (2) is, and two CTAs of eight warps hide its latency better than one of
  // eight beside eight (34.7 against 38.6 ms, 16 densities, 307 200 nodes).
  if (p <= 15) {
    if (want > 8) return p2e_launch<LOCAL, 4, 4, false>(nbox, g, hc, p, nrhs, s, exps, err, st);
    if (want > 4) return p2e_launch<LOCAL, 2, 4, true>(nbox, g, hc, p, nrhs, s, exps, err, st);
    return p2e_launch<LOCAL, 1, 4, true>(nbox, g, hc, p, nrhs, s, exps, err, st);
  }
  if (want > 8) return p2e_launch<LOCAL, 4, 6, false>(nbox, g, hc, p, nrhs, s, exps, err, st);
  if (want > 4) return p2e_launch<LOCAL, 2, 6, false>(nbox, g, hc, p, nrhs, s, exps, err, st);
  return p2e_launch<LOCAL, 1, 6, false>(nbox, g, hc, p, nrhs, s, exps, err, st);
}

}  // namespace

cudaError_t h3_launch_p2m(const qbxfmm_geometry& g, HelmCoeffs hc, int p, int nrhs,
                          const double2* s, double2* mp, cudaStream_t st)
{
  return p2e<false>(g.nsource_boxes, g, hc, p, nrhs, s, mp, nullptr, st);
}

cudaError_t h3_launch_p2l(const qbxfmm_geometry& g, HelmCoeffs hc, int p, int nrhs,
                          const double2* s, double2* lo, int32_t* err, cudaStream_t st)
{
  return p2e<true>(g.nttp_boxes, g, hc, p, nrhs, s, lo, err, st);
}

}  // namespace qbx
