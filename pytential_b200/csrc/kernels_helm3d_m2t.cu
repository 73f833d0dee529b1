// 3D Helmholtz: list-3 multipoles straight to the QBX targets, complex128, sm_100a.
//
// M2QBXL followed by QBXL2P is, per (target, its center, list-3 box), a linear
// functional of the box's multipole that no density enters.  Translating forms it once
// per density (a rotation, a coaxial translation and a back rotation of 256
// coefficients at order 15); here it is formed once as a row of weights and applied to
// the densities as a product.  The QBX local of order Q cut to its power series is the
// degree-Q Taylor polynomial about the center, so its value at the target t = c + a is
//   sum_{i <= Q} [s^i] u(c + s a),   u(x) = sum M_nm s_b^n h_n(k|x - x_b|) Y_nm(x - x_b):
// a truncated power series in one variable.  With e = (c - x_b)/d, eta = a/d,
// d = |c - x_b|, v(s) = e + s eta and x0 = k d,
//   h_n(k d|v|) Y_nm(v) = F_n(s) R_nm(s),  R_nm = |v|^n Y_nm(v)  (a polynomial in v),
//   F_n = h_n(x0 |v|) / |v|^n,             dF_n / d(|v|^2) = -(x0 / 2) F_{n+1},
// hence F_n(s) = sum_i h_{n+i}(x0) (-x0 / 2)^i (|v|^2 - 1)^i / i!, with
// |v|^2 - 1 = 2 (e.eta) s + |eta|^2 s^2, and the weight of M_nm is
//   w_nm = s_b^n sum_{i + j <= Q} g_{i+j} [s^i] R_nm [s^j] F_n = sum_i [s^i] R_nm Phi_{n,i}.
// g = 1 gives the cut series (the reference's default truncation).  Spherical waves
// sum_n j_n(k|a|) Lambda_n (fmmlib) have the same Taylor coefficients about the center,
// b_t = sum_{n + 2j = t} alpha_nj (k|a|)^t Lambda_n with j_n(x) = sum_j alpha_nj
// x^{n+2j}, and sum_n j_n Lambda_n = sum_t g_t b_t, g from back substitution.
// R_nm along n follows R_{n+1} = a_nm (v_z R_n - b_nm |v|^2 R_{n-1}) on truncated series.
#include <algorithm>

#include "../../include/qbxfmm_api.h"
#include "helm3.cuh"
#include "kernels.h"

namespace qbx {

namespace {

constexpr int M2T_NT = 128;
constexpr int M2T_TG = 8;     // targets per warp

// shared memory of one warp (in double2): Phi, the fourth power, and the radial values or,
// once Phi is formed, the series E of each lane
__host__ __device__ constexpr size_t m2t_he(int pf, int q)
{
  return M2T_TG * (pf + q + 1) > 32 * (q + 1) ? M2T_TG * (pf + q + 1) : 32 * (q + 1);
}

__host__ __device__ constexpr size_t m2t_warp_smem(int pf, int q)
{
  return (size_t)M2T_TG * ((pf + 1) * (q + 1) + (q + 1)) + m2t_he(pf, q);
}

// A CTA holds one octet of a chunk's targets; its four warps split the list-3 boxes
// (fixed-order sum at the end), so that one long list is spread over four warps.
// A warp holds 8 targets x 4 lanes: lane l carries target l / 4 and the columns
// m = 4 j + l % 4 (both signs).  At each (j, n) a lane's weights w_{n,m} and w_{n,-m} are,
// as they stand, the A fragment of an 8 x 4 FP64 tensor-core product (row = target,
// inner index = column), whose B fragment is the box's M_{n,+-m} of 8 densities: DG
// groups of 8 densities (MMA), or DG densities by plain multiply-adds and a sum over
// the four lanes at the end.
// OFF: M2P at the non-QBX targets (eval_multipoles), each its own center, Q = 0.
template <int Q, int DG, bool MMA, bool OFF>
__global__ void __launch_bounds__(M2T_NT, 3)
k_h3_m2t(qbxfmm_geometry g, HelmCoeffs hc, int pf, int nrhs, const double2* __restrict__ mpoles,
         double2* __restrict__ pot, int32_t* err)
{
  static_assert(!OFF || Q == 0);
  extern __shared__ double2 smem2[];
  const int ncf = (pf + 1) * (pf + 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tg = lane >> 2, kq = lane & 3;
  double2* rec = smem2;                                          // [(pf+1)(pf+2)/2]
  const int nrec = (pf + 1) * (pf + 2) / 2;
  double2* Phi = smem2 + nrec + (size_t)warp * m2t_warp_smem(pf, Q);   // [n][i][target]
  double2* P4 = Phi + (size_t)M2T_TG * (pf + 1) * (Q + 1) + tg;  // [i][target]
  double2* H = P4 - tg + M2T_TG * (Q + 1);                       // [n][target]
  double2* E = H + lane;                                         // [i][lane]
  constexpr int NWARP = M2T_NT / 32, OCT = QBXFMM_CENTER_CHUNK / M2T_TG;
  const int chunk = blockIdx.x / OCT, oct = blockIdx.x - chunk * OCT;
  const int itb = (OFF ? g.nonqbx_chunk_target_box : g.tsqbx_chunk_target_box)[chunk];
  const int cnt = (OFF ? g.nonqbx_chunk_count : g.tsqbx_chunk_count)[chunk];
  if (oct * M2T_TG >= cnt) return;
  const int l0 = g.list3_starts[itb], l1 = g.list3_starts[itb + 1];
  if (l1 <= l0) return;
  h3_rec_table(pf, rec, threadIdx.x, M2T_NT);
  __syncthreads();
  const int ti = oct * M2T_TG + tg;
  const int pi = (OFF ? g.nonqbx_chunk_start : g.tsqbx_chunk_start)[chunk] + min(ti, cnt - 1);
  bool active = ti < cnt;
  int t = pi;
  double cc[3], a[3] = {0.0, 0.0, 0.0};
  if (OFF) {
    load_point<3>(g.nonqbx_targets, g.nfiltered_targets, t, cc);
  } else {
    t = g.tsqbx_targets[pi];
    int ctr = g.tsqbx_centers[pi];
    if ((unsigned)ctr >= (unsigned)g.ncenters || (unsigned)t >= (unsigned)g.ntargets) {
      report(err, QBX_DEVERR_BAD_CENTER);
      active = false;
      t = ctr = 0;
    }
    load_point<3>(g.centers, g.ncenters, ctr, cc);
    load_point<3>(g.targets, g.ntargets, t, a);
#pragma unroll
    for (int d = 0; d < 3; ++d) a[d] -= cc[d];
  }
  const int r0 = blockIdx.y * (MMA ? 8 * DG : DG);
  double gw[Q + 1];
  m2t_taylor_weights<Q>(hc.taylor != 0, hc.k * sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]), gw);

  double vre[DG][2], vim[DG][2];     // MMA: two densities per lane and group; else [.][0]
#pragma unroll
  for (int d = 0; d < DG; ++d) vre[d][0] = vre[d][1] = vim[d][0] = vim[d][1] = 0.0;

  for (int li = l0 + warp; li < l1; li += NWARP) {
    const int sb = g.list3_lists[li];
    if ((unsigned)sb >= (unsigned)g.nboxes) {
      report(err, QBX_DEVERR_BAD_BOX);
      continue;
    }
    double cb[3];
    load_point<3>(g.box_centers, g.nboxes, sb, cb);
    const double sc = h3_scale(hc.k, level_width(g, g.box_levels[sb]));
    double e[3] = {cc[0] - cb[0], cc[1] - cb[1], cc[2] - cb[2]};
    const double dist = sqrt(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]);
    const double di = 1.0 / dist, x0 = hc.k * dist;
    double eta[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      e[d] *= di;
      eta[d] = a[d] * di;
    }
    const double c1 = 2.0 * (e[0] * eta[0] + e[1] * eta[1] + e[2] * eta[2]);
    const double c2s = eta[0] * eta[0] + eta[1] * eta[1] + eta[2] * eta[2];
    // h_n(x0), n <= pf + Q: every lane of a target runs the recurrence, lane n % 4 stores
    __syncwarp();
    {
      double s, c;
      sincos(x0, &s, &c);
      const double xi = 1.0 / x0;
      double2 hm = c2(s * xi, -c * xi), hn = c2((s - c * x0) * xi * xi, -(s * x0 + c) * xi * xi);
      double f = xi;
      for (int n = 0; n <= pf + Q; ++n) {
        if ((n & 3) == kq) H[n * M2T_TG + tg] = hm;
        f += 2.0 * xi;                                   // (2n + 3) / x0
        const double2 nx = c2(f * hn.x - hm.x, f * hn.y - hm.y);
        hm = hn;
        hn = nx;
      }
    }
    __syncwarp();
    {
      // D[i][i'] = sum_u g_{i'+i+u} d_i[u], d_i[u] the coefficient of s^{i+u} in
      // (-x0/2)^i (|v|^2 - 1)^i / i!;  Phi_{n,i'} = s_b^n sum_i h_{n+i} D[i][i']
      double D[Q + 1][Q + 1];
      double dc[Q + 1];
#pragma unroll
      for (int u = 0; u <= Q; ++u) dc[u] = u == 0 ? 1.0 : 0.0;
#pragma unroll
      for (int i = 0; i <= Q; ++i) {
        if (i > 0) {
          const double f = -0.5 * x0 * rcp(i), f1 = f * c1, f2 = f * c2s;
#pragma unroll
          for (int u = Q; u >= 1; --u) dc[u] = fma(f1, dc[u], f2 * dc[u - 1]);
          dc[0] *= f1;
        }
#pragma unroll
        for (int ip = 0; ip + i <= Q; ++ip) {
          double v = 0.0;
#pragma unroll
          for (int u = 0; u <= i; ++u)
            if (ip + i + u <= Q) v = fma(gw[ip + i + u], dc[u], v);
          D[i][ip] = v;
        }
      }
      double sn = 1.0;
      for (int i = 0; i < kq; ++i) sn *= sc;
      const double s4 = (sc * sc) * (sc * sc);
      for (int n = kq; n <= pf; n += 4, sn *= s4) {
        double2 ph[Q + 1];
#pragma unroll
        for (int ip = 0; ip <= Q; ++ip) ph[ip] = c2(0.0);
#pragma unroll
        for (int i = 0; i <= Q; ++i) {
          const double2 h = H[(n + i) * M2T_TG + tg];
#pragma unroll
          for (int ip = 0; ip + i <= Q; ++ip) ph[ip] = caxpy(D[i][ip], h, ph[ip]);
        }
#pragma unroll
        for (int ip = 0; ip <= Q; ++ip) Phi[(n * (Q + 1) + ip) * M2T_TG + tg] = cscale(sn, ph[ip]);
      }
    }
    __syncwarp();

    // E = ((e_x + i e_y) + s (eta_x + i eta_y))^m as a truncated series: m = kq, then by
    // the fourth power from one group of columns to the next
    const double2 X0 = c2(e[0], e[1]), X1 = c2(eta[0], eta[1]);
    {
      double2 W[Q + 1];
#pragma unroll
      for (int i = 0; i <= Q; ++i) W[i] = c2(i == 0 ? 1.0 : 0.0);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (u == kq) {
#pragma unroll
          for (int i = 0; i <= Q; ++i) E[i * 32] = W[i];
        }
#pragma unroll
        for (int i = Q; i >= 1; --i) W[i] = cfma(X0, W[i], cmul(X1, W[i - 1]));
        W[0] = cmul(X0, W[0]);
      }
      if (kq == 0) {
#pragma unroll
        for (int i = 0; i <= Q; ++i) P4[i * M2T_TG] = W[i];
      }
    }
    __syncwarp();
    const double2* Mb = mpoles + ((size_t)sb * nrhs + r0) * ncf;
    for (int j = 0; 4 * j <= pf; ++j) {
      const int m = 4 * j + kq;
      const double cm = m <= pf ? rec[idx3(m, m)].x : 0.0;
      double2 cur[Q + 1], prev[Q + 1];
#pragma unroll
      for (int i = 0; i <= Q; ++i) cur[i] = prev[i] = c2(0.0);
      double2 mp[DG], mm[DG];
      auto fetch = [&](int n) {
        const int o = n * n + n;
#pragma unroll
        for (int d = 0; d < DG; ++d) {
          const int r = MMA ? 8 * d + tg : d;
          const bool ok = m <= n && r0 + r < nrhs;
          mp[d] = ok ? __ldg(Mb + (size_t)r * ncf + o + m) : c2(0.0);
          mm[d] = ok && m > 0 ? __ldg(Mb + (size_t)r * ncf + o - m) : c2(0.0);
        }
      };
      fetch(4 * j);
#pragma unroll 1
      for (int n = 4 * j; n <= pf; ++n) {
        if (n == m) {
#pragma unroll
          for (int i = 0; i <= Q; ++i) cur[i] = cscale(cm, E[i * 32]);
        }
        double2 p = c2(0.0), q = c2(0.0);
#pragma unroll
        for (int i = 0; i <= Q; ++i) {
          const double2 ph = Phi[(n * (Q + 1) + i) * M2T_TG + tg];
          p = caxpy(cur[i].x, ph, p);
          q = caxpy(cur[i].y, ph, q);
        }
        const double2 wp = c2(p.x - q.y, p.y + q.x), wm = c2(p.x + q.y, p.y - q.x);
        double2 bp[DG], bm[DG];
#pragma unroll
        for (int d = 0; d < DG; ++d) {
          bp[d] = mp[d];
          bm[d] = mm[d];
        }
        if (n < pf) {
          fetch(n + 1);
          const double2 ab = rec[idx3(n + 1, min(m, n + 1))];
          const double z0 = ab.x * e[2], z1 = ab.x * eta[2], b = -ab.x * ab.y;
#pragma unroll
          for (int i = Q; i >= 0; --i) {
            double2 u = prev[i];
            if (i >= 1) u = caxpy(c1, prev[i - 1], u);
            if (i >= 2) u = caxpy(c2s, prev[i - 2], u);
            double2 v = cscale(b, u);
            v = caxpy(z0, cur[i], v);
            if (i >= 1) v = caxpy(z1, cur[i - 1], v);
            prev[i] = v;       // read above only at lower orders from here on
          }
#pragma unroll
          for (int i = 0; i <= Q; ++i) {
            const double2 v = prev[i];
            prev[i] = cur[i];
            cur[i] = v;
          }
        }
#pragma unroll
        for (int d = 0; d < DG; ++d) {
          if constexpr (MMA) {
            h3_dmma(vre[d][0], vre[d][1], wp.x, bp[d].x);
            h3_dmma(vim[d][0], vim[d][1], wp.x, bp[d].y);
            h3_dmma(vre[d][0], vre[d][1], -wp.y, bp[d].y);
            h3_dmma(vim[d][0], vim[d][1], wp.y, bp[d].x);
            h3_dmma(vre[d][0], vre[d][1], wm.x, bm[d].x);
            h3_dmma(vim[d][0], vim[d][1], wm.x, bm[d].y);
            h3_dmma(vre[d][0], vre[d][1], -wm.y, bm[d].y);
            h3_dmma(vim[d][0], vim[d][1], wm.y, bm[d].x);
          } else {
            double2 v = c2(vre[d][0], vim[d][0]);
            v = cfma(wm, bm[d], cfma(wp, bp[d], v));
            vre[d][0] = v.x;
            vim[d][0] = v.y;
          }
        }
      }
      if (4 * j + 4 <= pf) {
#pragma unroll
        for (int i = Q; i >= 0; --i) {
          double2 v = cmul(P4[0], E[i * 32]);
#pragma unroll
          for (int u = 1; u <= i; ++u) v = cfma(P4[u * M2T_TG], E[(i - u) * 32], v);
          E[i * 32] = v;
        }
      }
    }
  }
  // sum over the warps (the warps' scratch is free)
  __syncthreads();
  double2* red = smem2 + nrec;                 // [NWARP][2 DG or DG][32]
  constexpr int NV = MMA ? 2 * DG : DG;
#pragma unroll
  for (int d = 0; d < NV; ++d) {
    double2 v = MMA ? c2(vre[d / 2][d & 1], vim[d / 2][d & 1]) : c2(vre[d % DG][0], vim[d % DG][0]);
    if constexpr (!MMA) {                      // and over the four lanes of a target
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
    }
    red[(warp * NV + d) * 32 + lane] = v;
  }
  __syncthreads();
  for (int d = warp; d < NV; d += NWARP) {
    const int r = MMA ? r0 + 8 * (d / 2) + 2 * kq + (d & 1) : r0 + d;
    if (!active || r >= nrhs || (!MMA && kq != 0)) continue;
    double2 v = red[d * 32 + lane];
    for (int w = 1; w < NWARP; ++w) v = cadd(v, red[(w * NV + d) * 32 + lane]);
    double2* P = pot + (size_t)r * (OFF ? g.nfiltered_targets : g.ntargets) + t;
    *P = cadd(*P, v);
  }
}

template <int Q, int DG, bool MMA, bool OFF>
cudaError_t m2t_launch(const qbxfmm_geometry& g, HelmCoeffs hc, int pf, int nrhs,
                       const double2* mp, double2* pot, int32_t* err, cudaStream_t st)
{
  constexpr int ND = MMA ? 8 * DG : DG;
  const size_t scratch = std::max(m2t_warp_smem(pf, Q), (size_t)(MMA ? 2 * DG : DG) * 32);
  const size_t sh = ((size_t)(pf + 1) * (pf + 2) / 2 + (M2T_NT / 32) * scratch) * sizeof(double2);
  cudaError_t e = cudaFuncSetAttribute(k_h3_m2t<Q, DG, MMA, OFF>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  if (e != cudaSuccess) return e;
  const int chunks = OFF ? g.nnonqbx_chunks : g.ntsqbx_chunks;
  dim3 grid(chunks * (QBXFMM_CENTER_CHUNK / M2T_TG), (nrhs + ND - 1) / ND);
  k_h3_m2t<Q, DG, MMA, OFF><<<grid, M2T_NT, sh, st>>>(g, hc, pf, nrhs, mp, pot, err);
  return cudaGetLastError();
}

template <int Q, bool OFF = false>
cudaError_t m2t_q(const qbxfmm_geometry& g, HelmCoeffs hc, int pf, int nrhs, const double2* mp,
                  double2* pot, int32_t* err, cudaStream_t st)
{
  // a tensor-core group of 8 densities costs as much as 8 plain ones: plain for the few
  if (nrhs > 8) return m2t_launch<Q, 2, true, OFF>(g, hc, pf, nrhs, mp, pot, err, st);
  if (nrhs > 4) return m2t_launch<Q, 1, true, OFF>(g, hc, pf, nrhs, mp, pot, err, st);
  if (nrhs > 2) return m2t_launch<Q, 4, false, OFF>(g, hc, pf, nrhs, mp, pot, err, st);
  if (nrhs > 1) return m2t_launch<Q, 2, false, OFF>(g, hc, pf, nrhs, mp, pot, err, st);
  return m2t_launch<Q, 1, false, OFF>(g, hc, pf, nrhs, mp, pot, err, st);
}

}  // namespace

// Bound by the FP64 pipe at the ladder's recurrences.  One warp per chunk and list-3 quarter
// with the whole ladder in one lane per target took 825 us for 1500 points beside 24 300
// nodes at order 15 (too few warps); 555 us here.
cudaError_t h3_launch_eval_multipoles(const qbxfmm_geometry& g, HelmCoeffs hc, int p, int nrhs,
                                      const double2* mp, double2* pot, int32_t* err, cudaStream_t st)
{
  if (g.nnonqbx_chunks == 0) return cudaSuccess;
  if (p > H3_MAXP) return cudaErrorInvalidValue;
  return m2t_q<0, true>(g, hc, p, nrhs, mp, pot, err, st);
}

bool h3_m2t_wins(const qbxfmm_geometry& g)
{
  return g.ntsqbx_chunks > 0 && g.ntsqbx_chunks <= 8 * g.nqbx_chunks;
}

cudaError_t h3_launch_m2t(const qbxfmm_geometry& g, HelmCoeffs hc, int pf, int q, int nrhs,
                          const double2* mp, double2* pot_tree, int32_t* err, cudaStream_t st)
{
  if (g.ntsqbx_chunks == 0) return cudaSuccess;
  if (pf > H3_MAXP) return cudaErrorInvalidValue;
  switch (q) {
    case 0: return m2t_q<0>(g, hc, pf, nrhs, mp, pot_tree, err, st);
    case 1: return m2t_q<1>(g, hc, pf, nrhs, mp, pot_tree, err, st);
    case 2: return m2t_q<2>(g, hc, pf, nrhs, mp, pot_tree, err, st);
    case 3: return m2t_q<3>(g, hc, pf, nrhs, mp, pot_tree, err, st);
    case 4: return m2t_q<4>(g, hc, pf, nrhs, mp, pot_tree, err, st);
    case 5: return m2t_q<5>(g, hc, pf, nrhs, mp, pot_tree, err, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace qbx
