// 3D Helmholtz target-specific near field (eval_target_specific_qbx_locals,
// pytential/qbx/fmm.py:391-394; the reference's native module
// pytential/qbx/target_specific/impl.pyx:363-563), complex128, sm_100a.
//
// Per (target t, its center c, list-1 source y), a = t - c, b = y - c, the order-Q QBX
// expansion of the source evaluated at the target without forming it: the Taylor
// coefficients b_t of e^{ikr}/r along the line from c to t, weighted by g_t
// (m2t_taylor_weights: 1 for the reference's default truncation).  With x0 = k|b|,
// x = (a.b)/|b|^2, z = -|a|^2 / (2 |b|^2), X = x0 x, Z = x0 z,
//   K_S = ik sum_i h_i(x0) W_i,
//   K_D = -(i k^2 / |b|) sum_i h_{i+1}(x0) ((b.nu) W_i - (a.nu) W'_i),
//   W_i  = sum_{u <= Q - i}     g_{i+u}   C(i,u) X^{i-u} Z^u / i!,
//   W'_i = sum_{u <= Q - 1 - i} g_{i+1+u} C(i,u) X^{i-u} Z^u / i!:
// real polynomials of two ratios beside one Hankel recurrence (the Legendre form took
// three complex sums with two recurrences, about 230 FP64 instructions a pair; this
// takes about 150).
//
// A warp holds one octet of the chunk's targets x 4 sources: lane l evaluates the pair
// (target l / 4, source l % 4), which is the A fragment of an FP64 tensor-core product
// with the sources' strengths, columns (density, re / im), as in the M2L kernel.  The
// products run on the tensor pipe beside the FP64 pipe, which bounds the kernel.  Source
// tiles are double buffered with cp.async.
#include <algorithm>

#include "../../include/qbxfmm_api.h"
#include "helm3.cuh"
#include "kernels.h"

namespace qbx {

namespace {

constexpr int NEAR_NT = 128;
constexpr int NEAR_TS = 64;      // sources per tile, two tiles staged

// C(i, u) / i! = 1 / (u! (i - u)!)
constexpr double near_c(int i, int u)
{
  double v = 1.0;
  for (int k = 2; k <= u; ++k) v /= k;
  for (int k = 2; k <= i - u; ++k) v /= k;
  return v;
}

template <int Q>
struct NearC {
  double c[Q + 1][Q + 1];
};

template <int Q>
constexpr NearC<Q> near_table()
{
  NearC<Q> t{};
  for (int i = 0; i <= Q; ++i)
    for (int u = 0; u <= i; ++u) t.c[i][u] = near_c(i, u);
  return t;
}

// sum_{u <= U} C(i,u)/i! g_{i+o+u} X^{i-u} Z^u; zp[u] = Z^u
template <int Q, bool CUT>
QBX_D double near_w(int i, int U, int o, double X, const double* zp, const double* gw)
{
  constexpr NearC<Q> C = near_table<Q>();
  double r = CUT ? C.c[i][0] : C.c[i][0] * gw[i + o];
#pragma unroll
  for (int u = 1; u <= Q; ++u) {
    if (u > U || u > i) break;
    const double c = CUT ? C.c[i][u] : C.c[i][u] * gw[i + o + u];
    r = fma(r, X, c * zp[u]);
  }
#pragma unroll
  for (int e = 0; e < Q; ++e)          // X^{i - U}
    if (e < i - U) r *= X;
  return r;
}

QBX_D void near_cp16(void* dst, const void* src, bool on)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(on ? 16 : 0)
               : "memory");
}

QBX_D void near_cp8(void* dst, const void* src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

template <int Q, int NT, bool CUT>
__global__ void __launch_bounds__(NEAR_NT)
k_h3_near(qbxfmm_geometry g, HelmCoeffs hc, int nrhs, const double2* __restrict__ strengths,
          double2* __restrict__ pot_tree, int32_t* err)
{
  constexpr int SS = 8 * NT + 4;                 // row stride of the strengths (doubles)
  constexpr int NR = 4 * NT;
  constexpr int TILE = NEAR_TS * (SS + 6);       // strengths [TS][SS], y and nu [6][TS]
  extern __shared__ double2 smem2[];
  double* tiles = reinterpret_cast<double*>(smem2);              // [2][TILE]
  __shared__ int s_src[2][NEAR_TS];
  __shared__ int s_pref[MAXB + 1], s_start[MAXB];
  const int chunk = blockIdx.x, r0 = blockIdx.y * NR;
  const int itb = g.tsqbx_chunk_target_box[chunk];
  const int cnt = g.tsqbx_chunk_count[chunk], i0 = g.tsqbx_chunk_start[chunk];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = lane >> 2, kq = lane & 3;
  const bool busy = 8 * warp < cnt;              // this warp's octet exists
  bool active = 8 * warp + row < cnt;
  const int pi = i0 + max(0, min(8 * warp + row, cnt - 1));
  int t = g.tsqbx_targets[pi], ctr = g.tsqbx_centers[pi];
  if ((unsigned)ctr >= (unsigned)g.ncenters || (unsigned)t >= (unsigned)g.ntargets) {
    report(err, QBX_DEVERR_BAD_CENTER);
    active = false;
    t = ctr = 0;
  }
  double cc[3], a[3];
  load_point<3>(g.centers, g.ncenters, ctr, cc);
  load_point<3>(g.targets, g.ntargets, t, a);
#pragma unroll
  for (int d = 0; d < 3; ++d) a[d] -= cc[d];
  const double aa = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
  double gw[Q + 1];
  m2t_taylor_weights<Q>(CUT, hc.k * sqrt(aa), gw);
  const bool chg = hc.cq.x != 0.0 || hc.cq.y != 0.0;
  const bool dip = hc.cd.x != 0.0 || hc.cd.y != 0.0;
  // ik cq, -i k^2 cd
  const double2 kS = c2(-hc.k * hc.cq.y, hc.k * hc.cq.x);
  const double2 kD = c2(hc.k * hc.k * hc.cd.y, -hc.k * hc.k * hc.cd.x);
  const double kinv = 1.0 / hc.k;
  double acc[NT][2];
#pragma unroll
  for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = 0.0;

  const int l0 = g.list1_starts[itb], l1 = g.list1_starts[itb + 1];
  for (int gb = l0; gb < l1; gb += MAXB) {
    const int nb = min(MAXB, l1 - gb);
    __syncthreads();
    h3_list_prefix(g, g.list1_lists, gb, nb, s_pref, s_start, err);
    __syncthreads();
    const int total = s_pref[nb];
    // source indices of tile t; then its copies (positions, normals, strengths) by cp.async
    auto index = [&](int t) {
      const int v = t * NEAR_TS + threadIdx.x;
      if (threadIdx.x < NEAR_TS)
        s_src[t & 1][threadIdx.x] = v < total ? h3_stream_source(v, nb, s_pref, s_start) : -1;
    };
    auto fetch = [&](int t) {
      double* S = tiles + (t & 1) * TILE;
      double* Y = S + NEAR_TS * SS;
      for (int e = threadIdx.x; e < NEAR_TS * NR; e += NEAR_NT) {
        const int j = e & (NEAR_TS - 1), r = e / NEAR_TS, s = s_src[t & 1][j];
        const bool on = s >= 0 && r0 + r < nrhs;
        near_cp16(S + j * SS + 2 * r, strengths + (on ? (size_t)(r0 + r) * g.nsources + s : 0), on);
      }
      for (int e = threadIdx.x; e < NEAR_TS * 6; e += NEAR_NT) {
        const int j = e & (NEAR_TS - 1), d = e / NEAR_TS, s = s_src[t & 1][j];
        const double* from = d < 3 ? g.sources + (size_t)d * g.nsources
                                   : g.source_normals + (size_t)(d - 3) * g.nsources;
        if (d < 3 || dip) near_cp8(Y + d * NEAR_TS + j, from + max(s, 0));
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const int ntile = (total + NEAR_TS - 1) / NEAR_TS;
    if (ntile > 0) {
      index(0);
      index(1);
      __syncthreads();
      fetch(0);
    }
    for (int tl = 0; tl < ntile; ++tl) {
      const int ns = min(NEAR_TS, total - tl * NEAR_TS);
      const double* S = tiles + (tl & 1) * TILE;
      const double* Y = S + NEAR_TS * SS;
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      __syncthreads();                           // tile tl is here, the other buffer is free
      if (tl + 1 < ntile) fetch(tl + 1);
      if (busy) {
        for (int j0 = 0; j0 < ns; j0 += 4) {
          const int j = j0 + kq;
          const double b0 = Y[j] - cc[0], b1 = Y[NEAR_TS + j] - cc[1], b2 = Y[2 * NEAR_TS + j] - cc[2];
          const double bs = b0 * b0 + b1 * b1 + b2 * b2;
          const double rho = rsqrt_h(bs), rho2 = rho * rho;
          const double x0 = hc.k * bs * rho, xi = kinv * rho;
          const double X = (a[0] * b0 + a[1] * b1 + a[2] * b2) * rho2 * x0;
          double zp[Q + 1];
          zp[0] = 1.0;
#pragma unroll
          for (int u = 1; u <= Q; ++u) zp[u] = u == 1 ? -0.5 * aa * rho2 * x0 : zp[u - 1] * zp[1];
          double sn, cs;
          sincos(x0, &sn, &cs);
          double2 hp = c2(sn * xi, -cs * xi);
          double2 hn = c2((sn - cs * x0) * xi * xi, -(sn * x0 + cs) * xi * xi);
          double bn = 0.0, an = 0.0;
          if (dip) {
            const double n0 = Y[3 * NEAR_TS + j], n1 = Y[4 * NEAR_TS + j], n2 = Y[5 * NEAR_TS + j];
            bn = b0 * n0 + b1 * n1 + b2 * n2;
            an = a[0] * n0 + a[1] * n1 + a[2] * n2;
          }
          double2 vS = c2(0.0), vD = c2(0.0);
#pragma unroll
          for (int i = 0; i <= Q; ++i) {
            const double w = near_w<Q, CUT>(i, min(i, Q - i), 0, X, zp, gw);
            if (chg) vS = caxpy(w, hp, vS);
            if (dip) {
              double e = bn * w;
              if (i < Q) e = fma(-an, near_w<Q, CUT>(i, min(i, Q - 1 - i), 1, X, zp, gw), e);
              vD = caxpy(e, hn, vD);
            }
            const double f = (2.0 * i + 3.0) * xi;
            const double2 nx = c2(f * hn.x - hp.x, f * hn.y - hp.y);
            hp = hn;
            hn = nx;
          }
          double2 K = c2(0.0);
          if (chg) K = cmul(kS, vS);
          if (dip) K = cfma(kD, cscale(rho, vD), K);
          if (j >= ns || bs == 0.0) K = c2(0.0);
          const double* B = S + j * SS;
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            // columns (density, part): i sigma has (-im, re) there
            const double bx = B[8 * n + (row ^ 1)];
            h3_dmma(acc[n][0], acc[n][1], K.x, B[8 * n + row]);
            h3_dmma(acc[n][0], acc[n][1], K.y, (row & 1) ? bx : -bx);
          }
        }
      }
      __syncthreads();                           // (the copies of tile tl + 1 have their indices)
      index(tl + 2);
    }
  }
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const int r = r0 + 4 * n + kq;
    if (!active || r >= nrhs) continue;
    double2* P = pot_tree + (size_t)r * g.ntargets + t;
    *P = cadd(*P, c2(acc[n][0], acc[n][1]));
  }
}

template <int Q, int NT>
cudaError_t near_launch(const qbxfmm_geometry& g, HelmCoeffs hc, int nrhs, const double2* s,
                        double2* pt, int32_t* err, cudaStream_t st)
{
  const size_t sh = (size_t)2 * NEAR_TS * (8 * NT + 4 + 6) * sizeof(double);
  auto k = hc.taylor ? k_h3_near<Q, NT, true> : k_h3_near<Q, NT, false>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  if (e != cudaSuccess) return e;
  k<<<dim3(g.ntsqbx_chunks, (nrhs + 4 * NT - 1) / (4 * NT)), NEAR_NT, sh, st>>>(g, hc, nrhs, s, pt,
                                                                                err);
  return cudaGetLastError();
}

template <int Q>
cudaError_t near_q(const qbxfmm_geometry& g, HelmCoeffs hc, int nrhs, const double2* s, double2* pt,
                   int32_t* err, cudaStream_t st)
{
  const int want = hc.rb_ts > 0 ? hc.rb_ts : nrhs;     // the plan's tuning, else by nrhs
  if (want > 8) return near_launch<Q, 4>(g, hc, nrhs, s, pt, err, st);
  if (want > 4) return near_launch<Q, 2>(g, hc, nrhs, s, pt, err, st);
  return near_launch<Q, 1>(g, hc, nrhs, s, pt, err, st);
}

}  // namespace

cudaError_t h3_launch_tsqbx(const qbxfmm_geometry& g, HelmCoeffs hc, int q, int nrhs,
                            const double2* s, double2* pt, int32_t* err, cudaStream_t st)
{
  if (g.ntsqbx_chunks == 0) return cudaSuccess;
  switch (q) {
    case 0: return near_q<0>(g, hc, nrhs, s, pt, err, st);
    case 1: return near_q<1>(g, hc, nrhs, s, pt, err, st);
    case 2: return near_q<2>(g, hc, nrhs, s, pt, err, st);
    case 3: return near_q<3>(g, hc, nrhs, s, pt, err, st);
    case 4: return near_q<4>(g, hc, nrhs, s, pt, err, st);
    case 5: return near_q<5>(g, hc, nrhs, s, pt, err, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace qbx
