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
// products run on the tensor pipe beside the FP64 pipe, which bounds the kernel.
#include <algorithm>

#include "../../include/qbxfmm_api.h"
#include "helm3.cuh"
#include "kernels.h"

namespace qbx {

namespace {

constexpr int NEAR_NT = 128;

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

template <int Q, int NT, bool CUT>
__global__ void __launch_bounds__(NEAR_NT)
k_h3_near(qbxfmm_geometry g, HelmCoeffs hc, int nrhs, const double2* __restrict__ strengths,
          double2* __restrict__ pot_tree, int32_t* err)
{
  constexpr int SS = 8 * NT + 4;                 // row stride of the strengths (doubles)
  constexpr int NR = 4 * NT;
  extern __shared__ double2 smem2[];
  double* S = reinterpret_cast<double*>(smem2);  // [NEAR_NT][SS]
  __shared__ double2 s_a[NEAR_NT], s_b[NEAR_NT], s_c[NEAR_NT];   // (y0, y1), (y2, nu0), (nu1, nu2)
  __shared__ int s_src[NEAR_NT];
  __shared__ int s_pref[MAXB + 1], s_start[MAXB];
  const int chunk = blockIdx.x, r0 = blockIdx.y * NR;
  const int itb = g.tsqbx_chunk_target_box[chunk];
  const int cnt = g.tsqbx_chunk_count[chunk], i0 = g.tsqbx_chunk_start[chunk];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = lane >> 2, kq = lane & 3;
  // with 1 or 2 octets of targets the four warps share an octet's sources: warp's octet, its
  // part of the sources and the number of parts
  const int noct = (cnt + 7) >> 3, parts = noct <= 2 ? 4 / max(noct, 1) : 1;
  const int oct = warp / parts, part = warp - oct * parts;
  const bool busy = oct < noct;
  bool active = 8 * oct + row < cnt;
  const int pi = i0 + max(0, min(8 * oct + row, cnt - 1));
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
    for (int base = 0; base < total; base += NEAR_NT) {
      const int ns = min(NEAR_NT, total - base);
      if ((int)threadIdx.x < ns) {
        const int s = h3_stream_source(base + threadIdx.x, nb, s_pref, s_start);
        double y[3], nv[3] = {0, 0, 0};
        load_point<3>(g.sources, g.nsources, s, y);
        if (dip) load_point<3>(g.source_normals, g.nsources, s, nv);
        s_a[threadIdx.x] = c2(y[0], y[1]);
        s_b[threadIdx.x] = c2(y[2], nv[0]);
        s_c[threadIdx.x] = c2(nv[1], nv[2]);
        s_src[threadIdx.x] = s;
      } else {
        s_src[threadIdx.x] = -1;
      }
      __syncthreads();
      // strengths, sources fastest: runs of one box are contiguous
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int s = s_src[threadIdx.x];
        double2 v = c2(0.0);
        if (s >= 0 && r0 + r < nrhs) v = __ldg(strengths + (size_t)(r0 + r) * g.nsources + s);
        *reinterpret_cast<double2*>(S + threadIdx.x * SS + 2 * r) = v;
      }
      __syncthreads();
      if (busy) {
        for (int j0 = 4 * part; j0 < ns; j0 += 4 * parts) {
          const int j = j0 + kq;
          const double2 ya = s_a[j], yb = s_b[j], yc = s_c[j];
          const double b0 = ya.x - cc[0], b1 = ya.y - cc[1], b2 = yb.x - cc[2];
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
            bn = b0 * yb.y + b1 * yc.x + b2 * yc.y;
            an = a[0] * yb.y + a[1] * yc.x + a[2] * yc.y;
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
          // columns (density, part): i sigma has (-im, re) there
#pragma unroll
          for (int n = 0; n < NT; ++n) h3_dmma(acc[n][0], acc[n][1], K.x, B[8 * n + row]);
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            const double bx = B[8 * n + (row ^ 1)];
            h3_dmma(acc[n][0], acc[n][1], K.y, (row & 1) ? bx : -bx);
          }
        }
      }
      __syncthreads();
    }
  }
  if (parts > 1) {             // (the last tile's barrier freed S) the parts in order
#pragma unroll
    for (int n = 0; n < NT; ++n)
      *reinterpret_cast<double2*>(S + ((warp * NT + n) * 32 + lane) * 2) = c2(acc[n][0], acc[n][1]);
    __syncthreads();
    if (part > 0) return;
    for (int w = 1; w < parts; ++w)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const double2 v =
            *reinterpret_cast<const double2*>(S + (((warp + w) * NT + n) * 32 + lane) * 2);
        acc[n][0] += v.x;
        acc[n][1] += v.y;
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
  const size_t sh = (size_t)NEAR_NT * (8 * NT + 4) * sizeof(double);
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
