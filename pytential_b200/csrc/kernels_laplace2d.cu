// 2D Laplace box stages (form_multipoles, coarsen_multipoles, multipole_to_local,
// refine_locals; pytential/qbx/fmm.py:441-478, 519-523), sm_100a.  At most 21 coefficients.
//
// In 2D these stages are bound by latency, not by arithmetic: a few hundred boxes and a
// launch per level of M2M and L2L.  A warp holds an expansion, lane l its coefficient l: the
// powers of the shift by squaring in every lane (they were one thread's chain before a CTA
// barrier), and the binomials taken into factorials on both sides, so that a shift is a
// plain convolution,
//   M2M  out_l = (l-1)! sum_{1<=k<=l} [ratio^k M_k / (k-1)!] [t^{l-k} / (l-k)!] - M_0 t^l / l
//   L2L  out_l = ratio^l / l! sum_{k>=l} [k! L_k] [s^{k-l} / (k-l)!]
//   M2L  out_l = tau^-l (-1)^l (sum_k (k+l-1)!/l! [M_k tau^-k / (k-1)!] - M_0 / l),
//        out_0 = sum_k M_k tau^-k + M_0 log(tau rho)
// 1024 nodes, order 10, a launch: P2M 11.1 us, M2M 12.4 (6 levels), M2L 36.9 and L2L 6.7 before;
// with the wider near field the whole apply 209 -> 146 us.
#include "laplace.cuh"
#include "kernels.h"

namespace qbx {

namespace {

constexpr int NT = 128, NW = NT / 32;
constexpr int L2_MAXP = 20;

struct Factorials {
  double f[2 * L2_MAXP], r[L2_MAXP + 1];     // n!, 1 / n!
};

constexpr Factorials factorials()
{
  Factorials t{};
  double v = 1.0;
  for (int n = 0; n < 2 * L2_MAXP; ++n) {
    if (n > 0) v *= n;
    t.f[n] = v;
    if (n <= L2_MAXP) t.r[n] = 1.0 / v;
  }
  return t;
}

__constant__ Factorials c_fact = factorials();

// z^n, 0 <= n < 32
QBX_D double2 cpow_n(double2 z, int n)
{
  double2 r = (n & 1) ? z : c2(1.0);
#pragma unroll
  for (int b = 1; b < 5; ++b) {
    z = cmul(z, z);
    if ((n >> b) & 1) r = cmul(r, z);
  }
  return r;
}

QBX_D double pow_n(double z, int n)
{
  double r = (n & 1) ? z : 1.0;
#pragma unroll
  for (int b = 1; b < 5; ++b) {
    z *= z;
    if ((n >> b) & 1) r *= z;
  }
  return r;
}

// a box per CTA, a source per thread: every coefficient's terms, then a warp sums each
template <bool DIP>
__global__ void __launch_bounds__(NT)
k_p2m2(qbxfmm_geometry g, SourceCoeffs sc, int p, int nrhs, const double* __restrict__ strengths,
       double2* __restrict__ mpoles)
{
  extern __shared__ double2 tab[];           // [p + 1][NT + 1]
  constexpr int TS = NT + 1;
  const int b = g.source_boxes[blockIdx.x], r = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double rinv = 1.0 / level_width(g, g.box_levels[b]);
  double c[2];
  load_point<2>(g.box_centers, g.nboxes, b, c);
  const int s0 = g.box_source_starts[b], ns = g.box_source_counts_nonchild[b];
  double2* M = mpoles + ((size_t)b * nrhs + r) * (p + 1);
  for (int base = 0; base < ns; base += NT) {
    const int j = base + threadIdx.x;
    double2 u = c2(0.0), nu = c2(0.0);
    double q = 0.0;
    if (j < ns) {
      double y[2], nv[2] = {0.0, 0.0};
      load_point<2>(g.sources, g.nsources, s0 + j, y);
      if (DIP) load_point<2>(g.source_normals, g.nsources, s0 + j, nv);
      q = __ldg(strengths + (size_t)r * g.nsources + s0 + j);
      u = c2((y[0] - c[0]) * rinv, (y[1] - c[1]) * rinv);
      nu = c2(-sc.cd * q * rinv * nv[0], -sc.cd * q * rinv * nv[1]);
    }
    const double f = sc.cq * q;
    double2 a = c2(1.0);
    if (base > 0) __syncthreads();
    tab[threadIdx.x] = c2(f);
    for (int k = 1; k <= p; ++k) {
      const double2 prev = a;
      a = cmul(a, u);
      double2 v = cscale(-f * rcp(k), a);
      if (DIP) v = cfma(nu, prev, v);
      tab[k * TS + threadIdx.x] = v;
    }
    __syncthreads();
    const int used = min(NT, ns - base);
    for (int k = warp; k <= p; k += NW) {
      double2 v = c2(0.0);
      for (int i = lane; i < used; i += 32) v = cadd(v, tab[k * TS + i]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
      if (lane == 0) M[k] = cadd(M[k], v);
    }
  }
}

// a parent per CTA, a child per warp
__global__ void __launch_bounds__(NT)
k_m2m2(qbxfmm_geometry g, int p, int nrhs, int i0, double2* __restrict__ mpoles)
{
  __shared__ double2 s_m[NW][32], s_t[NW][32], s_out[NW][32];
  const int b = g.source_parent_boxes[i0 + blockIdx.x], r = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ch = g.box_child_ids[(size_t)warp * g.nboxes + b];
  double2 out = c2(0.0);
  if (ch != 0 && g.box_source_counts_cumul[ch] != 0) {
    double2 m = c2(0.0);
    if (lane <= p) m = mpoles[((size_t)ch * nrhs + r) * (p + 1) + lane];
    const int lev = g.box_levels[b];
    const double rho = level_width(g, lev), ratio = level_width(g, lev + 1) / rho;
    double cp[2], cc[2];
    load_point<2>(g.box_centers, g.nboxes, b, cp);
    load_point<2>(g.box_centers, g.nboxes, ch, cc);
    const double2 t = cpow_n(c2((cc[0] - cp[0]) / rho, (cc[1] - cp[1]) / rho), lane);
    const int l = min(lane, L2_MAXP);
    s_m[warp][lane] = cscale(pow_n(ratio, lane) * c_fact.r[max(l - 1, 0)], m);
    s_t[warp][lane] = cscale(c_fact.r[l], t);
    const double2 m0 = c2(__shfl_sync(0xffffffffu, m.x, 0), __shfl_sync(0xffffffffu, m.y, 0));
    __syncwarp();
    if (lane <= p) {
#pragma unroll 4
      for (int k = 1; k <= p; ++k)
        if (k <= lane) out = cfma(s_m[warp][k], s_t[warp][lane - k], out);
      out = lane == 0 ? m0
                      : csub(cscale(c_fact.f[lane - 1], out), cscale(rcp(lane), cmul(m0, t)));
    }
  }
  s_out[warp][lane] = out;
  __syncthreads();
  if (warp == 0 && lane <= p) {
    for (int w = 1; w < NW; ++w) out = cadd(out, s_out[w][lane]);
    double2* M = mpoles + ((size_t)b * nrhs + r) * (p + 1) + lane;
    *M = cadd(*M, out);
  }
}

// a target-or-parent box per CTA, the list-2 boxes dealt to its warps
__global__ void __launch_bounds__(NT)
k_m2l2(qbxfmm_geometry g, int p, int nrhs, const double2* __restrict__ mpoles,
       double2* __restrict__ locals, int32_t* err)
{
  __shared__ double2 s_m[NW][32], s_out[NW][32];
  __shared__ double s_f[2 * L2_MAXP];
  const int i = blockIdx.x, r = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l0 = g.list2_starts[i], l1 = g.list2_starts[i + 1];
  if (l1 <= l0) return;
  const int tb = g.target_or_target_parent_boxes[i];
  const double rho = level_width(g, g.box_levels[tb]), rinv = 1.0 / rho;
  double ct[2];
  load_point<2>(g.box_centers, g.nboxes, tb, ct);
  for (int n = threadIdx.x; n < 2 * L2_MAXP; n += NT) s_f[n] = c_fact.f[n];
  __syncthreads();
  const int l = min(lane, L2_MAXP);
  const double rl = c_fact.r[l], rl1 = c_fact.r[max(l - 1, 0)], sg = (lane & 1) ? -1.0 : 1.0;
  const double invl = lane > 0 ? rcp(lane) : 0.0;
  double2 acc = c2(0.0);
  // the next box's center and coefficient are in flight during a box's sum
  double cs[2] = {0.0, 0.0}, cn[2] = {0.0, 0.0};
  double2 m = c2(0.0), mn = c2(0.0);
  bool ok = false, okn = false;
  auto fetch = [&](int li) {
    okn = false;
    if (li >= l1) return;
    const int sb = g.list2_lists[li];
    if ((unsigned)sb >= (unsigned)g.nboxes) {
      if (lane == 0) report(err, QBX_DEVERR_BAD_BOX);
      return;
    }
    okn = true;
    load_point<2>(g.box_centers, g.nboxes, sb, cn);
    mn = lane <= p ? __ldg(mpoles + ((size_t)sb * nrhs + r) * (p + 1) + lane) : c2(0.0);
  };
  fetch(l0 + warp);
  for (int li = l0 + warp; li < l1; li += NW) {
    ok = okn;
    m = mn;
    cs[0] = cn[0];
    cs[1] = cn[1];
    fetch(li + NW);
    if (!ok) continue;
    const double d0 = (ct[0] - cs[0]) * rinv, d1 = (ct[1] - cs[1]) * rinv;
    const double2 tp = cpow_n(cinv(c2(d0, d1)), lane);
    const double2 m0 = c2(__shfl_sync(0xffffffffu, m.x, 0), __shfl_sync(0xffffffffu, m.y, 0));
    __syncwarp();
    s_m[warp][lane] = cscale(rl1, cmul(m, tp));
    __syncwarp();
    if (lane <= p) {
      double2 s = c2(0.0);
#pragma unroll 4
      for (int k = 1; k <= p; ++k) s = caxpy(s_f[k + lane - 1], s_m[warp][k], s);
      s = cscale(rl, s);
      if (lane == 0)
        acc = cadd(acc, cfma(m0, clog_(c2(d0 * rho, d1 * rho)), s));
      else
        acc = cfma(cscale(sg, csub(s, cscale(invl, m0))), tp, acc);
    }
  }
  s_out[warp][lane] = acc;
  __syncthreads();
  if (warp == 0 && lane <= p) {
    for (int w = 1; w < NW; ++w) acc = cadd(acc, s_out[w][lane]);
    double2* L = locals + ((size_t)tb * nrhs + r) * (p + 1) + lane;
    *L = cadd(*L, acc);
  }
}

// a child per warp
__global__ void __launch_bounds__(NT)
k_l2l2(qbxfmm_geometry g, int p, int nrhs, int i0, int i1, double2* __restrict__ locals)
{
  __shared__ double2 s_l[NW][32], s_t[NW][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = i0 + blockIdx.x * NW + warp, r = blockIdx.y;
  if (i >= i1) return;
  const int b = g.target_or_target_parent_boxes[i], par = g.box_parent_ids[b];
  double2 lp = c2(0.0);
  if (lane <= p) lp = locals[((size_t)par * nrhs + r) * (p + 1) + lane];
  const int lev = g.box_levels[b];
  const double rho = level_width(g, lev - 1), ratio = level_width(g, lev) / rho;
  double cp[2], cc[2];
  load_point<2>(g.box_centers, g.nboxes, par, cp);
  load_point<2>(g.box_centers, g.nboxes, b, cc);
  const int l = min(lane, L2_MAXP);
  s_l[warp][lane] = cscale(c_fact.f[l], lp);
  s_t[warp][lane] =
      cscale(c_fact.r[l], cpow_n(c2((cc[0] - cp[0]) / rho, (cc[1] - cp[1]) / rho), lane));
  __syncwarp();
  if (lane > p) return;
  double2 s = c2(0.0);
#pragma unroll 4
  for (int k = 0; k <= p; ++k)
    if (k >= lane) s = cfma(s_l[warp][k], s_t[warp][k - lane], s);
  double2* L = locals + ((size_t)b * nrhs + r) * (p + 1) + lane;
  *L = caxpy(pow_n(ratio, lane) * c_fact.r[l], s, *L);
}

}  // namespace

cudaError_t l2_launch_p2m(const qbxfmm_geometry& g, SourceCoeffs sc, int p, int nrhs,
                          const double* s, double2* mp, cudaStream_t st)
{
  if (g.nsource_boxes == 0) return cudaSuccess;
  if (p > L2_MAXP) return cudaErrorInvalidValue;
  const size_t sh = (size_t)(p + 1) * (NT + 1) * sizeof(double2);
  auto k = sc.cd != 0.0 ? k_p2m2<true> : k_p2m2<false>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  if (e != cudaSuccess) return e;
  k<<<dim3(g.nsource_boxes, nrhs), NT, sh, st>>>(g, sc, p, nrhs, s, mp);
  return cudaGetLastError();
}

cudaError_t l2_launch_m2m(const qbxfmm_geometry& g, const int32_t* lvl_host, int p, int nrhs,
                          double2* mp, cudaStream_t st)
{
  if (p > L2_MAXP) return cudaErrorInvalidValue;
  for (int lev = g.nlevels - 2; lev >= 0; --lev) {
    const int i0 = lvl_host[lev], i1 = lvl_host[lev + 1];
    if (i1 <= i0) continue;
    k_m2m2<<<dim3(i1 - i0, nrhs), NT, 0, st>>>(g, p, nrhs, i0, mp);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t l2_launch_m2l(const qbxfmm_geometry& g, int p, int nrhs, const double2* mp, double2* lo,
                          int32_t* err, cudaStream_t st)
{
  if (g.nttp_boxes == 0) return cudaSuccess;
  if (p > L2_MAXP) return cudaErrorInvalidValue;
  k_m2l2<<<dim3(g.nttp_boxes, nrhs), NT, 0, st>>>(g, p, nrhs, mp, lo, err);
  return cudaGetLastError();
}

cudaError_t l2_launch_l2l(const qbxfmm_geometry& g, const int32_t* lvl_host, int p, int nrhs,
                          double2* lo, cudaStream_t st)
{
  if (p > L2_MAXP) return cudaErrorInvalidValue;
  for (int lev = 1; lev < g.nlevels; ++lev) {
    const int i0 = lvl_host[lev], i1 = lvl_host[lev + 1];
    if (i1 <= i0) continue;
    k_l2l2<<<dim3((i1 - i0 + NW - 1) / NW, nrhs), NT, 0, st>>>(g, p, nrhs, i0, i1, lo);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace qbx
