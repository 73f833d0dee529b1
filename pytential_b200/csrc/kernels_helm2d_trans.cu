// 2D Helmholtz box translations M2M, M2L, L2L on the FP64 tensor cores, complex128, sm_100a.
//
// Eout_m[r] += fout(m) sum_n Z_{n-m}(d) fin(n) Ein_n[r], Z = J (M2M, L2L) or H (M2L): per
// source box a Toeplitz (2p + 1) x (2p + 1) matrix applied to the densities.  Its A
// fragments (8 rows m x 4 columns n) are read straight from the table Z_{-2p} .. Z_{2p} in
// shared memory, the B fragments (4 coefficients x (4 densities, re / im)) straight from
// the source box's coefficients in global memory, scaled in registers, and used for all row
// tiles, so nothing else is staged and no barrier separates the source boxes.  When 2p + 1
// is 1 mod 8 the last row runs on the FP64 pipe beside the products instead of a padded
// tile.  (By multiply-adds from staged blocks: 3.51 ms for 66 857 M2L pairs and 64
// densities, against 1.7 ms of products.)
//
// With the plan's tables (TAB: H of every list-2 offset and level, J of the eight shifts of a
// level, built once by qbxfmm_precompute_translations) a batch of up to 16 source boxes
// copies its tables by cp.async.  Without them the batch builds them: one warp runs the J
// recurrences, one the Y recurrences, one the powers of e^{i th}, a thread per box (serial
// chains of some 10 000 cycles, which bound M2M and L2L), then all threads combine them.
#include <algorithm>

#include "../../include/qbxfmm_api.h"
#include "helmholtz.cuh"
#include "helm3.cuh"
#include "kernels.h"

namespace qbx {

namespace {

QBX_D void cp_async16_h2(void* dst, const void* src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

constexpr int TR2_NT = 128;
constexpr int TR2_PB = 16;                   // source boxes per batch
constexpr int TR2_MAXP = 20;
constexpr size_t TR2_FEW = 2 * 148;          // CTAs of 64 densities that leave the GPU idle
constexpr int TR2_MT = (2 * TR2_MAXP + 1) / 8;

// Plan tables: shift [level][8][4p + 1] (M2M from child position c into its parent of the
// level: c; L2L from the parent into the child at position c of the level: 4 + c), m2l
// [level][class][4p + 1], cls: class of each list-2 entry
struct H2Tables {
  const double2* shift = nullptr;
  const double2* m2l = nullptr;
  const int32_t* cls = nullptr;
};

// position of a child in its parent: bit d set where its center's coordinate d is larger
QBX_D int h2_child_pos(double dx, double dy) { return (dx > 0.0 ? 1 : 0) | (dy > 0.0 ? 2 : 0); }

__global__ void __launch_bounds__(32)
k_h2_trans_tables(qbxfmm_geometry g, double k, int p, double2* __restrict__ shift,
                  double2* __restrict__ m2l, int32_t* __restrict__ cls, int npairs)
{
  const int NZ = 2 * p, ZW = 2 * NZ + 1;
  const int i = blockIdx.x * 32 + threadIdx.x;
  const int nshift = 8 * g.nlevels, nm2l = g.nlevels * g.m2l_nclasses;
  double Jb[2 * TR2_MAXP + 2], Yb[2 * TR2_MAXP + 2];
  if (i < nshift) {
    const int lev = i >> 3, c = i & 3;
    // M2M at parent level lev: parent - child; L2L at child level lev: child - parent
    const bool up = !(i & 4);
    const double q = 0.25 * level_width(g, up ? lev : lev - 1) * (up ? -1.0 : 1.0);
    h2_zfun(NZ, k, (c & 1) ? q : -q, (c & 2) ? q : -q, Jb, Yb, shift + (size_t)i * ZW, false);
  } else if (i < nshift + nm2l) {
    const int e = i - nshift, lev = e / g.m2l_nclasses, c = e - lev * g.m2l_nclasses;
    const double w = level_width(g, lev);
    h2_zfun(NZ, k, w * g.m2l_class_offsets[c], w * g.m2l_class_offsets[g.m2l_nclasses + c], Jb, Yb,
            m2l + (size_t)e * ZW, true);
  }
  for (int li = i; li < npairs; li += gridDim.x * 32) {
    const int pr = g.m2l_tgt_pairs[li];
    int lo = 0, hi = g.m2l_nclasses - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (g.m2l_class_starts[mid] <= pr) lo = mid;
      else hi = mid - 1;
    }
    cls[li] = lo;
  }
}

// KIND 0 = M2M, 1 = M2L, 2 = L2L; NTW tiles of 4 densities per warp.  SPLIT: the warps share
// the densities and deal the source boxes among them (fixed-order sum at the end); else
// each warp has its own densities.
template <int KIND, int NTW, bool SPLIT, bool TAB>
__global__ void __launch_bounds__(TR2_NT, 3)
k_h2_translate(qbxfmm_geometry g, double k, int p, int nrhs, int i0, H2Tables tab,
               const double2* __restrict__ ein, double2* __restrict__ eout, int32_t* err)
{
  constexpr int NR = (SPLIT ? 1 : 4) * NTW * 4;        // densities per CTA
  extern __shared__ double2 smem2[];
  const int NZ = 2 * p, ZW = 2 * NZ + 1, NC = 2 * p + 1;
  double2* Z = smem2;                                  // [PB][ZW]
  double2* Pw = Z + (size_t)TR2_PB * ZW;               // [PB][NZ + 1] e^{i m th}
  double* Js = reinterpret_cast<double*>(Pw + (size_t)TR2_PB * (NZ + 1));   // [PB][NZ + 1]
  double* Ys = Js + (size_t)TR2_PB * (NZ + 1);         // [PB][NZ + 1]
  __shared__ int s_src[TR2_PB];
  // the widths' powers: source side and target side (children of a box have one width)
  __shared__ double s_fin[TR2_MAXP + 1], s_fout[TR2_MAXP + 1];
  const int ib = i0 + blockIdx.x, r0 = blockIdx.y * NR;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int tb, l0, l1;
  if (KIND == 0) {
    tb = g.source_parent_boxes[ib];
    l0 = 0;
    l1 = 4;     // children
  } else if (KIND == 1) {
    tb = g.target_or_target_parent_boxes[ib];
    l0 = g.list2_starts[ib];
    l1 = g.list2_starts[ib + 1];
    if (l1 <= l0) return;
  } else {
    tb = g.target_or_target_parent_boxes[ib];
    l0 = 0;
    l1 = 1;     // parent
  }
  double ct[2];
  load_point<2>(g.box_centers, g.nboxes, tb, ct);
  const int lev = g.box_levels[tb];
  if (tid <= p) {
    const double rt = level_width(g, lev);
    const double rs = level_width(g, KIND == 0 ? lev + 1 : KIND == 1 ? lev : lev - 1);
    const double a = (double)tid;
    s_fin[tid] = KIND == 2 ? pow(rs, -a) : pow(rs, a);
    s_fout[tid] = KIND == 0 ? pow(rt, -a) : pow(rt, a);
  }
  const int row = lane >> 2, kq = lane & 3;
  const bool last = (NC & 7) == 1;                     // the last row beside the tiles
  const int mt = last ? NC >> 3 : (NC + 7) >> 3;       // <= TR2_MT
  const int t0 = SPLIT ? 0 : warp * NTW;
  const bool busy = r0 + 4 * t0 < nrhs;
  double acc[TR2_MT][NTW][2];
  double2 accl[NTW];
#pragma unroll
  for (int w = 0; w < NTW; ++w) {
    accl[w] = c2(0.0);
#pragma unroll
    for (int i = 0; i < TR2_MT; ++i) acc[i][w][0] = acc[i][w][1] = 0.0;
  }
  for (int lb = l0; lb < l1; lb += TR2_PB) {
    const int nbat = min(TR2_PB, l1 - lb);
    __syncthreads();
    if (tid < nbat) {
      int sb;
      if (KIND == 0) {
        sb = g.box_child_ids[(size_t)(lb + tid) * g.nboxes + tb];
        if (sb == 0 || g.box_source_counts_cumul[sb] == 0) sb = -1;
      } else if (KIND == 1) {
        sb = g.list2_lists[lb + tid];
        if ((unsigned)sb >= (unsigned)g.nboxes) {
          report(err, QBX_DEVERR_BAD_BOX);
          sb = -1;
        }
      } else {
        sb = g.box_parent_ids[tb];
      }
      s_src[tid] = sb;
    }
    __syncthreads();
    if constexpr (TAB) {
      for (int w = tid; w < nbat * ZW; w += TR2_NT) {
        const int bb = w / ZW, m = w - bb * ZW, sb = s_src[bb];
        if (sb < 0) continue;
        const double2* t;
        if (KIND == 1) {
          t = tab.m2l + ((size_t)lev * g.m2l_nclasses + tab.cls[lb + bb]) * ZW;
        } else {
          // position of the child in the parent
          double cs[2];
          load_point<2>(g.box_centers, g.nboxes, sb, cs);
          const double q = KIND == 0 ? -1.0 : 1.0;
          const int c = h2_child_pos(q * (ct[0] - cs[0]), q * (ct[1] - cs[1]));
          t = tab.shift + (size_t)(8 * lev + (KIND == 0 ? 0 : 4) + c) * ZW;
        }
        cp_async16_h2(Z + w, t + m);
      }
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    } else {
      if (lane < nbat && s_src[lane] >= 0) {
        double cs[2];
        load_point<2>(g.box_centers, g.nboxes, s_src[lane], cs);
        const double ux = ct[0] - cs[0], uy = ct[1] - cs[1];       // c_out - c_in
        const double r = sqrt(ux * ux + uy * uy);
        if (warp == 0) {
          double* J = Js + (size_t)lane * (NZ + 1);
          if (r == 0.0) {
            for (int m = 0; m <= NZ; ++m) J[m] = m == 0 && KIND != 1 ? 1.0 : 0.0;
          } else {
            bessel_jy(NZ, k * r, J, nullptr, false);
          }
        } else if (warp == 1) {
          if (KIND == 1) {
            double* Y = Ys + (size_t)lane * (NZ + 1);
            const double x = k * r, xinv = 1.0 / x;
            double a = 0.0, b = 0.0;
            if (r != 0.0) bessel_y01(x, a, b);
            Y[0] = a;
            Y[1] = b;
            for (int j = 1; j < NZ; ++j) {
              const double c = r == 0.0 ? 0.0 : 2.0 * j * xinv * b - a;
              a = b;
              b = c;
              Y[j + 1] = c;
            }
          }
        } else if (warp == 2) {
          double2* E = Pw + (size_t)lane * (NZ + 1);
          const double2 e1 = r == 0.0 ? c2(1.0) : c2(ux / r, uy / r);
          double2 e = c2(1.0);
          for (int m = 0; m <= NZ; ++m) {
            E[m] = e;
            e = cmul(e, e1);
          }
        }
      }
      __syncthreads();
      for (int w = tid; w < nbat * (NZ + 1); w += TR2_NT) {
        const int bb = w / (NZ + 1), m = w - bb * (NZ + 1);
        if (s_src[bb] < 0) continue;
        const double2 z = KIND == 1 ? c2(Js[w], Ys[w]) : c2(Js[w]), e = Pw[w];
        const double2 u = cmulc(z, e);                   // Z_m e^{-i m th}
        Z[(size_t)bb * ZW + NZ + m] = cmul(z, e);
        if (m > 0) Z[(size_t)bb * ZW + NZ - m] = (m & 1) ? c2(-u.x, -u.y) : u;
      }
    }
    __syncthreads();
    if (!busy) continue;
    for (int bb = SPLIT ? warp : 0; bb < nbat; bb += SPLIT ? 4 : 1) {
      const int sb = s_src[bb];
      if (sb < 0) continue;
      const double2* src = ein + ((size_t)sb * nrhs + r0) * NC;
      const double2* Zt = Z + (size_t)bb * ZW + NZ;    // Z_{n-m} at Zt[n - m]
      double2 nxt[NTW];
      auto fetch = [&](int n) {
#pragma unroll
        for (int w = 0; w < NTW; ++w) {
          const int r = 4 * (t0 + w) + (row >> 1);
          nxt[w] = (n < NC && r0 + r < nrhs) ? __ldg(src + (size_t)r * NC + n) : c2(0.0);
        }
      };
      fetch(kq);
      for (int n0 = 0; n0 < NC; n0 += 4) {
        const int n = min(n0 + kq, NC - 1);            // past the end: a finite Z times 0
        const double f = s_fin[abs(n - p)];
        double b[NTW], bx[NTW];
        double2 e[NTW];
#pragma unroll
        for (int w = 0; w < NTW; ++w) {
          // column (density, part): E, and i E for the imaginary part of Z
          e[w] = cscale(f, nxt[w]);
          b[w] = (row & 1) ? e[w].y : e[w].x;
          bx[w] = (row & 1) ? e[w].x : -e[w].y;
        }
        if (n0 + 4 < NC) fetch(n0 + 4 + kq);
#pragma unroll
        for (int i = 0; i < TR2_MT; ++i) {
          if (i >= mt) break;
          const double2 z = Zt[n - min(8 * i + row, NC - 1)];
#pragma unroll
          for (int w = 0; w < NTW; ++w) {
            h3_dmma(acc[i][w][0], acc[i][w][1], z.x, b[w]);
            h3_dmma(acc[i][w][0], acc[i][w][1], z.y, bx[w]);
          }
        }
        if (last) {
          const double2 z = Zt[n - (NC - 1)];
#pragma unroll
          for (int w = 0; w < NTW; ++w) accl[w] = cfma(z, e[w], accl[w]);
        }
      }
    }
  }
  if (last) {
    // over the four inner indices; lane (row, 0), row even: density 4 t + row / 2
#pragma unroll
    for (int w = 0; w < NTW; ++w)
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        accl[w].x += __shfl_xor_sync(0xffffffffu, accl[w].x, o);
        accl[w].y += __shfl_xor_sync(0xffffffffu, accl[w].y, o);
      }
  }
  double2* dst = eout + ((size_t)tb * nrhs + r0) * NC;
  double2* red = smem2;                                // SPLIT: [4][NR][NC]
  __syncthreads();
  auto put = [&](int r, int m, double2 v) {
    if (SPLIT) {
      red[((size_t)warp * NR + r) * NC + m] = v;
    } else if (r0 + r < nrhs) {
      double2* o = dst + (size_t)r * NC + m;
      *o = caxpy(s_fout[abs(m - p)], v, *o);
    }
  };
  if (busy) {
#pragma unroll
    for (int w = 0; w < NTW; ++w) {
#pragma unroll
      for (int i = 0; i < TR2_MT; ++i) {
        const int m = 8 * i + row;
        if (i < mt && m < NC) put(4 * (t0 + w) + kq, m, c2(acc[i][w][0], acc[i][w][1]));
      }
      if (last && kq == 0 && !(row & 1)) put(4 * (t0 + w) + (row >> 1), NC - 1, accl[w]);
    }
  }
  if (SPLIT) {
    __syncthreads();
    for (int e = tid; e < NR * NC; e += TR2_NT) {
      const int r = e / NC, m = e - r * NC;
      if (r0 + r >= nrhs) break;
      double2 v = red[e];
      for (int w = 1; w < 4; ++w) v = cadd(v, red[(size_t)w * NR * NC + e]);
      dst[e] = caxpy(s_fout[abs(m - p)], v, dst[e]);
    }
  }
}

template <int KIND, int NTW, bool SPLIT>
cudaError_t translate_launch(const qbxfmm_geometry& g, double k, int p, int nrhs, int i0, int nb,
                             const H2Tables& tab, const double2* ein, double2* eout, int32_t* err,
                             cudaStream_t st)
{
  constexpr int NR = (SPLIT ? 1 : 4) * NTW * 4;
  const bool have = tab.shift != nullptr;
  const size_t tabs = (size_t)TR2_PB * (4 * p + 1) + (have ? 0 : 2 * (size_t)TR2_PB * (2 * p + 1));
  const size_t red = SPLIT ? (size_t)4 * NR * (2 * p + 1) : 0;
  const size_t sh = std::max(tabs, red) * sizeof(double2);
  auto kern = have ? k_h2_translate<KIND, NTW, SPLIT, true> : k_h2_translate<KIND, NTW, SPLIT, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  if (e != cudaSuccess) return e;
  kern<<<dim3(nb, (nrhs + NR - 1) / NR), TR2_NT, sh, st>>>(g, k, p, nrhs, i0, tab, ein, eout, err);
  return cudaGetLastError();
}

template <int KIND>
cudaError_t translate(const qbxfmm_geometry& g, double k, int p, int nrhs, int i0, int nb,
                      const H2Tables& tab, const double2* ein, double2* eout, int32_t* err,
                      cudaStream_t st)
{
  if (p > TR2_MAXP) return cudaErrorInvalidValue;
  // More than 16 densities: each warp its own 16; else the warps deal the source boxes.  L2L
  // has one source box, so its warps always split densities.  Where a level's CTAs leave the
  // GPU idle, a CTA takes 16 densities instead of 64: its four warps M2M's children, or four
  // densities each (65 to 33 us an M2M level, 75 to 14 an L2L level, of such levels at 64
  // densities and order 20; larger levels are faster with 64, which share a table).
  const bool few = (size_t)nb * ((nrhs + 63) / 64) < TR2_FEW;
  if (KIND == 2) {
    if (!few && nrhs > 32)
      return translate_launch<KIND, 4, false>(g, k, p, nrhs, i0, nb, tab, ein, eout, err, st);
    if (!few && nrhs > 16)
      return translate_launch<KIND, 2, false>(g, k, p, nrhs, i0, nb, tab, ein, eout, err, st);
    return translate_launch<KIND, 1, false>(g, k, p, nrhs, i0, nb, tab, ein, eout, err, st);
  }
  if (nrhs > 16 && !(KIND == 0 && few))
    return translate_launch<KIND, 4, false>(g, k, p, nrhs, i0, nb, tab, ein, eout, err, st);
  if (nrhs > 8) return translate_launch<KIND, 4, true>(g, k, p, nrhs, i0, nb, tab, ein, eout, err, st);
  if (nrhs > 4) return translate_launch<KIND, 2, true>(g, k, p, nrhs, i0, nb, tab, ein, eout, err, st);
  return translate_launch<KIND, 1, true>(g, k, p, nrhs, i0, nb, tab, ein, eout, err, st);
}

// the sections of the translations buffer (double2), the classes last
H2Tables tables(const qbxfmm_geometry& g, int p, const void* translations)
{
  H2Tables t;
  if (!translations) return t;
  t.shift = static_cast<const double2*>(translations);
  t.m2l = t.shift + (size_t)8 * g.nlevels * (4 * p + 1);
  t.cls = reinterpret_cast<const int32_t*>(t.m2l + (size_t)g.nlevels * g.m2l_nclasses * (4 * p + 1));
  return t;
}

}  // namespace

size_t h2_translations_bytes(const qbxfmm_geometry& g, int p, int npairs)
{
  if (g.m2l_nclasses == 0 || p > TR2_MAXP) return 0;
  return (size_t)g.nlevels * (8 + g.m2l_nclasses) * (4 * p + 1) * sizeof(double2) +
         ((size_t)npairs + 3) / 4 * 4 * sizeof(int32_t);
}

cudaError_t h2_launch_translations(const qbxfmm_geometry& g, double k, int p, int npairs,
                                   void* translations, cudaStream_t st)
{
  const H2Tables t = tables(g, p, translations);
  const int n = g.nlevels * (8 + g.m2l_nclasses);
  k_h2_trans_tables<<<(n + 31) / 32, 32, 0, st>>>(g, k, p, const_cast<double2*>(t.shift),
                                                  const_cast<double2*>(t.m2l),
                                                  const_cast<int32_t*>(t.cls), npairs);
  return cudaGetLastError();
}

cudaError_t h2_launch_m2m(const qbxfmm_geometry& g, const int32_t* lvl_host, HelmCoeffs hc, int p,
                          int nrhs, const void* translations, double2* mp, int32_t* err,
                          cudaStream_t st)
{
  const H2Tables t = tables(g, p, translations);
  for (int lev = g.nlevels - 2; lev >= 0; --lev) {
    const int i0 = lvl_host[lev], i1 = lvl_host[lev + 1];
    if (i1 <= i0) continue;
    cudaError_t e = translate<0>(g, hc.k, p, nrhs, i0, i1 - i0, t, mp, mp, err, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t h2_launch_m2l(const qbxfmm_geometry& g, HelmCoeffs hc, int p, int nrhs,
                          const void* translations, const double2* mp, double2* lo, int32_t* err,
                          cudaStream_t st)
{
  if (g.nttp_boxes == 0) return cudaSuccess;
  return translate<1>(g, hc.k, p, nrhs, 0, g.nttp_boxes, tables(g, p, translations), mp, lo, err, st);
}

cudaError_t h2_launch_l2l(const qbxfmm_geometry& g, const int32_t* lvl_host, HelmCoeffs hc, int p,
                          int nrhs, const void* translations, double2* lo, int32_t* err,
                          cudaStream_t st)
{
  const H2Tables t = tables(g, p, translations);
  for (int lev = 1; lev < g.nlevels; ++lev) {
    const int i0 = lvl_host[lev], i1 = lvl_host[lev + 1];
    if (i1 <= i0) continue;
    cudaError_t e = translate<2>(g, hc.k, p, nrhs, i0, i1 - i0, t, lo, lo, err, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace qbx
