// Matrix form of the 3D Laplace box translations (M2L, M2M, L2L) on the FP64
// tensor cores (mma.sync m8n8k4 f64), sm_100a.
//
// With rscale-scaled coefficients a translation between boxes depends only on the
// translation vector in units of the box width: every list-2 pair with the same
// integer offset uses the same matrix (times 1/rho of the level, applied in the
// reduction), every M2M / L2L pair with the same child position uses the same
// matrix at every level.  A translation acts on the stored coefficients
// (m >= 0, the rest by conjugate symmetry) as a real-linear map, so each class is a
// real (2 ncoeff) x (2 ncoeff) matrix T acting on interleaved (re, im) vectors.
//
//   k_trans_build  : one CTA per class, T from the harmonic table of the class vector
//   k_trans_gemm   : M2L, a CTA per (class, rows, 64 pairs x rhs): C = T X with X the
//                    gathered source expansions
//   k_trans_reduce : deterministic sum of each output box's pair results (list order)
//   k_trans_gemm_pipe : M2M and L2L, a launch per level
//
// M2L classes related by a lattice symmetry (quarter turns about z, y and z
// reflections) share the matrix of their canonical offset: the GEMM applies the
// class's input map to the gathered columns and its output map to the products
// (m2l_symmetry_classes, laplace.cuh).
#include "laplace.cuh"
#include "kernels.h"

#include <algorithm>
#include <array>
#include <cstdlib>
#include <map>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

namespace qbx {

namespace {

constexpr int NT = 128;

QBX_D void dmma_8x8x4(double& d0, double& d1, double a, double b)
{
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

}  // namespace

// {{{ T construction

// kind 0 = M2L (class vector d = offset, S table of order 2p; value (-1)^j S),
// kind 1 = M2M (d = (child - parent) / rho_parent, R table of order p),
// kind 2 = L2L (same d, R table).
__global__ void __launch_bounds__(NT)
k_trans_build(int kind, int p, int ncf, int rp, int kp, int nclasses, const int32_t* __restrict__ offs,
              double* __restrict__ T)
{
  extern __shared__ double2 tab[];
  int cls = blockIdx.x;
  double d[3];
  if (kind == 0) {
    for (int k = 0; k < 3; ++k) d[k] = (double)offs[k * nclasses + cls];
  } else {
    // child position bits -> +-1/4 per axis (child centre relative to the parent)
    for (int k = 0; k < 3; ++k) d[k] = ((cls >> k) & 1) ? 0.25 : -0.25;
  }
  if (kind == 0) sh3_S_table(2 * p, d[0], d[1], d[2], tab, threadIdx.x, NT);
  else sh3_R_table(p, d[0], d[1], d[2], tab, threadIdx.x, NT);
  __syncthreads();
  double* Tc = T + (size_t)cls * rp * kp;
  const int R = 2 * ncf;
  for (int e = threadIdx.x; e < rp * kp; e += NT) {
    int row = e / kp, col = e - row * kp;
    double v = 0.0;
    if (row < R && col < R) {
      int co = row >> 1, ci = col >> 1;
      int no, mo, ni, mi;
      decode3(co, no, mo);
      decode3(ci, ni, mi);
      // unit input u at stored (ni, mi); its symmetric partner at -mi is u' = (-1)^mi conj(u)
      double2 u = (col & 1) ? c2(0.0, 1.0) : c2(1.0, 0.0);
      double2 up = cconj(u);
      if (mi & 1) up = c2(-up.x, -up.y);
      double2 val = c2(0.0);
      if (kind == 0) {
        // L_j^i = (-1)^j sum M_k^l S_{k+j}^{l+i}
        val = cmul(u, sh3_get(tab, ni + no, mi + mo));
        if (mi > 0) val = cadd(val, cmul(up, sh3_get(tab, ni + no, -mi + mo)));
        if (no & 1) val = c2(-val.x, -val.y);
      } else if (kind == 1) {
        // M'_n^m = sum (1/2)^k M_k^l conj(R_{n-k}^{m-l})
        double rk = ldexp(1.0, -ni);
        val = cmulc(u, sh3_get(tab, no - ni, mo - mi));
        if (mi > 0) val = cadd(val, cmulc(up, sh3_get(tab, no - ni, mo + mi)));
        val = cscale(rk, val);
      } else {
        // L''_k^l = (1/2)^k sum L_n^m conj(R_{n-k}^{m-l})
        double rk = ldexp(1.0, -no);
        val = cmulc(u, sh3_get(tab, ni - no, mi - mo));
        if (mi > 0) val = cadd(val, cmulc(up, sh3_get(tab, ni - no, -mi - mo)));
        val = cscale(rk, val);
      }
      v = (row & 1) ? val.y : val.x;
    }
    Tc[e] = v;
  }
}

// }}}

// {{{ GEMM

// C = T X for one group (class), one tile of 16 MI rows and one of 64 columns (pair x rhs):
// four warps of 8 MI x 32, operands in four cp.async stages of 16 k, k-contiguous with a row
// stride of 20 doubles (4 mod 16), free of bank conflicts as fragments.  A class symmetry
// permutes and negates parts of coefficients: of X when a fragment is read, of C in the
// epilogue.  The result is stored into cpair[pair * nrhs + r][0..rp).
// The form before (32 columns, operands staged between two barriers per 32 k, one row
// fragment loaded per product) took 4.53 ms for the M2L of 307 200 nodes at order 12 and
// 0.222 ms of 19 200 at order 10; this 3.35 and 0.191.
constexpr int GN = 64, GK = 16, GST = 4, GS = GK + 4;

template <int MI>
constexpr int gemm_stage() { return (16 * MI + GN) * GS; }

QBX_D void cp_async16_zfill(void* dst, const void* src, bool on)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(on ? 16 : 0)
               : "memory");
}

template <int MI>
__global__ void __launch_bounds__(NT)
k_trans_gemm(int ncf, int rp, int kp, int nrhs, const double* __restrict__ T,
             const int32_t* __restrict__ cls_code, const int32_t* __restrict__ group_starts,
             const int32_t* __restrict__ pair_src, const double2* __restrict__ ein,
             double* __restrict__ cpair, int32_t* err, int nboxes)
{
  constexpr int GM = 16 * MI;
  extern __shared__ double2 smem2[];
  double* sm = reinterpret_cast<double*>(smem2);       // [GST]{A [GM][GS], B [GN][GS]}
  __shared__ int s_src[GN];
  __shared__ uint8_t s_opi[M2L_SYM_MAXR], s_opo[M2L_SYM_MAXR];
  const int grp = blockIdx.z;
  const int p0 = group_starts[grp], ncol = (group_starts[grp + 1] - p0) * nrhs;
  const int c0 = blockIdx.x * GN, m0 = blockIdx.y * GM;
  if (c0 >= ncol) return;
  int mat = grp, sym = 0;
  if (cls_code) {
    const int code = cls_code[grp];
    mat = code >> 4;
    sym = code & 15;
  }
  const int R = 2 * ncf, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (sym) m2l_sym_tables(sym, R, s_opi, s_opo, tid, NT);
  for (int j = tid; j < GN; j += NT) {
    const int c = c0 + j;
    int src = -1;
    if (c < ncol) {
      src = pair_src[p0 + c / nrhs];
      if ((unsigned)src >= (unsigned)nboxes) {
        report(err, QBX_DEVERR_BAD_BOX);
        src = -1;
      }
    }
    s_src[j] = src;
  }
  __syncthreads();
  // this thread's 16-byte pieces of a chunk: rows / columns tid / 8 + 16 i, k = 2 (tid % 8)
  const double* Tg = T + (size_t)mat * rp * kp;
  const int kk = 2 * (tid & 7), rb = tid >> 3;
  const double* bp[GN / 16];
  bool bon[GN / 16];
#pragma unroll
  for (int i = 0; i < GN / 16; ++i) {
    const int src = s_src[rb + 16 * i];
    bon[i] = src >= 0;
    bp[i] = reinterpret_cast<const double*>(
                ein + ((size_t)(bon[i] ? src : 0) * nrhs + (c0 + rb + 16 * i) % nrhs) * ncf) + kk;
  }
  const double* ap = Tg + (size_t)(m0 + rb) * kp + kk;
  const int nk = (R + GK - 1) / GK;
  auto fetch = [&](int ck) {
    if (ck < nk) {
      double* A = sm + (ck % GST) * gemm_stage<MI>();
      double* B = A + GM * GS;
      const bool in = ck * GK + kk < R;                  // kp >= R; the rest is zero
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const bool on = in && m0 + rb + 16 * i < rp;
        cp_async16_zfill(A + (rb + 16 * i) * GS + kk, on ? ap + (size_t)16 * i * kp + ck * GK : Tg, on);
      }
#pragma unroll
      for (int i = 0; i < GN / 16; ++i) {
        const bool on = in && bon[i];
        cp_async16_zfill(B + (rb + 16 * i) * GS + kk, on ? bp[i] + ck * GK : Tg, on);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const int row = lane >> 2, tq = lane & 3, wm = warp & 1, wn = warp >> 1;
  double acc[MI][4][2];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  for (int i = 0; i < GST - 1; ++i) fetch(i);
  for (int ck = 0; ck < nk; ++ck) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(GST - 2) : "memory");
    __syncthreads();
    fetch(ck + GST - 1);                                 // into the stage read last round
    const double* A = sm + (ck % GST) * gemm_stage<MI>() + (wm * 8 * MI + row) * GS + tq;
    const double* B = sm + (ck % GST) * gemm_stage<MI>() + (GM + wn * 32 + row) * GS;
    const int kw = R - ck * GK;
#pragma unroll
    for (int k0 = 0; k0 < GK; k0 += 4) {
      if (k0 >= kw) break;
      double a[MI], b[4];
#pragma unroll
      for (int i = 0; i < MI; ++i) a[i] = A[i * 8 * GS + k0];
      int k = k0 + tq, neg = 0;
      if (sym && k < kw) {
        const int o = s_opi[ck * GK + k];
        k ^= o & 1;
        neg = (o & 2) << 30;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double x = B[j * 8 * GS + k];
        b[j] = __hiloint2double(__double2hiint(x) ^ neg, __double2loint(x));
      }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
  }
  // acc[i][j][v] = C[row m0 + (wm MI + i) 8 + row][column c0 + wn 32 + 8 j + 2 tq + v]; with a
  // class symmetry, its output map first (the other part of the row's coefficient, row ^ 1,
  // is in lane ^ 4)
  if (sym) {
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int rr = m0 + (wm * MI + i) * 8 + row, op = rr < R ? s_opo[rr] : 0;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const double other = __shfl_xor_sync(0xffffffffu, acc[i][j][v], 4);
          const double w = (op & 1) ? other : acc[i][j][v];
          acc[i][j][v] = (op & 2) ? -w : w;
        }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int c = c0 + wn * 32 + j * 8 + 2 * tq + v;
      if (c >= ncol) continue;
      const int pr = p0 + c / nrhs, r = c % nrhs;
      double* y = cpair + ((size_t)pr * nrhs + r) * rp;
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int rr = m0 + (wm * MI + i) * 8 + row;
        if (rr < rp) y[rr] = acc[i][j][v];
      }
    }
}

// Tiled form of M2M / L2L: CTA tile of 64 rows x 64 columns
// (box x rhs), K streamed in chunks of 16 through a cp.async pipeline of GT_ST stages (the
// synchronous form waited for two rounds of global loads per chunk: 8.8 us of 140 us a
// launch); warp (wm, wn) owns 32 x 32 of the tile as 4 x 4 m8n8 accumulators.  Both
// operands are staged k-contiguous with a row stride of 20 doubles (4 mod 16), free of
// bank conflicts as fragments.
//   L2L (SUM false): blockIdx.z = one of the level's eight groups; a group's children are
//   distinct, so each column is added into its child.
//   M2M (SUM true): a cluster of eight CTAs along z, one per child position of the
//   parents of the column tile; the eight products are summed in a fixed order through
//   distributed shared memory (rank q sums the rows 8 q .. 8 q + 7) and added into the
//   parents: one launch per level instead of eight that follow one another.
constexpr int GT_M = 64, GT_N = 64, GT_K = 16, GT_ST = 4;
constexpr int GT_S = GT_K + 4;               // row stride of a staged operand (doubles)
constexpr int GT_STAGE = (GT_M + GT_N) * GT_S;
constexpr int GT_CS = GT_N + 4;              // row stride of the result tile (doubles)

template <bool SUM>
__global__ void __launch_bounds__(NT)
k_trans_gemm_pipe(qbxfmm_geometry g, int ncf, int rp, int kp, int nrhs,
                  const double* __restrict__ T, int mat_mod, int g0, int i0, int i1,
                  double2* __restrict__ exps, int32_t* err)
{
  extern __shared__ double2 smem2[];
  double* sm = reinterpret_cast<double*>(smem2);
  __shared__ int s_src[GT_N], s_dst[GT_N];
  const int grp = g0 + blockIdx.z;
  const int p0 = SUM ? i0 : g.l2l_group_starts[grp], p1 = SUM ? i1 : g.l2l_group_starts[grp + 1];
  const int ncol = (p1 - p0) * nrhs;
  const int c0 = blockIdx.x * GT_N, m0 = blockIdx.y * GT_M;
  if (!SUM && c0 >= ncol) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int R = 2 * ncf;
  bool any = false;
  for (int j = tid; j < GT_N; j += NT) {
    const int c = c0 + j;
    int src = -1, dst = -1;
    if (c < ncol) {
      const int q = p0 + c / nrhs;
      if (SUM) {
        dst = g.source_parent_boxes[q];
        if ((unsigned)dst < (unsigned)g.nboxes) {
          src = g.box_child_ids[(size_t)blockIdx.z * g.nboxes + dst];
          if (src == 0) src = -1;                        // no such child
          else if ((unsigned)src >= (unsigned)g.nboxes) report(err, QBX_DEVERR_BAD_BOX), src = -1;
          else if (g.box_source_counts_cumul[src] == 0) src = -1;
        }
      } else {
        src = g.l2l_pair_src[q];
        dst = g.l2l_pair_dst[q];
        if ((unsigned)src >= (unsigned)g.nboxes) report(err, QBX_DEVERR_BAD_BOX), src = -1;
      }
      if ((unsigned)dst >= (unsigned)g.nboxes) report(err, QBX_DEVERR_BAD_BOX), dst = -1;
    }
    s_src[j] = src;
    s_dst[j] = dst;
    any |= src >= 0;
  }
  any = __syncthreads_or(any);
  const double* Tg = T + (size_t)(mat_mod > 0 ? grp % mat_mod : grp) * rp * kp;
  // this thread's 16-byte pieces of a chunk: rows / columns tid / 8 + 16 i, k = 2 (tid % 8)
  const int kk = 2 * (tid & 7), rb = tid >> 3;
  const double* ap[4];
  const double* bp[4];
  bool aon[4], bon[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = m0 + rb + 16 * i, src = s_src[rb + 16 * i];
    aon[i] = row < rp;
    ap[i] = Tg + (size_t)(aon[i] ? row : 0) * kp + kk;
    bon[i] = src >= 0;
    bp[i] = reinterpret_cast<const double*>(
                exps + ((size_t)(bon[i] ? src : 0) * nrhs + (c0 + rb + 16 * i) % nrhs) * ncf) + kk;
  }
  const int nk = any ? (R + GT_K - 1) / GT_K : 0;
  auto fetch = [&](int ck) {
    if (ck < nk) {
      double* A = sm + (ck % GT_ST) * GT_STAGE;
      double* B = A + GT_M * GT_S;
      const bool in = ck * GT_K + kk < R;                // kp >= R; the rest is zero
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const bool a = aon[i] && in, b = bon[i] && in;
        cp_async16_zfill(A + (rb + 16 * i) * GT_S + kk, a ? ap[i] + ck * GT_K : Tg, a);
        cp_async16_zfill(B + (rb + 16 * i) * GT_S + kk, b ? bp[i] + ck * GT_K : Tg, b);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const int row = lane >> 2, tq = lane & 3, wm = warp & 1, wn = warp >> 1;
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  for (int i = 0; i < GT_ST - 1; ++i) fetch(i);
  for (int ck = 0; ck < nk; ++ck) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(GT_ST - 2) : "memory");
    __syncthreads();
    fetch(ck + GT_ST - 1);                               // into the stage read last round
    const double* A = sm + (ck % GT_ST) * GT_STAGE + (wm * 32 + row) * GT_S + tq;
    const double* B = sm + (ck % GT_ST) * GT_STAGE + (GT_M + wn * 32 + row) * GT_S + tq;
#pragma unroll
    for (int k0 = 0; k0 < GT_K; k0 += 4) {
      double a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = A[i * 8 * GT_S + k0];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = B[j * 8 * GT_S + k0];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  // acc[i][j][v] = C[row m0 + wm 32 + 8 i + row][column c0 + wn 32 + 8 j + 2 tq + v]
  if constexpr (!SUM) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const int jc = wn * 32 + j * 8 + 2 * tq + v, dst = s_dst[jc];
        if (dst < 0) continue;
        double* y = reinterpret_cast<double*>(exps + ((size_t)dst * nrhs + (c0 + jc) % nrhs) * ncf);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int rr = m0 + wm * 32 + i * 8 + row;
          if (rr < R) y[rr] += acc[i][j][v];
        }
      }
  } else {
    cg::cluster_group cl = cg::this_cluster();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int v = 0; v < 2; ++v)
          sm[(wm * 32 + i * 8 + row) * GT_CS + wn * 32 + j * 8 + 2 * tq + v] = acc[i][j][v];
    cl.sync();
    const int rank = blockIdx.z;
    for (int e = tid; e < 8 * GT_N; e += NT) {
      const int jc = e >> 3, rl = 8 * rank + (e & 7), rr = m0 + rl;
      double v = 0.0;
      for (int z = 0; z < 8; ++z) v += cl.map_shared_rank(sm, z)[rl * GT_CS + jc];
      const int dst = s_dst[jc];
      if (dst < 0 || rr >= R) continue;
      double* y = reinterpret_cast<double*>(exps + ((size_t)dst * nrhs + (c0 + jc) % nrhs) * ncf);
      y[rr] += v;
    }
    cl.sync();
  }
}

// out box o (o = boxes[obase + blockIdx.x]): eout[o][r] += scale(o) sum_{pairs} cpair[pair][r]
// scale(o) = 1 / width(level(o)) when div_by_width, else 1.
__global__ void __launch_bounds__(NT)
k_trans_reduce(int ncf, int rp, int nrhs, const int32_t* __restrict__ boxes, int obase,
               const int32_t* __restrict__ starts, const int32_t* __restrict__ pairs,
               const double* __restrict__ cpair, double2* __restrict__ eout, int div_by_width,
               const int32_t* __restrict__ box_levels, double root_extent)
{
  int i = obase + blockIdx.x;
  int o = boxes[i];
  int r = blockIdx.y;
  double sc = div_by_width ? ldexp(1.0, box_levels[o]) / root_extent : 1.0;
  int R = 2 * ncf;
  double* y = reinterpret_cast<double*>(eout + ((size_t)o * nrhs + r) * ncf);
  const int q0 = starts[i], q1 = starts[i + 1];
  // the box's pair rows, staged once per chunk so that the loads of successive pairs
  // are independent
  constexpr int QC = 256;
  __shared__ const double* s_row[QC];
  for (int row0 = 0; row0 < R; row0 += NT) {
    const int row = row0 + threadIdx.x;
    double acc = 0.0;
    for (int qc = q0; qc < q1; qc += QC) {
      const int nq = min(QC, q1 - qc);
      __syncthreads();
      for (int t = threadIdx.x; t < nq; t += NT)
        s_row[t] = cpair + ((size_t)pairs[qc + t] * nrhs + r) * rp;
      __syncthreads();
      if (row < R) {
#pragma unroll 4
        for (int t = 0; t < nq; ++t) acc += s_row[t][row];
      }
    }
    if (row < R) y[row] += sc * acc;
  }
}

// }}}

// {{{ launchers

static void dims_from_ncf(int ncf, int& rp, int& kp)
{
  rp = (2 * ncf + 7) / 8 * 8;
  kp = (2 * ncf + 3) / 4 * 4;
}

TransCfg trans_cfg_laplace3(int p, int nclasses)
{
  TransCfg c;
  c.p = p;
  c.ncf = (p + 1) * (p + 2) / 2;
  dims_from_ncf(c.ncf, c.rp, c.kp);
  c.m2m_mat_mod = 8;
  c.m2m_base = nclasses;
  c.l2l_base = nclasses + 8;
  c.m2l_div_by_width = 1;
  c.nmatrices = nclasses + 16;
  return c;
}

TransCfg trans_cfg_helm3(int p, int nclasses, int nlevels)
{
  TransCfg c;
  c.p = p;
  c.ncf = (p + 1) * (p + 1);
  dims_from_ncf(c.ncf, c.rp, c.kp);
  c.m2m_mat_mod = 0;
  c.m2m_base = nclasses;
  c.l2l_base = nclasses + 8 * (size_t)nlevels;
  c.m2l_div_by_width = 0;
  c.nmatrices = nclasses + 16 * (size_t)nlevels;
  return c;
}

size_t trans_matrix_bytes(const TransCfg& c) { return c.nmatrices * c.rp * c.kp * sizeof(double); }

size_t trans_scratch_bytes(const TransCfg& c, int npairs, int nrhs)
{
  return (size_t)(npairs > 0 ? npairs : 1) * nrhs * c.rp * sizeof(double);
}

bool trans_supported(const TransCfg& c) { return c.rp <= 672; }

M2LSymClasses m2l_symmetry_classes(int nclasses, const std::vector<int32_t>& offs)
{
  M2LSymClasses r;
  r.cls_code.resize(nclasses);
  std::vector<std::array<int, 3>> canon;
  std::map<std::array<int, 3>, int> index;
  for (int c = 0; c < nclasses; ++c) {
    const int dx = offs[c], dy = offs[(size_t)nclasses + c], dz = offs[2 * (size_t)nclasses + c];
    const int a = std::max(std::abs(dx), std::abs(dy)), b = std::min(std::abs(dx), std::abs(dy));
    const std::array<int, 3> key = {a, b, std::abs(dz)};
    // (dx, dy) = R^q C^s (a, b)
    int code = -1;
    for (int q = 0; q < 4 && code < 0; ++q)
      for (int s = 0; s < 2 && code < 0; ++s) {
        int x = a, y = s ? -b : b;
        for (int i = 0; i < q; ++i) {
          const int t = x;
          x = -y;
          y = t;
        }
        if (x == dx && y == dy) code = q | s << 2 | (dz < 0 ? 8 : 0);
      }
    auto it = index.find(key);
    int ci;
    if (it == index.end()) {
      ci = (int)canon.size();
      index.emplace(key, ci);
      canon.push_back(key);
    } else {
      ci = it->second;
    }
    if (code < 0) {                      // not a lattice offset: no shared matrices
      r.ncanon = -1;
      return r;
    }
    r.cls_code[c] = ci << 4 | code;
  }
  r.ncanon = (int)canon.size();
  r.canon_off.resize(3 * (size_t)r.ncanon);
  for (int i = 0; i < r.ncanon; ++i)
    for (int k = 0; k < 3; ++k) r.canon_off[(size_t)k * r.ncanon + i] = canon[i][k];
  return r;
}

// T layout: [0, nm2l) M2L matrices (one per canonical offset), then M2M and L2L
// matrices (TransCfg bases); offs: [3][nm2l] on the device
cudaError_t launch_trans_build(const TransCfg& c, int nm2l, const int32_t* offs, double* T,
                               cudaStream_t st)
{
  int p = c.p;
  size_t sh = (size_t)(2 * p + 1) * (2 * p + 2) / 2 * sizeof(double2);
  size_t stride = (size_t)c.rp * c.kp;
  if (nm2l > 0)
    k_trans_build<<<nm2l, NT, sh, st>>>(0, p, c.ncf, c.rp, c.kp, nm2l, offs, T);
  k_trans_build<<<8, NT, sh, st>>>(1, p, c.ncf, c.rp, c.kp, 8, nullptr, T + c.m2m_base * stride);
  k_trans_build<<<8, NT, sh, st>>>(2, p, c.ncf, c.rp, c.kp, 8, nullptr, T + c.l2l_base * stride);
  return cudaGetLastError();
}

static cudaError_t m2l_products(const qbxfmm_geometry& g, const TransCfg& c, int nrhs,
                                const double* T, const int32_t* cls_code, int maxcols,
                                const double2* mp, double* cpair, int32_t* err, cudaStream_t st)
{
  if (maxcols <= 0) return cudaSuccess;
  // the tile height with the fewest rows past the end, the tallest of those
  const int mt = (c.rp + 7) / 8;
  int mi = 3;
  auto rows = [&](int m) { return (mt + 2 * m - 1) / (2 * m) * 2 * m; };
  for (int m = 4; m <= 6; ++m)
    if (rows(m) <= rows(mi)) mi = m;
  auto launch = [&](auto height) {
    constexpr int MI = decltype(height)::value;
    const size_t sh = (size_t)GST * gemm_stage<MI>() * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(k_trans_gemm<MI>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
    if (e != cudaSuccess) return e;
    const dim3 grid((maxcols + GN - 1) / GN, (c.rp + 16 * MI - 1) / (16 * MI), g.m2l_nclasses);
    k_trans_gemm<MI><<<grid, NT, sh, st>>>(c.ncf, c.rp, c.kp, nrhs, T, cls_code, g.m2l_class_starts,
                                           g.m2l_pair_src, mp, cpair, err, g.nboxes);
    return cudaGetLastError();
  };
  switch (mi) {
    case 3: return launch(std::integral_constant<int, 3>());
    case 4: return launch(std::integral_constant<int, 4>());
    case 5: return launch(std::integral_constant<int, 5>());
    default: return launch(std::integral_constant<int, 6>());
  }
}

cudaError_t launch_m2l_gemm(const qbxfmm_geometry& g, const TransHost& th, const TransCfg& c,
                            int nrhs, const double* T, const TransAux& aux, const double2* mp,
                            double2* lo, double* cpair, int32_t* err, cudaStream_t st)
{
  if (g.m2l_nclasses == 0) return cudaSuccess;
  cudaError_t e = m2l_products(g, c, nrhs, T, aux.cls_code, th.m2l_max_pairs * nrhs, mp, cpair, err,
                               st);
  if (e != cudaSuccess) return e;
  return launch_trans_reduce_m2l(g, c, nrhs, cpair, lo, st);
}

cudaError_t launch_trans_reduce_m2l(const qbxfmm_geometry& g, const TransCfg& c, int nrhs,
                                    const double* cpair, double2* lo, cudaStream_t st)
{
  if (g.nttp_boxes == 0) return cudaSuccess;
  k_trans_reduce<<<dim3(g.nttp_boxes, nrhs), NT, 0, st>>>(
      c.ncf, c.rp, nrhs, g.target_or_target_parent_boxes, 0, g.m2l_tgt_pair_starts,
      g.m2l_tgt_pairs, cpair, lo, c.m2l_div_by_width, g.box_levels, g.root_extent);
  return cudaGetLastError();
}

cudaError_t launch_trans_reduce_m2m(const qbxfmm_geometry& g, const TransHost& th, const TransCfg& c,
                                    int lev, int nrhs, const double* cpair, double2* mp,
                                    cudaStream_t st)
{
  int i0 = th.lvl_source_parent[lev], i1 = th.lvl_source_parent[lev + 1];
  if (i1 > i0)
    k_trans_reduce<<<dim3(i1 - i0, nrhs), NT, 0, st>>>(c.ncf, c.rp, nrhs, g.source_parent_boxes, i0,
                                                       g.m2m_par_pair_starts, g.m2m_par_pairs, cpair,
                                                       mp, 0, g.box_levels, g.root_extent);
  return cudaGetLastError();
}

template <bool SUM>
static cudaError_t gemm_pipe_launch(const qbxfmm_geometry& g, const TransCfg& c, int nrhs,
                                    const double* T, size_t mat_base, int g0, int i0, int i1,
                                    int maxcols, double2* exps, int32_t* err, cudaStream_t st)
{
  if (maxcols <= 0) return cudaSuccess;
  const size_t sh = (size_t)std::max(GT_ST * GT_STAGE, GT_M * GT_CS) * sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(k_trans_gemm_pipe<SUM>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((maxcols + GT_N - 1) / GT_N, (2 * c.ncf + GT_M - 1) / GT_M, 8);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = sh;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = SUM ? 8 : 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_trans_gemm_pipe<SUM>, g, c.ncf, c.rp, c.kp, nrhs,
                            T + mat_base * (size_t)c.rp * c.kp, c.m2m_mat_mod, g0, i0, i1, exps,
                            err);
}

// M2M without pair scratch: one launch per parent level
cudaError_t launch_m2m_direct(const qbxfmm_geometry& g, const TransHost& th, const TransCfg& c,
                              int nrhs, const double* T, double2* mp, int32_t* err, cudaStream_t st)
{
  for (int lev = g.nlevels - 2; lev >= 0; --lev) {
    if (th.m2m_level_max_group[lev] == 0) continue;
    const int i0 = th.lvl_source_parent[lev], i1 = th.lvl_source_parent[lev + 1];
    cudaError_t e = gemm_pipe_launch<true>(g, c, nrhs, T, c.m2m_base, lev * 8, i0, i1,
                                           (i1 - i0) * nrhs, mp, err, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// L2L on the tiled kernel (children are distinct across a level's eight groups)
cudaError_t launch_l2l_direct(const qbxfmm_geometry& g, const TransHost& th, const TransCfg& c,
                              int nrhs, const double* T, double2* lo, int32_t* err, cudaStream_t st)
{
  for (int lev = 1; lev < g.nlevels; ++lev) {
    cudaError_t e = gemm_pipe_launch<false>(g, c, nrhs, T, c.l2l_base, lev * 8, 0, 0,
                                            th.l2l_level_max_group[lev] * nrhs, lo, err, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}


bool trans_small(const TransCfg& c) { return c.ncf <= NT; }

// }}}

}  // namespace qbx
