// 2D Helmholtz: list-3 multipoles and box locals straight to the QBX targets, complex128,
// sm_100a.
//
// M2QBXL / L2QBXL followed by QBXL2P is, per (target t, its center c, box), a linear
// functional of the box's coefficients that no density enters: with Z = H (multipoles) or
// J (locals), Zt_m = J_m(k|t - c|) e^{i m th},
//   u(t) = sum_n E_n w_n,  w_n = f(n) sum_{|m| <= Q} Zt_m Z_{n-m}(c - c_b),
// f(n) = rho_b^{+-|n|}.  The (2p + 1)(2Q + 1) products are done once per (target, box)
// instead of once per density, and the densities see 2p + 1 of them: the rows w of the
// chunk's targets times the box's coefficients on the FP64 tensor cores, 8 targets x 4
// coefficients x (4 densities, re / im).  With 64 densities the expansions took 2.13 ms
// (M2QBXL), 0.65 ms (L2QBXL) and 0.14 ms (QBXL2P) of a 12.5 ms apply.
#include <algorithm>

#include "../../include/qbxfmm_api.h"
#include "helmholtz.cuh"
#include "helm3.cuh"
#include "kernels.h"

namespace qbx {

namespace {

constexpr int E2T_NT = 128;
constexpr int E2T_PB = 64;          // (target, box) pairs per batch
constexpr int E2T_MB = 8;           // boxes per batch
constexpr int E2T_MAXP = 20;
constexpr int E2T_NC = 2 * E2T_MAXP + 1;

// row stride of the weights (complex): the columns padded to 4, 4 mod 8
__host__ __device__ constexpr int e2t_stride(int p)
{
  const int c = (2 * p + 4) & ~3;
  return (c & 7) == 4 ? c : c + 4;
}

// Each warp: OC octets of the chunk's targets x NTW tiles of 4 densities.  OC = 1: warp =
// octet (up to 4 NTW densities); OC = 4: the warps split the density tiles.
template <int Q, bool FROM_LOCAL, int OC, int NTW>
__global__ void __launch_bounds__(E2T_NT)
k_h2_e2t(qbxfmm_geometry g, double k, int p, int nrhs, const double2* __restrict__ exps,
         double2* __restrict__ pot_tree, int32_t* err)
{
  constexpr int NQ = 2 * Q + 1;
  constexpr int NR = (OC == 1 ? 1 : 4) * NTW * 4;      // densities per CTA
  extern __shared__ double2 smem2[];
  const int NZ = p + Q, ZW = 2 * NZ + 1, NC = 2 * p + 1, WS = e2t_stride(p);
  double2* Zs = smem2;                                 // [PB][ZW]
  double2* W = Zs + (size_t)E2T_PB * ZW;               // [PB + 8][WS]
  __shared__ double2 s_zt[32][NQ];
  __shared__ double s_cc[2][32], s_fn[E2T_MB][E2T_NC];
  __shared__ int s_sb[E2T_MB], s_t[32];
  const int chunk = blockIdx.x, r0 = blockIdx.y * NR;
  const int itb = g.tsqbx_chunk_target_box[chunk];
  const int cnt = min(g.tsqbx_chunk_count[chunk], 32), i0 = g.tsqbx_chunk_start[chunk];
  const int l0 = FROM_LOCAL ? 0 : g.list3_starts[itb];
  const int l1 = FROM_LOCAL ? 1 : g.list3_starts[itb + 1];
  if (l1 <= l0 || cnt <= 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double Jb[2 * E2T_MAXP + 2], Yb[2 * E2T_MAXP + 2];
  if (tid < cnt) {
    int t = g.tsqbx_targets[i0 + tid], ctr = g.tsqbx_centers[i0 + tid];
    s_t[tid] = t;
    if ((unsigned)ctr >= (unsigned)g.ncenters || (unsigned)t >= (unsigned)g.ntargets) {
      report(err, QBX_DEVERR_BAD_CENTER);
      s_t[tid] = -1;
      t = ctr = 0;
    }
    double cc[2], x[2];
    load_point<2>(g.centers, g.ncenters, ctr, cc);
    load_point<2>(g.targets, g.ntargets, t, x);
    s_cc[0][tid] = cc[0];
    s_cc[1][tid] = cc[1];
    h2_zfun(Q, k, x[0] - cc[0], x[1] - cc[1], Jb, Yb, s_zt[tid], false);
  }
  // rows past the last pair are read as part of an octet and must be finite
  for (int e = tid; e < (E2T_PB + 8) * WS; e += E2T_NT) W[e] = c2(0.0);
  const int row = lane >> 2, kq = lane & 3;
  const int o0 = OC == 1 ? warp : 0, t0 = OC == 1 ? 0 : warp * NTW;
  const bool busy = 8 * o0 < cnt && r0 + 4 * t0 < nrhs;
  double acc[OC][NTW][2];
#pragma unroll
  for (int o = 0; o < OC; ++o)
#pragma unroll
    for (int w = 0; w < NTW; ++w) acc[o][w][0] = acc[o][w][1] = 0.0;

  const int per = min(E2T_MB, max(1, E2T_PB / cnt));   // boxes per batch
  for (int lb = l0; lb < l1; lb += per) {
    const int nbat = min(per, l1 - lb), npair = nbat * cnt;
    __syncthreads();
    if (tid < nbat) {
      int sb = FROM_LOCAL ? g.target_boxes[itb] : g.list3_lists[lb + tid];
      if ((unsigned)sb >= (unsigned)g.nboxes) {
        report(err, QBX_DEVERR_BAD_BOX);
        sb = -1;
      }
      s_sb[tid] = sb;
    }
    __syncthreads();
    for (int pi = tid; pi < npair; pi += E2T_NT) {
      const int bb = pi / cnt, t = pi - bb * cnt, sb = s_sb[bb];
      if (sb < 0) continue;
      double cs[2];
      load_point<2>(g.box_centers, g.nboxes, sb, cs);
      h2_zfun(NZ, k, s_cc[0][t] - cs[0], s_cc[1][t] - cs[1], Jb, Yb, Zs + (size_t)pi * ZW,
              !FROM_LOCAL);
    }
    for (int w = tid; w < nbat * NC; w += E2T_NT) {
      const int bb = w / NC, n = w - bb * NC, sb = s_sb[bb];
      if (sb < 0) continue;
      const double rho = level_width(g, g.box_levels[sb]);
      const double an = (double)abs(n - p);
      s_fn[bb][n] = FROM_LOCAL ? pow(rho, -an) : pow(rho, an);
    }
    __syncthreads();
    for (int e = tid; e < npair * NC; e += E2T_NT) {
      const int pi = e / NC, n = e - pi * NC, bb = pi / cnt, t = pi - bb * cnt;
      double2 v = c2(0.0);
      if (s_sb[bb] >= 0) {
        // coefficient n - p, order m = a - Q: Z_{n-m} at index NZ + (n - p) - (a - Q)
        const double2* Z = Zs + (size_t)pi * ZW + NZ + n - p + Q;
#pragma unroll
        for (int a = 0; a < NQ; ++a) v = cfma(s_zt[t][a], Z[-a], v);
        v = cscale(s_fn[bb][n], v);
      }
      W[pi * WS + n] = v;
    }
    __syncthreads();
    if (!busy) continue;
    for (int bb = 0; bb < nbat; ++bb) {
      const int sb = s_sb[bb];
      if (sb < 0) continue;
      const double2* Eb = exps + ((size_t)sb * nrhs + r0) * NC;
      const double2* Wb = W + (size_t)(bb * cnt + 8 * o0 + row) * WS + kq;
#pragma unroll 2
      for (int ks = 0; 4 * ks < NC; ++ks) {
        const int n = 4 * ks + kq;
        double2 e[NTW];
#pragma unroll
        for (int w = 0; w < NTW; ++w) {
          const int r = 4 * (t0 + w) + (row >> 1);
          e[w] = (n < NC && r0 + r < nrhs) ? __ldg(Eb + (size_t)r * NC + n) : c2(0.0);
        }
#pragma unroll
        for (int o = 0; o < OC; ++o) {
          if (8 * (o0 + o) >= cnt) break;
          const double2 wv = Wb[(size_t)8 * o * WS + 4 * ks];
#pragma unroll
          for (int w = 0; w < NTW; ++w) {
            // column (density, part): E, and i E for the imaginary part of the weight
            const double b = (row & 1) ? e[w].y : e[w].x, bx = (row & 1) ? e[w].x : -e[w].y;
            h3_dmma(acc[o][w][0], acc[o][w][1], wv.x, b);
            h3_dmma(acc[o][w][0], acc[o][w][1], wv.y, bx);
          }
        }
      }
    }
  }
  if (!busy) return;
#pragma unroll
  for (int o = 0; o < OC; ++o) {
    const int ti = 8 * (o0 + o) + row;
    if (ti >= cnt || s_t[ti] < 0) continue;
#pragma unroll
    for (int w = 0; w < NTW; ++w) {
      const int r = r0 + 4 * (t0 + w) + kq;
      if (r >= nrhs) continue;
      double2* P = pot_tree + (size_t)r * g.ntargets + s_t[ti];
      *P = cadd(*P, c2(acc[o][w][0], acc[o][w][1]));
    }
  }
}

template <int Q, bool FROM_LOCAL, int OC, int NTW>
cudaError_t e2t_launch(const qbxfmm_geometry& g, double k, int p, int nrhs, const double2* e,
                       double2* pot, int32_t* err, cudaStream_t st)
{
  constexpr int NR = (OC == 1 ? 1 : 4) * NTW * 4;
  const size_t sh = ((size_t)E2T_PB * (2 * (p + Q) + 1) + (size_t)(E2T_PB + 8) * e2t_stride(p)) *
                    sizeof(double2);
  cudaError_t rc = cudaFuncSetAttribute(k_h2_e2t<Q, FROM_LOCAL, OC, NTW>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  if (rc != cudaSuccess) return rc;
  k_h2_e2t<Q, FROM_LOCAL, OC, NTW><<<dim3(g.ntsqbx_chunks, (nrhs + NR - 1) / NR), E2T_NT, sh, st>>>(
      g, k, p, nrhs, e, pot, err);
  return cudaGetLastError();
}

template <int Q, bool FROM_LOCAL>
cudaError_t e2t_q(const qbxfmm_geometry& g, double k, int p, int nrhs, const double2* e, double2* pot,
                  int32_t* err, cudaStream_t st)
{
  if (nrhs > 16) return e2t_launch<Q, FROM_LOCAL, 4, 4>(g, k, p, nrhs, e, pot, err, st);
  if (nrhs > 8) return e2t_launch<Q, FROM_LOCAL, 1, 4>(g, k, p, nrhs, e, pot, err, st);
  if (nrhs > 4) return e2t_launch<Q, FROM_LOCAL, 1, 2>(g, k, p, nrhs, e, pot, err, st);
  return e2t_launch<Q, FROM_LOCAL, 1, 1>(g, k, p, nrhs, e, pot, err, st);
}

}  // namespace

// Less work than the expansions, but after the near field, which writes the same potential,
// where M2QBXL runs beside it: with few chunks the apply is as long as its longest stream, and
// the expansions are faster.  That line lies higher where no other targets' P2P and M2P take
// the GPU meanwhile, and where the expansions are little work: up to four densities, whose
// M2QBXL wastes no lanes, and low orders, by (2q + 1) (2p + 1) a density.  Time of the starfish's
// apply with the expansions over this form's:
//   no other targets, 350, 414, 498, 600, 680, 724, 759 and 964 chunks: 7 densities q 5, p 20
//   0.98 0.99 1.04 1.09 1.11 1.11 1.18 1.16; q 4, p 18 0.83 0.95 0.97 0.98 1.06 1.02 1.17 1.18;
//   q 3, p 15 0.82 0.90 0.94 0.96 0.99 0.95 1.10 1.06; q 1, p 6 0.85 0.82 0.86 0.87 0.91 0.86 0.96
//   1.06; 16 densities q 6, p 18 0.94 0.99 1.02 1.02 1.06 1.02 1.09 1.11; 64 densities, 296 and
//   733 chunks: q 6, p 20 1.04 1.21, q 3, p 15 0.94 1.08, q 2, p 8 0.91 0.92; 4 densities, q 5,
//   p 20, 414, 634, 733 and 1081: 0.81 0.90 0.94 1.13;
//   30 others, q 5, p 20, 84, 216, 326 and 414 chunks: 1 density 0.91 0.77 0.84 1.06, 16 0.86
//   0.78 0.93 1.07; 100 others, 216: 1 density 1.15, 2 1.05, 8 1.07; 1000 others, 300 chunks,
//   orders 0 to 8: 0.99 to 1.10.
bool h2_e2t_wins(const qbxfmm_geometry& g, int p, int q, int nrhs)
{
  if (g.ntsqbx_chunks == 0) return false;
  if (!h2_m2qbxl_fits(p, q, nrhs)) return true;
  const int work = (2 * q + 1) * (2 * p + 1);
  int per_sm = 5;
  if (g.nnonqbx_chunks > 0) per_sm = nrhs == 1 ? 1 : 2;
  else if (nrhs > 4 && work >= 400) per_sm = nrhs > 32 ? 2 : 3;
  else if (nrhs > 32 && work >= 160) per_sm = 4;
  return g.ntsqbx_chunks >= per_sm * 148 &&
         g.ntsqbx_chunks <= g.nqbx_chunks * (nrhs >= 4 ? 4 : 1);
}

cudaError_t h2_launch_e2t(const qbxfmm_geometry& g, double k, int p, int q, int nrhs,
                          bool from_local, const double2* exps, double2* pot_tree, int32_t* err,
                          cudaStream_t st)
{
  if (g.ntsqbx_chunks == 0) return cudaSuccess;
  if (p > E2T_MAXP) return cudaErrorInvalidValue;
#define QBX_E2T(Q)                                                                   \
  case Q:                                                                            \
    return from_local ? e2t_q<Q, true>(g, k, p, nrhs, exps, pot_tree, err, st)       \
                      : e2t_q<Q, false>(g, k, p, nrhs, exps, pot_tree, err, st);
  switch (q) {
    QBX_E2T(0) QBX_E2T(1) QBX_E2T(2) QBX_E2T(3) QBX_E2T(4)
    QBX_E2T(5) QBX_E2T(6) QBX_E2T(7) QBX_E2T(8)
    default: return cudaErrorInvalidValue;
  }
#undef QBX_E2T
}

}  // namespace qbx
