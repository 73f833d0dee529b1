// 3D Helmholtz, the reference's default (compressed Taylor) truncation: box locals
// straight to the QBX targets, complex128, sm_100a.
//
// L2QBXL followed by QBXL2P re-centers the box's order-p polynomial P (wave units, k x)
// at the QBX center, keeps the derivatives with z exponent <= 1 up to degree Q, rebuilds
// the others through the PDE and evaluates at the target.  That is a linear functional of P,
// the same for every density, with real weights:
//   u(t) = sum_{ABC} w_ABC P_ABC,  w_ABC = sum_{a,b,c<=1} c_abc binom(A,a) vx^(A-a)
//                                                binom(B,b) vy^(B-b) binom(C,c) vz^(C-c),
// v = k (center - box), c_abc the value at the target of the polynomial with the stored
// monomial (a, b, c) alone (the PDE rebuild transposed, 56 terms at Q = 5).  The chunk's
// targets (rows) times the monomials is a product on the FP64 tensor cores with the
// densities (columns); per center and density it was a separable shift in registers
// (31.8 ms for 307 200 targets and 16 densities, against 0.5 ms of products).
#include <algorithm>

#include "../../include/qbxfmm_api.h"
#include "helm3.cuh"
#include "kernels.h"
#include "taylor_h3.h"

namespace qbx {

namespace {

constexpr int L2T_NT = 128;
constexpr int L2T_RB = 8;          // densities per CTA: 16 columns of 8 bytes a row

// monomials ordered (C, A, B): all A, B of z exponent C before C + 1, B fastest
QBX_HD int l2t_off(int p, int C)
{
  int o = 0;
  for (int c = 0; c < C; ++c) o += (p - c + 1) * (p - c + 2) / 2;
  return o;
}

QBX_HD int l2t_rows(int p)
{
  const int nmono = (p + 1) * (p + 2) * (p + 3) / 6, two = 2 * (p + 1) * (p + 1);
  return (nmono > two ? nmono : two) + 4;
}

// row r's column c (density, re / im) is stored at c ^ 4 (r mod 4): four consecutive rows
// of a B fragment fall into different banks
QBX_HD int l2t_at(int r, int c) { return r * 16 + (c ^ (4 * (r & 3))); }

// One octet of the chunk's targets per warp.  Lane: target lane / 4, y exponents
// B = 4 u + lane % 4 (the inner index of a tensor-core step; A and C are the lane's
// loops).
template <int Q>
__global__ void __launch_bounds__(L2T_NT)
k_h3_l2t(qbxfmm_geometry g, HelmCoeffs hc, int p, int nrhs, const double2* __restrict__ locals,
         const double2* __restrict__ G0, double2* __restrict__ pot_tree, int32_t* err)
{
  extern __shared__ double2 smem2[];
  double* P = reinterpret_cast<double*>(smem2);          // [l2t_rows][16]
  __shared__ int s_off[H3T_MAXP + 2];
  __shared__ unsigned char s_st[H3T_MAXP2 * 3];          // stored exponents (c <= 1)
  const int ncf = (p + 1) * (p + 1), nmono = (p + 1) * (p + 2) * (p + 3) / 6;
  const int chunk = blockIdx.x, r0 = blockIdx.y * L2T_RB;
  const int itb = g.tsqbx_chunk_target_box[chunk];
  const int cnt = g.tsqbx_chunk_count[chunk];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if ((unsigned)itb >= (unsigned)g.ntarget_boxes) {
    if (tid == 0) report(err, QBX_DEVERR_BAD_BOX);
    return;
  }
  const int tb = g.target_boxes[itb];
  if ((unsigned)tb >= (unsigned)g.nboxes) {
    if (tid == 0) report(err, QBX_DEVERR_BAD_BOX);
    return;
  }
  const double k = hc.k;
  const double si = 1.0 / h3_scale(k, level_width(g, g.box_levels[tb]));
  if (tid <= p + 1) s_off[tid] = l2t_off(p, tid);
  if (tid == 0) {
    int s = 0;
    for (int c = 0; c <= 1 && c <= p; ++c)
      for (int a = 0; a + c <= p; ++a)
        for (int b = 0; a + b + c <= p; ++b, ++s) {
          s_st[3 * s] = (unsigned char)a;
          s_st[3 * s + 1] = (unsigned char)b;
          s_st[3 * s + 2] = (unsigned char)c;
        }
  }
  // the coefficients, unscaled, in the rows from ncf on (those of c >= 2, not yet formed)
  for (int e = tid; e < ncf * L2T_RB; e += L2T_NT) {
    const int r = e / ncf, c = e - r * ncf;
    int n, m;
    hq_decode(c, n, m);
    double2 v = c2(0.0);
    if (r0 + r < nrhs) {
      double f = 1.0;
      for (int i = 0; i < n; ++i) f *= si;
      v = cscale(f, __ldg(locals + ((size_t)tb * nrhs + r0 + r) * ncf + c));
    }
    *reinterpret_cast<double2*>(P + l2t_at(ncf + c, 2 * r)) = v;
  }
  for (int e = tid; e < 64; e += L2T_NT) P[(size_t)(l2t_rows(p) - 4) * 16 + e] = 0.0;
  __syncthreads();
  auto mono = [&](int a, int b, int c) {
    return s_off[c] + a * (p - c + 1) - a * (a - 1) / 2 + b;
  };
  // stored monomials: P_s = sum_nm G0[s][nm] b_nm over n <= a+b+c of its parity, |m| <= a+b
  // of the parity of a+b
  // (a thread per monomial, all densities: the table entries come from L2)
  for (int s = tid; s < ncf; s += L2T_NT) {
    const int a = s_st[3 * s], b = s_st[3 * s + 1], c = s_st[3 * s + 2];
    const int D = a + b + c, ab = a + b;
    double2 acc[L2T_RB];
#pragma unroll
    for (int r = 0; r < L2T_RB; ++r) acc[r] = c2(0.0);
    for (int n = D & 1; n <= D; n += 2) {
      const int mm = min(n, ab) - ((min(n, ab) + ab) & 1);
      const double2* G = G0 + (size_t)s * ncf + n * n + n;
#pragma unroll 4
      for (int m = -mm; m <= mm; m += 2) {
        const double2 gv = __ldg(G + m);
        const int at = ncf + n * n + n + m;
#pragma unroll
        for (int r = 0; r < L2T_RB; ++r)
          acc[r] = cfma(gv, *reinterpret_cast<const double2*>(P + l2t_at(at, 2 * r)), acc[r]);
      }
    }
    const int to = mono(a, b, c);
#pragma unroll
    for (int r = 0; r < L2T_RB; ++r) *reinterpret_cast<double2*>(P + l2t_at(to, 2 * r)) = acc[r];
  }
  __syncthreads();
  // the others from the PDE (Delta u + u = 0), by increasing exponent of z
  for (int c = 2; c <= p; ++c) {
    const int nab = (p - c + 1) * (p - c + 2) / 2;
    const double f = -1.0 / (c * (c - 1.0));
    for (int e = tid; e < nab * 16; e += L2T_NT) {
      const int w = e >> 4, col = e & 15;
      int a = 0, b = w;
      while (b >= p - c - a + 1) {
        b -= p - c - a + 1;
        ++a;
      }
      double v = P[l2t_at(mono(a, b, c - 2), col)];
      v = fma((a + 1.0) * (a + 2.0), P[l2t_at(mono(a + 2, b, c - 2), col)], v);
      v = fma((b + 1.0) * (b + 2.0), P[l2t_at(mono(a, b + 2, c - 2), col)], v);
      P[l2t_at(s_off[c] + w, col)] = f * v;
    }
    __syncthreads();
  }
  if (nmono + 4 < l2t_rows(p)) {        // rows past the last monomial that a fragment may read
    for (int e = tid; e < 64; e += L2T_NT) P[(size_t)nmono * 16 + e] = 0.0;
    __syncthreads();
  }
  if (8 * warp >= cnt) return;

  const int row = lane >> 2, kq = lane & 3;
  bool active = 8 * warp + row < cnt;
  const int pi = g.tsqbx_chunk_start[chunk] + min(8 * warp + row, cnt - 1);
  int t = g.tsqbx_targets[pi], ctr = g.tsqbx_centers[pi];
  if ((unsigned)ctr >= (unsigned)g.ncenters || (unsigned)t >= (unsigned)g.ntargets) {
    report(err, QBX_DEVERR_BAD_CENTER);
    active = false;
    t = ctr = 0;
  }
  double cc[3], x[3], cb[3];
  load_point<3>(g.centers, g.ncenters, ctr, cc);
  load_point<3>(g.targets, g.ntargets, t, x);
  load_point<3>(g.box_centers, g.nboxes, tb, cb);
  const double vx = k * (cc[0] - cb[0]), vy = k * (cc[1] - cb[1]), vz = k * (cc[2] - cb[2]);
  // c_abc: all monomials at the target, then the PDE transposed down to c <= 1
  double W[Q + 1][Q + 1][Q + 1];        // [c][a][b]
  {
    const double xa = k * (x[0] - cc[0]), ya = k * (x[1] - cc[1]), za = k * (x[2] - cc[2]);
    double pz = 1.0;
#pragma unroll
    for (int c = 0; c <= Q; ++c, pz *= za) {
      double px = pz;
#pragma unroll
      for (int a = 0; a + c <= Q; ++a, px *= xa) {
        double py = px;
#pragma unroll
        for (int b = 0; a + b + c <= Q; ++b, py *= ya) W[c][a][b] = py;
      }
    }
#pragma unroll
    for (int c = Q; c >= 2; --c)
#pragma unroll
      for (int a = 0; a + c <= Q; ++a)
#pragma unroll
        for (int b = 0; a + b + c <= Q; ++b) {
          const double w = -W[c][a][b] * (1.0 / (c * (c - 1.0)));
          W[c - 2][a][b] += w;
          W[c - 2][a + 2][b] = fma((a + 1.0) * (a + 2.0), w, W[c - 2][a + 2][b]);
          W[c - 2][a][b + 2] = fma((b + 1.0) * (b + 2.0), w, W[c - 2][a][b + 2]);
        }
  }
  double acc[2][2][2];                  // [parity of C][4 densities][two results]
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i >> 2][(i >> 1) & 1][i & 1] = 0.0;
  double py[Q + 1];                     // binom(B, b) vy^(B - b)
#pragma unroll
  for (int b = 0; b <= Q; ++b) py[b] = b == 0 ? 1.0 : 0.0;
  auto step = [](double* q, double v) {
#pragma unroll
    for (int b = Q; b >= 1; --b) q[b] = fma(v, q[b], q[b - 1]);
    q[0] *= v;
  };
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i < kq) step(py, vy);
  for (int u = 0; 4 * u <= p; ++u) {
    double px[Q + 1];                   // binom(A, a) vx^(A - a)
#pragma unroll
    for (int a = 0; a <= Q; ++a) px[a] = a == 0 ? 1.0 : 0.0;
    for (int A = 0; A + 4 * u <= p; ++A) {
      double y0 = 0.0, y1 = 0.0;
#pragma unroll
      for (int b = 0; b <= Q; ++b) {
        double t0 = 0.0, t1 = 0.0;
#pragma unroll
        for (int a = 0; a + b <= Q; ++a) {
          t0 = fma(W[0][a][b], px[a], t0);
          if (Q >= 1 && a + b + 1 <= Q) t1 = fma(W[Q >= 1 ? 1 : 0][a][b], px[a], t1);
        }
        y0 = fma(py[b], t0, y0);
        y1 = fma(py[b], t1, y1);
      }
      const int cmax = p - A - 4 * u - kq;           // the lane's last C
      double zc = 1.0, dz = 0.0;                     // vz^C and its derivative
      int idx = A * (p + 1) - A * (A - 1) / 2 + 4 * u + kq, tri = (p + 1) * (p + 2) / 2, ln = p + 1;
      for (int C = 0; C <= p - A - 4 * u; C += 2) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          // past the lane's (or the warp's) last C: weight 0, a row in bounds
          const bool on = C + h <= cmax;
          const double w = on ? fma(y1, dz, y0 * zc) : 0.0;
          const int rr = on ? idx : nmono;
          h3_dmma(acc[h][0][0], acc[h][0][1], w, P[l2t_at(rr, row)]);
          h3_dmma(acc[h][1][0], acc[h][1][1], w, P[l2t_at(rr, 8 + row)]);
          dz = fma(dz, vz, zc);
          zc *= vz;
          idx += tri - A;
          tri -= ln;
          --ln;
        }
      }
      step(px, vx);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) step(py, vy);
  }
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int r = r0 + 4 * n + kq;
    if (!active || r >= nrhs) continue;
    double2* O = pot_tree + (size_t)r * g.ntargets + t;
    *O = cadd(*O, c2(acc[0][n][0] + acc[1][n][0], acc[0][n][1] + acc[1][n][1]));
  }
}

template <int Q>
cudaError_t l2t_q(const qbxfmm_geometry& g, HelmCoeffs hc, int p, int nrhs, const double2* lo,
                  const double2* G0, double2* pot, int32_t* err, cudaStream_t st)
{
  const size_t sh = (size_t)l2t_rows(p) * 16 * sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(k_h3_l2t<Q>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sh);
  if (e != cudaSuccess) return e;
  k_h3_l2t<Q><<<dim3(g.ntsqbx_chunks, (nrhs + L2T_RB - 1) / L2T_RB), L2T_NT, sh, st>>>(
      g, hc, p, nrhs, lo, G0, pot, err);
  return cudaGetLastError();
}

}  // namespace

cudaError_t h3_launch_l2t_taylor(const qbxfmm_geometry& g, HelmCoeffs hc, int p, int q, int nrhs,
                                 const double2* lo, const double2* G0, double2* pot_tree,
                                 int32_t* err, cudaStream_t st)
{
  if (g.ntsqbx_chunks == 0) return cudaSuccess;
  if (p > H3T_MAXP) return cudaErrorInvalidValue;
  switch (q) {
    case 0: return l2t_q<0>(g, hc, p, nrhs, lo, G0, pot_tree, err, st);
    case 1: return l2t_q<1>(g, hc, p, nrhs, lo, G0, pot_tree, err, st);
    case 2: return l2t_q<2>(g, hc, p, nrhs, lo, G0, pot_tree, err, st);
    case 3: return l2t_q<3>(g, hc, p, nrhs, lo, G0, pot_tree, err, st);
    case 4: return l2t_q<4>(g, hc, p, nrhs, lo, G0, pot_tree, err, st);
    case 5: return l2t_q<5>(g, hc, p, nrhs, lo, G0, pot_tree, err, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace qbx
