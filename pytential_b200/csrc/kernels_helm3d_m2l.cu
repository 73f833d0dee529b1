// 3D Helmholtz M2L, complex128, on the FP64 tensor cores, sm_100a.
//
// Per list-2 pair: rotate the source's multipole so that the offset lies on the z axis,
// translate coaxially, rotate back.  With X_nm = e^{i m alpha} M_nm and
// T^n[m][mu] = eps_m eps_mu d^n_{m mu}(beta), T^n[-m][-mu] = T^n[m][mu], the sums and
// differences over +-m decouple,
//   X^e_a = (X_a + X_-a) / sqrt 2 (X_0 for a = 0),  X^o_a = (X_a - X_-a) / sqrt 2,
//   A^e_b = sum_a U[a][b] X^e_a,  A^o_b = sum_a V[a][b] X^o_a     (b = |mu|)
//   U[a][b] = T[a][b] + T[a][-b], V[a][b] = T[a][b] - T[a][-b]  (a, b > 0),
//   U[a][0] = sqrt 2 T[a][0], U[0][b] = sqrt 2 T[0][b], U[0][0] = T[0][0],
// so a rotation of order n is two real products of orders n + 1 and n instead of one of
// 2n + 1 (half the multiply-adds).  The coaxial blocks of +-mu are equal and act on A^e
// and A^o alike; the rotation back is U, V transposed.
//
// One CTA (16 warps) per target-or-parent box and 4 NT densities: the columns of every
// product are (density, re / im), 8 columns = 4 densities a tensor-core tile
// (mma.m8n8k4), so a lane's two results are one complex value.  The tables of a pair come
// by cp.async: U, V by direction (loaded while the next multipole is fetched), the
// coaxial blocks by (length, level) during the rotation back.  They are stored zero
// padded to multiples of 4 in the inner index with row strides of 4, 12 or 20 doubles
// (4 or 12 mod 16), which are free of bank conflicts read along rows (rotation back) and
// along columns (rotation); X and A rows likewise (8 NT + 4 doubles).
#include <algorithm>

#include "../../include/qbxfmm_api.h"
#include "helm3.cuh"
#include "kernels.h"

namespace qbx {

namespace {

constexpr int M2L_NTHR = 512;
constexpr double M2L_SQRT2 = 1.4142135623730950488;

QBX_HD int pad4(int s) { return (s + 3) & ~3; }
QBX_HD int blk_stride(int s) { return s <= 4 ? 4 : s <= 12 ? 12 : 20; }
QBX_HD int blk_size(int s) { return pad4(s) * blk_stride(s); }

// doubles of one direction's table: phases e^{i a alpha} (a = 0..p), U of n = 0..p, V of
// n = 1..p; of one coaxial table: real parts of mu = 0..p, imaginary parts
QBX_HD int m2l_dsize(int p)
{
  int v = 2 * (p + 1);
  for (int n = 0; n <= p; ++n) v += blk_size(n + 1) + (n > 0 ? blk_size(n) : 0);
  return v;
}

QBX_HD int m2l_csize(int p)
{
  int v = 0;
  for (int mu = 0; mu <= p; ++mu) v += 2 * blk_size(p + 1 - mu);
  return v;
}

// offsets of the blocks: U and V of order n in a direction's table, the real part of
// mu in a coaxial table (the imaginary part blk_size later)
QBX_HD int off_u(int n)
{
  int v = 0;
  for (int i = 0; i < n; ++i) v += blk_size(i + 1);
  return v;
}

QBX_HD int off_c(int p, int mu)
{
  int v = 0;
  for (int u = 0; u < mu; ++u) v += 2 * blk_size(p + 1 - u);
  return v;
}

QBX_D void cp_async16(void* dst, const void* src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// CTAs [0, ndir): U, V and phases of one direction; [ndir, ndir + ncoax): one coaxial
// table.  Inputs as k_h3_m2l_tables.
__global__ void __launch_bounds__(128)
k_h3_m2l_mma_tables(int pf, int ndir, int ncoax, const double* __restrict__ dirs,
                    const double* __restrict__ coaxp, const double* __restrict__ start,
                    const double* __restrict__ isq, const double* __restrict__ rt,
                    const double* __restrict__ gaunt, double* __restrict__ Dtab,
                    double* __restrict__ Ctab)
{
  __shared__ double2 s_rad[2 * H3_MAXP + 4];
  __shared__ double s_pw[H3_MAXP + 1];
  const int nm = 2 * pf + 1, nl = pf + 1, ncf = (pf + 1) * (pf + 1), tid = threadIdx.x;
  if ((int)blockIdx.x < ndir) {
    const double* u = dirs + 4 * blockIdx.x;
    const double cbeta = fmin(1.0, fmax(-1.0, u[2]));
    const double alpha = (u[0] == 0.0 && u[1] == 0.0) ? 0.0 : atan2(u[1], u[0]);
    const double beta = acos(cbeta);
    const double ch = cos(0.5 * beta), sh = sin(0.5 * beta);
    const int dsz = m2l_dsize(pf);
    double* D = Dtab + (size_t)blockIdx.x * dsz;
    for (int x = tid; x < dsz; x += 128) D[x] = 0.0;
    __syncthreads();
    double* U = D + 2 * (pf + 1);
    const int voff = off_u(pf + 1);
    for (int a = tid; a <= pf; a += 128) {
      double sn, cs;
      sincos(a * alpha, &sn, &cs);
      D[2 * a] = cs;
      D[2 * a + 1] = sn;
    }
    for (int t = tid; t < (pf + 1) * (pf + 1); t += 128) {
      const int a = t / (pf + 1), b = t % (pf + 1);
      const int n0 = max(a, b);
      // d^n_{a, +b} and d^n_{a, -b} by the recurrence along n
      double cur[2], prev[2] = {0.0, 0.0};
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int mu = s ? -b : b, ts = (a + pf) * nm + (mu + pf);
        double v = start[4 * ts];
        const int ec = (int)start[4 * ts + 1], es = (int)start[4 * ts + 2];
        for (int k = 0; k < ec; ++k) v *= ch;
        for (int k = 0; k < es; ++k) v *= sh;
        cur[s] = v;
      }
      // eps_m eps_mu, eps_m = (-1)^m for m > 0
      const double ea = (a & 1) ? -1.0 : 1.0, eb = (b & 1) ? -1.0 : 1.0;
      int uo = 0, vo = 0;
      for (int n = 0; n < n0; ++n) {
        uo += blk_size(n + 1);
        vo += n > 0 ? blk_size(n) : 0;
      }
      for (int n = n0; n <= pf; ++n) {
        const double tp = ea * eb * cur[0], tm = ea * cur[1];
        double w;
        if (a > 0 && b > 0) {
          w = tp + tm;
          U[voff + vo + (a - 1) * blk_stride(n) + (b - 1)] = tp - tm;
        } else {
          w = (a > 0 || b > 0) ? M2L_SQRT2 * tp : tp;
        }
        U[uo + a * blk_stride(n + 1) + b] = w;
        uo += blk_size(n + 1);
        vo += n > 0 ? blk_size(n) : 0;
        if (n == pf) break;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int mu = s ? -b : b;
          double nxt;
          if (n == 0) {
            nxt = cbeta * cur[s];
          } else {
            const double rn = 1.0 / n;
            const double wv = rn * isq[(n + 1) * (pf + 1) + a] * isq[(n + 1) * (pf + 1) + b];
            const double A = (2.0 * n + 1.0) * (n * (n + 1.0) * cbeta - (double)a * mu) * wv;
            const double C = (n + 1.0) * rn * rt[n * (pf + 1) + a] * rt[n * (pf + 1) + b];
            nxt = fma(A, cur[s], -C * prev[s]);
          }
          prev[s] = cur[s];
          cur[s] = nxt;
        }
      }
    }
    return;
  }
  const int c = blockIdx.x - ndir;
  if (c >= ncoax) return;
  const double kb = coaxp[2 * c], s = coaxp[2 * c + 1];
  const int L = 2 * pf;
  if (tid == 0) {
    h3_sph_h(L, kb, s_rad);
    for (int l = 0; l <= L; ++l)
      s_rad[l] = cmul(cscale(sqrt(FOUR_PI * (2.0 * l + 1.0)), ipow(l)), s_rad[l]);
  }
  for (int n = tid; n <= pf; n += 128) s_pw[n] = pow(s, (double)n);
  const int csz = m2l_csize(pf);
  double* C = Ctab + (size_t)c * csz;
  for (int x = tid; x < csz; x += 128) C[x] = 0.0;
  __syncthreads();
  for (int e = tid; e < (pf + 1) * (pf + 1) * (pf + 1); e += 128) {
    const int mu = e / ((pf + 1) * (pf + 1)), w = e - mu * (pf + 1) * (pf + 1);
    const int n = w / (pf + 1), nu = w % (pf + 1);
    if (n < mu || nu < mu) continue;
    const int o = nu * nu + nu + mu, lbase = abs(n - nu), jmax = min(n, nu);
    double2 tt = c2(0.0);
    for (int j = 0; j <= jmax; ++j)
      tt = caxpy(__ldg(gaunt + ((size_t)o * nl + j) * ncf + n * n + n + mu), s_rad[lbase + 2 * j], tt);
    tt = cscale(s_pw[nu] * s_pw[n], cmul(ipow(nu - n + 4 * pf), tt));
    const int sz = pf + 1 - mu, at = off_c(pf, mu) + (n - mu) * blk_stride(sz) + (nu - mu);
    C[at] = tt.x;
    C[at + blk_size(sz)] = tt.y;
  }
}

// tiles of 8 rows of the groups of orders a warp takes (order p - sub, then the rest)
template <int P15, int SUBS>
struct M2LGroups {
  // orders per warp: n_0 = p - sub, n_1 = sub + max(0, p - 15) and, past 15, n_2 = sub
  // (16 subs: n_0 = p - sub, n_1 = sub for the orders past 15)
  static constexpr int NG = SUBS == 16 ? (P15 ? 1 : 2) : (P15 ? 2 : 3);
  static constexpr int NTL = P15 ? 2 : 3;       // row tiles of n_0
  static constexpr int tiles(int g) { return g == 0 ? NTL : (g == 1 && SUBS == 8 && !P15 ? 2 : 1); }
};

template <int SUBS>
QBX_D int m2l_order(int p, int sub, int g)
{
  if (g == 0) return p - sub;                                    // < 0: none
  if (SUBS == 16) return sub < p - 15 ? sub : -1;
  if (g == 1) {
    const int n = sub + max(0, p - 15);
    return n <= p - 8 ? n : -1;
  }
  return sub < p - 15 ? sub : -1;
}

template <int SUBS>
QBX_D int m2l_column(int p, int sub, int g)     // mu of the coaxial step
{
  const int mu = g == 0 ? sub : SUBS == 16 ? 16 + sub : g == 1 ? 15 - sub : 16 + sub;
  return mu <= p ? mu : -1;
}

// NT tiles of 4 densities per CTA, NPW of them per warp: 16 warps = SUBS x NT / NPW.
// P15: p <= 15 (else p <= 17)
template <int NT, int NPW, bool P15>
__global__ void __launch_bounds__(M2L_NTHR)
k_h3_m2l_mma(qbxfmm_geometry g, int p, int nrhs, const double2* __restrict__ mp,
             double2* __restrict__ lo, const double* __restrict__ Dtab,
             const double* __restrict__ Ctab, const double* __restrict__ clsmap, int32_t* err)
{
  constexpr int SUBS = 16 * NPW / NT;
  using G = M2LGroups<P15, SUBS>;
  constexpr int XS = 8 * NT + 4;
  constexpr int PM = P15 ? 15 : 17;
  constexpr int KIT = ((PM + 1) * (PM + 2) / 2 * 4 * NT + M2L_NTHR - 1) / M2L_NTHR;
  extern __shared__ double2 smem2[];
  const int ncf = (p + 1) * (p + 1), ntri = (p + 1) * (p + 2) / 2;
  const int dsz = m2l_dsize(p), csz = m2l_csize(p);
  double* Td = reinterpret_cast<double*>(smem2);       // [dsz]
  double* Tc = Td + dsz;                               // [csz]
  double* X = Tc + csz;                                // [ncf + 4][XS]
  double* A = X + (size_t)(ncf + 4) * XS;              // [ncf + 4][XS]
  __shared__ int s_u[PM + 2], s_v[PM + 2], s_c[PM + 2], s_ae[PM + 2], s_ao[PM + 2];
  __shared__ unsigned char s_tn[(PM + 1) * (PM + 2) / 2], s_ta[(PM + 1) * (PM + 2) / 2];
  __shared__ int s_cls;

  const int i = blockIdx.x, r0 = blockIdx.y * 4 * NT;
  const int q0 = g.m2l_tgt_pair_starts[i], q1 = g.m2l_tgt_pair_starts[i + 1];
  if (q1 <= q0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row = lane >> 2, kq = lane & 3;
  const int sub = warp % SUBS, nt0 = (warp / SUBS) * NPW;
  if (tid <= p) {
    s_u[tid] = 2 * (p + 1) + off_u(tid);
    int v = 2 * (p + 1) + off_u(p + 1);
    for (int n = 1; n < tid; ++n) v += blk_size(n);
    s_v[tid] = v;
    s_c[tid] = off_c(p, tid);
    // rows of (n, mu): E at s_ae[mu] + n - mu, O at s_ao[mu] + n - mu
    s_ae[tid] = tid * (p + 1) - tid * (tid - 1) / 2;
    s_ao[tid] = ntri + (tid > 0 ? (tid - 1) * p - (tid - 1) * (tid - 2) / 2 : 0);
  }
  for (int c = tid; c < ntri; c += M2L_NTHR) {
    int n, m;
    decode3(c, n, m);
    s_tn[c] = (unsigned char)n;
    s_ta[c] = (unsigned char)m;
  }
  for (int x = tid; x < 4 * XS; x += M2L_NTHR) X[(size_t)ncf * XS + x] = A[(size_t)ncf * XS + x] = 0.0;

  auto find_class = [&](int q) {            // class of pair q into s_cls
    const int pr = g.m2l_tgt_pairs[q];
    for (int c = tid; c < g.m2l_nclasses; c += M2L_NTHR)
      if (g.m2l_class_starts[c] <= pr && pr < g.m2l_class_starts[c + 1]) s_cls = c;
  };
  auto load_table = [&](double* dst, const double* src, int n) {
    for (int x = 2 * tid; x < n; x += 2 * M2L_NTHR) cp_async16(dst + x, src + x);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  double acc[G::NG][G::NTL][NPW][4];        // (row, density): L_a (re, im), L_-a (re, im)
#pragma unroll
  for (int gi = 0; gi < G::NG; ++gi)
#pragma unroll
    for (int tl = 0; tl < G::NTL; ++tl)
#pragma unroll
      for (int w = 0; w < NPW; ++w)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[gi][tl][w][x] = 0.0;

  if (tid == 0) s_cls = 0;
  __syncthreads();
  find_class(q0);
  __syncthreads();
  int cls = s_cls;
  load_table(Tc, Ctab + (size_t)clsmap[2 * cls + 1] * csz, csz);
  for (int q = q0; q < q1; ++q) {
    load_table(Td, Dtab + (size_t)clsmap[2 * cls] * dsz, dsz);
    const int src = g.m2l_pair_src[g.m2l_tgt_pairs[q]];
    const bool bad = (unsigned)src >= (unsigned)g.nboxes;
    if (bad && tid == 0) report(err, QBX_DEVERR_BAD_BOX);
    double2 mv[KIT][2];
#pragma unroll
    for (int k = 0; k < KIT; ++k) {
      const int t = tid + k * M2L_NTHR, r = t / ntri, c = t - r * ntri;
      mv[k][0] = mv[k][1] = c2(0.0);
      if (r < 4 * NT && r0 + r < nrhs && !bad) {
        const double2* M = mp + ((size_t)src * nrhs + r0 + r) * ncf;
        const int n = s_tn[c], a = s_ta[c], o = n * n + n;
        mv[k][0] = __ldg(M + o + a);
        if (a > 0) mv[k][1] = __ldg(M + o - a);
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    // X^e, X^o
#pragma unroll
    for (int k = 0; k < KIT; ++k) {
      const int t = tid + k * M2L_NTHR, r = t / ntri, c = t - r * ntri;
      if (r >= 4 * NT) break;
      const int n = s_tn[c], a = s_ta[c];
      double2* E = reinterpret_cast<double2*>(X + (size_t)(n * n + a) * XS) + r;
      if (a == 0) {
        *E = mv[k][0];
      } else {
        const double2 ph = reinterpret_cast<const double2*>(Td)[a];
        const double2 u = cmul(ph, mv[k][0]), v = cmulc(mv[k][1], ph);
        *E = cscale(0.5 * M2L_SQRT2, cadd(u, v));
        double2* O = reinterpret_cast<double2*>(X + (size_t)(n * n + n + a) * XS) + r;
        *O = cscale(0.5 * M2L_SQRT2, csub(u, v));
      }
    }
    if (q + 1 < q1) find_class(q + 1);
    __syncthreads();
    if (q + 1 < q1) cls = s_cls;
    // rotation: A^e_b = sum_a U[a][b] X^e_a, A^o_b = sum_a V[a][b] X^o_a
#pragma unroll
    for (int gi = 0; gi < G::NG; ++gi) {
      const int n = m2l_order<SUBS>(p, sub, gi);
      if (n < 0) continue;
#pragma unroll
      for (int par = 0; par < 2; ++par) {
        const int s = n + 1 - par;
        if (s == 0) continue;
        const int stride = blk_stride(s), ks = pad4(s) >> 2;
        const double* T = Td + (par ? s_v[n] : s_u[n]) + kq * stride + row;
        const double* B = X + (size_t)(n * n + par * (n + 1) + kq) * XS + 8 * nt0 + row;
        double d[G::tiles(0)][NPW][2];
#pragma unroll
        for (int tl = 0; tl < G::tiles(gi); ++tl)
#pragma unroll
          for (int w = 0; w < NPW; ++w) d[tl][w][0] = d[tl][w][1] = 0.0;
        for (int k = 0; k < ks; ++k) {
          double b[NPW];
#pragma unroll
          for (int w = 0; w < NPW; ++w) b[w] = B[8 * w];
#pragma unroll
          for (int tl = 0; tl < G::tiles(gi); ++tl) {
            if (8 * tl >= s) break;
            const double a = T[8 * tl];
#pragma unroll
            for (int w = 0; w < NPW; ++w) h3_dmma(d[tl][w][0], d[tl][w][1], a, b[w]);
          }
          T += 4 * stride;
          B += 4 * XS;
        }
#pragma unroll
        for (int tl = 0; tl < G::tiles(gi); ++tl) {
          const int b = 8 * tl + row + par;
          if (b > n) continue;
          double* out = A + (size_t)((par ? s_ao[b] : s_ae[b]) + n - b) * XS + 8 * nt0 + 2 * kq;
#pragma unroll
          for (int w = 0; w < NPW; ++w)
            *reinterpret_cast<double2*>(out + 8 * w) = c2(d[tl][w][0], d[tl][w][1]);
        }
      }
    }
    __syncthreads();
    // coaxial translation: B_{nu mu} = sum_n C^mu[n][nu] A_{n mu}, e and o alike, into X
#pragma unroll
    for (int gi = 0; gi < G::NG; ++gi) {
      const int mu = m2l_column<SUBS>(p, sub, gi);
      if (mu < 0) continue;
      const int s = p + 1 - mu, stride = blk_stride(s), ks = pad4(s) >> 2, im = blk_size(s);
      const double* C = Tc + s_c[mu] + kq * stride + row;
      // columns (density, part): the product with Im C takes the other part, -im for re
      const int colx = 8 * nt0 + (row ^ 1);
      const double sg = (row & 1) ? 1.0 : -1.0;
#pragma unroll
      for (int par = 0; par < 2; ++par) {
        if (par && mu == 0) continue;
        const double* B = A + (size_t)((par ? s_ao[mu] : s_ae[mu]) + kq) * XS;
        const double* Ck = C;
        double d[G::NTL][NPW][2];
#pragma unroll
        for (int tl = 0; tl < G::NTL; ++tl)
#pragma unroll
          for (int w = 0; w < NPW; ++w) d[tl][w][0] = d[tl][w][1] = 0.0;
        for (int k = 0; k < ks; ++k) {
          double b[NPW], bx[NPW];
#pragma unroll
          for (int w = 0; w < NPW; ++w) {
            b[w] = B[8 * nt0 + row + 8 * w];
            bx[w] = sg * B[colx + 8 * w];
          }
#pragma unroll
          for (int tl = 0; tl < G::NTL; ++tl) {
            if (8 * tl >= s) break;
            const double cr = Ck[8 * tl], ci = Ck[im + 8 * tl];
#pragma unroll
            for (int w = 0; w < NPW; ++w) {
              h3_dmma(d[tl][w][0], d[tl][w][1], cr, b[w]);
              h3_dmma(d[tl][w][0], d[tl][w][1], ci, bx[w]);
            }
          }
          Ck += 4 * stride;
          B += 4 * XS;
        }
#pragma unroll
        for (int tl = 0; tl < G::NTL; ++tl) {
          const int nu = mu + 8 * tl + row;
          if (nu > p) continue;
          double* out = X + (size_t)(nu * nu + par * nu + mu) * XS + 8 * nt0 + 2 * kq;
#pragma unroll
          for (int w = 0; w < NPW; ++w)
            *reinterpret_cast<double2*>(out + 8 * w) = c2(d[tl][w][0], d[tl][w][1]);
        }
      }
    }
    __syncthreads();
    if (q + 1 < q1) load_table(Tc, Ctab + (size_t)clsmap[2 * cls + 1] * csz, csz);
    // rotation back: L^e_a = sum_b U[a][b] B^e_b, then e^{-+ i a alpha} (L^e +- L^o)
#pragma unroll
    for (int gi = 0; gi < G::NG; ++gi) {
      const int n = m2l_order<SUBS>(p, sub, gi);
      if (n < 0) continue;
#pragma unroll
      for (int tl = 0; tl < G::tiles(gi); ++tl) {
        if (8 * tl > n) break;
        double d[2][NPW][2];
        // V has the rows a = 1 .. n: its tile is read one row up, so that a lane's rows
        // agree (the row a = 0 of the odd part is not used)
#pragma unroll
        for (int par = 0; par < 2; ++par) {
          const int s = n + 1 - par;
#pragma unroll
          for (int w = 0; w < NPW; ++w) d[par][w][0] = d[par][w][1] = 0.0;
          if (s == 0) continue;
          const int stride = blk_stride(s), ks = pad4(s) >> 2;
          const int ra = 8 * tl + row - par;
          const double* T = Td + (par ? s_v[n] : s_u[n]) + max(ra, 0) * stride + kq;
          const double* B = X + (size_t)(n * n + par * (n + 1) + kq) * XS + 8 * nt0 + row;
          for (int k = 0; k < ks; ++k) {
            const double a = T[4 * k];
#pragma unroll
            for (int w = 0; w < NPW; ++w) h3_dmma(d[par][w][0], d[par][w][1], a, B[8 * w]);
            B += 4 * XS;
          }
        }
        const int a = 8 * tl + row;
        if (a > n) continue;
        const double2 ph = reinterpret_cast<const double2*>(Td)[a];
#pragma unroll
        for (int w = 0; w < NPW; ++w) {
          const double2 e = c2(d[0][w][0], d[0][w][1]);
          const double2 o = a > 0 ? c2(d[1][w][0], d[1][w][1]) : c2(0.0);
          double* ac = acc[gi][tl][w];
          const double2 lp = cmulc(cadd(e, o), ph), lm = cmul(csub(e, o), ph);
          ac[0] += lp.x;
          ac[1] += lp.y;
          ac[2] += lm.x;
          ac[3] += lm.y;
        }
      }
    }
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  const int tb = g.target_or_target_parent_boxes[i];
  if ((unsigned)tb >= (unsigned)g.nboxes) {
    if (tid == 0) report(err, QBX_DEVERR_BAD_BOX);
    return;
  }
#pragma unroll
  for (int gi = 0; gi < G::NG; ++gi) {
    const int n = m2l_order<SUBS>(p, sub, gi);
    if (n < 0) continue;
#pragma unroll
    for (int tl = 0; tl < G::tiles(gi); ++tl) {
      const int a = 8 * tl + row;
      if (a > n) continue;
#pragma unroll
      for (int w = 0; w < NPW; ++w) {
        const int r = r0 + 4 * (nt0 + w) + kq;
        if (r >= nrhs) continue;
        double2* out = lo + ((size_t)tb * nrhs + r) * ncf + n * n + n;
        const double f = a > 0 ? 0.5 * M2L_SQRT2 : 1.0;
        const double* ac = acc[gi][tl][w];
        out[a] = caxpy(f, c2(ac[0], ac[1]), out[a]);
        if (a > 0) out[-a] = caxpy(f, c2(ac[2], ac[3]), out[-a]);
      }
    }
  }
}

size_t m2l_mma_smem(int nt, int p)
{
  return (m2l_dsize(p) + m2l_csize(p) + 2 * ((size_t)(p + 1) * (p + 1) + 4) * (8 * nt + 4)) *
         sizeof(double);
}

template <int NT, int NPW, bool P15>
cudaError_t m2l_mma_launch(const qbxfmm_geometry& g, int p, int nrhs, const double2* mp,
                           double2* lo, const double* Dtab, const double* Ctab,
                           const double* clsmap, int32_t* err, cudaStream_t st)
{
  const size_t sh = m2l_mma_smem(NT, p);
  cudaError_t e = cudaFuncSetAttribute(k_h3_m2l_mma<NT, NPW, P15>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  if (e != cudaSuccess) return e;
  dim3 grid(g.nttp_boxes, (nrhs + 4 * NT - 1) / (4 * NT));
  k_h3_m2l_mma<NT, NPW, P15><<<grid, M2L_NTHR, sh, st>>>(g, p, nrhs, mp, lo, Dtab, Ctab, clsmap, err);
  return cudaGetLastError();
}

}  // namespace

size_t h3_m2l_mma_dsize(int p) { return m2l_dsize(p); }
size_t h3_m2l_mma_csize(int p) { return m2l_csize(p); }

cudaError_t h3_launch_m2l_mma(const qbxfmm_geometry& g, int p, int nrhs, const double2* mp,
                              double2* lo, const double* Dtab, const double* Ctab,
                              const double* clsmap, int32_t* err, cudaStream_t st, int rb)
{
  if (g.nttp_boxes == 0 || g.m2l_nclasses == 0) return cudaSuccess;
  // cp.async needs 16-byte aligned tables
  if (p > H3_MAXP || ((reinterpret_cast<uintptr_t>(Dtab) | reinterpret_cast<uintptr_t>(Ctab)) & 15))
    return cudaErrorInvalidValue;
  // densities per CTA: the plan's tuning, else 16, 8 or 4 by their number; 16 of order
  // 16 or more do not fit the shared memory
  const int want = rb > 0 ? rb : nrhs;
  if (p <= 15) {
    if (want > 8) return m2l_mma_launch<4, 2, true>(g, p, nrhs, mp, lo, Dtab, Ctab, clsmap, err, st);
    if (want > 4) return m2l_mma_launch<2, 1, true>(g, p, nrhs, mp, lo, Dtab, Ctab, clsmap, err, st);
    return m2l_mma_launch<1, 1, true>(g, p, nrhs, mp, lo, Dtab, Ctab, clsmap, err, st);
  }
  if (want > 4) return m2l_mma_launch<2, 1, false>(g, p, nrhs, mp, lo, Dtab, Ctab, clsmap, err, st);
  return m2l_mma_launch<1, 1, false>(g, p, nrhs, mp, lo, Dtab, Ctab, clsmap, err, st);
}

cudaError_t h3_launch_m2l_mma_tables(int pf, int ndir, int ncoax, const double* dirs,
                                     const double* coaxp, const double* start, const double* isq,
                                     const double* rt, const double* gaunt, double* Dtab,
                                     double* Ctab, cudaStream_t st)
{
  if (ndir + ncoax == 0) return cudaSuccess;
  k_h3_m2l_mma_tables<<<ndir + ncoax, 128, 0, st>>>(pf, ndir, ncoax, dirs, coaxp, start, isq, rt,
                                                    gaunt, Dtab, Ctab);
  return cudaGetLastError();
}

}  // namespace qbx
