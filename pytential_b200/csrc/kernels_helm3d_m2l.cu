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
// (mma.m8n8k4), so a lane's two results are one complex value.  A pair's coaxial table
// (by (length, level)), phases and raw multipole come by cp.async under the rotation back
// of the pair before it, U, V (by direction) while X is formed.  The tables are stored zero
// padded to multiples of 4 in the inner index with row strides of 4, 12 or 20 doubles
// (4 or 12 mod 16), which are free of bank conflicts read along rows (rotation back) and
// along columns (rotation); X and A rows likewise (8 NT + 4 doubles).
#include <algorithm>
#include <type_traits>

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

// the tables of each M2L pair: direction | coaxial << 16
__global__ void k_h3_m2l_pair_tables(qbxfmm_geometry g, const double* __restrict__ clsmap,
                                     int npairs, int32_t* __restrict__ out)
{
  const int pr = blockIdx.x * blockDim.x + threadIdx.x;
  if (pr >= npairs) return;
  // class of the pair: m2l_class_starts[c] <= pr < m2l_class_starts[c + 1]
  int lo = 0, hi = g.m2l_nclasses - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (g.m2l_class_starts[mid] <= pr) lo = mid;
    else hi = mid - 1;
  }
  out[pr] = (int)clsmap[2 * lo] | (int)clsmap[2 * lo + 1] << 16;
}

// orders (and columns) per warp: n_0 = p - sub, n_1 = sub + max(0, p - 15) and, past 15,
// n_2 = sub (16 subs: n_0 = p - sub, n_1 = sub for the orders past 15).  A product of s
// columns has ceil(s / 4) steps and ceil(s / 8) row tiles, so its code is straight-line for
// each number of steps KS (row tiles (KS + 1) / 2)
template <bool P15, int SUBS>
struct M2LGroups {
  static constexpr int NG = SUBS == 16 ? (P15 ? 1 : 2) : (P15 ? 2 : 3);
  static constexpr int KS0 = P15 ? 4 : 5;          // most steps of group 0
  static constexpr int ks(int g) { return g == 0 ? KS0 : (g == 1 && SUBS == 8 ? (P15 ? 2 : 3) : 1); }
  static constexpr int tiles(int g) { return (ks(g) + 1) / 2; }
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

// run f with the number of steps as a constant, 1 .. MAX
template <int MAX, typename F>
QBX_D void with_steps(int ks, F f)
{
  if constexpr (MAX == 1) {
    f(std::integral_constant<int, 1>());
  } else {
    if (ks == MAX) f(std::integral_constant<int, MAX>());
    else with_steps<MAX - 1>(ks, f);
  }
}

// run f with the group index as a constant, 0 .. N - 1
template <int N, typename F>
QBX_D void for_groups(F f)
{
  f(std::integral_constant<int, 0>());
  if constexpr (N > 1) f(std::integral_constant<int, 1>());
  if constexpr (N > 2) f(std::integral_constant<int, 2>());
}

constexpr int ks_stride(int ks) { return ks == 1 ? 4 : ks <= 3 ? 12 : 20; }

// NT tiles of 4 densities per CTA, NPW of them per warp: 16 warps = SUBS x NT / NPW.
// P15: p <= 15 (else p <= 17)
template <int NT, int NPW, bool P15>
__global__ void __launch_bounds__(M2L_NTHR)
k_h3_m2l_mma(qbxfmm_geometry g, int p, int nrhs, const double2* __restrict__ mp,
             double2* __restrict__ lo, const double* __restrict__ Dtab,
             const double* __restrict__ Ctab, const int32_t* __restrict__ pairtab, int32_t* err)
{
  constexpr int SUBS = 16 * NPW / NT;
  using G = M2LGroups<P15, SUBS>;
  constexpr int XS = 8 * NT + 4, NR = 4 * NT;
  constexpr int PM = P15 ? 15 : 17;
  constexpr int PARTS = 16 / NR;            // warps per density when X is formed
  extern __shared__ double2 smem2[];
  const int ncf = (p + 1) * (p + 1), ntri = (p + 1) * (p + 2) / 2;
  const int nph = 2 * (p + 1), dsz = m2l_dsize(p), csz = m2l_csize(p);
  double* Td = reinterpret_cast<double*>(smem2);       // [dsz - nph]: U, V
  double* Tc = Td + (dsz - nph);                       // [csz]
  double* X = Tc + csz;                                // [ncf + 4][XS]
  double* A = X + (size_t)(ncf + 4) * XS;              // [ncf + 4][XS]; raw multipole [NR][ncf]
  double* Ph = A + (size_t)(ncf + 4) * XS;             // [2][nph]: e^{i a alpha}
  __shared__ int s_u[PM + 2], s_v[PM + 2], s_c[PM + 2], s_ae[PM + 2], s_ao[PM + 2];
  __shared__ unsigned char s_tn[(PM + 1) * (PM + 2) / 2], s_ta[(PM + 1) * (PM + 2) / 2];

  const int i = blockIdx.x, r0 = blockIdx.y * NR;
  const int q0 = g.m2l_tgt_pair_starts[i], q1 = g.m2l_tgt_pair_starts[i + 1];
  if (q1 <= q0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row = lane >> 2, kq = lane & 3;
  const int sub = warp % SUBS, nt0 = (warp / SUBS) * NPW;
  if (tid <= p) {
    s_u[tid] = off_u(tid);
    int v = off_u(p + 1);
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
  // rows past the end are read against zero table entries: finite, and never written
  for (int x = tid; x < 4 * XS; x += M2L_NTHR) X[(size_t)ncf * XS + x] = A[(size_t)ncf * XS + x] = 0.0;

  auto copy = [&](double* dst, const double* src, int n) {
    for (int x = 2 * tid; x < n; x += 2 * M2L_NTHR) cp_async16(dst + x, src + x);
  };
  // the coaxial table, the phases and the raw multipole of pair q
  auto load_pair = [&](int q, int tab, int buf) {
    copy(Tc, Ctab + (size_t)(tab >> 16) * csz, csz);
    copy(Ph + buf * nph, Dtab + (size_t)(tab & 0xffff) * dsz, nph);
    const int src = g.m2l_pair_src[g.m2l_tgt_pairs[q]];
    const bool bad = (unsigned)src >= (unsigned)g.nboxes;
    if (bad && tid == 0) report(err, QBX_DEVERR_BAD_BOX);
    const double* M = reinterpret_cast<const double*>(mp + ((size_t)(bad ? 0 : src) * nrhs + r0) * ncf);
    const int have = bad ? 0 : 2 * ncf * min(NR, nrhs - r0);
    for (int x = 2 * tid; x < 2 * ncf * NR; x += 2 * M2L_NTHR) {
      if (x < have) cp_async16(A + x, M + x);
      else *reinterpret_cast<double2*>(A + x) = c2(0.0);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto load_rotation = [&](int tab) {
    copy(Td, Dtab + (size_t)(tab & 0xffff) * dsz + nph, dsz - nph);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  double acc[G::NG][G::tiles(0)][NPW][4];   // (row, density): L_a (re, im), L_-a (re, im)
#pragma unroll
  for (int gi = 0; gi < G::NG; ++gi)
#pragma unroll
    for (int tl = 0; tl < G::tiles(0); ++tl)
#pragma unroll
      for (int w = 0; w < NPW; ++w)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[gi][tl][w][x] = 0.0;

  int tab = pairtab[g.m2l_tgt_pairs[q0]];
  load_pair(q0, tab, 0);
  load_rotation(tab);
  for (int q = q0; q < q1; ++q) {
    const int buf = (q - q0) & 1;
    const int next = q + 1 < q1 ? pairtab[g.m2l_tgt_pairs[q + 1]] : 0;
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");   // all but the rotation table
    __syncthreads();
    // X^e, X^o from the raw multipole
    {
      const int r = warp % NR;
      const double2* M = reinterpret_cast<const double2*>(A) + (size_t)r * ncf;
      const double2* ph = reinterpret_cast<const double2*>(Ph + buf * nph);
      for (int c = lane + 32 * (warp / NR); c < ntri; c += 32 * PARTS) {
        const int n = s_tn[c], a = s_ta[c], o = n * n + n;
        double2* E = reinterpret_cast<double2*>(X + (size_t)(n * n + a) * XS) + r;
        if (a == 0) {
          *E = M[o];
        } else {
          const double2 f = cscale(0.5 * M2L_SQRT2, ph[a]);
          const double2 u = cmul(f, M[o + a]), v = cmulc(M[o - a], f);
          *E = cadd(u, v);
          reinterpret_cast<double2*>(X + (size_t)(o + a) * XS)[r] = csub(u, v);
        }
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    // rotation: A^e_b = sum_a U[a][b] X^e_a, A^o_b = sum_a V[a][b] X^o_a
    for_groups<G::NG>([&](auto group) {
      constexpr int gi = decltype(group)::value;
      const int n = m2l_order<SUBS>(p, sub, gi);
      if (n < 0) return;
#pragma unroll
      for (int par = 0; par < 2; ++par) {
        const int s = n + 1 - par;
        if (s == 0) continue;
        const double* Tn = Td + (par ? s_v[n] : s_u[n]) + row;
        const double* Bn = X + (size_t)(n * n + par * (n + 1) + kq) * XS + 8 * nt0 + row;
        with_steps<G::ks(gi)>((s + 3) >> 2, [&](auto steps) {
          constexpr int KS = decltype(steps)::value, TL = (KS + 1) / 2, ST = ks_stride(KS);
          double b[KS][NPW], a[KS][TL], d[TL][NPW][2];
#pragma unroll
          for (int k = 0; k < KS; ++k) {
#pragma unroll
            for (int w = 0; w < NPW; ++w) b[k][w] = Bn[4 * k * XS + 8 * w];
#pragma unroll
            for (int tl = 0; tl < TL; ++tl) a[k][tl] = Tn[(4 * k + kq) * ST + 8 * tl];
          }
#pragma unroll
          for (int tl = 0; tl < TL; ++tl)
#pragma unroll
            for (int w = 0; w < NPW; ++w) d[tl][w][0] = d[tl][w][1] = 0.0;
#pragma unroll
          for (int k = 0; k < KS; ++k)
#pragma unroll
            for (int tl = 0; tl < TL; ++tl)
#pragma unroll
              for (int w = 0; w < NPW; ++w) h3_dmma(d[tl][w][0], d[tl][w][1], a[k][tl], b[k][w]);
#pragma unroll
          for (int tl = 0; tl < TL; ++tl) {
            const int bb = 8 * tl + row + par;
            if (bb > n) continue;
            double* out = A + (size_t)((par ? s_ao[bb] : s_ae[bb]) + n - bb) * XS + 8 * nt0 + 2 * kq;
#pragma unroll
            for (int w = 0; w < NPW; ++w)
              *reinterpret_cast<double2*>(out + 8 * w) = c2(d[tl][w][0], d[tl][w][1]);
          }
        });
      }
    });
    __syncthreads();
    // coaxial translation: B_{nu mu} = sum_n C^mu[n][nu] A_{n mu}, e and o alike, into X
    for_groups<G::NG>([&](auto group) {
      constexpr int gi = decltype(group)::value;
      const int mu = m2l_column<SUBS>(p, sub, gi);
      if (mu < 0) return;
      const int s = p + 1 - mu, im = blk_size(s);
      // columns (density, part): the product with Im C takes the other part, -im for re
      const int col = 8 * nt0 + row, colx = 8 * nt0 + (row ^ 1);
      const double sg = (row & 1) ? 1.0 : -1.0;
      with_steps<G::KS0>((s + 3) >> 2, [&](auto steps) {
        constexpr int KS = decltype(steps)::value, TL = (KS + 1) / 2, ST = ks_stride(KS);
        const double* C = Tc + s_c[mu] + kq * ST + row;
#pragma unroll
        for (int par = 0; par < 2; ++par) {
          if (par && mu == 0) continue;
          const double* B = A + (size_t)((par ? s_ao[mu] : s_ae[mu]) + kq) * XS;
          double d[TL][NPW][2];
#pragma unroll
          for (int tl = 0; tl < TL; ++tl)
#pragma unroll
            for (int w = 0; w < NPW; ++w) d[tl][w][0] = d[tl][w][1] = 0.0;
#pragma unroll
          for (int k = 0; k < KS; ++k) {
            double b[NPW], bx[NPW];
#pragma unroll
            for (int w = 0; w < NPW; ++w) {
              b[w] = B[4 * k * XS + col + 8 * w];
              bx[w] = sg * B[4 * k * XS + colx + 8 * w];
            }
#pragma unroll
            for (int tl = 0; tl < TL; ++tl) {
              const double cr = C[4 * k * ST + 8 * tl], ci = C[im + 4 * k * ST + 8 * tl];
#pragma unroll
              for (int w = 0; w < NPW; ++w) h3_dmma(d[tl][w][0], d[tl][w][1], cr, b[w]);
#pragma unroll
              for (int w = 0; w < NPW; ++w) h3_dmma(d[tl][w][0], d[tl][w][1], ci, bx[w]);
            }
          }
#pragma unroll
          for (int tl = 0; tl < TL; ++tl) {
            const int nu = mu + 8 * tl + row;
            if (nu > p) continue;
            double* out = X + (size_t)(nu * nu + par * nu + mu) * XS + 8 * nt0 + 2 * kq;
#pragma unroll
            for (int w = 0; w < NPW; ++w)
              *reinterpret_cast<double2*>(out + 8 * w) = c2(d[tl][w][0], d[tl][w][1]);
          }
        }
      });
    });
    __syncthreads();
    // A and the coaxial table are free: the next pair's copies run under the rotation back
    if (q + 1 < q1) load_pair(q + 1, next, buf ^ 1);
    // rotation back: L^e_a = sum_b U[a][b] B^e_b, then e^{-+ i a alpha} (L^e +- L^o)
    for_groups<G::NG>([&](auto group) {
      constexpr int gi = decltype(group)::value;
      const int n = m2l_order<SUBS>(p, sub, gi);
      if (n < 0) return;
      with_steps<G::ks(gi)>((n + 4) >> 2, [&](auto steps) {
        constexpr int KS = decltype(steps)::value, TL = (KS + 1) / 2, ST = ks_stride(KS);
        // the odd part has one column and row less (row a = 0 is not used): the tile is
        // read one row up, so that a lane's rows agree
        const int so = blk_stride(n);
        const bool full = n > 4 * (KS - 1);            // the odd part's last step exists
        const double* Te = Td + s_u[n] + row * ST + kq;
        const double* To = Td + s_v[n] + kq;
        const double* Be = X + (size_t)(n * n + kq) * XS + 8 * nt0 + row;
        const double* Bo = Be + (size_t)(n + 1) * XS;
        double e[TL][NPW][2], o[TL][NPW][2];
#pragma unroll
        for (int tl = 0; tl < TL; ++tl)
#pragma unroll
          for (int w = 0; w < NPW; ++w)
            e[tl][w][0] = e[tl][w][1] = o[tl][w][0] = o[tl][w][1] = 0.0;
#pragma unroll
        for (int k = 0; k < KS; ++k) {
          double be[NPW], bo[NPW];
#pragma unroll
          for (int w = 0; w < NPW; ++w) {
            be[w] = Be[4 * k * XS + 8 * w];
            bo[w] = (k < KS - 1 || full) ? Bo[4 * k * XS + 8 * w] : 0.0;
          }
#pragma unroll
          for (int tl = 0; tl < TL; ++tl) {
            const double ae = Te[8 * tl * ST + 4 * k];
#pragma unroll
            for (int w = 0; w < NPW; ++w) h3_dmma(e[tl][w][0], e[tl][w][1], ae, be[w]);
            if (k < KS - 1 || full) {
              const double ao = To[max(8 * tl + row - 1, 0) * so + 4 * k];
#pragma unroll
              for (int w = 0; w < NPW; ++w) h3_dmma(o[tl][w][0], o[tl][w][1], ao, bo[w]);
            }
          }
        }
#pragma unroll
        for (int tl = 0; tl < TL; ++tl) {
          const int a = 8 * tl + row;
          if (a > n) continue;
          const double2 ph = reinterpret_cast<const double2*>(Ph + buf * nph)[a];
#pragma unroll
          for (int w = 0; w < NPW; ++w) {
            const double2 ve = c2(e[tl][w][0], e[tl][w][1]);
            const double2 vo = a > 0 ? c2(o[tl][w][0], o[tl][w][1]) : c2(0.0);
            double* ac = acc[gi][tl][w];
            const double2 lp = cmulc(cadd(ve, vo), ph), lm = cmul(csub(ve, vo), ph);
            ac[0] += lp.x;
            ac[1] += lp.y;
            ac[2] += lm.x;
            ac[3] += lm.y;
          }
        }
      });
    });
    __syncthreads();
    if (q + 1 < q1) load_rotation(next);
  }
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
  return (m2l_dsize(p) + 2 * (p + 1) + m2l_csize(p) +
          2 * ((size_t)(p + 1) * (p + 1) + 4) * (8 * nt + 4)) * sizeof(double);
}

template <int NT, int NPW, bool P15>
cudaError_t m2l_mma_launch(const qbxfmm_geometry& g, int p, int nrhs, const double2* mp,
                           double2* lo, const double* Dtab, const double* Ctab,
                           const int32_t* pairtab, int32_t* err, cudaStream_t st)
{
  const size_t sh = m2l_mma_smem(NT, p);
  cudaError_t e = cudaFuncSetAttribute(k_h3_m2l_mma<NT, NPW, P15>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  if (e != cudaSuccess) return e;
  dim3 grid(g.nttp_boxes, (nrhs + 4 * NT - 1) / (4 * NT));
  k_h3_m2l_mma<NT, NPW, P15><<<grid, M2L_NTHR, sh, st>>>(g, p, nrhs, mp, lo, Dtab, Ctab, pairtab, err);
  return cudaGetLastError();
}

}  // namespace

size_t h3_m2l_mma_dsize(int p) { return m2l_dsize(p); }
size_t h3_m2l_mma_csize(int p) { return m2l_csize(p); }

cudaError_t h3_launch_m2l_mma(const qbxfmm_geometry& g, int p, int nrhs, const double2* mp,
                              double2* lo, const double* Dtab, const double* Ctab,
                              const int32_t* pairtab, int32_t* err, cudaStream_t st, int rb)
{
  if (g.nttp_boxes == 0 || g.m2l_nclasses == 0) return cudaSuccess;
  // cp.async needs 16-byte aligned tables
  if (p > H3_MAXP || ((reinterpret_cast<uintptr_t>(Dtab) | reinterpret_cast<uintptr_t>(Ctab)) & 15))
    return cudaErrorInvalidValue;
  // densities per CTA: the plan's tuning, else 16, 8 or 4 by their number; 16 of order
  // 16 or more do not fit the shared memory
  const int want = rb > 0 ? rb : nrhs;
  if (p <= 15) {
    if (want > 8) return m2l_mma_launch<4, 2, true>(g, p, nrhs, mp, lo, Dtab, Ctab, pairtab, err, st);
    if (want > 4) return m2l_mma_launch<2, 1, true>(g, p, nrhs, mp, lo, Dtab, Ctab, pairtab, err, st);
    return m2l_mma_launch<1, 1, true>(g, p, nrhs, mp, lo, Dtab, Ctab, pairtab, err, st);
  }
  if (want > 4) return m2l_mma_launch<2, 1, false>(g, p, nrhs, mp, lo, Dtab, Ctab, pairtab, err, st);
  return m2l_mma_launch<1, 1, false>(g, p, nrhs, mp, lo, Dtab, Ctab, pairtab, err, st);
}

cudaError_t h3_launch_m2l_mma_tables(int pf, int ndir, int ncoax, const double* dirs,
                                     const double* coaxp, const double* start, const double* isq,
                                     const double* rt, const double* gaunt, double* Dtab,
                                     double* Ctab, const qbxfmm_geometry& g, const double* clsmap,
                                     int npairs, int32_t* pairtab, cudaStream_t st)
{
  if (ndir + ncoax == 0) return cudaSuccess;
  if (ndir > 0xffff || ncoax > 0x7fff) return cudaErrorInvalidValue;
  if (npairs > 0)
    k_h3_m2l_pair_tables<<<(npairs + 255) / 256, 256, 0, st>>>(g, clsmap, npairs, pairtab);
  k_h3_m2l_mma_tables<<<ndir + ncoax, 128, 0, st>>>(pf, ndir, ncoax, dirs, coaxp, start, isq, rt,
                                                    gaunt, Dtab, Ctab);
  return cudaGetLastError();
}

}  // namespace qbx
