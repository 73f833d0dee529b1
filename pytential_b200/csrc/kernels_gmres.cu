// GMRES: one iteration's orthogonalization and update for a batch of densities
// (pytential/linalg/gmres.py:224-299), sm_100a.
//
//   twice:  for every kept image A_j:  d = <A_j, w>,  w -= d A_j,  v -= d e_j  (v = r first)
//           w, v /= |w|
//   then    d = <w, r>,  r' = r - d w,  x += d v
// The steps over j depend on one another, so the time is a chain of reductions: with a
// library launch for each product, sum and difference an iteration over 12 kept images of 7
// densities and 6224 nodes took 0.9 ms beside an operator of 1 ms.  Here a cluster of eight
// CTAs holds a density's w and v in registers (up to 16384 entries, else in L2), the next
// image is loaded during a reduction, and a reduction is one exchange through distributed
// shared memory, summed in a fixed order: one launch an iteration.  Above 16384 entries a step
// reads and writes w and v as well, and eight SMs a density are few: the caller (gmres.py) takes
// the tensor operations where they are faster.
// 25 iterations with 7 densities of 6224 nodes: 48.6 -> 28.0 ms, 25 of them in the operator.
#include "../../include/qbxfmm_api.h"
#include "common.cuh"
#include "kernels.h"

#include <utility>

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

namespace qbx {

namespace {

constexpr int GM_CL = 8, GM_NT = 256, GM_W = GM_NT / 32;
constexpr int GM_MAXV = 64;                  // images per launch

struct GmresImages {
  const void* a[GM_MAXV];
  const void* e[GM_MAXV];
};

QBX_D double gm_mul(double a, double b) { return a * b; }
QBX_D double2 gm_mul(double2 a, double2 b) { return cmul(a, b); }
QBX_D double gm_dot(double a, double b, double s) { return fma(a, b, s); }
QBX_D double2 gm_dot(double2 a, double2 b, double2 s)      // conj(a) b
{
  return c2(fma(a.x, b.x, fma(a.y, b.y, s.x)), fma(a.x, b.y, fma(-a.y, b.x, s.y)));
}
QBX_D double gm_sub(double a, double b) { return a - b; }
QBX_D double2 gm_sub(double2 a, double2 b) { return csub(a, b); }
QBX_D double gm_add(double a, double b) { return a + b; }
QBX_D double2 gm_add(double2 a, double2 b) { return cadd(a, b); }
QBX_D double gm_scale(double f, double a) { return f * a; }
QBX_D double2 gm_scale(double f, double2 a) { return cscale(f, a); }
QBX_D double gm_abs(double a) { return fabs(a); }
QBX_D double gm_abs(double2 a) { return hypot(a.x, a.y); }
QBX_D double gm_xor(double a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
QBX_D double2 gm_xor(double2 a, int o) { return c2(gm_xor(a.x, o), gm_xor(a.y, o)); }

// E entries of w and v per thread in registers, or in global memory (E = 0).  first: w and v
// start from win and r; norm: normalize at the end of a sweep; last: update r and x.
template <typename T, int E>
__global__ void __cluster_dims__(GM_CL, 1, 1) __launch_bounds__(GM_NT)
k_gmres_step(GmresImages im, int count, int nsweep, bool first, bool norm, bool last, long long n,
             const T* __restrict__ win, const T* __restrict__ r, T* __restrict__ w, T* __restrict__ v,
             const uint8_t* __restrict__ active, T* __restrict__ rnew, T* __restrict__ x)
{
  cg::cluster_group cl = cg::this_cluster();
  // no CTA writes to another's shared memory before all have started; the loads of w and v
  // run meanwhile
  auto started = cl.barrier_arrive();
  __shared__ T s_warp[GM_W], s_part[2][GM_CL];
  const int rank = cl.block_rank(), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t off = (size_t)blockIdx.y * n;
  const long long i0 = rank * GM_NT + threadIdx.x;
  const int K = E > 0 ? E : (int)((n + GM_CL * GM_NT - 1) / (GM_CL * GM_NT));
  auto at = [&](int k) { return i0 + (long long)k * (GM_CL * GM_NT); };
  auto each = [&](auto f) {
    if constexpr (E > 0) {
#pragma unroll
      for (int k = 0; k < E; ++k) f(k);
    } else {
      for (int k = 0; k < K; ++k) f(k);
    }
  };
  T wr[E > 0 ? E : 1], vr[E > 0 ? E : 1], ar[E > 0 ? E : 1];
  auto W = [&](int k) -> T& {
    if constexpr (E > 0) return wr[k];
    else return w[off + at(k)];
  };
  auto V = [&](int k) -> T& {
    if constexpr (E > 0) return vr[k];
    else return v[off + at(k)];
  };
  const T zero = gm_scale(0.0, T());
  each([&](int k) {
    const bool in = at(k) < n;
    if constexpr (E > 0) {
      wr[k] = in ? (first ? win : w)[off + at(k)] : zero;
      vr[k] = in ? (first ? r : v)[off + at(k)] : zero;
    } else if (first && in) {
      W(k) = win[off + at(k)];
      V(k) = r[off + at(k)];
    }
  });
  cl.barrier_wait(std::move(started));
  int par = 0;
  auto reduce = [&](T s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = gm_add(s, gm_xor(s, o));
    if (lane == 0) s_warp[warp] = s;
    __syncthreads();
    if (warp == 0) {
      T t = s_warp[lane & (GM_W - 1)];
#pragma unroll
      for (int o = GM_W / 2; o > 0; o >>= 1) t = gm_add(t, gm_xor(t, o));
      if (lane < GM_CL) *cl.map_shared_rank(&s_part[par][rank], lane) = t;
    }
    cl.sync();
    T t = s_part[par][0];
    for (int c = 1; c < GM_CL; ++c) t = gm_add(t, s_part[par][c]);
    par ^= 1;
    return t;
  };
  auto fetch = [&](const void* p) {
    if constexpr (E > 0) {
#pragma unroll
      for (int k = 0; k < E; ++k)
        ar[k] = at(k) < n ? __ldg(static_cast<const T*>(p) + off + at(k)) : zero;
    }
  };
  auto A = [&](const void* p, int k) -> T {
    if constexpr (E > 0) return ar[k];
    else return __ldg(static_cast<const T*>(p) + off + at(k));
  };
  for (int sweep = 0; sweep < nsweep; ++sweep) {
    if (count > 0) fetch(im.a[0]);
    for (int j = 0; j < count; ++j) {
      T s = zero;
      each([&](int k) {
        if (E > 0 || at(k) < n) s = gm_dot(A(im.a[j], k), W(k), s);
      });
      // e_j is on its way during the reduction
      T er[E > 0 ? E : 1];
      if constexpr (E > 0) {
#pragma unroll
        for (int k = 0; k < E; ++k)
          er[k] = at(k) < n ? __ldg(static_cast<const T*>(im.e[j]) + off + at(k)) : zero;
      }
      const T d = reduce(s);
      each([&](int k) {
        if (E == 0 && at(k) >= n) return;
        W(k) = gm_sub(W(k), gm_mul(d, A(im.a[j], k)));
      });
      if (j + 1 < count) fetch(im.a[j + 1]);
      each([&](int k) {
        if (E == 0 && at(k) >= n) return;
        T ev;
        if constexpr (E > 0) ev = er[k];
        else ev = __ldg(static_cast<const T*>(im.e[j]) + off + at(k));
        V(k) = gm_sub(V(k), gm_mul(d, ev));
      });
    }
    if (norm) {
      T s = zero;
      each([&](int k) {
        if (E > 0 || at(k) < n) s = gm_dot(W(k), W(k), s);
      });
      const double nw = sqrt(gm_abs(reduce(s)));
      const double inv = active[blockIdx.y] && nw > 0.0 ? 1.0 / nw : 0.0;
      each([&](int k) {
        if (E == 0 && at(k) >= n) return;
        W(k) = gm_scale(inv, W(k));
        V(k) = gm_scale(inv, V(k));
      });
    }
  }
  T d = zero;
  if (last) {
    T s = zero;
    each([&](int k) {
      if (at(k) < n) s = gm_dot(W(k), r[off + at(k)], s);
    });
    d = reduce(s);
    if (!active[blockIdx.y]) d = zero;
  }
  each([&](int k) {
    if (at(k) >= n) return;
    const size_t o = off + at(k);
    const T wv = W(k), vv = V(k);
    if constexpr (E > 0) {
      w[o] = wv;
      v[o] = vv;
    }
    if (last) {
      if (rnew) rnew[o] = gm_sub(r[o], gm_mul(d, wv));
      x[o] = gm_add(x[o], gm_mul(d, vv));
    }
  });
}

template <typename T>
cudaError_t step(int nd, long long n, int count, const void* const* a, const void* const* e,
                 const T* win, const T* r, T* w, T* v, const uint8_t* active, T* rnew, T* x,
                 cudaStream_t st)
{
  const long long per = (n + GM_CL * GM_NT - 1) / (GM_CL * GM_NT);
  const dim3 grid(GM_CL, nd);
  auto launch = [&](int j0, int cnt, int nsweep, bool first, bool norm, bool last) {
    GmresImages im;
    for (int j = 0; j < cnt; ++j) {
      im.a[j] = a[j0 + j];
      im.e[j] = e[j0 + j];
    }
#define QBX_GM(E)                                                                                \
  k_gmres_step<T, E><<<grid, GM_NT, 0, st>>>(im, cnt, nsweep, first, norm, last, n, win, r, w, v, \
                                             active, rnew, x)
    if (per <= 4) QBX_GM(4);
    else if (per <= 8) QBX_GM(8);
    else QBX_GM(0);
#undef QBX_GM
    return cudaGetLastError();
  };
  if (count <= GM_MAXV) return launch(0, count, 2, true, true, true);
  for (int sweep = 0; sweep < 2; ++sweep)
    for (int j0 = 0; j0 < count; j0 += GM_MAXV) {
      const bool end = j0 + GM_MAXV >= count;
      cudaError_t err = launch(j0, end ? count - j0 : GM_MAXV, 1, sweep == 0 && j0 == 0, end,
                               end && sweep == 1);
      if (err != cudaSuccess) return err;
    }
  return cudaSuccess;
}

}  // namespace

cudaError_t launch_gmres_step(bool cplx, int nd, long long n, int count, const void* const* a,
                              const void* const* e, const void* win, const void* r, void* w, void* v,
                              const uint8_t* active, void* rnew, void* x, cudaStream_t st)
{
  if (cplx)
    return step<double2>(nd, n, count, a, e, (const double2*)win, (const double2*)r, (double2*)w,
                         (double2*)v, active, (double2*)rnew, (double2*)x, st);
  return step<double>(nd, n, count, a, e, (const double*)win, (const double*)r, (double*)w,
                      (double*)v, active, (double*)rnew, (double*)x, st);
}

}  // namespace qbx
