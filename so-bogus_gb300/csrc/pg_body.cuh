// The projected-gradient iteration shared by the persistent kernels (kernels_pg.cu describes its phases).
#pragma once

#include "internal.h"
#include "soc_device.cuh"
#include "soc_ops.cuh"
#include "spmv_chunk.cuh"

namespace bogus_gpu {

namespace {

template <class T>
__device__ __forceinline__ void load3cg(const T* p, int i, T* v) {
  v[0] = ldcg(p + 3 * i);
  v[1] = ldcg(p + 3 * i + 1);
  v[2] = ldcg(p + 3 * i + 2);
}
template <class T>
__device__ __forceinline__ void store3(T* p, int i, const T* v) {
  p[3 * i] = v[0];
  p[3 * i + 1] = v[1];
  p[3 * i + 2] = v[2];
}

// Positions, ST values apart: 3, or 4 (FP32, one 16-byte access) where a kernel gathers them padded.
template <int ST, class T>
__device__ __forceinline__ void load_pos(const T* p, int i, T* v) {
  if constexpr (ST == 4) {
    const float4 q = __ldcg(reinterpret_cast<const float4*>(p) + i);
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
  } else {
    load3cg(p, i, v);
  }
}
template <int ST, class T>
__device__ __forceinline__ void store_pos(T* p, int i, const T* v) {
  if constexpr (ST == 4) reinterpret_cast<float4*>(p)[i] = make_float4(v[0], v[1], v[2], 0.f);
  else store3(p, i, v);
}

// Position buffers 0, 1, 2 (X0..X2) and 4 (Wv, free in APGD / Descent: the speculative momentum point);
// 3 names the x_best buffer in PGOut::best_buf.
template <class T>
struct Bufs {
  const PGArgsT<T>& a;
  __device__ T* X(int k) const { return k == 0 ? a.X0 : (k == 1 ? a.X1 : (k == 2 ? a.X2 : a.Wv)); }
  __device__ T* MX(int k) const { return k == 0 ? a.MX0 : (k == 1 ? a.MX1 : (k == 2 ? a.MX2 : a.MX3)); }
};

__device__ __forceinline__ int third(int p, int q) {
  for (int k = 0; k < 3; ++k)
    if (k != p && k != q) return k;
  return 0;
}

// The first two of the product buffers {0, 1, 2, 3} other than p and q (p == q allowed).
__device__ __forceinline__ void two_free_mx(int p, int q, int& f0, int& f1) {
  f0 = -1;
  f1 = -1;
  for (int v = 0; v < 4; ++v) {
    if (v == p || v == q) continue;
    if (f0 < 0) f0 = v;
    else if (f1 < 0) f1 = v;
  }
}

// The first two of the position buffers {0, 1, 2, 4} other than p and q (p == q allowed).
__device__ __forceinline__ void two_free(int p, int q, int& f0, int& f1) {
  const int ids[4] = {0, 1, 2, 4};
  f0 = -1;
  f1 = -1;
  for (int k = 0; k < 4; ++k) {
    const int v = ids[k];
    if (v == p || v == q) continue;
    if (f0 < 0) f0 = v;
    else if (f1 < 0) f1 = v;
  }
}

}  // namespace

// Per-warp scratch of the FP32 correction products, allocated only in the kernel that uses them (HY).
template <bool HY>
__device__ __forceinline__ ChunkScratchT<float>* hy_scratch() { return nullptr; }
template <>
__device__ __forceinline__ ChunkScratchT<float>* hy_scratch<true>() {
  __shared__ ChunkScratchT<float> s[8];
  return s;
}

// W x_ref + the FP32 product of the correction, for row 32c + lane
template <class T>
__device__ __forceinline__ void add_wxref(const PGArgsT<T>& a, int c, const float* acc32, T* acc) {
  const int i = 32 * c + (threadIdx.x & 31);
  if (i < a.n) {
    acc[0] = ldcg(a.hy_wxref + 3 * i) + (double)acc32[0];
    acc[1] = ldcg(a.hy_wxref + 3 * i + 1) + (double)acc32[1];
    acc[2] = ldcg(a.hy_wxref + 3 * i + 2) + (double)acc32[2];
  }
}

// W v for row 32c + lane as W x_ref + W32 (v - x_ref)_32, d = (v - x_ref)_32: FP32 chains over the FP32 copy of
// W (interleaved, or the plain BSR values of the batched solves) in the chunk-segmented order, then added to the
// FP64 W x_ref.
template <class T, bool IL>
__device__ __forceinline__ void hy_product(const PGArgsT<T>& a, int c, const float* __restrict__ d,
                                           ChunkScratchT<float>& sh32, T* acc) {
  float acc32[3] = {0.f, 0.f, 0.f};
  if constexpr (IL) {
    const InterleavedBlocks<float> b32{a.icol, a.hy_ival, a.slot0};
    spmv_chunk<1, true>(a.rowptr, b32, a.n, c, sh32, [&](int j, float* x) { load3cg(d, j, x); }, acc32);
  } else {
    const PlainBlocks<float> b32{a.col, a.hy_ival};
    spmv_chunk<1, true>(a.rowptr, b32, a.n, c, sh32, [&](int j, float* x) { load3cg(d, j, x); }, acc32);
  }
  add_wxref(a, c, acc32, acc);
}

template <class T, bool IL>
struct BlocksOf;
template <class T>
struct BlocksOf<T, false> {
  static __device__ __forceinline__ PlainBlocks<T> make(const PGArgsT<T>& a) { return PlainBlocks<T>{a.col, a.val}; }
};
template <class T>
struct BlocksOf<T, true> {
  static __device__ __forceinline__ InterleavedBlocks<T> make(const PGArgsT<T>& a) {
    return InterleavedBlocks<T>{a.icol, a.ival, a.slot0};
  }
};

// IL: read W through its interleaved copy (single-problem solves) or the plain BSR arrays (batched and
// allocation-free solves). The arithmetic is the same.
// SC: the Standard and Conjugated variants (their own kernel instantiation, so that their code does not change the
// register allocation of the APGD / Descent / SPG kernels).
// HY: APGD with FP32 correction products (FP64 iterates, law and reductions; its own instantiation as well):
// W v = W x_ref + W32 (v - x_ref)_32, x_ref and W x_ref refreshed in FP64 every hy_refresh iterations.
// AHEAD: FP64 products with their loads two blocks ahead (spmv_chunk).
// RES: the FP32 copy of W lives in shared memory, each warp owning one chunk (ctx.chunk32, kernels_pg_resident32.cu); the
// FP32 points that its products gather (the positions of the FP32 solve, the corrections of HY) are 4 floats apart.
template <class T, bool IL, bool SC = false, bool HY = false, bool RES = false, bool AHEAD = false, class Ctx>
__device__ __forceinline__ int pg_body_inl(const PGArgsT<T>& a, Ctx& ctx) {
  constexpr int ST = RES && sizeof(T) == 4 ? 4 : 3;
  using Ops = SocOps<T>;
  const Bufs<T> B{a};
  ChunkScratchT<T>& sh = ctx.cs[threadIdx.x >> 5];
  const auto blocks = BlocksOf<T, IL>::make(a);
  // y = W x of chunk c for every lane (row 32c + lane), x gathered from a buffer written earlier in the kernel
  auto product = [&](int c, const T* __restrict__ xsrc, T* acc) {
    if constexpr (RES && sizeof(T) == 4) {
      ctx.chunk32.template product<1>(xsrc, acc, acc);
      return;
    }
    spmv_chunk<1, true, AHEAD>(a.rowptr, blocks, a.n, c, sh, [&](int j, T* x) { load3cg(xsrc, j, x); }, acc);
  };
  const int lane = threadIdx.x & 31;
  // HY: the FP32 correction v - x_ref of position buffer k (0, 1, 2 or 4), written beside every position that a
  // later product multiplies
  auto hy_d = [&](int k) -> float* { return a.hy_d + (size_t)(k == 4 ? 3 : k) * a.hy_stride; };
  auto store_corr = [&](int k, int i, const T* v) {
    if constexpr (HY) {
      T xr[3];
      load3cg(a.hy_xref, i, xr);
      const float d[3] = {(float)(v[0] - xr[0]), (float)(v[1] - xr[1]), (float)(v[2] - xr[2])};
      store_pos<RES ? 4 : 3>(hy_d(k), i, d);
    }
  };
  // W X(k) for row 32c + lane: the FP64 product or, HY, W x_ref + W32 (X(k) - x_ref)_32 (FP32 FMA chains in the
  // chunk-segmented order over the FP32 interleaved copy of W)
  auto product_k = [&](int c, int k, T* acc) {
    if constexpr (HY) {
      if constexpr (RES) {
        float acc32[3] = {0.f, 0.f, 0.f};
        ctx.chunk32.template product<1>(hy_d(k), acc32, acc32);
        add_wxref(a, c, acc32, acc);
      } else {
        hy_product<T, IL>(a, c, hy_d(k), hy_scratch<HY>()[threadIdx.x >> 5], acc);
      }
    } else {
      product(c, B.X(k), acc);
    }
  };
  const bool desaxce = a.desaxce != 0;
  const bool spg = a.variant == 4;
  const bool apgd = a.variant == 3;
  const int C = a.nchunks;
  const unsigned res_mask = a.use_inf ? 1u : 0u;

  auto put = [&](int q, int c, double v, bool is_max) {
    v = is_max ? warp_max_butterfly(v) : warp_sum_butterfly(v);
    if (lane == 0) ctx.csum()[q * C + c] = v;
  };
  // chunk sums of values 0 and 1 (value 0 the maximum when max0)
  auto put2 = [&](int c, double v0, double v1, bool max0) {
    if (max0) {
      put(0, c, v0, true);
      put(1, c, v1, false);
      return;
    }
    const double v = warp_sum2_butterfly(v0, v1);
    if ((lane & 15) == 0) ctx.csum()[(lane >> 4) * C + c] = v;
  };
  auto put4 = [&](int c, double v0, double v1, double v2, double v3) {
    const double v = warp_sum4_butterfly(v0, v1, v2, v3);
    if ((lane & 7) == 0) ctx.csum()[(lane >> 3) * C + c] = v;
  };
  auto sync = [&]() -> bool { return ctx.sync(); };
  auto sync_reduce = [&](int K, unsigned maxmask) -> bool { return ctx.sync_reduce(K, maxmask); };
  // split: the CTAs may go on before the scalars are published; read them after ctx.await_scalars()
  auto sync_reduce_split = [&](int K, unsigned maxmask) -> bool { return ctx.sync_reduce_split(K, maxmask); };
  auto scal = [&](int q) { return ctx.scal(q); };
  // ConstrainedSolverBase::eval: sum / (1 + n), or the maximum with the infinity norm
  const double n_plus_1 = (double)(1 + a.n);
  auto residual_of = [&](double reduced) { return a.use_inf ? reduced : ipipe::div_rn(reduced, n_plus_1); };
  unsigned ph[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  unsigned n_refresh = 0;  // HY: refreshes of x_ref
  auto finish = [&](double min_res, unsigned iters, int best_buf, int converged) -> int {
    if (ctx.writer()) {
      a.out->min_res = min_res;
      a.out->iters = iters;
      a.out->best_buf = best_buf;
      a.out->converged = converged;
#pragma unroll
      for (int k = 0; k < 9; ++k) a.out->phases[k] = ph[k];
      a.out->hy_refreshes = n_refresh;
    }
    return best_buf;
  };

  int ix = 0, iprev = 0, ixs = 1, imx = 0;

  // projectOnConstraints(x) (:90)
  ph[0]++;
  for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
    const int i = 32 * c + lane;
    if (i < a.n) {
      T x[3];
      load_pos<ST>(a.X0, i, x);
      Ops::project(__ldg(a.mu + i), x);
      store_pos<ST>(a.X0, i, x);
    }
  }
  if (!sync()) return -1;

  // Mx = W x (:93) and guess_alpha (:21-28): |W (x - 1)|^2, |x - 1|^2
  ph[1]++;
  for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
    const int i = 32 * c + lane;
    double v0 = 0.0, v1 = 0.0;
    T acc[3] = {T(0), T(0), T(0)}, accd[3] = {T(0), T(0), T(0)};
    if constexpr (RES && sizeof(T) == 4) {
      ctx.chunk32.template product<2>(a.X0, acc, accd);
    } else {
      spmv_chunk<2, true>(a.rowptr, blocks, a.n, c, sh, [&](int j, T* x) { load3cg(a.X0, j, x); }, acc, accd);
    }
    if (i < a.n) {
      store3(a.MX0, i, acc);
      v0 = Ops::sq3(accd);
      T x[3];
      load_pos<ST>(a.X0, i, x);
      const T d[3] = {x[0] - T(1), x[1] - T(1), x[2] - T(1)};
      v1 = Ops::sq3(d);
      if constexpr (HY) {
        store3(a.hy_wxref, i, acc);
        store3(a.hy_xref, i, x);
      }
    }
    put2(c, v0, v1, false);
  }
  if (!sync_reduce(2, 0u)) return -1;
  double alpha = 1.0;
  {
    const double nMx = scal(0);
    if (nMx > 1.e-16) alpha = dmin(1., ipipe::div_rn(scal(1), nMx));
  }
  if (a.max_iters == 0) {
    return finish(-1.0, 0, 0, 0);
  }

  // Row-local part A, given Mx_i: writes y, s0 and xs = P(x - alpha_t y) (APGD) and returns the residual
  // and objective terms; SPG additionally needs (xs - prev).y.
  auto phaseA = [&](int i, const T* Mx, double alpha_t, double& res_i, double& second_i) {
    T x[3], bb[3];
    load_pos<ST>(B.X(ix), i, x);
    bb[0] = __ldg(a.b + 3 * i);
    bb[1] = __ldg(a.b + 3 * i + 1);
    bb[2] = __ldg(a.b + 3 * i + 2);
    const T mu = __ldg(a.mu + i), sc = __ldg(a.scaling + i);
    T y[3] = {Mx[0] + bb[0], Mx[1] + bb[1], Mx[2] + bb[2]};
    const T lx[3] = {x[0] * sc, x[1] * sc, x[2] * sc};
    res_i = Ops::law_eval(desaxce, mu, lx, y);
    const T s0 = Ops::cov(desaxce, mu, y);
    y[0] = desaxce ? y[0] + s0 : Ops::plus0(y[0]);
    y[1] = Ops::plus0(y[1]);
    y[2] = Ops::plus0(y[2]);
    const T na = T(-alpha_t);
    T xs[3] = {fma(na, y[0], x[0]), fma(na, y[1], x[1]), fma(na, y[2], x[2])};
    Ops::project(mu, xs);
    store3(a.Y, i, y);
    if (desaxce) a.S0[i] = s0;
    store_pos<ST>(B.X(ixs), i, xs);
    store_corr(ixs, i, xs);
    if (spg) {
      T pv[3];
      load_pos<ST>(B.X(iprev), i, pv);
      const T d[3] = {xs[0] - pv[0], xs[1] - pv[1], xs[2] - pv[2]};
      second_i = Ops::dot3(d, y);
    } else {
      const T t0 = Ops::half(Mx[0]) + bb[0];
      const T t[3] = {desaxce ? t0 + s0 : Ops::plus0(t0), Ops::plus0(Ops::half(Mx[1]) + bb[1]),
                      Ops::plus0(Ops::half(Mx[2]) + bb[2])};
      second_i = Ops::dot3(x, t);
    }
  };

  auto runA = [&](double alpha_t, bool split) -> bool {  // A as its own pass (Mx already in MX(imx))
    ph[2]++;
    for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
      const int i = 32 * c + lane;
      double r = 0.0, q = 0.0;
      if (i < a.n) {
        T Mx[3];
        load3cg(B.MX(imx), i, Mx);
        phaseA(i, Mx, alpha_t, r, q);
      }
      put2(c, r, q, res_mask != 0);
    }
    return split ? sync_reduce_split(2, res_mask) : sync_reduce(2, res_mask);
  };

  double min_res = -1.0, theta = 1.0;
  bool best_pending = false;
  unsigned it = 0;

  if constexpr (SC) {
    // ------------------------------------------------ Standard (:157-209) and Conjugated (:211-286)
    // Single-problem solves only (the host rejects them elsewhere): the Conjugated variant's first reduction
    // has 5 quantities. x = X(ix), the line search's trial point X(ixs) (the two swap when a search ends),
    // Mx = MX(imx), its product MX(1 - imx). Standard: pg = X(2), W pg = MX(2). Conjugated: prev_pg = X(2),
    // prev_dir = MX(2) (formed in A as (x - x_old) / alpha of the last search, x_old still in X(ixs)),
    // dir = X(4).
    const bool conj = a.variant == 2;
    double alpha_s = 1.0, alpha_prev = 1.0, prev_n2 = 0.0;
    bool have_prev = false;
    for (;;) {
      // A: y = Mx + b, the residual, s = COV(y), y += s, J; xs = P(x - y), pg = x - xs (:164-176, :218-231)
      ph[2]++;
      for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
        const int i = 32 * c + lane;
        double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        if (i < a.n) {
          T x[3], Mx[3], bb[3];
          load_pos<ST>(B.X(ix), i, x);
          load3cg(B.MX(imx), i, Mx);
          bb[0] = __ldg(a.b + 3 * i);
          bb[1] = __ldg(a.b + 3 * i + 1);
          bb[2] = __ldg(a.b + 3 * i + 2);
          const T mu = __ldg(a.mu + i), sc = __ldg(a.scaling + i);
          T y[3] = {Mx[0] + bb[0], Mx[1] + bb[1], Mx[2] + bb[2]};
          const T lx[3] = {x[0] * sc, x[1] * sc, x[2] * sc};
          v[0] = Ops::law_eval(desaxce, mu, lx, y);
          const T s0 = Ops::cov(desaxce, mu, y);
          y[0] = y[0] + s0;
          y[1] = Ops::plus0(y[1]);
          y[2] = Ops::plus0(y[2]);
          const T t[3] = {(Ops::half(Mx[0]) + bb[0]) + s0, Ops::plus0(Ops::half(Mx[1]) + bb[1]),
                          Ops::plus0(Ops::half(Mx[2]) + bb[2])};
          v[1] = Ops::dot3(x, t);
          T xs[3] = {x[0] - y[0], x[1] - y[1], x[2] - y[2]};
          Ops::project(mu, xs);
          const T pg[3] = {x[0] - xs[0], x[1] - xs[1], x[2] - xs[2]};
          store3(a.Y, i, y);
          a.S0[i] = s0;
          if (!conj) {
            v[2] = Ops::dot3(y, pg);
          } else {
            v[2] = Ops::sq3(pg);
            if (have_prev) {
              T xo[3], ppg[3];
              load_pos<ST>(B.X(ixs), i, xo);
              load_pos<ST>(B.X(2), i, ppg);
              const T pd[3] = {(x[0] - xo[0]) / T(alpha_prev), (x[1] - xo[1]) / T(alpha_prev),
                               (x[2] - xo[2]) / T(alpha_prev)};
              store3(B.MX(2), i, pd);
              const T dg[3] = {pg[0] - ppg[0], pg[1] - ppg[1], pg[2] - ppg[2]};
              v[3] = Ops::dot3(pd, dg);
              v[4] = Ops::dot3(pg, ppg);
            }
          }
          store_pos<ST>(B.X(2), i, pg);
        }
        put(0, c, v[0], res_mask != 0);
        put(1, c, v[1], false);
        put(2, c, v[2], false);
        if (conj) {
          put(3, c, v[3], false);
          put(4, c, v[4], false);
        }
      }
      if (!sync_reduce(conj ? 5 : 3, res_mask)) return -1;
      const double res = residual_of(scal(0)), J = scal(1), s2 = scal(2);
      const double den_c = conj ? scal(3) : 0.0, xp = conj ? scal(4) : 0.0;
      if (a.trace && ctx.writer()) a.trace[it] = res;
      if (it == 0 || less_from_zero(res, min_res)) {
        min_res = res;
        best_pending = true;
      }
      if (res < a.tol) return finish(min_res, it, ix, 1);
      // the step direction
      double beta = 0.0;
      bool neg_y = false;
      if (!conj) {
        // Mpg = W pg, pg.Mpg (:177-181); pg *= beta with beta = -y.pg / pg.Mpg
        ph[3]++;
        for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
          const int i = 32 * c + lane;
          double v0 = 0.0;
          T acc[3] = {T(0), T(0), T(0)};
          product(c, B.X(2), acc);
          if (i < a.n) {
            T pg[3];
            load_pos<ST>(B.X(2), i, pg);
            store3(B.MX(2), i, acc);
            v0 = Ops::dot3(pg, acc);
          }
          put(0, c, v0, false);
        }
        if (!sync_reduce(1, 0u)) return -1;
        beta = -s2 / scal(0);
      } else if (prev_n2 == 0.) {
        neg_y = true;  // dir = -y (:232-233)
      } else {
        // dir = beta prev_dir - y, with dir = -y when it is not a descent direction (:235-245)
        beta = (den_c < 1.e-12) ? dmax(0., (s2 - xp)) / prev_n2 : dmax(0., (s2 - xp)) / den_c;
        const T bc = T(beta);
        ph[7]++;
        for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
          const int i = 32 * c + lane;
          double v0 = 0.0;
          if (i < a.n) {
            T pd[3], y[3];
            load3cg(B.MX(2), i, pd);
            load3cg(a.Y, i, y);
            const T dir[3] = {bc * pd[0] - y[0], bc * pd[1] - y[1], bc * pd[2] - y[2]};
            store_pos<ST>(B.X(4), i, dir);
            v0 = Ops::dot3(dir, y);
          }
          put(0, c, v0, false);
        }
        if (!sync_reduce(1, 0u)) return -1;
        neg_y = scal(0) >= 0.;
      }
      if (conj) prev_n2 = s2;
      // Armijo line search (:93-107 of the same file's line-search helper): xs = P(x + alpha dir), W xs,
      // Js = xs.((W xs / 2 + (b + s)) + 0) against J + armijo (y.(xs - x))
      alpha_s = conj ? alpha_s * a.opt : dmin(1., alpha_s * a.opt);
      const T bt = T(beta);
      for (unsigned ls = 0; ls < a.ls_iters; ++ls) {
        const T al = T(alpha_s);
        ph[4]++;
        for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
          const int i = 32 * c + lane;
          if (i < a.n) {
            T x[3], d[3];
            load_pos<ST>(B.X(ix), i, x);
            if (!conj) {
              T pg[3];
              load_pos<ST>(B.X(2), i, pg);
              d[0] = pg[0] * bt; d[1] = pg[1] * bt; d[2] = pg[2] * bt;
            } else if (neg_y) {
              T y[3];
              load3cg(a.Y, i, y);
              d[0] = -y[0]; d[1] = -y[1]; d[2] = -y[2];
            } else {
              load_pos<ST>(B.X(4), i, d);
            }
            T xs[3] = {fma(al, d[0], x[0]), fma(al, d[1], x[1]), fma(al, d[2], x[2])};
            Ops::project(__ldg(a.mu + i), xs);
            store_pos<ST>(B.X(ixs), i, xs);
            if (best_pending) store_pos<ST>(a.XB, i, x);
          }
        }
        best_pending = false;
        if (!sync()) return -1;
        ph[3]++;
        for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
          const int i = 32 * c + lane;
          double v0 = 0.0, v1 = 0.0;
          T acc[3] = {T(0), T(0), T(0)};
          product(c, B.X(ixs), acc);
          if (i < a.n) {
            store3(B.MX(1 - imx), i, acc);
            T x[3], xs[3], y[3];
            load_pos<ST>(B.X(ix), i, x);
            load_pos<ST>(B.X(ixs), i, xs);
            load3cg(a.Y, i, y);
            const T s0 = ldcg(a.S0 + i);
            const T bs[3] = {__ldg(a.b + 3 * i) + s0, Ops::plus0(__ldg(a.b + 3 * i + 1)),
                             Ops::plus0(__ldg(a.b + 3 * i + 2))};
            const T t[3] = {Ops::plus0(Ops::half(acc[0]) + bs[0]), Ops::plus0(Ops::half(acc[1]) + bs[1]),
                            Ops::plus0(Ops::half(acc[2]) + bs[2])};
            v0 = Ops::dot3(xs, t);
            const T dd[3] = {xs[0] - x[0], xs[1] - x[1], xs[2] - x[2]};
            v1 = Ops::dot3(y, dd);
          }
          put2(c, v0, v1, false);
        }
        if (!sync_reduce(2, 0u)) return -1;
        if (scal(0) < J + a.armijo * scal(1)) break;
        alpha_s *= a.pess;
      }
      // x = xs, Mx = W xs
      const int t2 = ix;
      ix = ixs;
      ixs = t2;
      imx = 1 - imx;
      alpha_prev = alpha_s;
      have_prev = true;
      ++it;
      if (it >= a.max_iters) break;
    }
    return finish(min_res, it, 3, 0);
  }

  if (!spg) {
    // ---------------------------------------------------------------- APGD / Descent
    // APGD's momentum point x = xs + beta (xs - prev) (:137-139) is formed speculatively by every trial
    // product (C) into the spare buffer ispec, with beta from the Nesterov sequence (it needs no reduction);
    // when the line search ends with momentum, that buffer becomes x without a pass of its own.
    // A (alone or fused with E) ends with a split reduction: the trial product of the next C phase does not
    // need the residual and objective, so a warp reads them (iteration top: trace, best iterate, convergence)
    // after the product of its first chunk, or after the phase when it gets no chunk.
    int ispec = 4;
    // momentum product by linearity: imp holds W prev (prev = x after the projection: MX(imx)); each trial
    // product goes to ims and the momentum product fma(beta, W xs - W prev, W xs) to imn
    const bool lin = apgd && a.lin_momentum != 0;
    int imp = imx, ims = 1, imn = 2;
    unsigned next_refresh = HY ? a.hy_refresh : 0u;  // HY: the first iteration whose momentum step refreshes x_ref
    double alpha_t = alpha * a.opt;
    // stall test of the FP32 part (stall_iters > 0; compiled into the FP32 kernels only): consecutive iterations
    // whose residual repeats the previous one bit for bit or whose line search ran out of trials
    // HY: the part ends (for the plain FP64 solve to take over) when the best residual has not improved by 1 %
    // in 10 refresh intervals, the noise of the FP32 corrections having become the limit
    constexpr bool kStallTest = sizeof(T) == 4 || HY;
    unsigned stall_run = 0;
    bool exhausted = false;
    double prev_res = 0.0;
    double hy_best = 0.0;
    unsigned hy_best_it = 0;
    if (!runA(alpha_t, true)) return -1;
    for (;;) {
      double res = 0.0, J = 0.0;
      bool top_done = false, converged = false, stalled = false;
      auto top = [&]() -> bool {
        if (top_done) return true;
        if (!ctx.await_scalars()) return false;
        res = residual_of(scal(0));
        J = scal(1);
        if (a.trace && ctx.writer()) a.trace[it] = res;
        if (it == 0 || less_from_zero(res, min_res)) {
          min_res = res;
          best_pending = true;
        }
        converged = less_from_zero(res, a.tol);
        if (sizeof(T) == 4 && a.stall_iters) {
          stall_run = ((it > 0 && res == prev_res) || exhausted) ? stall_run + 1 : 0;
          prev_res = res;
          stalled = !converged && stall_run >= a.stall_iters;
        }
        if constexpr (HY) {
          if (it == 0 || res < 0.99 * hy_best) {
            hy_best = res;
            hy_best_it = it;
          }
          stalled = !converged && it - hy_best_it >= 10u * a.hy_refresh;
        }
        top_done = true;
        return true;
      };
      alpha = alpha_t;
      unsigned ls = 0;
      double decr2 = 0.0;
      double theta_spec = theta;
      const double beta_spec = apgd ? nesterov_inertia(theta_spec, 0.0) : 0.0;
      const T bt = T(beta_spec);
      if (lin) two_free_mx(imx, imp, ims, imn);
      const int ims_t = lin ? ims : 1 - imx;
      for (;;) {
        // C: Mxs = W xs, the line-search terms and the speculative momentum point (and its product, lin)
        for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
          const int i = 32 * c + lane;
          double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
          T acc[3] = {T(0), T(0), T(0)};
          product_k(c, ixs, acc);
          if (!top()) return -1;
          if (converged || (kStallTest && stalled)) break;
          if (i < a.n) {
            store3(B.MX(ims_t), i, acc);
            T x[3], xs[3], pv[3], y[3];
            load_pos<ST>(B.X(ix), i, x);
            load_pos<ST>(B.X(ixs), i, xs);
            load_pos<ST>(B.X(iprev), i, pv);
            load3cg(a.Y, i, y);
            const T t0 = Ops::half(acc[0]) + __ldg(a.b + 3 * i);
            const T t[3] = {desaxce ? t0 + ldcg(a.S0 + i) : Ops::plus0(t0),
                            Ops::plus0(Ops::half(acc[1]) + __ldg(a.b + 3 * i + 1)),
                            Ops::plus0(Ops::half(acc[2]) + __ldg(a.b + 3 * i + 2))};
            v0 = Ops::dot3(xs, t);
            const T d[3] = {xs[0] - x[0], xs[1] - x[1], xs[2] - x[2]};
            v1 = Ops::dot3(y, d);
            v2 = Ops::sq3(d);
            const T d2[3] = {xs[0] - pv[0], xs[1] - pv[1], xs[2] - pv[2]};
            v3 = Ops::dot3(d2, y);
            if (best_pending) store_pos<ST>(a.XB, i, x);
            if (apgd) {
              const T xn[3] = {fma(bt, xs[0] - pv[0], xs[0]), fma(bt, xs[1] - pv[1], xs[1]), fma(bt, xs[2] - pv[2], xs[2])};
              store_pos<ST>(B.X(ispec), i, xn);
              store_corr(ispec, i, xn);
              if (lin) {
                T mp[3];
                load3cg(B.MX(imp), i, mp);
                const T mn[3] = {fma(bt, acc[0] - mp[0], acc[0]), fma(bt, acc[1] - mp[1], acc[1]),
                                 fma(bt, acc[2] - mp[2], acc[2])};
                store3(B.MX(imn), i, mn);
              }
            }
          }
          put4(c, v0, v1, v2, v3);
        }
        if (!top()) return -1;
        if (converged) return finish(min_res, it, best_pending ? ix : 3, 1);
        if (kStallTest && stalled) return finish(min_res, it, best_pending ? ix : 3, 0);
        ph[3]++;
        best_pending = false;
        if (!sync_reduce(4, 0u)) return -1;
        const double Js = scal(0), decr = scal(1), nrm = scal(2);
        decr2 = scal(3);
        if (Js < (J + decr) + ipipe::div_rn(.5, alpha) * nrm) break;
        ++ls;
        alpha *= a.pess;
        if (ls >= a.ls_iters) break;
        // B: retry with a smaller step
        ph[4]++;
        for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
          const int i = 32 * c + lane;
          if (i < a.n) {
            T x[3], y[3];
            load_pos<ST>(B.X(ix), i, x);
            load3cg(a.Y, i, y);
            const T na = T(-alpha);
            T xs[3] = {fma(na, y[0], x[0]), fma(na, y[1], x[1]), fma(na, y[2], x[2])};
            Ops::project(__ldg(a.mu + i), xs);
            store_pos<ST>(B.X(ixs), i, xs);
            store_corr(ixs, i, xs);
          }
        }
        if (!sync()) return -1;
      }
      if (sizeof(T) == 4) exhausted = ls > 0 && ls >= a.ls_iters;
      ++it;
      const bool more = it < a.max_iters;
      if (apgd && negative(decr2)) {
        theta = theta_spec;  // nesterov_inertia(theta, 0) (:137), whose value beta_spec already holds
        const int nix = ispec, nprev = ixs;
        ix = nix;
        iprev = nprev;
        two_free(ix, iprev, ixs, ispec);
        if (!more) break;
        alpha_t = alpha * a.opt;
        if (lin) {
          // W x formed in C: A alone
          imx = imn;
          imp = ims;
          if (!runA(alpha_t, true)) return -1;
          continue;
        }
        // E + A: Mx = W x, then A of the next iteration on the same rows (HY: at a refresh the FP64 product,
        // which becomes W x_ref, with x_ref = x)
        const bool refresh = HY && it >= next_refresh;
        ph[6]++;
        for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
          const int i = 32 * c + lane;
          double r = 0.0, q = 0.0;
          T acc[3] = {T(0), T(0), T(0)};
          if constexpr (HY) {
            if (refresh) {
              product(c, B.X(ix), acc);
              if (i < a.n) {
                T xr[3];
                load_pos<ST>(B.X(ix), i, xr);
                store3(a.hy_xref, i, xr);
                store3(a.hy_wxref, i, acc);
              }
            } else {
              product_k(c, ix, acc);
            }
          } else {
            product(c, B.X(ix), acc);
          }
          if (i < a.n) {
            store3(B.MX(imx), i, acc);
            phaseA(i, acc, alpha_t, r, q);
          }
          put2(c, r, q, res_mask != 0);
        }
        if (refresh) {
          next_refresh = it + a.hy_refresh;
          ++n_refresh;
        }
        if (!sync_reduce_split(2, res_mask)) return -1;
      } else {
        theta = 1.;
        ix = ixs;
        iprev = ixs;
        if (lin) {
          imx = ims;
          imp = ims;
        } else {
          imx = 1 - imx;
        }
        two_free(ix, iprev, ixs, ispec);
        if (!more) break;
        alpha_t = alpha * a.opt;
        if (!runA(alpha_t, true)) return -1;
      }
    }
    return finish(min_res, it, 3, 0);
  }

  // ------------------------------------------------------------------ SPG (:288-351)
  const double a_min = 1.e-6, a_max = 1.e6;
  unsigned repeats = 0;  // stall test of the FP32 part (stall_iters > 0; FP32 kernels): the residual repeats in a row
  double prev_res = 0.0;
  for (;;) {
    if (!runA(alpha, false)) return -1;  // y, residual, s, xs = P(x - alpha y), (xs - prev).y
    const double res = residual_of(scal(0)), decr = scal(1);
    if (a.trace && ctx.writer()) a.trace[it] = res;
    if (it == 0 || less_from_zero(res, min_res)) {
      min_res = res;
      best_pending = true;
    }
    if (less_from_zero(res, a.tol)) {
      return finish(min_res, it, best_pending ? ix : 3, 1);
    }
    if (sizeof(T) == 4 && a.stall_iters) {
      repeats = (it > 0 && res == prev_res) ? repeats + 1 : 0;
      prev_res = res;
      if (repeats >= a.stall_iters) return finish(min_res, it, best_pending ? ix : 3, 0);
    }
    const bool mom = negative(decr);
    const double beta = mom ? nesterov_inertia(theta, 0.0) : 0.0;
    if (!mom) theta = 1.;
    // D: w and the new x (over the old x); keep the best iterate first
    ph[7]++;
    for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
      const int i = 32 * c + lane;
      if (i < a.n) {
        T x[3], xs[3], pv[3], w[3], xn[3];
        load_pos<ST>(B.X(ix), i, x);
        load_pos<ST>(B.X(ixs), i, xs);
        load_pos<ST>(B.X(iprev), i, pv);
        if (best_pending) store_pos<ST>(a.XB, i, x);
        const T bt = T(beta);
        for (int k = 0; k < 3; ++k) {
          if (mom) {
            w[k] = fma(bt, xs[k] - pv[k], xs[k]) - x[k];
            xn[k] = x[k] + w[k];
          } else {
            w[k] = xs[k] - x[k];
            xn[k] = xs[k];
          }
        }
        store_pos<ST>(a.Wv, i, w);
        store_pos<ST>(B.X(ix), i, xn);
      }
    }
    best_pending = false;
    if (!sync()) return -1;
    // E: Mx_new = W x; z = -Mx_old + Mx_new; w.z, |z|^2
    ph[8]++;
    for (int c = ctx.first_chunk(); c < C; c = ctx.next_chunk(c)) {
      const int i = 32 * c + lane;
      double v0 = 0.0, v1 = 0.0;
      T acc[3] = {T(0), T(0), T(0)};
      product(c, B.X(ix), acc);
      if (i < a.n) {
        T mo[3], w[3];
        store3(B.MX(1 - imx), i, acc);
        load3cg(B.MX(imx), i, mo);
        load_pos<ST>(a.Wv, i, w);
        const T z[3] = {-mo[0] + acc[0], -mo[1] + acc[1], -mo[2] + acc[2]};
        v0 = Ops::dot3(w, z);
        v1 = Ops::sq3(z);
      }
      put2(c, v0, v1, false);
    }
    if (!sync_reduce(2, 0u)) return -1;
    imx = 1 - imx;
    iprev = ixs;
    ixs = third(ix, iprev);
    alpha = ipipe::div_rn(scal(0), scal(1));
    alpha = dmin(a_max, dmax(a_min, alpha));
    ++it;
    if (it >= a.max_iters) break;
  }
  return finish(min_res, it, 3, 0);
}

}  // namespace bogus_gpu
