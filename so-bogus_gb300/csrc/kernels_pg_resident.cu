// Projected-gradient solve (APGD / Descent / SPG, Core/BlockSolvers/ProjectedGradient.impl.hpp:74-155, 288-351) of a
// problem small enough to stay in the SMs: one cooperative launch of one CTA per SM in which every 32-contact chunk
// is owned by a team of three warps for the whole solve.
//
// What bounds such a problem is latency, not throughput: with a chunk or a few per SM, a warp of k_pg_persistent
// waits for each block of W it loads (some 15 round trips to L2 per product), runs the nine FMAs of a block one after
// another (64 cycles each, the latency of GB300's FP64 unit, which one SM's four sub-partitions share at one warp
// instruction per 19 cycles), and re-reads its contacts' vectors in every phase. Here
//   - W stays in shared memory: a chunk's interleaved blocks and their columns are copied once, so a product's only
//     loads from outside the SM are the gathers of x, issued two groups of three steps ahead of their FMAs;
//   - each gathered point is loaded once per team: warp r takes step r of a group and passes it through shared
//     memory (a gather of 32 scattered contacts holds the load unit for as long as the step's FMAs take);
//   - the product is split by row component: warp r of the team accumulates component r of every row (3 FMAs per
//     block in place of 9), and the row-local work by quantity (the law's residual, the step and the objective in the
//     A phase; the three line-search terms and the momentum point in the C phase);
//   - the contacts' vectors stay in registers (a small shared array passes them between the team's warps); global
//     memory carries only the two gathered points, padded to 32 bytes per contact for one 256-bit load each, and
//     the chunk sums;
//   - reductions use the flat barrier (every CTA combines the chunk sums itself), and one warp per CTA takes the
//     line-search and momentum decisions and publishes them in shared memory.
// Every value goes through the same operations in the same order as in k_pg_persistent (kernels_pg.cu, which has the
// phases and the reference's line numbers), so the results are identical.
// us per APGD iteration on GB300 (2.31 products), k_pg_persistent / this kernel: 33 contacts 40 / 17, 500 44 / 18,
// 2 000 54 / 22, 10 000 57 / 28, 20 000 65 / 35. At 2 000 contacts, of 44 500 cycles: products 20 000 (7 200 of them
// the chain of FMAs), law and vectors 9 300, barriers 7 000, sums 4 400, decisions 4 000.
#include "internal.h"
#include "soc_device.cuh"
#include "resident.cuh"
#include "cluster_reduce.cuh"

namespace bogus_gpu {

namespace {

struct TeamShared {
  TeamCore core;
  double xs[3][32], y[3][32];  // the last step; the second product of the guess (pieces, then values) before
};

// Scalars of the iteration, written by one warp per CTA after each reduction.
struct Control {
  double stripes[32];
  double alpha, alpha_t, alpha_less, theta, theta_next, beta, J, min_res, half_over_alpha, half_over_less;
  int go, best;
  unsigned phases[9];
};

enum { kAccept = 0, kMomentum = 1, kRetry = 2, kStop = 3 };

// The CTA's part in a solve: rank among the CTAs (parties) that share the problem, and its chunks, one per team.
struct Place {
  int rank;
  unsigned parties;
  int first, stride, count;  // chunks list[first + k stride] (list null: the index itself), k < count
  const int* list;
  unsigned long long* progress;  // ResidentReduce::progress
  __device__ int chunk(int k) const {
    const int j = first + k * stride;
    return list ? __ldg(list + j) : j;
  }
};

// The CTA's shared memory: the scalars, the teams' arrays, (cluster) the two gathered points of all contacts and the
// chunk sums, the chunks' blocks.
__host__ __device__ inline size_t teams_offset() { return (sizeof(Control) + 15) / 16 * 16; }
__host__ __device__ inline size_t points_offset(int teams) { return teams_offset() + (size_t)teams * sizeof(TeamShared); }
__host__ __device__ inline size_t cluster_bytes(int chunks) { return (size_t)chunks * (2 * 32 * 4 + 2 * 4) * sizeof(double); }

// CL: the CTAs of the problem are one cluster.
template <bool CL>
__device__ __forceinline__ void resident_solve(const PGArgs& a, int teams, const Place& place, unsigned char* smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int team = warp / kTeamWarps, role = warp - kTeamWarps * team;
  Control& ctl = *reinterpret_cast<Control*>(smem);
  const bool has = team < place.count;
  const int c = has ? place.chunk(team) : 0;
  TeamShared& sh = reinterpret_cast<TeamShared*>(smem + teams_offset())[team < teams ? team : 0];
  const int C = a.nchunks;
  const int i = 32 * c + lane;
  const bool on = has && i < a.n;
  const bool desaxce = a.desaxce != 0, spg = a.variant == 4, apgd = a.variant == 3;
  const unsigned res_mask = a.use_inf ? 1u : 0u;
  const bool writer = place.rank == 0 && threadIdx.x == 0;
  // the gathered points: x (or the momentum point) and the trial point xs
  double* const gx = CL ? reinterpret_cast<double*>(smem + points_offset(teams)) : a.MX0;
  double* const gs = gx + 4 * (size_t)(CL ? 32 * C : a.n);
  auto put_point = [&](double* g, const double* v) {
    if constexpr (CL) {
#pragma unroll 4
      for (int r = 0; r < (int)place.parties; ++r) store_cluster3(g, r, v);
    } else {
      store_padded(g, v);
    }
  };
  const size_t ip = on ? 4 * (size_t)i : 0;

  auto own_point = [&](const double* g, double* v) {
    if constexpr (CL) {
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] = g[k];
    } else {
      load_padded(g, v);
    }
  };

  ResidentChunk chunk{sh.core, lane, role, team};
  if (has) {
    size_t before = 0;  // the CTA's chunks one after another, behind the teams' arrays
    for (int k = 0; k < team; ++k) before += (size_t)steps_of(a.rowptr, a.n, place.chunk(k));
    chunk.load(a.rowptr, a.col, a.val, a.n, c,
               smem + points_offset(teams) + (CL ? cluster_bytes(C) : 0) + before * kStepBytes);
  }
  const double (*const part)[64] = sh.core.part;
  // W g for this chunk's contacts, all components to every warp of the team
  auto team_product = [&](const double* g, double* out) {
    if constexpr (CL) chunk.product_local<1>(g);
    else chunk.product<1>(g);
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k] = part[k][lane];
  };

  // ---- barriers ----------------------------------------------------------------------------------------------
  auto red = [&] {
    if constexpr (CL)
      return ClusterReduce{gs + 4 * (size_t)32 * C, C, ctl.stripes, lane, warp, nwarps, (int)place.parties};
    else
      return ResidentReduce{MonoBarrier{a.mono, a.gb.status, place.parties + a.phantom_ctas}, a.csum, C, ctl.stripes, lane, warp,
                            nwarps, place.progress};
  }();
  auto put = [&](int q, double v) { red.put(q, c, v); };
  auto reduce = [&](int K, unsigned maxmask, auto side, auto decide) { return red.reduce(K, maxmask, side, decide); };
  auto sync = [&]() { return red.sync(); };

  // ---- per-contact state, the same in the team's three warps ------------------------------------------------
  // (x and prev in registers; xs, y and the products in the team's shared memory; b, mu and the scalings are read
  // where they are used, from L1)
  double x[3] = {0.0, 0.0, 0.0}, pv[3], Mx[3] = {0.0, 0.0, 0.0};
  double s0 = 0.0;  // COV(y)_N of the last A (warp 0)
  if (on) {
#pragma unroll
    for (int k = 0; k < 3; ++k) x[k] = a.X0[3 * (size_t)i + k];
    project_cone(__ldg(a.mu + i), x);  // projectOnConstraints(x) (:90)
    if (role == 1) put_point(gx + ip, x);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) pv[k] = x[k];
  auto load_b = [&](double* b) {
#pragma unroll
    for (int k = 0; k < 3; ++k) b[k] = __ldg(a.b + 3 * (size_t)i + k);
  };
  auto store_best = [&]() {
    if (on && role == 1)
      for (int k = 0; k < 3; ++k) a.XB[3 * (size_t)i + k] = x[k];
  };
  auto count = [&](int k) {
    if (threadIdx.x == 0) ++ctl.phases[k];
  };
  auto finish = [&](unsigned iters, int converged) {
    if (!writer) return;
    a.out->min_res = ctl.min_res;
    a.out->iters = iters;
    a.out->best_buf = 3;
    a.out->converged = converged;
#pragma unroll
    for (int k = 0; k < 9; ++k) a.out->phases[k] = ctl.phases[k];
    a.out->hy_refreshes = 0;
  };
  if (threadIdx.x == 0) {
    ctl.theta = 1.0;
    ctl.min_res = -1.0;
    for (int k = 0; k < 9; ++k) ctl.phases[k] = k == 0 ? 1u : 0u;
  }
  if (!sync()) return;

  // Mx = W x (:93) and guess_alpha (:21-28)
  count(1);
  if (has) {
    if constexpr (CL) chunk.product_local<2>(gx, sh.xs[0]);
    else chunk.product<2>(gx, sh.xs[0]);
#pragma unroll
    for (int k = 0; k < 3; ++k) Mx[k] = part[k][lane];
    if (role == 0) {
      const double* second = sh.xs[0] + lane;
      const double d[3] = {second[0], second[64], second[128]};
      put(0, on ? sq3(d) : 0.0);
    } else if (role == 1) {
      const double d[3] = {x[0] - 1.0, x[1] - 1.0, x[2] - 1.0};
      put(1, on ? sq3(d) : 0.0);
    }
  }
  if (!reduce(2, 0u, [] {}, [&](double total) {
        const double nMx = total_of(total, 0), n1 = total_of(total, 1);
        double alpha = 1.0;
        if (nMx > 1.e-16) alpha = dmin(1., ipipe::div_rn(n1, nMx));
        if (lane == 0) {
          ctl.alpha = alpha;
          ctl.alpha_t = spg ? alpha : alpha * a.opt;
        }
      }))
    return;
  if (a.max_iters == 0) {
    store_best();
    finish(0, 0);
    return;
  }

  unsigned it = 0;
  const double n_plus_1 = (double)(1 + a.n);
  // A (:110-125): the residual (warp 0), xs = P(x - alpha_t y) with y += COV(y) (warp 1; SPG: (xs - prev).y), the
  // objective (warp 2); y, xs and s0 go to the other warps
  auto phaseA = [&]() {
    if (!has) return;
    double v = 0.0;
    if (on) {
      const double mu = __ldg(a.mu + i);
      double b[3];
      load_b(b);
      if (role == 0) {
        const double scal = __ldg(a.scaling + i);
        const double yr[3] = {Mx[0] + b[0], Mx[1] + b[1], Mx[2] + b[2]};
        const double lx[3] = {x[0] * scal, x[1] * scal, x[2] * scal};
        v = law_eval(desaxce, mu, lx, yr);
        s0 = duality_cov(desaxce, mu, yr);
      } else if (role == 1) {
        double yn[3] = {Mx[0] + b[0], Mx[1] + b[1], Mx[2] + b[2]};
        const double sn = duality_cov(desaxce, mu, yn);
        yn[0] = desaxce ? yn[0] + sn : ipipe::plus_zero(yn[0]);
        yn[1] = ipipe::plus_zero(yn[1]);
        yn[2] = ipipe::plus_zero(yn[2]);
        const double na = neg(ctl.alpha_t);
        double p[3] = {fma(na, yn[0], x[0]), fma(na, yn[1], x[1]), fma(na, yn[2], x[2])};
        project_cone(mu, p);
        put_point(gs + ip, p);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          sh.xs[k][lane] = p[k];
          sh.y[k][lane] = yn[k];
        }
        if (spg) {
          const double d[3] = {p[0] - pv[0], p[1] - pv[1], p[2] - pv[2]};
          v = dot3(d, yn);
        }
      } else if (!spg) {
        double first = ipipe::scale2<-1>(Mx[0]) + b[0];
        if (desaxce) {
          const double yr[3] = {Mx[0] + b[0], Mx[1] + b[1], Mx[2] + b[2]};
          first = first + duality_cov(true, mu, yr);
        } else {
          first = ipipe::plus_zero(first);
        }
        const double t[3] = {first, ipipe::plus_zero(ipipe::scale2<-1>(Mx[1]) + b[1]),
                             ipipe::plus_zero(ipipe::scale2<-1>(Mx[2]) + b[2])};
        v = dot3(x, t);
      }
    }
    if (role == 0) {
      if (a.use_inf) red.put_max(0, c, v);
      else put(0, v);
    } else if (role == (spg ? 1 : 2)) {
      put(1, v);
    }
  };
  // beside A's barrier: the momentum weight that follows from theta, and 1 / 2 alpha for the line search
  auto before_top = [&]() {
    double theta = ctl.theta, beta = 0.0;
    if (spg || apgd) beta = nesterov_inertia(theta, 0.0);
    const double hoa = ipipe::div_rn(.5, ctl.alpha_t);
    if (lane == 0) {
      ctl.beta = beta;
      ctl.theta_next = theta;
      ctl.half_over_alpha = hoa;
    }
  };
  // after A's reduction: the residual, the best iterate, the trace, the objective
  auto top = [&](double total) {
    const double reduced = total_of(total, 0), second = total_of(total, 1);
    const double res = a.use_inf ? reduced : ipipe::div_rn(reduced, n_plus_1);
    const bool best = it == 0 || less_from_zero(res, ctl.min_res);
    const bool stop = less_from_zero(res, a.tol);
    const bool mom = spg ? negative(second) : apgd;
    __syncwarp();
    if (lane == 0) {
      if (a.trace && place.rank == 0) a.trace[it] = res;
      if (best) ctl.min_res = res;
      ctl.best = best;
      ctl.go = stop ? kStop : (mom ? kMomentum : kAccept);
      ctl.J = second;
      if (spg) ctl.theta = mom ? ctl.theta_next : 1.0;
      else ctl.alpha = ctl.alpha_t;
    }
  };
  auto shared3 = [&](const double (*v)[32], double* out) {
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k] = on ? v[k][lane] : 0.0;
  };

  count(2);
  phaseA();
  if (!spg) {
    // ---------------------------------------------------------------------------------------- APGD / Descent
    for (;;) {
      if (!reduce(2, res_mask, before_top, top)) return;
      if (ctl.go == kStop) {
        if (ctl.best) store_best();
        finish(it, 1);
        return;
      }
      bool pending = ctl.best != 0;
      unsigned ls = 0;
      int next;
      for (;;) {
        // C (:127-139): Mxs = W xs; Js (warp 0), y.(xs - x) and |xs - x|^2 (warp 1), (xs - prev).y and the momentum
        // point (warp 2)
        count(3);
        if (has) {
          double xs[3], Ms[3];
          team_product(gs, Ms);
          shared3(sh.xs, xs);
          if (role == 0) {
            double b[3] = {0.0, 0.0, 0.0};
            if (on) load_b(b);
            const double first = ipipe::scale2<-1>(Ms[0]) + b[0];
            const double t[3] = {desaxce ? first + s0 : ipipe::plus_zero(first),
                                 ipipe::plus_zero(ipipe::scale2<-1>(Ms[1]) + b[1]),
                                 ipipe::plus_zero(ipipe::scale2<-1>(Ms[2]) + b[2])};
            put(0, on ? dot3(xs, t) : 0.0);
          } else if (role == 1) {
            double y[3];
            shared3(sh.y, y);
            const double d[3] = {xs[0] - x[0], xs[1] - x[1], xs[2] - x[2]};
            const double v = warp_sum2_butterfly(on ? dot3(y, d) : 0.0, on ? sq3(d) : 0.0);
            red.put_totals(1, c, v);
            if (pending) store_best();
          } else {
            double y[3];
            shared3(sh.y, y);
            const double bt = ctl.beta;
            const double d[3] = {xs[0] - pv[0], xs[1] - pv[1], xs[2] - pv[2]};
            if (apgd && on) {
              const double xn[3] = {fma(bt, d[0], xs[0]), fma(bt, d[1], xs[1]), fma(bt, d[2], xs[2])};
              put_point(gx + ip, xn);
            }
            put(3, on ? dot3(d, y) : 0.0);
          }
        }
        pending = false;
        if (!reduce(4, 0u,
                    [&] {  // the step that a rejection takes, and its 1 / 2 alpha
                      const double smaller = ctl.alpha * a.pess;
                      const double hoa = ipipe::div_rn(.5, smaller);
                      if (lane == 0) {
                        ctl.alpha_less = smaller;
                        ctl.half_over_less = hoa;
                      }
                    },
                    [&](double total) {
                      const double Js = total_of(total, 0), decr = total_of(total, 1), nrm = total_of(total, 2);
                      const double decr2 = total_of(total, 3);
                      const bool accept = Js < (ctl.J + decr) + ctl.half_over_alpha * nrm;
                      const bool retry = !accept && ls + 1 < a.ls_iters;
                      const double alpha = accept ? ctl.alpha : ctl.alpha_less;
                      const double alpha_t = alpha * a.opt;
                      const bool mom = apgd && negative(decr2);
                      __syncwarp();
                      if (lane == 0) {
                        ctl.alpha = alpha;
                        ctl.go = retry ? kRetry : (mom ? kMomentum : kAccept);
                        if (retry) {
                          ctl.half_over_alpha = ctl.half_over_less;
                        } else {
                          ctl.theta = mom ? ctl.theta_next : 1.0;
                          ctl.alpha_t = alpha_t;
                        }
                      }
                    }))
          return;
        next = ctl.go;
        if (next != kRetry) break;
        ++ls;
        // B: retry with a smaller step
        count(4);
        if (on && role == 1) {
          const double na = neg(ctl.alpha);
          double p[3] = {fma(na, sh.y[0][lane], x[0]), fma(na, sh.y[1][lane], x[1]), fma(na, sh.y[2][lane], x[2])};
          project_cone(__ldg(a.mu + i), p);
          put_point(gs + ip, p);
#pragma unroll
          for (int k = 0; k < 3; ++k) sh.xs[k][lane] = p[k];
        }
        if (!sync()) return;
      }
      ++it;
      if (it >= a.max_iters) break;
      if (on && next == kMomentum) own_point(gx + ip, x);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double xs = on ? sh.xs[k][lane] : 0.0;
        if (next != kMomentum) {
          x[k] = xs;
          Mx[k] = part[k][lane];
        }
        pv[k] = xs;
      }
      if (next == kMomentum) {
        // E + A: Mx = W x (:141), then A of the next iteration
        count(6);
        if (has) team_product(gx, Mx);
      } else {
        count(2);
        if (has) team_sync(team);  // phaseA writes the shared xs that the team's warps have just read
      }
      phaseA();
    }
    finish(it, 0);
    return;
  }

  // ---------------------------------------------------------------------------------------------- SPG (:288-351)
  for (;;) {
    if (!reduce(2, res_mask, before_top, top)) return;
    if (ctl.go == kStop) {
      if (ctl.best) store_best();
      finish(it, 1);
      return;
    }
    // D: w and the new x
    count(7);
    const bool mom = ctl.go == kMomentum;
    const double bt = ctl.beta;
    if (ctl.best) store_best();
    double xs[3], Ms[3] = {0.0, 0.0, 0.0};
    shared3(sh.xs, xs);
    double w[3] = {0.0, 0.0, 0.0};
    if (on && role == 1) {
      double xn[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (mom) {
          w[k] = fma(bt, xs[k] - pv[k], xs[k]) - x[k];
          xn[k] = x[k] + w[k];
        } else {
          w[k] = xs[k] - x[k];
          xn[k] = xs[k];
        }
      }
      put_point(gx + ip, xn);
    }
    if (!sync()) return;
    // E: Mx_new = W x; z = -Mx_old + Mx_new; w.z (warp 1), |z|^2 (warp 0)
    count(8);
    if (on) own_point(gx + ip, x);
    if (has) {
      team_product(gx, Ms);
      const double z[3] = {-Mx[0] + Ms[0], -Mx[1] + Ms[1], -Mx[2] + Ms[2]};
      if (role == 0) put(1, on ? sq3(z) : 0.0);
      else if (role == 1) put(0, on ? dot3(w, z) : 0.0);
    }
    if (!reduce(2, 0u, [] {}, [&](double total) {
          double alpha = ipipe::div_rn(total_of(total, 0), total_of(total, 1));
          alpha = dmin(1.e6, dmax(1.e-6, alpha));
          if (lane == 0) ctl.alpha_t = alpha;
        }))
      return;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      Mx[k] = Ms[k];
      pv[k] = xs[k];
    }
    ++it;
    if (it >= a.max_iters) break;
    count(2);
    phaseA();
  }
  finish(it, 0);
}

// One problem on the whole grid.
__global__ void __launch_bounds__(32 * kTeamWarps * kMaxTeams, 1) k_pg_resident(PGArgs a, int teams) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int first = __ldg(a.cta_ptr + blockIdx.x);
  const Place place{(int)blockIdx.x, gridDim.x, first, 1, __ldg(a.cta_ptr + blockIdx.x + 1) - first, a.cta_list, nullptr};
  resident_solve<false>(a, teams, place, smem);
}

// One problem of at most kClusterChunks chunks on one cluster, a CTA per chunk. With so few chunks the trips through L2
// count most: an arrival at the counter and the poll that sees it (1.35 us a barrier), the chunk sums read back, the
// gathered points. Here the hardware's cluster barrier separates the phases, every CTA holds all points and chunk sums
// in its own shared memory (a chunk's team writes them into each CTA's), and a product gathers from there.
// us per iteration on GB300, k_pg_resident / this kernel, APGD and SPG: 33 contacts 16.6 / 12.6 and 12.2 / 9.9, 200 17.9 /
// 13.0 and 13.4 / 10.5, 500 18.3 / 14.4 and 13.5 / 11.3. With two or three chunks per CTA, to go beyond 16, the SM's one
// FP64 unit costs more than the barriers do: 1000 contacts 20.1 / 21.7, 1500 20.3 / 26.7.
__global__ void __launch_bounds__(32 * kMinWarps, 1) k_pg_resident_cluster(PGArgs a, int teams) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int rank = (int)blockIdx.x, ctas = (int)gridDim.x;
  const Place place{rank, gridDim.x, rank, ctas, (a.nchunks - rank + ctas - 1) / ctas, nullptr, nullptr};
  cluster_arrive();  // every CTA's shared memory is there before the first store into it
  cluster_wait();
  resident_solve<true>(a, teams, place, smem);
  __syncwarp();
  cluster_arrive();  // and stays until the last
  cluster_wait();
}

// A batch: every CTA works through its own list of jobs, a job being its part in one problem (the chunks rank,
// rank + ctas, ...). The lists hold the problems in one global order, so a CTA waits in a problem's barriers only for
// CTAs that are at this problem or at earlier ones. The wait for earlier ones is as long as their solves are: it ends in
// a timeout only when no CTA of the launch passes a barrier for the length of the limit (mono[nproblems] counts them).
__global__ void __launch_bounds__(32 * kTeamWarps * kMaxTeams, 1)
    k_pg_resident_batch(PGBatchArgs ba, const int* job_ptr, const ResidentJob* jobs, unsigned long long* mono, int teams) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ PGArgs a;
  for (int j = __ldg(job_ptr + blockIdx.x); j < __ldg(job_ptr + blockIdx.x + 1); ++j) {
    const ResidentJob job = jobs[j];
    const size_t c0 = ba.contact_ptr[job.problem];
    const int n = (int)(ba.contact_ptr[job.problem + 1] - c0);
    __syncthreads();
    if (threadIdx.x == 0) {
      a = ba.base;
      a.n = n;
      a.nchunks = (n + 31) / 32;
      a.rowptr = ba.base.rowptr + c0;
      a.b = ba.base.b + 3 * c0;
      a.mu = ba.base.mu + c0;
      a.scaling = ba.base.scaling + c0;
      a.X0 = ba.base.X0 + 3 * c0;
      a.MX0 = ba.base.MX0 + 8 * c0;  // two gathered points, padded
      a.XB = ba.base.XB + 3 * c0;
      a.csum = ba.base.csum + 8 * (size_t)ba.chunk_ptr[job.problem];
      a.trace = nullptr;
      a.out = ba.base.out + job.problem;
      a.mono = mono + job.problem;
    }
    __syncthreads();
    const int mine = a.nchunks > job.rank ? (a.nchunks - job.rank + job.ctas - 1) / job.ctas : 0;
    const Place place{job.rank, (unsigned)job.ctas, job.rank, job.ctas, mine, nullptr, mono + ba.nproblems};
    resident_solve<false>(a, teams, place, smem);
    // the best iterate over the initial one, by the lanes that stored it
    const int warp = threadIdx.x >> 5, i = 32 * (job.rank + (warp / kTeamWarps) * job.ctas) + (threadIdx.x & 31);
    if (warp / kTeamWarps < mine && warp % kTeamWarps == 1 && i < n)
      for (int k = 0; k < 3; ++k) ba.r[3 * (c0 + i) + k] = a.XB[3 * i + k];
  }
}

// teams per CTA, and the largest sum of S over a CTA's chunks
size_t resident_smem(int teams, int steps) {
  return points_offset(teams) + (size_t)steps * kStepBytes;
}

}  // namespace

// Whether the resident kernel takes CTAs with up to `teams` chunks of up to `steps` steps (S) in sum and `longest` each:
// a team per chunk, every chunk's blocks in shared memory, a lane's row starts in 64 bits, columns in 16.
bool pg_resident_fits(int device, int teams, int steps, int longest, int n) {
  return teams >= 1 && teams <= kMaxTeams && longest <= 64 && n <= 65536 &&
         resident_smem(teams, steps) <= resident_shared_limit(device);
}

int pg_resident_max_teams() { return kMaxTeams; }

namespace {
cudaError_t launch_resident(const void* fn, void** args, int ctas, int teams, int steps, cudaStream_t s) {
  const size_t bytes = resident_smem(teams, steps);
  const cudaError_t e = allow_resident_shared(fn);
  if (e != cudaSuccess) return e;
  const int warps = kTeamWarps * teams > kMinWarps ? kTeamWarps * teams : kMinWarps;
  return cudaLaunchCooperativeKernel(fn, dim3(ctas), dim3(32 * warps), args, bytes, s);
}
cudaLaunchConfig_t cluster_config(int ctas, size_t bytes, cudaStream_t s, cudaLaunchAttribute* at) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)ctas;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(32 * kMinWarps);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}
}  // namespace

cudaError_t launch_pg_resident(const PGArgs& a, int ctas, int teams, int steps, cudaStream_t s) {
  PGArgs copy = a;
  void* args[] = {&copy, &teams};
  return launch_resident((const void*)k_pg_resident, args, ctas, teams, steps, s);
}

// One CTA per chunk, a cluster of up to 16 (more than the portable 8).
bool pg_resident_cluster_fits(int device, int chunks, int longest) {
  if (chunks < 1 || chunks > kClusterChunks || longest > 64) return false;
  const size_t bytes = resident_smem(1, longest) + cluster_bytes(chunks);
  if (bytes > resident_shared_limit(device)) return false;
  const void* fn = (const void*)k_pg_resident_cluster;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      allow_resident_shared(fn) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  cudaLaunchAttribute at{};
  cudaLaunchConfig_t cfg = cluster_config(chunks, bytes, nullptr, &at);
  int active = 0;
  if (cudaOccupancyMaxActiveClusters(&active, fn, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return active >= 1;
}

cudaError_t launch_pg_resident_cluster(const PGArgs& a, int longest, cudaStream_t s) {
  cudaLaunchAttribute at{};
  cudaLaunchConfig_t cfg = cluster_config(a.nchunks, resident_smem(1, longest) + cluster_bytes(a.nchunks), s, &at);
  return cudaLaunchKernelEx(&cfg, k_pg_resident_cluster, a, 1);
}

cudaError_t launch_pg_resident_batch(const PGBatchArgs& b, const int* job_ptr, const ResidentJob* jobs,
                                     unsigned long long* mono, int ctas, int teams, int steps, cudaStream_t s) {
  PGBatchArgs copy = b;
  void* args[] = {&copy, &job_ptr, &jobs, &mono, &teams};
  return launch_resident((const void*)k_pg_resident_batch, args, ctas, teams, steps, s);
}

// Sets this file's copy of the device-side wait limit on the current device.
BOGUS_GPU_WAIT_LIMIT_SETTER(set_wait_limit_pg_resident)

}  // namespace bogus_gpu
