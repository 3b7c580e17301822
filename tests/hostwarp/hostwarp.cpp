// Test helper: device code that orders the warps of a CTA, compiled for the host. Every lane is a thread, the barriers
// and warp votes of CUDA are barriers among those threads, and a CTA's shared memory is a block of the simulated
// cluster's, so an order that the code does not enforce is an order that a test can bring about.
#include <algorithm>
#include <atomic>
#include <barrier>
#include <chrono>
#include <memory>
#include <optional>
#include <thread>
#include <utility>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
using std::min;

namespace sim {
constexpr int kDoubles = 512;  // shared memory of a CTA
struct Warp {
  std::barrier<> meet{32};
  double swap[32];
};
struct Cta {
  explicit Cta(int warps) : threads(32 * warps), w(warps) {}
  std::barrier<> threads;
  std::vector<Warp> w;
  double smem[kDoubles] = {};
};
struct Cluster {
  Cluster(int ctas, int warps) : all(32 * warps * ctas) {
    for (int r = 0; r < ctas; ++r) cta.push_back(std::make_unique<Cta>(warps));
  }
  std::vector<std::unique_ptr<Cta>> cta;
  std::barrier<> all;
};
thread_local Cluster* cluster;
thread_local Cta* cta;
thread_local Warp* warp;
thread_local int lane;
thread_local std::optional<std::barrier<>::arrival_token> token;
}  // namespace sim

inline void __syncwarp() { sim::warp->meet.arrive_and_wait(); }
inline void __syncthreads() { sim::cta->threads.arrive_and_wait(); }
inline double shfl(double v, int src) {
  sim::warp->swap[sim::lane] = v;
  __syncwarp();
  const double r = sim::warp->swap[src];
  __syncwarp();
  return r;
}

inline unsigned __ballot_sync(unsigned, bool on) {
  sim::warp->swap[sim::lane] = on;
  __syncwarp();
  unsigned m = 0;
  for (int l = 0; l < 32; ++l) m |= (sim::warp->swap[l] != 0.0 ? 1u : 0u) << l;
  __syncwarp();
  return m;
}
inline double __shfl_sync(unsigned, double v, int src) { return shfl(v, src); }
inline bool __any_sync(unsigned mask, bool on) { return __ballot_sync(mask, on) != 0; }
inline int atomicCAS(int* p, int expected, int v) {
  std::atomic_ref<int>(*p).compare_exchange_strong(expected, v);
  return expected;
}

namespace bogus_gpu {
inline void store_cluster(const double* p, int rank, double v) {
  sim::cluster->cta[rank]->smem[p - sim::cta->smem] = v;
}
inline void cluster_arrive() { sim::token.emplace(sim::cluster->all.arrive()); }
inline void cluster_wait() { sim::cluster->all.wait(std::move(*sim::token)); }
inline double warp_sum_butterfly(double v) {
  for (int off = 16; off >= 1; off >>= 1) v = v + shfl(v, sim::lane ^ off);
  return v;
}
inline double warp_max_butterfly(double v) {
  for (int off = 16; off >= 1; off >>= 1) {
    const double o = shfl(v, sim::lane ^ off);
    v = (v < o) ? o : v;
  }
  return v;
}
}  // namespace bogus_gpu

#include "cluster_reduce.cuh"
#include "warp_wait.cuh"

using namespace bogus_gpu;

namespace {
// f(rank, warp, lane) on every lane of a cluster
template <class F>
void run_cluster(int ctas, int warps, F&& f) {
  sim::Cluster cl(ctas, warps);
  std::vector<std::thread> threads;
  for (int r = 0; r < ctas; ++r)
    for (int w = 0; w < warps; ++w)
      for (int l = 0; l < 32; ++l)
        threads.emplace_back([&, r, w, l] {
          sim::cluster = &cl;
          sim::cta = cl.cta[r].get();
          sim::warp = &sim::cta->w[w];
          sim::lane = l;
          f(r, w, l);
        });
  for (auto& t : threads) t.join();
}
}  // namespace

extern "C" {

// `rounds` reductions of C chunks on a cluster of two CTAs whose last warps take their time over the side work: the side
// work reads what the last decision wrote and leaves a value that the next decision reads. Returns the number of
// decisions and side works that met a value of another round, or that saw another total than the chunks' sum.
int hw_cluster_reduce(int C, int rounds) {
  constexpr int kCtas = 2, kWarps = 2;
  std::atomic<int> wrong{0};
  std::atomic<int> side_value[kCtas] = {}, decided[kCtas] = {};
  run_cluster(kCtas, kWarps, [&](int r, int w, int l) {
    ClusterReduce red{sim::cta->smem + 64, C, sim::cta->smem, l, w, kWarps, kCtas};
    double expected = 0.0;
    for (int c = 0; c < C; ++c) expected += 32.0 * (c + 1);  // whole numbers: the same in any order
    for (int k = 1; k <= rounds; ++k) {
      if (w == 0)
        for (int c = r; c < C; c += kCtas) red.put(0, c, c + 1.0);
      red.reduce(
          1, 0u,
          [&] {
            std::this_thread::sleep_for(std::chrono::milliseconds(l == 0 ? 60 : 0));
            if (l != 0) return;
            if (decided[r] != k - 1) ++wrong;
            side_value[r] = k;
          },
          [&](double total) {
            if (l != 0) return;
            if (side_value[r] != k || total != expected) ++wrong;
            decided[r] = k;
          });
    }
  });
  return wrong;
}

// One maximum over two chunks of 32 values, one chunk per CTA of a cluster of two; the decision's total in each CTA.
void hw_cluster_max(const double* values, double* totals) {
  run_cluster(2, 2, [&](int r, int w, int l) {
    ClusterReduce red{sim::cta->smem + 64, 2, sim::cta->smem, l, w, 2, 2};
    if (w == 0) red.put_max(0, r, values[32 * r + l]);
    red.reduce(2, 1u, [] {}, [&](double total) {
      if (l == 0) totals[r] = total;
    });
  });
}

// A warp's wait with the lanes of `late` past the limit and those of `stopped` told to stop, *status as given; returns
// whether every lane (1), no lane (0) or only some (-1) gave up.
int hw_warp_gives_up(unsigned late, unsigned stopped, int* status) {
  std::atomic<int> gave{0};
  run_cluster(1, 1, [&](int, int, int l) {
    gave += warp_gives_up((late >> l) & 1u, (stopped >> l) & 1u, l, status, 5) ? 1 : 0;
  });
  return gave == 32 ? 1 : gave == 0 ? 0 : -1;
}

}  // extern "C"
