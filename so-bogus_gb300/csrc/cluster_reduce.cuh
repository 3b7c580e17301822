// Reductions and barriers of a problem that one cluster of CTAs solves (kernels_pg_resident.cu).
#pragma once

#include <cstddef>

#ifdef __CUDACC__
#include "device_common.cuh"
#endif

namespace bogus_gpu {

#ifdef __CUDACC__
// Stores into the shared memory of every CTA of the cluster (the address is this CTA's own).
__device__ __forceinline__ void store_cluster(const double* p, int rank, double v) {
  asm volatile("{ .reg .b32 r; mapa.shared::cluster.u32 r, %0, %1; st.shared::cluster.f64 [r], %2; }" ::"r"(
                   (unsigned)__cvta_generic_to_shared(p)),
               "r"(rank), "d"(v)
               : "memory");
}
__device__ __forceinline__ void store_cluster3(const double* p, int rank, const double* x) {
  asm volatile(
      "{ .reg .b32 r; mapa.shared::cluster.u32 r, %0, %1; st.shared::cluster.v2.f64 [r], {%2, %3}; "
      "st.shared::cluster.f64 [r+16], %4; }" ::"r"((unsigned)__cvta_generic_to_shared(p)),
      "r"(rank), "d"(x[0]), "d"(x[1]), "d"(x[2])
      : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
#endif

// ResidentReduce for a cluster: the hardware's barrier in place of the counter in global memory, and the chunk sums
// written to every CTA's shared memory. At most 16 CTAs and kClusterChunks chunks (two per stripe), so warp 0 reduces
// alone: lane 8 q + k forms stripe k of quantity q.
constexpr int kClusterChunks = 16;
struct ClusterReduce {
  double* csum;  // 2 x 4 x C doubles of this CTA's shared memory
  const int C;
  double* stripes;
  const int lane, warp, nwarps, parties;
  unsigned phase = 0;
  __device__ double* sums() const { return csum + (size_t)(phase & 1u) * 4 * C; }
  // v: quantity q of chunk c, in every lane
  __device__ void put_total(int q, int c, double v) {
    if (lane < parties) store_cluster(sums() + q * C + c, lane, v);
  }
  // quantity q in lanes 0-15, q + 1 in the others
  __device__ void put_totals(int q, int c, double v) {
    if ((lane & 15) < parties) store_cluster(sums() + (q + (lane >> 4)) * C + c, lane & 15, v);
  }
  __device__ void put(int q, int c, double v) { put_total(q, c, warp_sum_butterfly(v)); }
  // With a NaN among the values the lanes' maxima differ (a sum is NaN in all of them): every CTA gets the first lane's, as
  // the kernels that store it once do. CTAs with different totals would take different branches, and one that ends while
  // another still writes to its shared memory faults the launch.
  __device__ void put_max(int q, int c, double v) { put_total(q, c, __shfl_sync(0xffffffffu, warp_max_butterfly(v), 0)); }
  // The last warp, which has no chunk, prepares the next decision (side) before it arrives: the barrier orders arrivals
  // only, so what it wrote after its own would not be there for warp 0. Nothing in the phase before the barrier reads or
  // writes what side writes, and nothing but the decision before that phase writes what it reads.
  template <class Side>
  __device__ void arrive_and_wait(Side&& side) {
    if (warp == nwarps - 1) side();
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  }
  __device__ bool sync() {
    arrive_and_wait([] {});
    ++phase;
    return true;
  }
  template <class Side, class Decide>
  __device__ bool reduce(int K, unsigned maxmask, Side&& side, Decide&& decide) {
    arrive_and_wait(side);
    if (warp == 0) {
      // stripe k: chunks [k per, (k + 1) per); what a warp's butterfly over the two and zeros gives
      const double* s = sums();
      const int q = lane >> 3, k = lane & 7, per = (C + 7) / 8, b = k * per, e = min(C, b + per);
      const bool mx = (maxmask >> q) & 1u;
      double v = 0.0;
      if (q < K && b < e) {
        const double v0 = s[q * C + b], v1 = b + 1 < e ? s[q * C + b + 1] : 0.0;
        if (mx) {
          const double m0 = v0 < 0.0 ? 0.0 : v0, m1 = v1 < 0.0 ? 0.0 : v1;
          v = m0 < m1 ? m1 : m0;
        } else {
          v = (0.0 + v0) + (0.0 + v1);
        }
      }
      stripes[lane] = v;
      __syncwarp();
      const int t = lane < K ? lane : 0;
      const bool tmx = (maxmask >> t) & 1u;
      double total = stripes[8 * t];
#pragma unroll
      for (int j = 1; j < 8; ++j) {
        const double w = stripes[8 * t + j];
        total = tmx ? ((w < total) ? total : w) : total + w;
      }
      decide(total);
    }
    __syncthreads();
    ++phase;
    return true;
  }
};

}  // namespace bogus_gpu
