// Persistent projected-gradient solvers: the whole solve of PgMethod<APGD / Descent / SPG>
// (Core/BlockSolvers/ProjectedGradient.impl.hpp:74-155, 288-351) runs in one cooperative launch.
//
// Work split: warp w of the grid owns the 32-contact chunks w, w + W, w + 2W, ... in every phase, lane l
// contact 32c + l. A phase is one pass over the contacts (row-local vector work) or over W (SpMV with the
// row-local work fused into its epilogue). Global dot products are reduced in the canonical order: a
// butterfly per chunk inside the warp, then the 8-stripe combination. Up to kFlatChunks chunks every CTA runs it
// itself once all have arrived (flat_barrier, flat_combine); beyond, the last CTAs to reach the barrier take a stripe
// each and the last of those publishes the scalars (mono_barrier_combine). Either way every CTA takes the same
// line-search / momentum decisions on identical values. Waits are bounded, so a fault elsewhere ends the kernel
// with BOGUS_GPU_TIMEOUT instead of a hang.
//
// Phases of one APGD iteration (reference line numbers in ProjectedGradient.impl.hpp):
//   A   y = Mx + b, residual (:110-111), s = COV(y), y += s, J (:113-115), xs = P(x - a y) (:123-125)
//   C   Mxs = W xs; Js, y.(xs-x), |xs-x|^2 (:127-132), (xs-prev).y (:135); APGD also writes the
//       momentum point x = xs + beta (xs - prev) (:137-139) to a spare buffer ........... barrier+reduce
//   B   line-search retry: xs = P(x - a y) ............................................ barrier
//   E+A Mx = W x (:141) fused with A of the next iteration ............................. barrier+reduce
// With momentum, the spare buffer becomes x (a buffer swap); without, x = xs and Mx = Mxs are swaps and A
// runs as its own pass. Phase counter 5 (a separate momentum pass) is no longer used.
#include "pg_body.cuh"

namespace bogus_gpu {

// Single problem: the whole GPU, phases separated by bounded grid barriers on monotonic counters
// (mono_barrier); at a reducing barrier the last CTAs to arrive combine the chunk sums, one stripe each, and
// the last of them publishes the scalars in global memory. After a split reduction the CTAs go on once every
// CTA has arrived, and each warp waits for the publication only where it reads the scalars. Each CTA takes
// its 32-contact chunks from its own list (cta_ptr / cta_list: the chunks dealt largest first to the CTAs in
// serpentine rounds, so every SM's total is the same to within about one chunk), its warps sharing the list
// through a shared-memory counter per phase parity; without lists (the allocation-free entry point) warps
// take chunks from a global ticket counter per phase parity, cleared by the last CTA of the barrier that ends
// the phase, in largest-first order (chunk_order). Every cross-phase dependency goes through a barrier, and
// the reduction order does not depend on which warp handles a chunk.
template <class T>
struct GridCtx {
  const PGArgsT<T>& a;
  double* smem8;
  double* sscal;       // the scalars of the last flat reduction
  ChunkScratchT<T>* cs;
  unsigned* s_cnt;     // 2 shared-memory counters (phase parity) over the CTA's chunk list
  unsigned phase = 0;  // barriers passed (identical in every CTA)
  __device__ int ticket() {
    int c = 0;
    if ((threadIdx.x & 31) == 0) {
      if (a.cta_ptr) {
        const int k = (int)atomicAdd(s_cnt + (phase & 1u), 1u);
        const int b0 = __ldg(a.cta_ptr + blockIdx.x), b1 = __ldg(a.cta_ptr + blockIdx.x + 1);
        c = b0 + k < b1 ? __ldg(a.cta_list + b0 + k) : a.nchunks;
      } else {
        c = (int)atomicAdd(a.tickets + (phase & 1u), 1u);
        if (a.chunk_order) c = c < a.nchunks ? __ldg(a.chunk_order + c) : a.nchunks;
      }
    }
    return __shfl_sync(0xffffffffu, c, 0);
  }
  // after a barrier (every warp of the CTA is past its draws of this phase): the counter of this phase's
  // parity is free for the phase after next
  __device__ void reset_cta_counter() {
    if (a.cta_ptr && threadIdx.x == 0) s_cnt[phase & 1u] = 0u;
  }
  __device__ int first_chunk() { return ticket(); }
  __device__ int next_chunk(int) { return ticket(); }
  __device__ bool writer() const { return blockIdx.x == 0 && threadIdx.x == 0; }
  __device__ void clear_tickets() {
    if (threadIdx.x == 0) a.tickets[phase & 1u] = 0u;
  }
  unsigned reductions = 0;  // reductions published or pending (identical in every CTA)
  bool pending = false;     // this warp has not yet waited for the last (split) reduction
  __device__ double* csum() const { return a.csum + (a.flat ? (size_t)(phase & 1u) * 4 * a.nchunks : 0); }
  __device__ MonoBarrier mb() const { return MonoBarrier{a.mono, a.gb.status, gridDim.x + a.phantom_ctas}; }
  __device__ bool sync() {
    const bool ok = a.flat ? flat_barrier(mb(), phase) : mono_barrier(mb(), phase, [&] { clear_tickets(); });
    reset_cta_counter();
    ++phase;
    return ok;
  }
  __device__ bool reduce(int K, unsigned maxmask, bool split) {
    if (a.flat) {
      if (!flat_barrier(mb(), phase)) return false;
      flat_combine(csum(), (size_t)a.nchunks, a.nchunks, a.nchunks, K, maxmask, smem8, sscal);
      reset_cta_counter();
      ++phase;
      return true;
    }
    const bool ok = mono_barrier_combine(mb(), phase, reductions, split, a.csum, (size_t)a.nchunks, a.nchunks,
                                         a.nchunks, K, maxmask, a.stripes, a.scal, [&] { clear_tickets(); });
    reset_cta_counter();
    ++phase;
    ++reductions;
    pending = split;
    return ok;
  }
  __device__ bool sync_reduce(int K, unsigned maxmask) { return reduce(K, maxmask, false); }
  __device__ bool sync_reduce_split(int K, unsigned maxmask) { return reduce(K, maxmask, true); }
  __device__ bool await_scalars() {
    if (!pending) return true;
    pending = false;
    return mono_await(mb(), reductions);
  }
  __device__ double scal(int q) const { return a.flat ? sscal[q] : ldcg(a.scal + q); }
};

// The solver body; the hybrid instantiation is inlined by force (the compiler's own choice outlines it, with
// 500-odd bytes of spills), the others as the compiler decides.
template <class T, bool IL, bool SC = false, bool HY = false, class Ctx>
__device__ int pg_body(const PGArgsT<T>& a, Ctx& ctx) {
  return pg_body_inl<T, IL, SC, HY>(a, ctx);
}

// Occupancy target: 3 resident CTAs per SM (see pg_max_grid). FEW (FP64, at most 2 CTAs per SM launched, a chunk or less
// per warp): the registers of the third CTA hold the next two blocks and points instead, since a warp's own latency
// counts there. us per APGD iteration on GB300 without / with (before the reductions' loads came together, which took
// 38 000 to 65.9): 26 000 contacts 69.7 / 58.7, 38 000 80.4 / 70.6, 50 000 85.7 / 78.0, 77 000 98.2 / 92.3.
template <class T, bool IL, bool SC = false, bool HY = false, bool FEW = false>
__global__ void __launch_bounds__(256, FEW ? 2 : 3) k_pg_persistent(PGArgsT<T> a) {
  __shared__ double smem8[32], sscal[4];
  __shared__ ChunkScratchT<T> cs[8];
  __shared__ unsigned s_cnt[2];
  if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0u;
  __syncthreads();
  GridCtx<T> ctx{a, smem8, sscal, cs, s_cnt};
  pg_body_inl<T, IL, SC, HY, false, FEW>(a, ctx);
}

// One problem per CTA (batched solves): phases separated by __syncthreads, scalars reduced by the CTA's
// 8 warps (the same 8-stripe combination) and kept in shared memory.
template <class T>
struct BlockCtx {
  const PGArgsT<T>& a;
  double* smem8;
  double* sscal;
  ChunkScratchT<T>* cs;
  __device__ int first_chunk() const { return threadIdx.x >> 5; }
  __device__ int next_chunk(int c) const { return c + 8; }
  __device__ bool writer() const { return threadIdx.x == 0; }
  __device__ double* csum() const { return a.csum; }
  __device__ bool sync() {
    __syncthreads();
    return true;
  }
  __device__ bool sync_reduce(int K, unsigned maxmask) {
    __syncthreads();
    block8_combine_k(a.csum, a.nchunks, K, maxmask, smem8, sscal);
    return true;
  }
  __device__ bool sync_reduce_split(int K, unsigned maxmask) { return sync_reduce(K, maxmask); }
  __device__ bool await_scalars() const { return true; }
  __device__ double scal(int q) const { return sscal[q]; }
};

// Batched solves: CTAs take problems from a queue (largest first); each runs the complete solve of its
// problem with the same arithmetic as the single-problem kernel, then writes the best iterate to r.
template <class T, bool HY = false>
__global__ void __launch_bounds__(256) k_pg_batched(PGBatchArgsT<T> ba) {
  __shared__ double smem8[32], sscal[8];
  __shared__ ChunkScratchT<T> cs[8];
  __shared__ int s_job;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_job = atomicAdd(ba.next, 1);
    __syncthreads();
    const int job = s_job;
    if (job >= ba.nproblems) return;
    const int p = ba.queue[job];
    const int c0 = ba.contact_ptr[p];
    const int n = ba.contact_ptr[p + 1] - c0;
    PGArgsT<T> a = ba.base;
    a.n = n;
    a.nchunks = (n + 31) / 32;
    a.rowptr = ba.base.rowptr + c0;
    a.b = ba.base.b + 3 * (size_t)c0;
    a.mu = ba.base.mu + c0;
    a.scaling = ba.base.scaling + c0;
    a.X0 = ba.base.X0 + 3 * (size_t)c0;
    a.X1 = ba.base.X1 + 3 * (size_t)c0;
    a.X2 = ba.base.X2 + 3 * (size_t)c0;
    a.MX0 = ba.base.MX0 + 3 * (size_t)c0;
    a.MX1 = ba.base.MX1 + 3 * (size_t)c0;
    if (ba.base.lin_momentum) {
      a.MX2 = ba.base.MX2 + 3 * (size_t)c0;
      a.MX3 = ba.base.MX3 + 3 * (size_t)c0;
    }
    a.Y = ba.base.Y + 3 * (size_t)c0;
    a.S0 = ba.base.S0 + c0;
    a.XB = ba.base.XB + 3 * (size_t)c0;
    a.Wv = ba.base.Wv + 3 * (size_t)c0;
    a.csum = ba.base.csum + 4 * (size_t)ba.chunk_ptr[p];
    a.trace = nullptr;
    a.out = ba.base.out + p;
    if constexpr (HY) {
      a.hy_d = ba.base.hy_d + 3 * (size_t)c0;
      a.hy_xref = ba.base.hy_xref + 3 * (size_t)c0;
      a.hy_wxref = ba.base.hy_wxref + 3 * (size_t)c0;
    }
    BlockCtx<T> ctx{a, smem8, sscal, cs};
    int best;
    if constexpr (HY) {
      best = pg_body_inl<T, false, false, true>(a, ctx);
    } else {
      best = pg_body<T, false>(a, ctx);
    }
    __syncthreads();
    if (n == 0) continue;
    const T* src = best == 3 ? a.XB : (best == 4 ? a.Wv : (best == 0 ? a.X0 : (best == 1 ? a.X1 : a.X2)));
    T* dst = ba.r + 3 * (size_t)c0;
    for (int k = threadIdx.x; k < 3 * n; k += blockDim.x) dst[k] = ldcg(src + k);
  }
}

// Team schedule: CTAs [team * size, team * size + size) solve one problem at a time with the single-problem
// context (dynamic chunk tickets, bounded barrier, chunk sums combined by the team's last CTAs to arrive
// (grid_barrier_combine), scalars published in the team's slot), on counters of their own. The last CTA to reach the barrier before a job takes the next problem from the queue. The
// arithmetic is that of the other schedules, so each problem's result is the same bit for bit.
template <class T>
struct TeamCtx {
  const PGArgsT<T>& a;
  double* smem8;
  ChunkScratchT<T>* cs;
  unsigned* tickets;        // 2
  unsigned* combine_count;  // 1
  double* sc;               // 8 scalars, then 32 stripe sums
  GridBarrier gb;
  int rank;
  unsigned phase = 0;
  __device__ int ticket() {
    int c = 0;
    if ((threadIdx.x & 31) == 0) c = (int)atomicAdd(tickets + (phase & 1u), 1u);
    return __shfl_sync(0xffffffffu, c, 0);
  }
  __device__ int first_chunk() { return ticket(); }
  __device__ int next_chunk(int) { return ticket(); }
  __device__ bool writer() const { return rank == 0 && threadIdx.x == 0; }
  __device__ double* csum() const { return a.csum; }
  __device__ void clear_tickets() {
    if (threadIdx.x == 0) tickets[phase & 1u] = 0u;
  }
  __device__ bool sync() {
    const bool ok = grid_barrier(gb, [&] { clear_tickets(); });
    ++phase;
    return ok;
  }
  __device__ bool sync_reduce(int K, unsigned maxmask) {
    const bool ok = grid_barrier_combine(gb, combine_count, a.csum, (size_t)a.nchunks, a.nchunks, a.nchunks, K, maxmask,
                                         sc + 8, sc, [&] { clear_tickets(); });
    ++phase;
    return ok;
  }
  __device__ bool sync_reduce_split(int K, unsigned maxmask) { return sync_reduce(K, maxmask); }
  __device__ bool await_scalars() const { return true; }
  __device__ double scal(int q) const { return ldcg(sc + q); }
};

template <class T, bool HY = false>
__global__ void __launch_bounds__(256, 3) k_pg_team(PGBatchArgsT<T> ba, PGTeamArgs ta) {
  __shared__ double smem8[32];
  __shared__ ChunkScratchT<T> cs[8];
  const int team = blockIdx.x / ta.size, rank = blockIdx.x - team * ta.size;
  unsigned* cnt = ta.counters + 8 * (size_t)team;
  const GridBarrier gb{cnt, cnt + 1, ta.status, (unsigned)ta.size};
  for (;;) {
    // the last CTA to arrive takes the next problem and clears the team's chunk tickets: the final phase of the
    // previous problem (a converged solve leaves its last product phase without a closing barrier) may have
    // drawn tickets that no barrier cleared
    if (!grid_barrier(gb, [&] {
          if (threadIdx.x == 0) {
            ta.job[team] = (int)atomicAdd((unsigned*)ba.next, 1u);
            cnt[2] = 0u;
            cnt[3] = 0u;
          }
        }))
      return;
    const int job = *(volatile int*)(ta.job + team);
    if (job >= ba.nproblems) return;
    const int p = ba.queue[job];
    const int c0 = ba.contact_ptr[p];
    const int n = ba.contact_ptr[p + 1] - c0;
    PGArgsT<T> a = ba.base;
    a.n = n;
    a.nchunks = (n + 31) / 32;
    a.rowptr = ba.base.rowptr + c0;
    a.b = ba.base.b + 3 * (size_t)c0;
    a.mu = ba.base.mu + c0;
    a.scaling = ba.base.scaling + c0;
    a.X0 = ba.base.X0 + 3 * (size_t)c0;
    a.X1 = ba.base.X1 + 3 * (size_t)c0;
    a.X2 = ba.base.X2 + 3 * (size_t)c0;
    a.MX0 = ba.base.MX0 + 3 * (size_t)c0;
    a.MX1 = ba.base.MX1 + 3 * (size_t)c0;
    if (ba.base.lin_momentum) {
      a.MX2 = ba.base.MX2 + 3 * (size_t)c0;
      a.MX3 = ba.base.MX3 + 3 * (size_t)c0;
    }
    a.Y = ba.base.Y + 3 * (size_t)c0;
    a.S0 = ba.base.S0 + c0;
    a.XB = ba.base.XB + 3 * (size_t)c0;
    a.Wv = ba.base.Wv + 3 * (size_t)c0;
    a.csum = ba.base.csum + 4 * (size_t)ba.chunk_ptr[p];
    a.trace = nullptr;
    a.out = ba.base.out + p;
    if constexpr (HY) {
      a.hy_d = ba.base.hy_d + 3 * (size_t)c0;
      a.hy_xref = ba.base.hy_xref + 3 * (size_t)c0;
      a.hy_wxref = ba.base.hy_wxref + 3 * (size_t)c0;
    }
    TeamCtx<T> ctx{a, smem8, cs, cnt + 2, cnt + 4, ta.scal + 40 * (size_t)team, gb, rank};
    int best;
    if constexpr (HY) {
      best = pg_body_inl<T, false, false, true>(a, ctx);
    } else {
      best = pg_body<T, false>(a, ctx);
    }
    if (best < 0) return;  // a wait ran out (status recorded)
    if (n == 0) continue;
    const T* src = best == 3 ? a.XB : (best == 4 ? a.Wv : (best == 0 ? a.X0 : (best == 1 ? a.X1 : a.X2)));
    T* dst = ba.r + 3 * (size_t)c0;
    for (int k = rank * (int)blockDim.x + (int)threadIdx.x; k < 3 * n; k += ta.size * (int)blockDim.x)
      dst[k] = ldcg(src + k);
  }
}

// Resident 256-thread CTAs per SM that both kernels reach (the FP64 batched kernels and their instantiations with
// FP32 correction products share launch shapes).
template <class K1, class K2>
cudaError_t occupancy_min(int* per, K1 k1, K2 k2) {
  int a = 0, b = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k1, 256, 0);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k2, 256, 0);
  *per = a < b ? a : b;
  return e;
}

template <class T>
cudaError_t launch_team_t(const PGBatchArgsT<T>& b, const PGTeamArgs& t, int grid, cudaStream_t s) {
  PGBatchArgsT<T> bc = b;
  PGTeamArgs tc = t;
  void* args[] = {&bc, &tc};
  const void* fn = (const void*)k_pg_team<T>;
  if constexpr (sizeof(T) == 8) {
    if (b.base.hy_refresh) {
      if (b.base.variant != 3 || b.base.lin_momentum || !b.base.hy_ival || !b.base.hy_d || !b.base.hy_xref ||
          !b.base.hy_wxref)
        return cudaErrorInvalidValue;
      fn = (const void*)k_pg_team<T, true>;
    }
  }
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(256), args, 0, s);
}

cudaError_t launch_pg_team(const PGBatchArgs& b, const PGTeamArgs& t, int grid, cudaStream_t s) {
  return launch_team_t(b, t, grid, s);
}

cudaError_t launch_pg_team(const PGBatchArgs32& b, const PGTeamArgs& t, int grid, cudaStream_t s) {
  return launch_team_t(b, t, grid, s);
}

int pg_team_per_sm(int device, bool fp32) {
  int per = 0;
  (void)device;
  const cudaError_t e = fp32 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pg_team<float>, 256, 0)
                             : occupancy_min(&per, k_pg_team<double>, k_pg_team<double, true>);
  return e == cudaSuccess ? per : 0;
}

int pg_batched_per_sm(int device, bool fp32) {
  int per = 0;
  (void)device;
  const cudaError_t e = fp32 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pg_batched<float>, 256, 0)
                             : occupancy_min(&per, k_pg_batched<double>, k_pg_batched<double, true>);
  return e == cudaSuccess ? per : 0;
}

int pg_team_grid(int device, bool fp32) {
  int sms = 0, per = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  const cudaError_t e = fp32 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pg_team<float>, 256, 0)
                             : occupancy_min(&per, k_pg_team<double>, k_pg_team<double, true>);
  if (e != cudaSuccess) return 0;
  const int cap = 3;
  if (per > cap) per = cap;
  return per * sms;
}

cudaError_t launch_pg_batched(const PGBatchArgs& b, int grid, cudaStream_t s) {
  if (b.base.hy_refresh) {
    if (b.base.variant != 3 || b.base.lin_momentum || !b.base.hy_ival || !b.base.hy_d || !b.base.hy_xref ||
        !b.base.hy_wxref)
      return cudaErrorInvalidValue;
    k_pg_batched<double, true><<<grid, 256, 0, s>>>(b);
  } else {
    k_pg_batched<double><<<grid, 256, 0, s>>>(b);
  }
  return cudaGetLastError();
}

cudaError_t launch_pg_batched(const PGBatchArgs32& b, int grid, cudaStream_t s) {
  k_pg_batched<float><<<grid, 256, 0, s>>>(b);
  return cudaGetLastError();
}

int pg_batched_grid(int device, bool fp32) {
  int sms = 0, per = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  const cudaError_t e = fp32 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pg_batched<float>, 256, 0)
                             : occupancy_min(&per, k_pg_batched<double>, k_pg_batched<double, true>);
  if (e != cudaSuccess) return 0;
  return per * sms;
}

cudaError_t launch_pg_persistent(const PGArgs& a, int grid, cudaStream_t s) {
  PGArgs copy = a;
  void* args[] = {&copy};
  const bool sc = a.variant == 0 || a.variant == 2;  // Standard, Conjugated
  const bool hy = a.hy_refresh != 0;                 // FP32 correction products (APGD)
  if ((sc || hy) && !a.slot0) return cudaErrorInvalidValue;  // they run on the interleaved copy only
  if (hy && (a.variant != 3 || a.lin_momentum || !a.hy_ival || !a.hy_d || !a.hy_xref || !a.hy_wxref))
    return cudaErrorInvalidValue;
  int device = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  const bool few = a.slot0 && grid <= 2 * sms;
  const void* fn = sc ? (const void*)k_pg_persistent<double, true, true>
                      : (hy ? (const void*)k_pg_persistent<double, true, false, true>
                            : few ? (const void*)k_pg_persistent<double, true, false, false, true>
                                  : (a.slot0 ? (const void*)k_pg_persistent<double, true>
                                             : (const void*)k_pg_persistent<double, false>));
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(256), args, 0, s);
}

cudaError_t launch_pg_persistent(const PGArgs32& a, int grid, cudaStream_t s) {
  if (!a.slot0) return cudaErrorInvalidValue;  // the FP32 solve reads the interleaved copy only
  PGArgs32 copy = a;
  void* args[] = {&copy};
  return cudaLaunchCooperativeKernel((const void*)k_pg_persistent<float, true>, dim3(grid), dim3(256), args, 0, s);
}

int pg_max_grid(int device, bool fp32, bool interleaved) {
  int sms = 0, per = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  const void* fn = fp32 ? (const void*)k_pg_persistent<float, true>
                        : (interleaved ? (const void*)k_pg_persistent<double, true>
                                       : (const void*)k_pg_persistent<double, false>);
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, 256, 0);
  if (e != cudaSuccess) return 0;
  // Measured on the 200 000-contact problem: 3 resident CTAs per SM for FP64 (0.388 ms per APGD iteration
  // against 0.411 with 2 and 0.502 with 1; later 0.215 ms against 0.249 with 4 CTAs at 64 registers). FP32:
  // 3 CTAs at 80 registers with the block values and x loaded two blocks ahead, 0.120 ms per iteration, against
  // 0.126 at 4 CTAs (64 registers, one block ahead), 0.137 at 4 CTAs with only x ahead, 0.141 with 5 at 48
  // registers and 0.232 with 2.
  const int cap = 3;
  if (per > cap) per = cap;
  return per * sms;
}

// Sets this file's copy of the device-side wait limit on the current device.
BOGUS_GPU_WAIT_LIMIT_SETTER(set_wait_limit_pg)

}  // namespace bogus_gpu
