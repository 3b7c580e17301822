// The FP32-refined solve of a problem whose FP32 copy of W fits the SMs' shared memory (about 52 000 contacts of 4 per
// body): the FP32 part, and the FP64 iterations with FP32 correction products. One cooperative launch of one CTA per SM,
// every 32-contact chunk owned by one warp for the whole solve.
//
// k_pg_persistent<float> is bound by what surrounds its products: each block's values, columns and row starts are loaded
// again in every pass, x takes three scattered loads, and each of an SM's three CTAs repeats the flat reduction. Here the
// chunk's values and 16-bit columns are copied to shared memory once, the points that products gather are 16 bytes per
// contact (one load each, six steps ahead), and an SM reduces once. FP32 FMAs need no split over warps (4 cycles each).
// The iteration is pg_body_inl's with the products in the canonical chunk-segmented order, so the results are
// identical. us per FP32 iteration on GB300, k_pg_persistent<float> / this kernel (APGD): 300 contacts 30.6 / 18.4, 2000
// 34.4 / 20.7, 10 000 36.1 / 21.6, 30 000 42.8 / 22.7, 50 000 55.6 / 29.9. 100 iterations with correction products at
// 50 000: 6.9 / 4.5 ms. It is faster wherever it fits; what bounds it now is the two barriers and reductions of an
// iteration (about 17 us of it, the time of 40 contacts) and, above 40 000, the chunk's own serial chain.
#include "pg_body.cuh"

namespace bogus_gpu {

namespace {

constexpr int kMaxWarps = 16;      // chunks per CTA
constexpr int kPartBytes = 6 * 64 * 4;
constexpr int kStep32Bytes = 32 * (36 + 2);

// A chunk of the FP32 copy of W in shared memory, owned by one warp.
struct Chunk32 {
  float (*part)[64] = nullptr;   // pieces of the rows by component (slot: rank of the row among the nonempty + lane)
  float* wv = nullptr;           // value e of step s: wv[32 (9 s + e) + lane]
  unsigned short* wc = nullptr;  // column of step s: wc[32 s + lane]
  int lane = 0, S = 0, nv = 0, slot0 = 0, piece0 = 0, pieces = 0;
  unsigned long long starts = 0;  // bit s: the lane's block s opens a row that its block s - 1 does not belong to

  // Copies chunk c of the interleaved FP32 copy (InterleavedBlocks) and finds this lane's segment and row.
  __device__ void load(const int* rowptr, const int* icol, const float* ival, const long long* slots, int n, int c,
                       unsigned char* blocks) {
    const int r0 = 32 * c, r1 = min(r0 + 32, n);
    const int B0 = __ldg(rowptr + r0), nblk = __ldg(rowptr + r1) - B0;
    S = nblk > 0 ? (nblk + 31) / 32 : 1;
    wv = reinterpret_cast<float*>(blocks);
    wc = reinterpret_cast<unsigned short*>(wv + (size_t)S * 32 * 9);
    const long long base = __ldg(slots + c);
    const float4* sv = reinterpret_cast<const float4*>(ival + 9 * base);
    for (int k = lane; k < S * 32 * 9 / 4; k += 32) reinterpret_cast<float4*>(wv)[k] = __ldcs(sv + k);
    const int k0 = lane * S;
    nv = max(0, min(S, nblk - k0));
    for (int s = 0; s < S; ++s)  // past the lane's blocks: a valid column (the lane drops the result)
      wc[32 * s + lane] = (unsigned short)(s < nv ? __ldcs(icol + base + 32 * s + lane) : r0);
    // row starts: row t's in lane t
    const int rs = __ldg(rowptr + min(r0 + lane, r1)) - B0, re = __ldg(rowptr + min(r0 + lane + 1, r1)) - B0;
    const unsigned filled = __ballot_sync(0xffffffffu, rs < re);
    int first = 0;
    for (int t = 0; t < 32; ++t) {
      const int st = __shfl_sync(0xffffffffu, rs, t);
      if (nv > 0 && st <= k0) first = t;  // the last row that starts at or before the segment
      if (nv > 0 && st > k0 && st < k0 + nv) starts |= 1ull << (st - k0);
    }
    slot0 = __popc(filled & ((1u << first) - 1u)) + lane;
    if (rs < re) {
      const int lf = rs / S;
      piece0 = __popc(filled & ((1u << lane) - 1u)) + lf;
      pieces = (re - 1) / S - lf + 1;
    }
    __syncwarp();
  }

  // Row `lane` of the chunk's product with the points g (4 floats per contact); NP = 2: also with g - 1. acc, acc2 are
  // left alone where the row has no block.
  template <int NP>
  __device__ __forceinline__ void product(const float* __restrict__ g, float* acc, float* acc2) const {
    constexpr int D = 6;
    const float4* pt = reinterpret_cast<const float4*>(g);
    int slot = slot0;
    unsigned long long open = starts;
    float p[3] = {0.f, 0.f, 0.f}, q[3] = {0.f, 0.f, 0.f};
    float4 ring[D];
#pragma unroll
    for (int d = 0; d < D; ++d) ring[d] = __ldcg(pt + wc[32 * min(d, S - 1) + lane]);
    auto step = [&](int s, const float4& x) {
      const bool starts_row = open & 1ull;
      open >>= 1;
      if (starts_row) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          part[r][slot] = p[r];
          p[r] = 0.f;
          if (NP == 2) {
            part[3 + r][slot] = q[r];
            q[r] = 0.f;
          }
        }
        ++slot;
      }
      const float* b = wv + 288 * s + lane;
      const bool valid = s < nv;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const float b0 = b[32 * (3 * r)], b1 = b[32 * (3 * r + 1)], b2 = b[32 * (3 * r + 2)];
        const float pn = fmaf(b2, x.z, fmaf(b1, x.y, fmaf(b0, x.x, p[r])));
        p[r] = valid ? pn : p[r];
        if (NP == 2) {
          const float qn = fmaf(b2, x.z - 1.f, fmaf(b1, x.y - 1.f, fmaf(b0, x.x - 1.f, q[r])));
          q[r] = valid ? qn : q[r];
        }
      }
    };
    int s = 0;
    for (; s + D <= S; s += D) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const float4 x = ring[d];
        ring[d] = __ldcg(pt + wc[32 * min(s + d + D, S - 1) + lane]);
        step(s + d, x);
      }
    }
#pragma unroll
    for (int d = 0; d < D - 1; ++d)
      if (s + d < S) step(s + d, ring[d]);
    if (nv > 0) {
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        part[r][slot] = p[r];
        if (NP == 2) part[3 + r][slot] = q[r];
      }
    }
    __syncwarp();
    if (pieces > 0) {
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        float v = zero_plus(part[r][piece0]);
        for (int k = 1; k < pieces; ++k) v = v + part[r][piece0 + k];
        acc[r] = v;
        if (NP == 2) {
          float w = zero_plus(part[3 + r][piece0]);
          for (int k = 1; k < pieces; ++k) w = w + part[3 + r][piece0 + k];
          acc2[r] = w;
        }
      }
    }
    __syncwarp();
  }
};

// One warp per chunk, phases separated by the flat barrier.
template <class T>
struct Resident32Ctx {
  const PGArgsT<T>& a;
  double* smem32;
  double* sscal;
  ChunkScratchT<T>* cs;  // FP64 products of HY (guess, refreshes): per-warp scratch in global memory
  Chunk32 chunk32;
  int own;  // this warp's chunk (nchunks: none)
  unsigned phase = 0;
  __device__ int first_chunk() const { return own; }
  __device__ int next_chunk(int) const { return a.nchunks; }
  __device__ bool writer() const { return blockIdx.x == 0 && threadIdx.x == 0; }
  __device__ double* csum() const { return a.csum + (size_t)(phase & 1u) * 4 * a.nchunks; }
  __device__ MonoBarrier mb() const { return MonoBarrier{a.mono, a.gb.status, gridDim.x + a.phantom_ctas}; }
  __device__ bool sync() {
    const bool ok = flat_barrier(mb(), phase);
    ++phase;
    return ok;
  }
  __device__ bool sync_reduce(int K, unsigned maxmask) {
    if (!flat_barrier(mb(), phase)) return false;
    flat_combine(csum(), (size_t)a.nchunks, a.nchunks, a.nchunks, K, maxmask, smem32, sscal);
    ++phase;
    return true;
  }
  __device__ bool sync_reduce_split(int K, unsigned maxmask) { return sync_reduce(K, maxmask); }
  __device__ bool await_scalars() const { return true; }
  __device__ double scal(int q) const { return sscal[q]; }
};

template <class T, bool HY>
__global__ void __launch_bounds__(32 * kMaxWarps, 1) k_pg_resident32(PGArgsT<T> a, ChunkScratchT<T>* scratch) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double smem32[32], sscal[4];
  const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int first = __ldg(a.cta_ptr + blockIdx.x), count = __ldg(a.cta_ptr + blockIdx.x + 1) - first;
  Resident32Ctx<T> ctx{a, smem32, sscal, scratch + (size_t)blockIdx.x * nwarps, Chunk32{}, a.nchunks};
  if (warp < count) {
    ctx.own = __ldg(a.cta_list + first + warp);
    size_t before = 0;
    for (int k = 0; k < warp; ++k) {
      const int c = __ldg(a.cta_list + first + k);
      const int nblk = __ldg(a.rowptr + min(32 * c + 32, a.n)) - __ldg(a.rowptr + 32 * c);
      before += nblk > 0 ? (nblk + 31) / 32 : 1;
    }
    ctx.chunk32.lane = threadIdx.x & 31;
    ctx.chunk32.part = reinterpret_cast<float(*)[64]>(smem + (size_t)warp * kPartBytes);
    const float* values;
    if constexpr (HY) values = a.hy_ival;
    else values = a.ival;
    ctx.chunk32.load(a.rowptr, a.icol, values, a.slot0, a.n, ctx.own,
                     smem + (size_t)nwarps * kPartBytes + before * kStep32Bytes);
  }
  pg_body_inl<T, true, false, HY, true>(a, ctx);
}

int warps_of(int chunks) { return chunks > 8 ? chunks : 8; }
size_t resident32_smem(int chunks, int steps) {
  return (size_t)warps_of(chunks) * kPartBytes + (size_t)steps * kStep32Bytes;
}

template <class T, bool HY>
cudaError_t launch32(const PGArgsT<T>& a, int ctas, int chunks, int steps, ChunkScratchT<T>* scratch, cudaStream_t s) {
  const size_t bytes = resident32_smem(chunks, steps);
  const void* fn = (const void*)k_pg_resident32<T, HY>;
  const cudaError_t e = allow_resident_shared(fn);
  if (e != cudaSuccess) return e;
  PGArgsT<T> copy = a;
  void* args[] = {&copy, &scratch};
  return cudaLaunchCooperativeKernel(fn, dim3(ctas), dim3(32 * warps_of(chunks)), args, bytes, s);
}

// Positions between 3 doubles and 4 floats per contact.
__global__ void k_pad_positions(int n, const double* __restrict__ src, float4* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = make_float4((float)src[3 * (size_t)i], (float)src[3 * (size_t)i + 1], (float)src[3 * (size_t)i + 2], 0.f);
}
__global__ void k_unpad_positions(int n, const float4* __restrict__ src, double* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 v = src[i];
  dst[3 * (size_t)i] = v.x;
  dst[3 * (size_t)i + 1] = v.y;
  dst[3 * (size_t)i + 2] = v.z;
}

}  // namespace

bool pg_resident32_fits(int device, int chunks, int steps, int longest, int n) {
  return chunks >= 1 && chunks <= kMaxWarps && longest <= 64 && n <= 65536 &&
         resident32_smem(chunks, steps) <= resident_shared_limit(device);
}

size_t pg_resident32_scratch(int ctas, int chunks) { return sizeof(ChunkScratch) * (size_t)ctas * warps_of(chunks); }

cudaError_t launch_pg_resident32(const PGArgs32& a, int ctas, int chunks, int steps, cudaStream_t s) {
  return launch32<float, false>(a, ctas, chunks, steps, nullptr, s);
}

cudaError_t launch_pg_resident32(const PGArgs& a, int ctas, int chunks, int steps, void* scratch, cudaStream_t s) {
  if (!a.hy_refresh || a.variant != 3 || a.lin_momentum || !a.slot0 || !a.hy_ival || !a.hy_d || !a.hy_xref || !a.hy_wxref)
    return cudaErrorInvalidValue;
  return launch32<double, true>(a, ctas, chunks, steps, static_cast<ChunkScratch*>(scratch), s);
}

cudaError_t launch_pad_positions(int n, const double* src, float* dst, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_pad_positions<<<(n + 255) / 256, 256, 0, s>>>(n, src, reinterpret_cast<float4*>(dst));
  return cudaGetLastError();
}
cudaError_t launch_unpad_positions(int n, const float* src, double* dst, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_unpad_positions<<<(n + 255) / 256, 256, 0, s>>>(n, reinterpret_cast<const float4*>(src), dst);
  return cudaGetLastError();
}

// Sets this file's copy of the device-side wait limit on the current device.
BOGUS_GPU_WAIT_LIMIT_SETTER(set_wait_limit_pg_resident32)

}  // namespace bogus_gpu
