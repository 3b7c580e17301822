// A 32-contact chunk of W owned by a team of three warps of one SM for the whole of a kernel: its blocks in shared
// memory, and the product with a gathered point in the canonical chunk-segmented order (spmv_chunk.cuh).
//
// Warp r of the team accumulates component r of every row (3 FMAs per block in place of 9: the FP64 unit's latency is
// 64 cycles whatever the lanes), and gathers every third point for all three (a gather of 32 scattered contacts holds
// the load unit for as long as a step's FMAs take). Points are 32 bytes per contact, one 256-bit load each, issued two
// groups of three steps ahead of their FMAs. A product of a 2 000-contact chunk (20 steps) takes 8 600 cycles on
// GB300: 4 000 in the chain of FMAs, 2 600 from the first column to the first FMA and from the last to the exchanged
// result, the rest in shared-memory loads and the team's barriers.
#pragma once

#include "device_common.cuh"
#include "fp64_int.cuh"

namespace bogus_gpu {

constexpr int kTeamWarps = 3;
constexpr int kMaxTeams = 5;
constexpr int kMinWarps = 8;  // a stripe of the reductions each; those past the teams' warps do nothing else

// Shared memory of one team, beside its chunk's blocks.
struct TeamCore {
  // pieces of the rows, by component (slot: rank of the row among the nonempty + lane), then the product itself
  double part[kTeamWarps][64];
  double stage[2][3][3][32];  // the gathered points of two groups of three steps
  int st[36];                 // row starts of the chunk, relative to its first block
};
constexpr int kStepBytes = 32 * (72 + 2);  // block values and 16-bit columns of a step

__device__ __forceinline__ void team_sync(int team) {
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(32 * kTeamWarps) : "memory");
}

// A gathered point: 32 bytes per contact, the fourth value unused.
__device__ __forceinline__ void load_padded(const double* p, double* x) {
  double pad;
  asm volatile("ld.relaxed.gpu.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(pad)
               : "l"(p));
}
__device__ __forceinline__ void store_padded(double* p, const double* x) {
  __stcg(reinterpret_cast<double2*>(p), make_double2(x[0], x[1]));
  __stcg(p + 2, x[2]);
}

// S of chunk c (spmv_chunk.cuh)
__device__ __forceinline__ int steps_of(const int* rowptr, int n, int c) {
  const int nblk = __ldg(rowptr + min(32 * c + 32, n)) - __ldg(rowptr + 32 * c);
  return nblk > 0 ? (nblk + 31) / 32 : 1;
}

struct ResidentChunk {
  TeamCore& sh;
  const int lane, role, team;
  double* wv = nullptr;          // value e of step s: wv[32 (9 s + e) + lane]
  unsigned short* wc = nullptr;  // column of step s: wc[32 s + lane]
  int S = 0, nv = 0, slot0 = 0, piece0 = 0, pieces = 0;
  unsigned long long starts = 0;  // bit s: the lane's block s opens a row that its block s - 1 does not belong to

  // Copies the blocks of chunk c of a BSR matrix of n <= 65536 rows (at most 64 steps) to `blocks` and finds this lane's
  // segment and row.
  __device__ void load(const int* rowptr, const int* col, const double* val, int n, int c, unsigned char* blocks) {
    const int r0 = 32 * c, r1 = min(r0 + 32, n);
    const int B0 = __ldg(rowptr + r0);
    const int nblk = __ldg(rowptr + r1) - B0;
    S = nblk > 0 ? (nblk + 31) / 32 : 1;
    wv = reinterpret_cast<double*>(blocks);
    wc = reinterpret_cast<unsigned short*>(wv + (size_t)S * 32 * 9);
    if (role == 0) {
      sh.st[lane] = __ldg(rowptr + min(r0 + lane, r1)) - B0;
      if (lane == 0) sh.st[32] = nblk;
    }
    const int tid = 32 * role + lane;
    // block k is met by lane k / S at step k % S; the padding past the last block gets a valid column (its lane
    // drops the result)
    for (int k = tid; k < nblk * 9; k += 32 * kTeamWarps) {
      const int b = k / 9, e = k - 9 * b, l = b / S;
      wv[32 * (9 * (b - l * S) + e) + l] = __ldcs(val + 9 * (size_t)B0 + k);
    }
    for (int k = nblk * 9 + tid; k < S * 32 * 9; k += 32 * kTeamWarps) {
      const int b = k / 9, e = k - 9 * b, l = b / S;
      wv[32 * (9 * (b - l * S) + e) + l] = 0.0;
    }
    for (int k = tid; k < S * 32; k += 32 * kTeamWarps) {
      const int l = k / S;
      wc[32 * (k - l * S) + l] = (unsigned short)(k < nblk ? __ldcs(col + B0 + k) : r0);
    }
    team_sync(team);
    const int k0 = lane * S;
    nv = max(0, min(S, nblk - k0));
    const int rs = sh.st[lane], re = sh.st[lane + 1];
    const unsigned filled = __ballot_sync(0xffffffffu, rs < re);
    auto rank = [&](int t) { return __popc(filled & ((1u << t) - 1u)); };
    if (nv > 0) {
      int lo = 0, hi = 31;  // row containing block k0: last t with st[t] <= k0
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sh.st[mid] <= k0) lo = mid;
        else hi = mid - 1;
      }
      slot0 = rank(lo) + lane;
      for (int t = lo + 1; t < 32 && sh.st[t] < k0 + nv; ++t)
        if (sh.st[t] > k0) starts |= 1ull << (sh.st[t] - k0);
    }
    if (rs < re) {
      const int lf = rs / S;
      piece0 = rank(lane) + lf;
      pieces = (re - 1) / S - lf + 1;
    }
  }

  // group k: steps 3 k .. 3 k + 2, this warp's gather the step 3 k + role (past the end: any contact)
  __device__ __forceinline__ const double* point(const double* g, int k) const {
    return g + 4 * (size_t)wc[32 * min(3 * k + role, S - 1) + lane];
  }
  __device__ __forceinline__ void put_stage(int k, const double* x) {
#pragma unroll
    for (int e = 0; e < 3; ++e) sh.stage[k & 1][role][e][lane] = x[e];
  }

  // The chunk's product with the gathered point g: component r of row `lane` in sh.part[r][lane] for every warp of the
  // team. NP = 2: also the product with g - 1, in part2 (3 x 64 doubles). A lane past its segment runs the FMAs on
  // the padding and keeps its sum, so a step has no divergence.
  template <int NP>
  __device__ __forceinline__ void product(const double* __restrict__ g, double* part2_all = nullptr) {
    double* part2 = part2_all + 64 * role;
    int slot = slot0;
    double p = 0.0, q = 0.0;
    const double* bl = wv + 32 * 3 * role + lane;
    unsigned long long open = starts;
    auto step = [&](int s, const double* b, const double* x) {
      const bool starts_row = open & 1ull;
      open >>= 1;
      if (starts_row) sh.part[role][slot] = p;
      p = starts_row ? 0.0 : p;
      const bool valid = s < nv;
      const double pn = fma(b[2], x[2], fma(b[1], x[1], fma(b[0], x[0], p)));
      p = valid ? pn : p;
      if (NP == 2) {
        if (starts_row) part2[slot] = q;
        q = starts_row ? 0.0 : q;
        const double qn = fma(b[2], x[2] - 1.0, fma(b[1], x[1] - 1.0, fma(b[0], x[0] - 1.0, q)));
        q = valid ? qn : q;
      }
      slot += starts_row ? 1 : 0;
    };
    auto consume = [&](int k) {
      double b[3][3], x[3][3];  // all loads of the group before its chain of FMAs
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const double* be = bl + 288 * min(3 * k + e, S - 1);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          b[e][r] = be[32 * r];
          x[e][r] = sh.stage[k & 1][e][r][lane];
        }
      }
#pragma unroll
      for (int e = 0; e < 3; ++e)
        if (3 * k + e < S) step(3 * k + e, b[e], x[e]);
      team_sync(team);
    };
    // even groups pass through u, odd ones through v (no copies between them: a copy would wait for the load)
    const int groups = (S + 2) / 3;
    double u[3], v[3];
    load_padded(point(g, 0), u);
    load_padded(point(g, 1), v);
    put_stage(0, u);
    load_padded(point(g, 2), u);
    team_sync(team);
    for (int k = 0; k < groups; k += 2) {
      if (k + 1 < groups) {
        put_stage(1, v);
        load_padded(point(g, k + 3), v);
      }
      consume(k);
      if (k + 1 >= groups) break;
      if (k + 2 < groups) {
        put_stage(0, u);
        load_padded(point(g, k + 4), u);
      }
      consume(k + 1);
    }
    exchange<NP>(slot, p, q, part2);
  }

  // The same product with points in the CTA's own shared memory: every warp reads all of them itself, the next group of
  // three steps while the FMAs of one run, so the team meets only at the end. No warp of the team may still read the
  // previous product.
  template <int NP>
  __device__ __forceinline__ void product_local(const double* g, double* part2_all = nullptr) {
    double* part2 = part2_all + 64 * role;
    int slot = slot0;
    double p = 0.0, q = 0.0;
    const double* bl = wv + 32 * 3 * role + lane;
    unsigned long long open = starts;
    struct Group {
      double b[3][3], x[3][3];
    };
    auto load = [&](int k, Group& t) {
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const int s = min(3 * k + e, S - 1);
        const double* pt = g + 4 * (size_t)wc[32 * s + lane];
        const double2 xy = *reinterpret_cast<const double2*>(pt);
        t.x[e][0] = xy.x;
        t.x[e][1] = xy.y;
        t.x[e][2] = pt[2];
#pragma unroll
        for (int r = 0; r < 3; ++r) t.b[e][r] = bl[288 * s + 32 * r];
      }
    };
    auto consume = [&](int k, const Group& t) {
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const int s = 3 * k + e;
        if (s >= S) break;
        const bool starts_row = open & 1ull;
        open >>= 1;
        if (starts_row) sh.part[role][slot] = p;
        p = starts_row ? 0.0 : p;
        const bool valid = s < nv;
        const double pn = fma(t.b[e][2], t.x[e][2], fma(t.b[e][1], t.x[e][1], fma(t.b[e][0], t.x[e][0], p)));
        p = valid ? pn : p;
        if (NP == 2) {
          if (starts_row) part2[slot] = q;
          q = starts_row ? 0.0 : q;
          const double qn =
              fma(t.b[e][2], t.x[e][2] - 1.0, fma(t.b[e][1], t.x[e][1] - 1.0, fma(t.b[e][0], t.x[e][0] - 1.0, q)));
          q = valid ? qn : q;
        }
        slot += starts_row ? 1 : 0;
      }
    };
    const int groups = (S + 2) / 3;
    Group u, v;
    load(0, u);
    for (int k = 0; k < groups; k += 2) {
      if (k + 1 < groups) load(k + 1, v);
      consume(k, u);
      if (k + 1 >= groups) break;
      if (k + 2 < groups) load(k + 2, u);
      consume(k + 1, v);
    }
    exchange<NP>(slot, p, q, part2);
  }

  // The last pieces, the rows' sums, and the result to every warp of the team.
  template <int NP>
  __device__ __forceinline__ void exchange(int slot, double p, double q, double* part2) {
    if (nv > 0) {
      sh.part[role][slot] = p;
      if (NP == 2) part2[slot] = q;
    }
    __syncwarp();
    double a = 0.0, a2 = 0.0;
    if (pieces > 0) {
      a = ipipe::plus_zero(sh.part[role][piece0]);
      for (int k = 1; k < pieces; ++k) a = a + sh.part[role][piece0 + k];
      if (NP == 2) {
        a2 = ipipe::plus_zero(part2[piece0]);
        for (int k = 1; k < pieces; ++k) a2 = a2 + part2[piece0 + k];
      }
    }
    __syncwarp();
    sh.part[role][lane] = a;
    if (NP == 2) part2[lane] = a2;
    team_sync(team);
  }
};

// Barriers and reductions of kernels whose CTAs own chunks: the flat barrier, one stripe per warp, the totals and the
// decision by warp 0. Every thread of the CTA calls; chunk sums alternate between two buffers of 4 C.
struct ResidentReduce {
  const MonoBarrier mb;
  double* csum;
  const int C;
  double* stripes;  // 32 shared doubles
  const int lane, warp, nwarps;
  // CTAs that share a problem may still be at others when this one arrives first: a counter that every CTA advances at
  // every barrier of every problem (null where all CTAs start together). While it moves, the wait of the first barrier
  // does not count as a hang; past it all CTAs are here and the limit holds as it is.
  unsigned long long* progress = nullptr;
  unsigned phase = 0;  // barriers passed
  __device__ double* sums() const { return csum + (size_t)(phase & 1u) * 4 * C; }
  // v: quantity q of chunk c, in lane 0
  __device__ void put_total(int q, int c, double v) {
    if (lane == 0) sums()[q * C + c] = v;
  }
  // quantity q in lanes 0-15, q + 1 in the others
  __device__ void put_totals(int q, int c, double v) {
    if ((lane & 15) == 0) sums()[(q + (lane >> 4)) * C + c] = v;
  }
  // sum of v over the warp as chunk c's value of quantity q
  __device__ void put(int q, int c, double v) { put_total(q, c, warp_sum_butterfly(v)); }
  __device__ void put_max(int q, int c, double v) { put_total(q, c, warp_max_butterfly(v)); }
  // The last warp prepares the next decision (side) while thread 0 waits for the other CTAs.
  template <class Side>
  __device__ bool arrive_and_wait(Side&& side) {
    bool ok = true;
    __syncthreads();
    if (warp == nwarps - 1) side();
    if (threadIdx.x == 0) {
      if (progress) red_add_relaxed_u64(progress, 1ull);
      if (mb.parties > 1u) ok = flat_wait(mb, phase, phase == 0 ? progress : nullptr);
    }
    return __syncthreads_and(ok) != 0;
  }
  __device__ bool sync() {
    const bool ok = arrive_and_wait([] {});
    ++phase;
    return ok;
  }
  // Barrier, K <= 4 quantities (value 0 a maximum where maxmask; K == 2 then), then decide(total) by warp 0, lane q < K
  // holding quantity q's total (read the others with total_of).
  template <class Side, class Decide>
  __device__ bool reduce(int K, unsigned maxmask, Side&& side, Decide&& decide) {
    if (!arrive_and_wait(side)) return false;
    const double* s = sums();
    const int per = (C + 7) / 8;
    if (warp < 8) {
      const int st = warp, b = st * per, e = min(C, b + per);
      double p[4] = {0.0, 0.0, 0.0, 0.0};
      for (int k = b + lane; k < e; k += 32) {
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = q < K ? ldcg(s + q * C + k) : 0.0;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q < K) p[q] = (maxmask >> q) & 1u ? ((v[q] < p[q]) ? p[q] : v[q]) : p[q] + v[q];
      }
      if (b >= e) {
        if (lane < K) stripes[8 * lane + st] = 0.0;
      } else if (maxmask) {
        const double v0 = warp_max_butterfly(p[0]), v1 = warp_sum_butterfly(p[1]);
        if (lane < 2) stripes[8 * lane + st] = lane ? v1 : v0;
      } else if (K > 2) {
        const double v = warp_sum4_butterfly(p[0], p[1], p[2], p[3]);
        if ((lane & 7) == 0) stripes[lane + st] = v;
      } else {
        const double v = warp_sum2_butterfly(p[0], p[1]);
        if ((lane & 15) == 0) stripes[lane / 2 + st] = v;
      }
    }
    __syncthreads();
    if (warp == 0) {
      const int q = lane < K ? lane : 0;
      const bool mx = (maxmask >> q) & 1u;
      double total = stripes[8 * q];
#pragma unroll
      for (int k = 1; k < 8; ++k) {
        const double v = stripes[8 * q + k];
        total = mx ? ((v < total) ? total : v) : total + v;
      }
      decide(total);
    }
    __syncthreads();
    ++phase;
    return true;
  }
};
__device__ __forceinline__ double total_of(double total, int q) { return __shfl_sync(0xffffffffu, total, q); }

}  // namespace bogus_gpu
