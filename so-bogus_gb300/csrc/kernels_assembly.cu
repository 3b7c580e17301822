// Delassus assembly W = H M^-1 H^T and b = w - H M^-1 f on the device
// (DualFrictionProblem::computeFrom, Interfaces/FrictionProblem.cpp:30-40; block products of
// Core/Block/SparseMatrixMatrixProduct.impl.hpp:295-349).
//
// Each contact has at most two body slots ordered by body index, with a 3 x ndof Jacobian block per slot.
// Order of evaluation (shared with the CPU oracle):
//   T_(j,t)[m][c]  = chain over q of fma(Minv_k[m][q], H_(j,t)[c][q])            (M^-1 H^T first)
//   W_ij[r][c]     = chain over the shared bodies (increasing), then m, of fma(H_(i,ti)[r][m], T_(j,tj)[m][c])
// The pattern comes from the bodies' contact lists: row i is the merge of its bodies' lists (one thread per row, once to
// count and once to fill both W and its lower triangle). One thread computes one lower block from the slot pairs that share
// a body and writes it to the lower triangle and, in both places, to W; the transposed place is found by bisection of
// its row's sorted columns.
// Bound by launches and the upload of H at the sizes of a time step, by the writes of W where a body is in many contacts.
// computeFrom on GB300, ms, with the pattern built on the host / here: 15 001 contacts on a new handle 6.6 / 1.5, on the same
// 6.0 / 0.75; 33 contacts 0.22 / 0.23 and 0.15 / 0.145; one body in 1000 contacts 22.5 / 0.74, in 6000 900 / 6.5 (with the
// transposed blocks placed by atomics and each row's sorted by one thread, as launch_full_pattern does for a matrix that
// the caller gives, 210 and 10 300).
#include "internal.h"

namespace bogus_gpu {

__global__ void k_assembly_T(int n, int d, const double* __restrict__ minv, const int* __restrict__ cb,
                             const double* __restrict__ H, double* __restrict__ T) {
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;  // 2 * contact + t
  if (slot >= 2 * n) return;
  const int k = cb[slot];
  if (k < 0) return;
  const double* Mi = minv + (size_t)k * d * d;
  const double* Hs = H + (size_t)slot * 3 * d;
  double* Ts = T + (size_t)slot * d * 3;
  for (int m = 0; m < d; ++m)
    for (int c = 0; c < 3; ++c) {
      double a = 0.0;
      for (int q = 0; q < d; ++q) a = fma(Mi[m * d + q], Hs[c * d + q], a);
      Ts[m * 3 + c] = a;
    }
}

cudaError_t launch_assembly_T(int n, int d, const double* minv, const int* cb, const double* H, double* T,
                              cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_assembly_T<<<(2 * n + 127) / 128, 128, 0, s>>>(n, d, minv, cb, H, T);
  return cudaGetLastError();
}

// H slots of the contacts from the caller's blocks: slot 0 the body of smaller index (a repeated body counts once)
__global__ void k_assembly_slots(int n, int d, const int* __restrict__ cb, const int* __restrict__ objA,
                                 const double* __restrict__ HA, const double* __restrict__ HB, double* __restrict__ H) {
  const int hs = 3 * d;
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= 2LL * n * hs) return;
  const int slot = (int)(e / hs), i = slot >> 1, k = (int)(e - (long long)slot * hs);
  const int body = cb[slot];
  H[e] = body < 0 ? 0.0 : (body == objA[i] ? HA : HB)[(size_t)i * hs + k];
}

cudaError_t launch_assembly_slots(int n, int d, const int* cb, const int* objA, const double* HA, const double* HB,
                                  double* H, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const long long m = 6LL * n * d;
  k_assembly_slots<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(n, d, cb, objA, HA, HB, H);
  return cudaGetLastError();
}

// Calls f(j) for the contacts that share a body with contact i, itself among them, in increasing order. bptr, bent: the
// bodies' lists of 2 contact + slot in increasing order.
template <class F>
__device__ __forceinline__ void for_row(int i, const int* __restrict__ cb, const int* __restrict__ bptr,
                                        const int* __restrict__ bent, F&& f) {
  constexpr int kNone = 0x7fffffff;
  const int b0 = cb[2 * i], b1 = cb[2 * i + 1];
  int p = b0 >= 0 ? bptr[b0] : 0, q = b1 >= 0 ? bptr[b1] : 0;
  const int pe = b0 >= 0 ? bptr[b0 + 1] : 0, qe = b1 >= 0 ? bptr[b1 + 1] : 0;
  int jp = p < pe ? bent[p] >> 1 : kNone, jq = q < qe ? bent[q] >> 1 : kNone;
  while (true) {
    const int j = jp < jq ? jp : jq;
    if (j == kNone) break;
    f(j);
    if (jp == j) jp = ++p < pe ? bent[p] >> 1 : kNone;
    if (jq == j) jq = ++q < qe ? bent[q] >> 1 : kNone;
  }
}

// lower[i], full[i]: blocks of row i up to its diagonal, and all of them
__global__ void k_row_count(int n, const int* __restrict__ cb, const int* __restrict__ bptr,
                            const int* __restrict__ bent, int* __restrict__ lower, int* __restrict__ full) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int l = 0, c = 0;
  for_row(i, cb, bptr, bent, [&](int j) {
    l += j <= i ? 1 : 0;
    ++c;
  });
  lower[i] = l;
  full[i] = c;
}

__global__ void k_row_fill(int n, const int* __restrict__ cb, const int* __restrict__ bptr,
                           const int* __restrict__ bent, const int* __restrict__ lptr, int* __restrict__ lrow,
                           int* __restrict__ lcol, const int* __restrict__ fptr, int* __restrict__ fcol) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int k = lptr[i], p = fptr[i];
  for_row(i, cb, bptr, bent, [&](int j) {
    fcol[p++] = j;
    if (j > i) return;
    lrow[k] = i;
    lcol[k++] = j;
  });
}

cudaError_t launch_row_count(int n, const int* cb, const int* bptr, const int* bent, int* lower, int* full,
                             cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_row_count<<<(n + 127) / 128, 128, 0, s>>>(n, cb, bptr, bent, lower, full);
  return cudaGetLastError();
}
cudaError_t launch_row_fill(int n, const int* cb, const int* bptr, const int* bent, const int* lptr, int* lrow,
                            int* lcol, const int* fptr, int* fcol, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_row_fill<<<(n + 127) / 128, 128, 0, s>>>(n, cb, bptr, bent, lptr, lrow, lcol, fptr, fcol);
  return cudaGetLastError();
}

// D > 0: dofs fixed at compile time, a slot pair's H and T in registers for its nine chains
template <int D>
__global__ void k_assembly_W(int nlow, int dofs, const int* __restrict__ lptr, const int* __restrict__ row,
                             const int* __restrict__ col, const int* __restrict__ fptr, const int* __restrict__ fcol,
                             const int* __restrict__ cb, const double* __restrict__ H, const double* __restrict__ T,
                             double* __restrict__ lval, double* __restrict__ fval) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nlow) return;
  const int d = D > 0 ? D : dofs;
  const int i = row[k], j = col[k];
  double B[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int ti = 0; ti < 2; ++ti)
    for (int tj = 0; tj < 2; ++tj) {
      const int body = cb[2 * i + ti];
      if (body < 0 || body != cb[2 * j + tj]) continue;
      const double* Hi = H + (size_t)(2 * i + ti) * 3 * d;
      const double* Tj = T + (size_t)(2 * j + tj) * d * 3;
#pragma unroll
      for (int m = 0; m < (D > 0 ? D : 1); ++m)
        for (int mm = m; mm < d; mm += (D > 0 ? D : 1)) {
#pragma unroll
          for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) B[3 * r + c] = fma(Hi[r * d + mm], Tj[mm * 3 + c], B[3 * r + c]);
        }
    }
  double* L = lval + 9 * (size_t)k;
  double* F = fval + 9 * ((size_t)fptr[i] + (k - lptr[i]));
#pragma unroll
  for (int e = 0; e < 9; ++e) L[e] = F[e] = B[e];
  if (j == i) return;
  int lo = fptr[j] + (lptr[j + 1] - lptr[j]), hi = fptr[j + 1] - 1;  // column i is past the diagonal of row j
  while (lo < hi) {
    const int mid = lo + (hi - lo) / 2;
    if (fcol[mid] < i) lo = mid + 1;
    else hi = mid;
  }
  double* Ft = fval + 9 * (size_t)lo;
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) Ft[3 * r + c] = B[3 * c + r];
}

cudaError_t launch_assembly_W(int nlow, int ndof, const int* lptr, const int* row, const int* col, const int* fptr,
                              const int* fcol, const int* cb, const double* H, const double* T, double* lval,
                              double* fval, cudaStream_t s) {
  if (nlow == 0) return cudaSuccess;
  const int g = (nlow + 127) / 128;
  if (ndof == 6) k_assembly_W<6><<<g, 128, 0, s>>>(nlow, ndof, lptr, row, col, fptr, fcol, cb, H, T, lval, fval);
  else k_assembly_W<0><<<g, 128, 0, s>>>(nlow, ndof, lptr, row, col, fptr, fcol, cb, H, T, lval, fval);
  return cudaGetLastError();
}

__global__ void k_assembly_mf(int nb, int d, const double* __restrict__ minv, const double* __restrict__ f,
                              double* __restrict__ mf) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nb * d) return;
  const int k = t / d, m = t % d;
  double a = 0.0;
  for (int q = 0; q < d; ++q) a = fma(minv[(size_t)k * d * d + m * d + q], f ? f[(size_t)k * d + q] : 0.0, a);
  mf[t] = a;
}

__global__ void k_assembly_b(int n, int d, const int* __restrict__ cb, const double* __restrict__ H,
                             const double* __restrict__ mf, const double* __restrict__ w, double* __restrict__ b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int r = 0; r < 3; ++r) {
    double a = 0.0;
    for (int t = 0; t < 2; ++t) {
      const int k = cb[2 * i + t];
      if (k < 0) continue;
      const double* Hs = H + (size_t)(2 * i + t) * 3 * d;
      for (int m = 0; m < d; ++m) a = fma(Hs[r * d + m], mf[(size_t)k * d + m], a);
    }
    b[3 * i + r] = w[3 * i + r] - a;
  }
}

cudaError_t launch_assembly_b(int n, int nbodies, int ndof, const double* minv, const double* f, const int* cb,
                              const double* H, const double* w, double* mf, double* b, cudaStream_t s) {
  if (nbodies > 0) k_assembly_mf<<<(nbodies * ndof + 127) / 128, 128, 0, s>>>(nbodies, ndof, minv, f, mf);
  if (n > 0) k_assembly_b<<<(n + 127) / 128, 128, 0, s>>>(n, ndof, cb, H, mf, w, b);
  return cudaGetLastError();
}

}  // namespace bogus_gpu
