// Triangular solves of small mixed factorisations (2 to kInvMaxSteps block columns) by explicit
// inverses.
//
// A wavefront sweep (tc_solve.cuh) is a chain of super blocks, about 36 us each whatever the number
// of right-hand sides, and its factors take transposed copies, scaled blocks and planes to prepare.
// While L^-1 and U^-1 of the whole matrix cost little, a solve is two dense products with them that
// all SMs share: X = U^-1 (L^-1 (P B)), 4-6 us each.  The inverses are formed by columns:
// full_inverse_kernel solves for 8 columns per CTA by blocks of 128 rows, with the diagonal blocks'
// inverses that the factorisation made anyway.  FP32 FMAs throughout.
#pragma once
#include "common.cuh"

namespace hprmat {

constexpr int kInvNB = 128;
constexpr int kInvCols = 8;

struct InvArgs {
  const float2* W;    // factors as the LU stores them (column-major, ld)
  long ld;
  const float2* dinv;  // diagonal blocks' inverses: [2 s + u], 128 x 128 column-major
  const int* sig;     // L's rows of block column s in final order: sig[s * sig_ld + row]
  long sig_ld;
  int N;
  float2* out;  // L^-1, then U^-1 (ldo x N each, column-major)
  long ldo;
};

__host__ __device__ constexpr size_t full_inverse_smem(int N) {
  return ((size_t)((N + kInvNB - 1) / kInvNB) * kInvNB + kInvNB) * kInvCols * sizeof(float2);
}

// Grid (N / 8, 2): columns c0 .. c0 + 7 of L^-1 (y = 0) or U^-1 (y = 1).  256 threads: row r of a
// block row, four of the columns.  FMA-bound on the SM that has the longest chain: 2 N^3 / 3
// complex FMAs over 148 SMs.
__global__ void __launch_bounds__(256) full_inverse_kernel(InvArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* X = reinterpret_cast<float2*>(smem_raw);  // [block rows * 128][8]
  const int N = a.N, ns = (N + kInvNB - 1) / kInvNB;
  float2* rhs = X + (size_t)ns * kInvNB * kInvCols;  // [128][8]
  const bool upper = blockIdx.y == 1;
  const int c0 = blockIdx.x * kInvCols, J0 = c0 / kInvNB;
  const int tid = threadIdx.x, r = tid & (kInvNB - 1), h = (tid >> 7) * 4;  // columns h .. h + 3
  const int nchain = upper ? J0 + 1 : ns - J0;
  for (int i = tid; i < ns * kInvNB * kInvCols; i += 256) X[i] = make_float2(0.f, 0.f);
  __syncthreads();
  const float2* D0 = a.dinv + (size_t)(2 * J0 + (upper ? 1 : 0)) * kInvNB * kInvNB + (size_t)(c0 % kInvNB) * kInvNB;
#pragma unroll
  for (int q = 0; q < 4; ++q) X[(size_t)(J0 * kInvNB + r) * kInvCols + h + q] = D0[(size_t)(h + q) * kInvNB + r];
  __syncthreads();
  auto product = [](float2 (&acc)[4], float2 t, const float2* x, bool subtract) {
    const float4 x01 = reinterpret_cast<const float4*>(x)[0], x23 = reinterpret_cast<const float4*>(x)[1];
    if (subtract) t = make_float2(-t.x, -t.y);
    cfma(acc[0], t, make_float2(x01.x, x01.y));
    cfma(acc[1], t, make_float2(x01.z, x01.w));
    cfma(acc[2], t, make_float2(x23.x, x23.y));
    cfma(acc[3], t, make_float2(x23.z, x23.w));
  };
  for (int s = 1; s < nchain; ++s) {
    const int J = upper ? J0 - s : J0 + s;
    const int row = J * kInvNB + r;
    float2 acc[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] = make_float2(0.f, 0.f);
    if (row < N) {
      for (int p = 0; p < s; ++p) {
        const int K = upper ? J0 - p : J0 + p;
        const int kn = min(kInvNB, N - K * kInvNB);
        const float2* src = a.W + (upper ? row : a.sig[(size_t)K * a.sig_ld + row]) + (size_t)K * kInvNB * a.ld;
        const float2* xk = X + (size_t)K * kInvNB * kInvCols + h;
        int k = 0;
        for (; k + 16 <= kn; k += 16) {
          float2 t[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) t[e] = src[(size_t)(k + e) * a.ld];
#pragma unroll
          for (int e = 0; e < 16; ++e) product(acc, t[e], xk + (size_t)(k + e) * kInvCols, true);
        }
        for (; k < kn; ++k) product(acc, src[(size_t)k * a.ld], xk + (size_t)k * kInvCols, true);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) rhs[r * kInvCols + h + q] = acc[q];
    __syncthreads();
    const float2* D = a.dinv + (size_t)(2 * J + (upper ? 1 : 0)) * kInvNB * kInvNB + r;
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] = make_float2(0.f, 0.f);
    for (int k = 0; k < kInvNB; k += 16) {
      float2 t[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) t[e] = D[(size_t)(k + e) * kInvNB];
#pragma unroll
      for (int e = 0; e < 16; ++e) product(acc, t[e], rhs + (k + e) * kInvCols + h, false);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) X[(size_t)row * kInvCols + h + q] = acc[q];
    __syncthreads();
  }
  float2* out = a.out + (upper ? (size_t)a.ldo * N : 0);
  for (int i = tid; i < N; i += 256)
#pragma unroll
    for (int q = 0; q < kInvCols; ++q)
      if (c0 + q < N) out[(size_t)i + (size_t)(c0 + q) * a.ldo] = X[(size_t)i * kInvCols + q];
}

__host__ __device__ constexpr size_t inv_apply_smem(int N) {  // B's columns; reused for the warps' sums
  return ((size_t)N * kInvCols > 8 * 32 * kInvCols ? (size_t)N * kInvCols : 8 * 32 * kInvCols) * sizeof(float2);
}

// out = T B for T = L^-1 (lower) or U^-1 (upper), N x N; rows of B taken through perm if given.
// Grid (N / 32, nrhs / 8): 32 rows (lanes) x 8 columns per CTA, the 8 warps taking every eighth
// column of T, whose zero part is skipped.
__global__ void __launch_bounds__(256) inv_apply_kernel(const float2* __restrict__ T, long ldt, int N, bool upper,
                                                        const int* __restrict__ perm, const float2* __restrict__ B,
                                                        long ldb, int nrhs, float2* __restrict__ out, long ldo) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* bs = reinterpret_cast<float2*>(smem_raw);  // [k - klo][8]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = blockIdx.x * 32, cb = blockIdx.y * kInvCols;
  const int klo = upper ? r0 : 0, khi = upper ? N : min(N, r0 + 32);
  {
    const int c = tid & 7;
    const bool cv = cb + c < nrhs;
    const float2* b = B + (size_t)(cv ? cb + c : 0) * ldb;
    for (int k = klo + (tid >> 3); k < khi; k += 32)
      bs[(size_t)(k - klo) * kInvCols + c] = cv ? b[perm ? perm[k] : k] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  float2 acc[kInvCols];
#pragma unroll
  for (int q = 0; q < kInvCols; ++q) acc[q] = make_float2(0.f, 0.f);
  const int row = r0 + lane;
  const float2* t = T + (row < N ? row : N - 1);
  auto step = [&](float2 v, int k) {
    const float4* x = reinterpret_cast<const float4*>(bs + (size_t)(k - klo) * kInvCols);
#pragma unroll
    for (int q = 0; q < kInvCols / 2; ++q) {
      const float4 b = x[q];
      cfma(acc[2 * q], v, make_float2(b.x, b.y));
      cfma(acc[2 * q + 1], v, make_float2(b.z, b.w));
    }
  };
  int k = klo + warp;
  for (; k + 56 < khi; k += 64) {
    float2 v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = t[(size_t)(k + 8 * e) * ldt];
#pragma unroll
    for (int e = 0; e < 8; ++e) step(v[e], k + 8 * e);
  }
  for (; k < khi; k += 8) step(t[(size_t)k * ldt], k);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kInvCols; ++q) bs[(warp * kInvCols + q) * 32 + lane] = acc[q];
  __syncthreads();
  const int c = warp;
  float2 s = make_float2(0.f, 0.f);
#pragma unroll
  for (int w = 0; w < 8; ++w) s = cadd(s, bs[(w * kInvCols + c) * 32 + lane]);
  if (row < N && cb + c < nrhs) out[(size_t)row + (size_t)(cb + c) * ldo] = s;
}

}  // namespace hprmat
