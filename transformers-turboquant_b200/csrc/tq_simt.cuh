// Building blocks of the fp32 CUDA-core kernels: a register-tiled [64 x D] x [D x D]
// product against a matrix held in shared memory, and the SM count.
#pragma once
#include "tq_common.cuh"

namespace tq {

// Column permutation of the shared-memory copy of a transposed matrix: the thread that
// owns coordinates tx*8..tx*8+7 reads two float4 at [tx*4] and [D/2 + tx*4], which is
// bank-conflict free across tx.
template <int D>
__device__ __forceinline__ int perm_col(int j) {
  const int tx = j >> 3, e = j & 7;
  return (e >> 2) * (D / 2) + tx * 4 + (e & 3);
}

// Four floats of a matrix that may start at any 4-byte address (one load where it is 16-byte aligned, as tensors are).
__device__ __forceinline__ float4 ldg4(const float* p) {
  if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0) return __ldg(reinterpret_cast<const float4*>(p));
  return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

// Copy a row-major [D, D] fp32 matrix into shared memory as the right-hand side of
// tile_gemm.  TRANSPOSE: MT[i][perm(j)] = M[j][i] (for x @ M^T); else MT[i][perm(j)] = M[i][j].
template <int D, bool TRANSPOSE>
__device__ void load_matrix(const float* __restrict__ M, float* __restrict__ MT, int tid, int nthreads) {
  if constexpr (TRANSPOSE) {
    // Lanes take consecutive rows and 32 bytes of each: a whole sector read, and stores to 32 columns of one row of MT
    // (two to a bank).  Lanes along a row instead store 32 deep into one bank, and one load at a time costs a trip to L2
    // each: the two made half of a launch of one tile per CTA.
    constexpr int N = D * (D / 8), kAhead = 4;  // pieces whose loads are in flight together
    for (int e0 = tid; e0 < N; e0 += kAhead * nthreads) {
      float4 u[kAhead], v[kAhead];
#pragma unroll
      for (int x = 0; x < kAhead; ++x) {
        const int e = e0 + x * nthreads;
        if (e < N) {
          const float* src = M + e % D * D + e / D * 8;
          u[x] = ldg4(src);
          v[x] = ldg4(src + 4);
        }
      }
#pragma unroll
      for (int x = 0; x < kAhead; ++x) {
        const int e = e0 + x * nthreads, b = e / D * 8, col = perm_col<D>(e % D);
        if (e < N) {
          const float w[8] = {u[x].x, u[x].y, u[x].z, u[x].w, v[x].x, v[x].y, v[x].z, v[x].w};
#pragma unroll
          for (int i = 0; i < 8; ++i) MT[(b + i) * D + col] = w[i];
        }
      }
    }
  } else {
    constexpr int N = D * (D / 4), kAhead = 8;
    for (int e0 = tid; e0 < N; e0 += kAhead * nthreads) {
      float4 v[kAhead];
#pragma unroll
      for (int x = 0; x < kAhead; ++x)
        if (e0 + x * nthreads < N) v[x] = ldg4(M + 4 * (e0 + x * nthreads));
#pragma unroll
      for (int x = 0; x < kAhead; ++x) {
        const int e = e0 + x * nthreads;  // the permutation keeps groups of four columns together
        if (e < N) *reinterpret_cast<float4*>(MT + e / (D / 4) * D + perm_col<D>(e % (D / 4) * 4)) = v[x];
      }
    }
  }
}

// Two fp32 multiply-adds in one instruction (each rounded as fmaf rounds): d = a * b + d
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  return v;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}

// acc[r][c] = sum_i X[row0+r][i] * MT[i][cols of this thread]
template <int D, int XS>
__device__ __forceinline__ void tile_gemm(const float* __restrict__ X, const float* __restrict__ MT,
                                          int row0, int tx, float (&acc)[4][8]) {
  unsigned long long a2[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) a2[r][c] = 0ull;
#pragma unroll 2
  for (int i4 = 0; i4 < D; i4 += 4) {
    float4 xv[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) xv[r] = *reinterpret_cast<const float4*>(X + (row0 + r) * XS + i4);
#pragma unroll
    for (int ii = 0; ii < 4; ++ii) {
      const ulonglong2 m0 = *reinterpret_cast<const ulonglong2*>(MT + (i4 + ii) * D + tx * 4);
      const ulonglong2 m1 = *reinterpret_cast<const ulonglong2*>(MT + (i4 + ii) * D + D / 2 + tx * 4);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float xs = ii == 0 ? xv[r].x : ii == 1 ? xv[r].y : ii == 2 ? xv[r].z : xv[r].w;
        const unsigned long long x2 = pack2(xs, xs);
        fma2(a2[r][0], x2, m0.x);
        fma2(a2[r][1], x2, m0.y);
        fma2(a2[r][2], x2, m1.x);
        fma2(a2[r][3], x2, m1.y);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) unpack2(a2[r][c], acc[r][2 * c], acc[r][2 * c + 1]);
}


inline int sm_count() {
  static int cached = 0;
  if (!cached) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev);
    if (cached <= 0) cached = 148;
  }
  return cached;
}

}  // namespace tq
