// FP32 matrix products on the CUDA cores: one 128 x 128 tile of op(A) op(B)
// per CTA of 256 threads.
//
// Each output is one FP32 chain of fused multiply-adds over ascending k from
// its initial value, whatever the tile it lies in: the result does not depend
// on the tiling, and a split of K is the caller's choice.  8 x 8 outputs a
// thread as column pairs (packed __ffma2_rn: two correctly rounded
// multiply-adds an instruction), 16 columns of K a stage, the next stage
// prefetched into registers while the current one is used from shared memory.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace sg {

constexpr int BM = 128, BN = 128, BK = 16, NTHR = 256;
constexpr int LDS_ = BM + 4;
struct alignas(16) Smem { float a[2][BK][LDS_]; float b[2][BK][LDS_]; };

// Operand tile of 128 rows (of the output dimension) x BK.  KMAJ: X[r][k]
// (ld between r), else X[k][r] (ld between k).  vec: 16-byte loads are
// aligned.  Entries past `rows` or `ke` read as zero.
template <bool KMAJ>
__device__ __forceinline__ void load_tile(const float* __restrict__ X, int64_t ld, int r0, int rows, int k0, int ke,
                                          bool vec, float4 (&v)[2]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int idx = threadIdx.x + h * NTHR;
    const int r = KMAJ ? r0 + (idx >> 2) : r0 + (idx & 31) * 4;
    const int k = KMAJ ? k0 + (idx & 3) * 4 : k0 + (idx >> 5);
    v[h] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (KMAJ) {
      if (r >= rows || k >= ke) continue;
      const float* p = X + (int64_t)r * ld + k;
      if (vec && k + 3 < ke) {
        v[h] = *reinterpret_cast<const float4*>(p);
      } else {
        v[h].x = p[0];
        if (k + 1 < ke) v[h].y = p[1];
        if (k + 2 < ke) v[h].z = p[2];
        if (k + 3 < ke) v[h].w = p[3];
      }
    } else {
      if (k >= ke || r >= rows) continue;
      const float* p = X + (int64_t)k * ld + r;
      if (vec && r + 3 < rows) {
        v[h] = *reinterpret_cast<const float4*>(p);
      } else {
        v[h].x = p[0];
        if (r + 1 < rows) v[h].y = p[1];
        if (r + 2 < rows) v[h].z = p[2];
        if (r + 3 < rows) v[h].w = p[3];
      }
    }
  }
}

template <bool KMAJ>
__device__ __forceinline__ void store_tile(float (*s)[LDS_], const float4 (&v)[2]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int idx = threadIdx.x + h * NTHR;
    if (KMAJ) {
      const int r = idx >> 2, k = (idx & 3) * 4;
      s[k][r] = v[h].x; s[k + 1][r] = v[h].y; s[k + 2][r] = v[h].z; s[k + 3][r] = v[h].w;
    } else {
      *reinterpret_cast<float4*>(&s[idx >> 5][(idx & 31) * 4]) = v[h];
    }
  }
}

__device__ __forceinline__ bool vec_ok(const float* p, int64_t ld) {
  return ((uintptr_t)p & 15) == 0 && (ld & 3) == 0;
}

// Output (i, j) of a thread: row row_of(i), column pair col_of(j), col_of(j) + 1.
__device__ __forceinline__ int row_of(int i) { return (i >> 2) * 64 + (threadIdx.x >> 4) * 4 + (i & 3); }
__device__ __forceinline__ int col_of(int j) { return (j >> 1) * 64 + (threadIdx.x & 15) * 4 + (j & 1) * 2; }

// acc += op(A)[m0.., kb..ke) op(B)[kb..ke), n0..]; A_KM: A[m][k], else A[k][m];
// B_KM: B[n][k], else B[k][n].
template <bool A_KM, bool B_KM>
__device__ __forceinline__ void tile(const float* __restrict__ A, int64_t lda, const float* __restrict__ B,
                                     int64_t ldb, int M, int N, int kb, int ke, int m0, int n0, Smem& sm,
                                     float2 (&acc)[8][4]) {
  const bool va = vec_ok(A, lda) && (!A_KM || (kb & 3) == 0), vb = vec_ok(B, ldb) && (!B_KM || (kb & 3) == 0);
  float4 pa[2], pb[2];
  load_tile<A_KM>(A, lda, m0, M, kb, ke, va, pa);
  load_tile<B_KM>(B, ldb, n0, N, kb, ke, vb, pb);
  int buf = 0;
  store_tile<A_KM>(sm.a[0], pa);
  store_tile<B_KM>(sm.b[0], pb);
  __syncthreads();
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  for (int k0 = kb; k0 < ke; k0 += BK) {
    const bool more = k0 + BK < ke;
    if (more) {
      load_tile<A_KM>(A, lda, m0, M, k0 + BK, ke, va, pa);
      load_tile<B_KM>(B, ldb, n0, N, k0 + BK, ke, vb, pb);
    }
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      const float4 a0 = *reinterpret_cast<const float4*>(&sm.a[buf][k][ty * 4]);
      const float4 a1 = *reinterpret_cast<const float4*>(&sm.a[buf][k][64 + ty * 4]);
      const float4 b0 = *reinterpret_cast<const float4*>(&sm.b[buf][k][tx * 4]);
      const float4 b1 = *reinterpret_cast<const float4*>(&sm.b[buf][k][64 + tx * 4]);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float2 b[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y),
                           make_float2(b1.z, b1.w)};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 aa = make_float2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(aa, b[j], acc[i][j]);
      }
    }
    if (more) {
      store_tile<A_KM>(sm.a[buf ^ 1], pa);
      store_tile<B_KM>(sm.b[buf ^ 1], pb);
      __syncthreads();
      buf ^= 1;
    }
  }
}

}  // namespace sg
