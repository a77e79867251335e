// Sample-space SR (minSR) linear algebra on one GPU:
//   column means and centring/scaling of O, the Gram matrix T = O~ O~^T + lambda I
//   on the CUDA cores (the tensor-core ones are in gram.cu and fp64_tc.cu, with the
//   Cholesky), blocked forward/backward substitution, and dp = O~^T x.  Also the plain energy
//   gradient <E O> - <E><O>.
#include "common.cuh"

namespace {

constexpr int TB = 64;   // output tile
constexpr int TK = 16;   // k chunk

// FP32 inputs: products are accumulated in FP32 over 4 consecutive k and then
// folded into a double-float (hi, lo) pair with Knuth's TwoSum, which keeps the
// Gram matrix accurate to ~FP64 level (its smallest eigenvalues sit at the
// diagonal shift, ~1e-6 of its norm) at ~2.5x the FP32 cost instead of the
// 64x of native FP64 arithmetic on GB300.  FP64 inputs accumulate natively.
template <typename TA>
struct TileAcc {
  TA acc[4][4];
  float lo[4][4];
  float hi[4][4];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int r = 0; r < 4; ++r) { acc[q][r] = 0; lo[q][r] = 0.f; hi[q][r] = 0.f; }
  }
  __device__ __forceinline__ void fold() {
    if constexpr (sizeof(TA) == 4) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float a = hi[q][r], b = (float)acc[q][r];
          const float s = a + b;
          const float bb = s - a;
          const float err = (a - (s - bb)) + (b - bb);
          hi[q][r] = s;
          lo[q][r] += err;
          acc[q][r] = 0;
        }
    }
  }
  __device__ __forceinline__ double value(int q, int r) const {
    if constexpr (sizeof(TA) == 4) return (double)hi[q][r] + (double)lo[q][r] + (double)acc[q][r];
    return (double)acc[q][r];
  }
};

// Column kernels: a CTA of 8 warps takes 32 NC columns, lane = column (NC of
// them, 32 apart), warp w the rows w, w + 8, ...; the warps' sums meet in
// shared memory.  (One thread per column leaves all but Np / 256 CTAs' worth of
// the GPU idle and each thread waiting on one load at a time.)  NC = 4 reads 512
// consecutive bytes of an FP32 row, which HBM pages want (one 128-byte piece a
// row read 8192 x 115200 in 4.3 ms of centring); NC = 1 where that would leave
// fewer CTAs than the GPU holds.  An FP64 instruction costs a warp 64 clocks
// on GB300, so FP32 inputs are summed in three FP32 words (Sum3), which become
// one FP64 number at the end; rows whose terms leave the range in which that
// is finer than FP64 sums are added in FP64.
// 8192 x 115200 FP32: centring 10.7 and O~^T x 3.6 ms before; three
// respectively one passes over 3.8 GB take 1.7 and 0.6 at the measured rate.
constexpr int CW = 8;                    // warps a CTA
constexpr int CB = 128;                  // rows a block of the loops below
constexpr int64_t CWIDE = 128 * 304;     // columns from which NC = 4: two CTAs on each of 152 SMs

// Terms of a group of rows are summed in FP32 words while the largest lies in
// [2^-85, 2^96): sums of 2^28 rows stay below FP32's largest number, and what
// the parts of a product lose below FP32's least (2^-149 each) stays below
// 2^-60 of that term.
constexpr unsigned TERM_LO = (127u - 85u) << 23, TERM_HI = (127u + 96u) << 23;

// x = h + m + l exactly, 24 + 24 + 5 bits, for |x| in [2^-70, 2^70) or 0: the
// parts are normal floats or 0.  False for any other x.
__device__ __forceinline__ bool split_f64(double x, float& h, float& m, float& l) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x), sg = (unsigned)hi & 0x80000000u;
  const int e = ((hi >> 20) & 0x7ff) - 1023;
  h = m = l = 0.f;
  if (e < -70 || e >= 70) return x == 0.0;
  h = __uint_as_float(sg | (unsigned)(e + 127) << 23 | ((unsigned)(hi & 0xfffff) << 3) | (lo >> 29));
  m = __uint2float_rn((lo >> 5) & 0xffffffu) * __uint_as_float(sg | (unsigned)(e - 47 + 127) << 23);
  l = __uint2float_rn(lo & 31u) * __uint_as_float(sg | (unsigned)(e - 52 + 127) << 23);
  return true;
}

// Sums over all rows of the lane's NC columns, in every warp.  load(i, j): the
// value at row i, column group j; begin(i0), called by all threads before the
// rows [i0, i0 + CB): whether they may be summed in FP32 words; add(S, i - i0,
// x): adds x's term to S and returns its leading part (FP32 inputs; LOW: terms
// below TERM_LO are inexact); term(i - i0, x): the term in FP64.
template <typename T, int NC, bool LOW, typename B, typename L, typename A, typename F>
__device__ __forceinline__ void column_sums(int64_t Ns, double (*part)[NC * 32], double (&sum)[NC], B begin, L load,
                                            A add, F term) {
  constexpr int CU = 16 / NC;            // rows in flight
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  vmc::Sum3 acc[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) sum[j] = 0.0;
  for (int64_t i0 = 0; i0 < Ns; i0 += CB) {
    const bool words = begin(i0);
#pragma unroll 1
    for (int u0 = 0; u0 < CB / CW; u0 += CU) {
      T x[CU][NC];
#pragma unroll
      for (int u = 0; u < CU; ++u)
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const int64_t i = i0 + (u0 + u) * CW + warp;
          x[u][j] = i < Ns ? load(i, j) : T(0);
        }
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        bool f64 = true;
        if constexpr (sizeof(T) == 4) {
          if (words) {
            const vmc::Sum3 was = acc[j];
            unsigned mx = 0;
#pragma unroll
            for (int u = 0; u < CU; ++u)
              mx = max(mx, __float_as_uint(add(acc[j], (u0 + u) * CW + warp, x[u][j])) & 0x7fffffffu);
            f64 = mx >= TERM_HI;
            if (LOW && mx < TERM_LO)
#pragma unroll
              for (int u = 0; u < CU; ++u) f64 |= x[u][j] != T(0);   // all zero: nothing is lost
            if (f64) acc[j] = was;
          }
        }
        if (f64)
#pragma unroll
          for (int u = 0; u < CU; ++u) sum[j] += term((u0 + u) * CW + warp, x[u][j]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < NC; ++j) part[warp][j * 32 + lane] = sizeof(T) == 4 ? sum[j] + acc[j].value() : sum[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < CW; ++w) t += part[w][j * 32 + lane];
    sum[j] = t;
  }
}

// mean[p] = (1/Ns) sum_i O[i][p];  Oc[i][p] = (O[i][p] - mean[p]) * scale, FP32
// in double-float arithmetic.  An entry whose rounding to FP32 that arithmetic's
// own error (below 2^-43 of the entry and of the scaled mean) could change takes
// the FP64 expression, so that the result is always that expression rounded:
// about one entry in 10^5, tested for 16 entries at once (8192 samples, 115 K
// columns: below 1 ms of a solve of 90).  So do entries whose distance from the
// mean leaves [2^-80, 2^120): below it the remainders underflow FP32 (where the
// mean is that small too: a larger one widens the test), above it the
// difference overflows.
// O may be Oc (neither is __restrict__): a warp has read its rows before it
// writes them, and no other warp of any CTA reads their columns' entries again.
template <typename T, int NC>
__global__ void __launch_bounds__(32 * CW) k_center(const T* O, int64_t Ns, int64_t Np, int64_t ldo, T* Oc,
                                                    int64_t ldc, double* __restrict__ mean, double scale) {
  __shared__ double part[CW][NC * 32];
  __shared__ float again[sizeof(T) == 4 ? 16 : 1][32 * CW];
  constexpr int CU = 16 / NC;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t p0 = (int64_t)blockIdx.x * (32 * NC) + lane;
  int64_t off[NC];       // columns past the end read the last one
#pragma unroll
  for (int j = 0; j < NC; ++j) off[j] = p0 + 32 * j < Np ? p0 + 32 * j : Np - 1;
  double sum[NC];
  auto load = [&](int64_t i, int j) { return O[i * ldo + off[j]]; };
  column_sums<T, NC, false>(
      Ns, part, sum, [](int64_t) { return true; }, load,
      [](vmc::Sum3& S, int, T v) {
        S.add((float)v);
        return (float)v;
      },
      [](int, T v) { return (double)v; });
  double m[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    m[j] = sum[j] / (double)Ns;
    if (mean && warp == 0 && p0 + 32 * j < Np) mean[p0 + 32 * j] = m[j];
  }
  if (!Oc) return;
  float mh[NC], ml[NC];
  const float sh = (float)scale, sl = (float)(scale - (double)sh);
#pragma unroll
  for (int j = 0; j < NC; ++j) { mh[j] = (float)m[j]; ml[j] = (float)(m[j] - (double)mh[j]); }
  float dm[NC], d0[NC], d1[NC];     // |d| in [d0, d1): too small (an exact 0 - 0 is not)
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    dm[j] = fabsf(mh[j] * sh) * 0x1p-43f;
    d0[j] = mh[j] == 0.f ? 0x1p-149f : 0.f;
    d1[j] = fabsf(mh[j]) < 0x1p-80f ? 0x1p-80f : 0.f;
  }
  for (int64_t i0 = warp; i0 < Ns; i0 += CW * CU) {
    T x[CU][NC];
#pragma unroll
    for (int u = 0; u < CU; ++u)
#pragma unroll
      for (int j = 0; j < NC; ++j) x[u][j] = i0 + u * CW < Ns ? load(i0 + u * CW, j) : T(0);
    bool unsure = false;
#pragma unroll
    for (int u = 0; u < CU; ++u)
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        T v;
        if constexpr (sizeof(T) == 4) {
          float d = x[u][j];
          const float e = vmc::two_sum(d, -mh[j]) - ml[j];
          const float q = d * sh;
          const float r = fmaf(e, sh, fmaf(d, sl, fmaf(d, sh, -q)));
          const float w = fmaf(fabsf(q), 0x1p-43f, dm[j]);
          v = q + (r + w);
          unsure |= v != q + (r - w) || !(fabsf(d) < 0x1p120f) || (fabsf(d) < d1[j] && fabsf(d) >= d0[j]);
        } else {
          v = (x[u][j] - m[j]) * scale;
        }
        if (i0 + u * CW < Ns && p0 + 32 * j < Np) Oc[(i0 + u * CW) * ldc + p0 + 32 * j] = v;
      }
    if constexpr (sizeof(T) == 4) {
      if (__any_sync(VMC_FULL_MASK, unsure)) {
        // O may be Oc: the entries come from registers, through shared memory
        // for a loop that is not unrolled
#pragma unroll
        for (int u = 0; u < CU; ++u)
#pragma unroll
          for (int j = 0; j < NC; ++j) again[u * NC + j][threadIdx.x] = x[u][j];
#pragma unroll 1
        for (int u = 0; u < CU && i0 + u * CW < Ns; ++u)
#pragma unroll
          for (int j = 0; j < NC; ++j)
            if (p0 + 32 * j < Np)
              Oc[(i0 + u * CW) * ldc + p0 + 32 * j] =
                  (float)(((double)again[u * NC + j][threadIdx.x] - m[j]) * scale);
      }
    }
  }
}

// g[p] = (1/Ns) sum_i E[i] O[i][p] - Ebar * mean_i O[i][p]
template <typename TI>
__global__ void k_egrad(const TI* __restrict__ O, int64_t Ns, int64_t Np, int64_t ldo, const double* __restrict__ E,
                        double Ebar, double* __restrict__ g) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= Np) return;
  double se = 0.0, so = 0.0;
  for (int64_t i = 0; i < Ns; ++i) {
    double o = (double)O[i * ldo + p];
    se += E[i] * o;
    so += o;
  }
  g[p] = se / (double)Ns - Ebar * so / (double)Ns;
}

// C[i][j] (+)= sign * sum_{k<K} A[i][k] * A[j][k] for lower-triangular 64x64 tiles
// (tile row >= tile col).  A row-major with leading dim lda; rows offset by
// row0 for both operands; columns of C offset by col0 as well.  Tiles of the
// strict upper triangle are mirrored when mirror != 0.
template <typename TI, typename TA>
__global__ void k_syrk(const TI* __restrict__ A, int64_t lda, int64_t n, int64_t K, double* __restrict__ C,
                       int64_t ldc, int64_t off, double sgn, double diag, int mirror) {
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (bj > bi) return;
  __shared__ TA As[TK][TB + 1];
  __shared__ TA Bs[TK][TB + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t i0 = off + (int64_t)bi * TB, j0 = off + (int64_t)bj * TB;
  TileAcc<TA> T;
  T.zero();
  for (int64_t k0 = 0; k0 < K; k0 += TK) {
    for (int idx = threadIdx.x; idx < TB * TK; idx += 256) {
      int r = idx / TK, kk = idx - r * TK;
      int64_t gk = k0 + kk;
      int64_t gi = i0 + r, gj = j0 + r;
      As[kk][r] = (gi < off + n && gk < K) ? (TA)A[gi * lda + gk] : (TA)0;
      Bs[kk][r] = (gj < off + n && gk < K) ? (TA)A[gj * lda + gk] : (TA)0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      TA a[4], b[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) { a[q] = As[kk][ty * 4 + q]; b[q] = Bs[kk][tx * 4 + q]; }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) T.acc[q][r] += a[q] * b[r];
      if ((kk & 3) == 3) T.fold();
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      int64_t gi = i0 + ty * 4 + q, gj = j0 + tx * 4 + r;
      if (gi < off + n && gj < off + n && gj <= gi) {
        double v = C[gi * ldc + gj] + sgn * T.value(q, r);
        if (gi == gj) v += diag;
        C[gi * ldc + gj] = v;
        if (mirror && gi != gj) C[gj * ldc + gi] = v;
      }
    }
}

// Blocked triangular solves (panels of TRSV_NB rows), one launch per panel:
// with the panel's solved values every remaining row is updated, and CTA 0,
// whose rows are the next diagonal block, goes on to solve that block.  An
// FP64 instruction takes a warp 64 clocks on GB300, so the block is solved as
// two chains of 32 steps (one warp, a row a lane: a product with the
// reciprocal diagonal, a shuffle and a multiply-add a step) with the 32 x 32
// product between them spread over four warps.
constexpr int TRSV_NB = 64;

// Solves the diagonal block Ls (its rows and columns past the matrix are those
// of the identity) for the right-hand side bs, in place; rd, part: scratch.
// All 256 threads call it, with bs and Ls visible to all of them.
template <bool TRANS>
__device__ __forceinline__ void trsv_block(const double (*Ls)[TRSV_NB + 1], double* bs, double* rd,
                                           double (*part)[TRSV_NB]) {
  const int tid = threadIdx.x, l = tid & 31, warp = tid >> 5;
  if (tid < TRSV_NB) rd[tid] = 1.0 / Ls[tid][tid];
  __syncthreads();
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    const int o = (TRANS ? 1 - h : h) * 32;      // rows of this half
    if (warp == 0) {
      double b = bs[o + l];
      const double r = rd[o + l];
#pragma unroll 8
      for (int s = 0; s < 32; ++s) {
        const int j = TRANS ? 31 - s : s;
        const double xj = __shfl_sync(VMC_FULL_MASK, b * r, j);
        const double c = TRANS ? Ls[o + j][o + l] : Ls[o + l][o + j];
        if (l == j) b = xj;
        else if (TRANS ? l < j : l > j) b = fma(-c, xj, b);
      }
      bs[o + l] = b;
    }
    __syncthreads();
    if (h == 0) {   // the other half's right-hand side: a row a lane, eight columns a warp
      const int p = 32 - o;
      if (warp < 4) {
        double acc = 0.0;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          const int j = o + warp * 8 + s;
          acc = fma(TRANS ? Ls[j][p + l] : Ls[p + l][j], bs[j], acc);
        }
        part[warp][l] = acc;
      }
      __syncthreads();
      if (warp == 0) bs[p + l] -= (part[0][l] + part[1][l]) + (part[2][l] + part[3][l]);
      __syncwarp();
    }
  }
}

__device__ __forceinline__ void trsv_load(double (*Ls)[TRSV_NB + 1], const double* __restrict__ L, int64_t ldc,
                                          int64_t k0, int nb) {
#pragma unroll
  for (int q = 0; q < TRSV_NB * TRSV_NB / 256; ++q) {
    const int idx = q * 256 + threadIdx.x, r = idx >> 6, c = idx & 63;
    Ls[r][c] = (r < nb && c < nb) ? L[(k0 + r) * ldc + k0 + c] : (r == c ? 1.0 : 0.0);
  }
}

// Forward: rows i >= k1 take b[i] -= sum_j L[i][k0 + j] b[k0 + j] over the 64
// solved values before k1 (none when k1 = 0), a warp per row, 64 rows a CTA;
// CTA 0 then solves the block at k1.
__global__ void __launch_bounds__(256) k_trsv_fwd(const double* __restrict__ L, int64_t ldc, int64_t n, int64_t k1,
                                                  double* __restrict__ b) {
  __shared__ double Ls[TRSV_NB][TRSV_NB + 1];
  __shared__ double bs[TRSV_NB], rd[TRSV_NB];
  __shared__ double part[4][TRSV_NB];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i0 = k1 + (int64_t)blockIdx.x * TRSV_NB;
  const int nb = (int)(n - k1 < TRSV_NB ? n - k1 : TRSV_NB);
  if (blockIdx.x == 0) trsv_load(Ls, L, ldc, k1, nb);
  double x0 = 0.0, x1 = 0.0;
  if (k1 > 0) { x0 = b[k1 - TRSV_NB + lane]; x1 = b[k1 - 32 + lane]; }
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int r = warp * 8 + q;
    const int64_t i = i0 + r;
    double v = 0.0;
    if (i < n) {
      if (k1 > 0) {
        const double* row = L + i * ldc + k1 - TRSV_NB;
        double acc = row[lane] * x0;
        acc = vmc::warp_sum(fma(row[lane + 32], x1, acc));
        v = b[i] - acc;
      } else {
        v = b[i];
      }
    }
    if (lane == 0) {
      if (blockIdx.x == 0) bs[r] = v;
      else if (i < n) b[i] = v;
    }
  }
  if (blockIdx.x != 0) return;
  __syncthreads();
  trsv_block<false>(Ls, bs, rd, part);
  if (threadIdx.x < nb) b[k1 + threadIdx.x] = bs[threadIdx.x];
}

// Backward: columns j < k1 + 64 take b[j] -= sum_i L[k1 + 64 + i][j] b[k1 + 64 + i]
// over the block of solved values that starts at k1 + 64 (none past n), a
// thread per column and 16 of the block's rows, 64 columns a CTA; CTA 0 holds
// the columns [k1, k1 + 64) and solves that block of L^T.
__global__ void __launch_bounds__(256) k_trsv_bwd(const double* __restrict__ L, int64_t ldc, int64_t n, int64_t k1,
                                                  double* __restrict__ b) {
  __shared__ double Ls[TRSV_NB][TRSV_NB + 1];
  __shared__ double bs[TRSV_NB], rd[TRSV_NB];
  __shared__ double part[4][TRSV_NB];
  const int64_t j0 = k1 - (int64_t)blockIdx.x * TRSV_NB;
  const int64_t s0 = k1 + TRSV_NB;
  const int nb = (int)(n - k1 < TRSV_NB ? n - k1 : TRSV_NB);
  const int ns = (int)(n - s0 < TRSV_NB ? (n > s0 ? n - s0 : 0) : TRSV_NB);
  if (blockIdx.x == 0) trsv_load(Ls, L, ldc, k1, nb);
  const int c = threadIdx.x & 63, h = threadIdx.x >> 6;
  double acc = 0.0;
  if (c < nb || blockIdx.x != 0) {
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int i = h * 16 + q;
      if (i < ns) acc = fma(L[(s0 + i) * ldc + j0 + c], b[s0 + i], acc);
    }
  }
  part[h][c] = acc;
  __syncthreads();
  if (h == 0) {
    double v = 0.0;
    if (c < nb || blockIdx.x != 0) v = b[j0 + c] - ((part[0][c] + part[1][c]) + (part[2][c] + part[3][c]));
    if (blockIdx.x == 0) bs[c] = v;
    else b[j0 + c] = v;
  }
  if (blockIdx.x != 0) return;
  __syncthreads();
  trsv_block<true>(Ls, bs, rd, part);
  if (threadIdx.x < nb) b[k1 + threadIdx.x] = bs[threadIdx.x];
}

// dp[p] = sum_i Oc[i][p] * x[i]; FP32 rows: the product with x = h + m + l (exact,
// split once a CTA and block of rows) as two exact products and the last bits'
template <typename T, int NC>
__global__ void __launch_bounds__(32 * CW) k_gemv_t(const T* __restrict__ Oc, int64_t Ns, int64_t Np, int64_t ldc,
                                                    const double* __restrict__ x, double* __restrict__ dp) {
  __shared__ double part[CW][NC * 32];
  __shared__ float4 xs[2][CB];     // two blocks: the next is written while the last is still read
  __shared__ double xd[2][CB];
  const int64_t p0 = (int64_t)blockIdx.x * (32 * NC) + (threadIdx.x & 31);
  int64_t off[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) off[j] = p0 + 32 * j < Np ? p0 + 32 * j : Np - 1;
  double sum[NC];
  int buf = 1;
  auto begin = [&](int64_t i0) {
    buf ^= 1;
    bool out = false;
    if (threadIdx.x < CB) {
      const double v = i0 + threadIdx.x < Ns ? x[i0 + threadIdx.x] : 0.0;
      xd[buf][threadIdx.x] = v;
      if constexpr (sizeof(T) == 4) {
        float h, m, l;
        out = !split_f64(v, h, m, l);
        xs[buf][threadIdx.x] = make_float4(h, m, l, 0.f);
      }
    }
    return __syncthreads_or(out) == 0;
  };
  auto load = [&](int64_t i, int j) { return Oc[i * ldc + off[j]]; };
  column_sums<T, NC, true>(
      Ns, part, sum, begin, load,
      [&](vmc::Sum3& S, int r, T v) {
        const float o = (float)v;
        const float4 f = xs[buf][r];
        const float p = __fmul_rn(o, f.x), q = __fmul_rn(o, f.y);
        S.add(p);
        S.low(fmaf(o, f.x, -p));
        S.low(q);
        S.d += fmaf(o, f.z, fmaf(o, f.y, -q));
        return p;
      },
      [&](int r, T v) { return (double)v * xd[buf][r]; });
#pragma unroll
  for (int j = 0; j < NC; ++j)
    if (p0 + 32 * j < Np && threadIdx.x < 32) dp[p0 + 32 * j] = sum[j];
}

__global__ void k_rhs(const double* __restrict__ E, int64_t Ns, double Ebar, double scale, double* __restrict__ b) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < Ns) b[i] = (E[i] - Ebar) * scale;
}

__global__ void k_zero(double* __restrict__ p, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = 0.0;
}

}  // namespace

extern "C" {

// Centre and scale O (Ns x Np, ld ldo) into Oc (ld ldc): Oc = (O - mean)/sqrt(Ns).
// dtype codes: 0 = float64, 1 = float32 (for both O and Oc).
int vmc_sr_center(const void* O, int dtype, int64_t Ns, int64_t Np, int64_t ldo, void* Oc, int64_t ldc, double* mean,
                  void* stream) {
  if (Ns <= 0 || Np <= 0 || ldo < Np || ldc < Np || !O || !Oc) return VMC_ERR_ARGS;
  const double scale = 1.0 / sqrt((double)Ns);
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned g1 = (unsigned)((Np + 31) / 32), g4 = (unsigned)((Np + 127) / 128);
  if (dtype == 0)
    k_center<double, 1><<<g1, 32 * CW, 0, st>>>((const double*)O, Ns, Np, ldo, (double*)Oc, ldc, mean, scale);
  else if (dtype == 1 && Np >= CWIDE)
    k_center<float, 4><<<g4, 32 * CW, 0, st>>>((const float*)O, Ns, Np, ldo, (float*)Oc, ldc, mean, scale);
  else if (dtype == 1)
    k_center<float, 1><<<g1, 32 * CW, 0, st>>>((const float*)O, Ns, Np, ldo, (float*)Oc, ldc, mean, scale);
  else
    return VMC_ERR_ARGS;
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

// T (Ns x Ns, FP64, ld ldt) = (accumulate ? T : 0) + Oc Oc^T (+ diag_shift on the diagonal).
int vmc_sr_gram(const void* Oc, int dtype, int64_t Ns, int64_t Np, int64_t ldc, double* T, int64_t ldt,
                double diag_shift, int accumulate, void* stream) {
  if (Ns <= 0 || Np < 0 || ldc < Np || ldt < Ns || !Oc || !T) return VMC_ERR_ARGS;
  cudaStream_t s = (cudaStream_t)stream;
  if (!accumulate) {
    int64_t n = Ns * ldt;
    k_zero<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(T, n);
  }
  int64_t nt = (Ns + TB - 1) / TB;
  if (nt > 65535) return VMC_ERR_ARGS;
  dim3 grid((unsigned)nt, (unsigned)nt);
  if (dtype == 0)
    k_syrk<double, double><<<grid, 256, 0, s>>>((const double*)Oc, ldc, Ns, Np, T, ldt, 0, 1.0, diag_shift, 1);
  else if (dtype == 1)
    k_syrk<float, float><<<grid, 256, 0, s>>>((const float*)Oc, ldc, Ns, Np, T, ldt, 0, 1.0, diag_shift, 1);
  else
    return VMC_ERR_ARGS;
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

// Solve L L^T x = b in place on b (L from vmc_sr_cholesky).
int vmc_sr_cholesky_solve(const double* L, int64_t n, int64_t ldt, double* b, void* stream) {
  if (n <= 0 || ldt < n || !L || !b) return VMC_ERR_ARGS;
  cudaStream_t st = (cudaStream_t)stream;
  for (int64_t k1 = 0; k1 < n; k1 += TRSV_NB)   // L y = b
    k_trsv_fwd<<<(unsigned)((n - k1 + TRSV_NB - 1) / TRSV_NB), 256, 0, st>>>(L, ldt, n, k1, b);
  for (int64_t k1 = ((n - 1) / TRSV_NB) * TRSV_NB; k1 >= 0; k1 -= TRSV_NB)   // L^T x = y
    k_trsv_bwd<<<(unsigned)(k1 / TRSV_NB + 1), 256, 0, st>>>(L, ldt, n, k1, b);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

// b = (E - Ebar)/sqrt(Ns)
int vmc_sr_rhs(const double* E, int64_t Ns, double Ebar, double* b, void* stream) {
  if (Ns <= 0 || !E || !b) return VMC_ERR_ARGS;
  k_rhs<<<(unsigned)((Ns + 255) / 256), 256, 0, (cudaStream_t)stream>>>(E, Ns, Ebar, 1.0 / sqrt((double)Ns), b);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

// dp = Oc^T x
int vmc_sr_update(const void* Oc, int dtype, int64_t Ns, int64_t Np, int64_t ldc, const double* x, double* dp,
                  void* stream) {
  if (Ns <= 0 || Np <= 0 || ldc < Np || !Oc || !x || !dp) return VMC_ERR_ARGS;
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned g1 = (unsigned)((Np + 31) / 32), g4 = (unsigned)((Np + 127) / 128);
  if (dtype == 0)
    k_gemv_t<double, 1><<<g1, 32 * CW, 0, st>>>((const double*)Oc, Ns, Np, ldc, x, dp);
  else if (dtype == 1 && Np >= CWIDE)
    k_gemv_t<float, 4><<<g4, 32 * CW, 0, st>>>((const float*)Oc, Ns, Np, ldc, x, dp);
  else if (dtype == 1)
    k_gemv_t<float, 1><<<g1, 32 * CW, 0, st>>>((const float*)Oc, Ns, Np, ldc, x, dp);
  else
    return VMC_ERR_ARGS;
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

// g = <E O> - Ebar <O>
int vmc_energy_gradient(const void* O, int dtype, int64_t Ns, int64_t Np, int64_t ldo, const double* E, double Ebar,
                        double* g, void* stream) {
  if (Ns <= 0 || Np <= 0 || ldo < Np || !O || !E || !g) return VMC_ERR_ARGS;
  unsigned grid = (unsigned)((Np + 255) / 256);
  if (dtype == 0)
    k_egrad<double><<<grid, 256, 0, (cudaStream_t)stream>>>((const double*)O, Ns, Np, ldo, E, Ebar, g);
  else if (dtype == 1)
    k_egrad<float><<<grid, 256, 0, (cudaStream_t)stream>>>((const float*)O, Ns, Np, ldo, E, Ebar, g);
  else
    return VMC_ERR_ARGS;
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// General GEMM for the factored (Kronecker) SR pieces, CUDA cores:
//   C = beta * C + alpha * (op(A) op(B)) [elementwise * D]
// op(A) is M x K (ta = 0: A[m][k] row-major; ta = 1: A[k][m]), op(B) is K x N
// (tb = 0: B[k][n]; tb = 1: B[n][k]); optional per-k scale s[k] on op(A).
// Inputs FP32 or FP64 (accumulated in FP64 for FP64 inputs, FP32 per 64x64x16
// tile step otherwise), C and D FP64.  lower != 0 computes only tiles with
// tile-row >= tile-col and mirrors them (symmetric results).
// ---------------------------------------------------------------------------
namespace {
template <typename TI, typename TA>
__global__ void k_gemm_gen(int ta, int tb, int64_t M, int64_t N, int64_t K, double alpha, const TI* __restrict__ A,
                           int64_t lda, const TI* __restrict__ Bm, int64_t ldb, const TI* __restrict__ sk,
                           double beta, double* __restrict__ C, int64_t ldc, const double* __restrict__ D,
                           int64_t ldd, int lower) {
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (lower && bj > bi) return;
  __shared__ TA As[TK][TB + 1];
  __shared__ TA Bs[TK][TB + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t m0 = (int64_t)bi * TB, n0 = (int64_t)bj * TB;
  TileAcc<TA> T;
  T.zero();
  for (int64_t k0 = 0; k0 < K; k0 += TK) {
    for (int idx = threadIdx.x; idx < TB * TK; idx += 256) {
      int r, kk;
      if (ta) { kk = idx / TB; r = idx - kk * TB; } else { r = idx / TK; kk = idx - r * TK; }
      const int64_t gm = m0 + r, gk = k0 + kk;
      TA v = 0;
      if (gm < M && gk < K) {
        v = (TA)(ta ? A[gk * lda + gm] : A[gm * lda + gk]);
        if (sk) v *= (TA)sk[gk];
      }
      As[kk][r] = v;
    }
    for (int idx = threadIdx.x; idx < TB * TK; idx += 256) {
      int c, kk;
      if (tb) { c = idx / TK; kk = idx - c * TK; } else { kk = idx / TB; c = idx - kk * TB; }
      const int64_t gn = n0 + c, gk = k0 + kk;
      Bs[kk][c] = (gn < N && gk < K) ? (TA)(tb ? Bm[gn * ldb + gk] : Bm[gk * ldb + gn]) : (TA)0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      TA a[4], b[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) { a[q] = As[kk][ty * 4 + q]; b[q] = Bs[kk][tx * 4 + q]; }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) T.acc[q][r] += a[q] * b[r];
      if ((kk & 3) == 3) T.fold();
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t gm = m0 + ty * 4 + q, gn = n0 + tx * 4 + r;
      if (gm >= M || gn >= N) continue;
      if (lower && gn > gm) continue;
      double v = alpha * T.value(q, r);
      if (D) v *= D[gm * ldd + gn];
      const double out = (beta == 0.0 ? 0.0 : beta * C[gm * ldc + gn]) + v;
      C[gm * ldc + gn] = out;
      if (lower && gm != gn) C[gn * ldc + gm] = out;
    }
}

// The same product for FP32 inputs: the sums of k_gemm_gen<float, float> (four
// products in FP32, then a TwoSum into the double-float accumulator, ascending
// k; equal to the bit), tiled 64 x 64 with 8 x 4 outputs a thread and the next
// 16 columns of K prefetched.  A multiply-add costs 2.75 FP32 instructions (the
// fold is 7 per four), so operand traffic is amortised over 32 outputs: the
// head's four products at 8192 samples 16.4 -> 9.2 ms.
constexpr int DG_T = 64, DG_K = 16, DG_THREADS = 128;

// operand tile of 64 rows x 16: KM: X[r][k], else X[k][r]; sk scales the columns of K
template <bool KM>
__device__ __forceinline__ void dg_load(const float* __restrict__ X, int64_t ld, int64_t r0, int64_t rows, int64_t k0,
                                        int64_t K, const float* __restrict__ sk, float (&v)[8]) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int idx = threadIdx.x + q * DG_THREADS;
    const int64_t r = r0 + (KM ? idx >> 4 : idx & 63), k = k0 + (KM ? idx & 15 : idx >> 6);
    float x = 0.f;
    if (r < rows && k < K) {
      x = KM ? X[r * ld + k] : X[k * ld + r];
      if (sk) x *= sk[k];
    }
    v[q] = x;
  }
}
template <bool KM>
__device__ __forceinline__ void dg_store(float (*s)[DG_T + 4], const float (&v)[8]) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int idx = threadIdx.x + q * DG_THREADS;
    s[KM ? idx & 15 : idx >> 6][KM ? idx >> 4 : idx & 63] = v[q];
  }
}

template <bool TA, bool TB_>
__global__ void __launch_bounds__(DG_THREADS) k_gemm_df(int64_t M, int64_t N, int64_t K, double alpha,
                                                        const float* __restrict__ A, int64_t lda,
                                                        const float* __restrict__ Bm, int64_t ldb,
                                                        const float* __restrict__ sk, double beta,
                                                        double* __restrict__ C, int64_t ldc,
                                                        const double* __restrict__ D, int64_t ldd, int lower) {
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (lower && bj > bi) return;
  __shared__ alignas(16) float As[2][DG_K][DG_T + 4], Bs[2][DG_K][DG_T + 4];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t m0 = (int64_t)bi * DG_T, n0 = (int64_t)bj * DG_T;
  float hi[8][4], lo[8][4];
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int r = 0; r < 4; ++r) hi[q][r] = lo[q][r] = 0.f;
  float pa[8], pb[8];
  dg_load<!TA>(A, lda, m0, M, 0, K, sk, pa);
  dg_load<TB_>(Bm, ldb, n0, N, 0, K, nullptr, pb);
  dg_store<!TA>(As[0], pa);
  dg_store<TB_>(Bs[0], pb);
  __syncthreads();
  int buf = 0;
  for (int64_t k0 = 0; k0 < K; k0 += DG_K) {
    const bool more = k0 + DG_K < K;
    if (more) {
      dg_load<!TA>(A, lda, m0, M, k0 + DG_K, K, sk, pa);
      dg_load<TB_>(Bm, ldb, n0, N, k0 + DG_K, K, nullptr, pb);
    }
#pragma unroll
    for (int g = 0; g < DG_K / 4; ++g) {
      float acc[8][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float* ar = As[buf][g * 4 + u];
        const float4 a0 = *reinterpret_cast<const float4*>(ar + ty * 4);
        const float4 a1 = *reinterpret_cast<const float4*>(ar + 32 + ty * 4);
        const float4 b0 = *reinterpret_cast<const float4*>(&Bs[buf][g * 4 + u][tx * 4]);
        const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        const float b[4] = {b0.x, b0.y, b0.z, b0.w};
#pragma unroll
        for (int q = 0; q < 8; ++q)
#pragma unroll
          for (int r = 0; r < 4; ++r) acc[q][r] = u == 0 ? a[q] * b[r] : fmaf(a[q], b[r], acc[q][r]);
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float x = hi[q][r], y = acc[q][r];
          const float t = x + y, bb = t - x;
          lo[q][r] += (x - (t - bb)) + (y - bb);
          hi[q][r] = t;
        }
    }
    if (more) {
      dg_store<!TA>(As[buf ^ 1], pa);
      dg_store<TB_>(Bs[buf ^ 1], pb);
      __syncthreads();
      buf ^= 1;
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t gm = m0 + (q >> 2) * 32 + ty * 4 + (q & 3), gn = n0 + tx * 4 + r;
      if (gm >= M || gn >= N) continue;
      if (lower && gn > gm) continue;
      double v = alpha * ((double)hi[q][r] + (double)lo[q][r]);
      if (D) v *= D[gm * ldd + gn];
      const double out = (beta == 0.0 ? 0.0 : beta * C[gm * ldc + gn]) + v;
      C[gm * ldc + gn] = out;
      if (lower && gm != gn) C[gn * ldc + gm] = out;
    }
}

// T[a][b] += alpha * (-v[a] - v[b] + c0)
__global__ void k_rank_corr(int64_t n, double* __restrict__ T, int64_t ldt, const double* __restrict__ v, double c0,
                            double alpha) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n * n) return;
  const int64_t a = idx / n, b = idx - a * n;
  T[a * ldt + b] += alpha * (c0 - v[a] - v[b]);
}

// v[a] = sum_k P[a][k] * H[a][k]
template <typename TI>
__global__ void k_rowdot(int64_t n, int64_t K, const double* __restrict__ P, int64_t ldp, const TI* __restrict__ H,
                         int64_t ldh, double* __restrict__ v) {
  const int64_t a = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (a >= n) return;
  double s = 0.0;
  for (int64_t k = lane; k < K; k += 32) s += P[a * ldp + k] * (double)H[a * ldh + k];
  s = vmc::warp_sum(s);
  if (lane == 0) v[a] = s;
}
}  // namespace

extern "C" {

int vmc_gemm(int ta, int tb, int64_t M, int64_t N, int64_t K, double alpha, const void* A, int64_t lda, const void* B,
             int64_t ldb, const void* sk, int dtype, double beta, double* C, int64_t ldc, const double* D,
             int64_t ldd, int lower, void* stream) {
  if (M <= 0 || N <= 0 || K < 0 || !A || !B || !C || (dtype != 0 && dtype != 1)) return VMC_ERR_ARGS;
  if (lower && M != N) return VMC_ERR_ARGS;
  const int64_t mt = (M + TB - 1) / TB, nt = (N + TB - 1) / TB;
  if (mt > 65535) return VMC_ERR_ARGS;
  dim3 grid((unsigned)nt, (unsigned)mt);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == 0)
    k_gemm_gen<double, double><<<grid, 256, 0, s>>>(ta, tb, M, N, K, alpha, (const double*)A, lda, (const double*)B,
                                                     ldb, (const double*)sk, beta, C, ldc, D, ldd, lower);
  else if (ta && tb)
    k_gemm_df<true, true><<<grid, DG_THREADS, 0, s>>>(M, N, K, alpha, (const float*)A, lda, (const float*)B, ldb,
                                                      (const float*)sk, beta, C, ldc, D, ldd, lower);
  else if (ta)
    k_gemm_df<true, false><<<grid, DG_THREADS, 0, s>>>(M, N, K, alpha, (const float*)A, lda, (const float*)B, ldb,
                                                       (const float*)sk, beta, C, ldc, D, ldd, lower);
  else if (tb)
    k_gemm_df<false, true><<<grid, DG_THREADS, 0, s>>>(M, N, K, alpha, (const float*)A, lda, (const float*)B, ldb,
                                                       (const float*)sk, beta, C, ldc, D, ldd, lower);
  else
    k_gemm_df<false, false><<<grid, DG_THREADS, 0, s>>>(M, N, K, alpha, (const float*)A, lda, (const float*)B, ldb,
                                                        (const float*)sk, beta, C, ldc, D, ldd, lower);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

int vmc_sr_kron_correction(int64_t n, double* T, int64_t ldt, const double* P, int64_t ldp, const void* H, int dtype,
                           int64_t ldh, int64_t K, double mu_sq, double alpha, double* v_work, void* stream) {
  if (n <= 0 || K <= 0 || !T || !P || !H || !v_work || (dtype != 0 && dtype != 1)) return VMC_ERR_ARGS;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == 0)
    k_rowdot<double><<<(unsigned)((n + 7) / 8), 256, 0, s>>>(n, K, P, ldp, (const double*)H, ldh, v_work);
  else
    k_rowdot<float><<<(unsigned)((n + 7) / 8), 256, 0, s>>>(n, K, P, ldp, (const float*)H, ldh, v_work);
  const int64_t nn = n * n;
  k_rank_corr<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(n, T, ldt, v_work, mu_sq, alpha);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

}  // extern "C"
