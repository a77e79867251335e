// Sample-space SR Gram matrix on the tensor cores:
//
//   T (Ns x Ns, FP64) [+]= alpha * (X X^T) o D  (+ shift I)
//
// for an FP32 matrix X (Ns x K): the per-sample log-derivatives, centred and
// scaled (the dense block of O), or the Kronecker factor G of the NNBF output
// layer (with D = H H^T).  Fixed-point split (the Ozaki scheme's idea): each
// row i gets a shared power-of-two exponent E_i (its largest |x| below
// 2^E_i), and y = x 2^-E_i is written as three 7-bit integer digits,
//   y = 2^-6 a0 + 2^-13 a1 + 2^-20 a2,  a_s in [-64, 64]
// (to 2^-20 of the row's largest entry), each digit scaled by its power of two
// exactly representable in BF16.  The product y_i y_j is taken as all nine
// digit products (hi, mid, lo the three planes), so the result is exactly the
// Gram matrix of the rounded rows and stays positive semidefinite.  The
// leading term hi hi is an integer multiple of 2^-12 of magnitude <= 1, so its
// FP32 running sum over a 2048-column chunk (<= 2^23 units) is exact: it
// accumulates in its own TMEM accumulator with no rounding at all.  The eight
// small terms (2^-7 of it and below) share a second accumulator, where FP32
// rounding is ~2^-25 of 2^-7 of the result.
// Both are drained every 2048 columns of K into a running sum of each output,
// two FP32 numbers in registers (exact error terms, ~2^-48 of the sum): an FP64
// instruction holds a warp's scheduler for 64 clocks, and the drain into FP64 T
// with its conversions, exponents and scattered read-modify-writes took as
// long as the chunk's products (8192 samples, 115 K + 8 K columns: 58.7 -> 38.2
// ms).  The FP64 result, scaled by 2^(E_i + E_j), is formed once a tile and goes
// through shared memory so that T and D are read and written along their rows.
//
// Tile: 128 x 128 outputs per CTA, lower triangle of tiles only (the upper
// triangle is written as the mirror image).  K atoms of 64 BF16 (128 bytes per
// row) are staged by TMA (SWIZZLE_128B) through a 2-stage pipeline; each stage
// holds the three planes of the 128 rows of both operands (96 KB).  Warp 0
// issues the copies, warp 1 (one thread) the tcgen05 MMAs into two TMEM
// buffers used alternately per K chunk (each 2 x 128 columns: leading and
// small products), warps 2..9 (two a TMEM lane quadrant) hold the running sums.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include "common.cuh"
#include "tc.cuh"

namespace {

constexpr int GT = 128;                       // tile rows / cols
constexpr int KA = 64;                        // bf16 per K atom (128 bytes)
constexpr int PLANE = GT * KA * 2;            // 16 KB: one plane of one operand, one atom
constexpr int STAGE = 6 * PLANE;              // A hi/mid/lo + B hi/mid/lo
constexpr int NSTAGE = 2;
constexpr int CHUNK_ATOMS = 32;               // 2048 columns of K per FP32 accumulation
constexpr int GR_THREADS = 320;
constexpr int EC = GT / 2;                    // columns per epilogue warp
constexpr int GR_SMEM = NSTAGE * STAGE + 1024 + 256;

// Row exponents: E[r] = ilogb(max_k |X[r][k]|) + 1 (0 for a zero row or a
// padding row), one CTA per row; eight loads a thread in flight.
__global__ void __launch_bounds__(256) k_row_exp(const float* __restrict__ X, int64_t rows, int64_t rows_pad, int64_t K,
                                                 int64_t ldx, int* __restrict__ E) {
  __shared__ unsigned wmax[8];
  const int64_t r = (int64_t)blockIdx.y * INT32_MAX + blockIdx.x;
  if (r >= rows_pad) return;
  const float* x = X + r * ldx;
  float m = 0.f;
  if (r < rows) {
    int64_t c = threadIdx.x;
    for (; c + 7 * 256 < K; c += 8 * 256) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = x[c + u * 256];
#pragma unroll
      for (int u = 0; u < 8; ++u) m = fmaxf(m, fabsf(v[u]));
    }
    for (; c < K; c += 256) m = fmaxf(m, fabsf(x[c]));
  }
  const unsigned b = __reduce_max_sync(VMC_FULL_MASK, __float_as_uint(m));   // m >= 0: ordered as its bits
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned t = wmax[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) t = max(t, wmax[w]);
    m = __uint_as_float(t);
    E[r] = (m > 0.f && m < INFINITY) ? ilogbf(m) + 1 : 0;
  }
}

// x -> (hi, mid, lo) planes of the fixed-point digits of x 2^-E[r] (plane p at
// P + p * plane), row-major with row stride kp; rows >= `rows` and columns >=
// K are zero.  Every step below is exact in FP32: scaling by powers of two,
// rounding to an integer, and the subtraction of that integer from a value
// within 0.5 of it.  HBM is the limit (10 bytes an entry; 8192 x
// 123 K: 4.2 ms with a division and three ldexp an entry, 2.0 now with the row
// exponents): SPLIT_CU columns a
// thread in flight, a row's blocks along x and the rows along y and z.
constexpr int SPLIT_CU = 8;

__global__ void __launch_bounds__(256) k_split3(const float* __restrict__ X, int64_t rows, int64_t rows_pad, int64_t K,
                                                int64_t ldx, int64_t kp, const int* __restrict__ E,
                                                __nv_bfloat16* __restrict__ P) {
  const int64_t r = (int64_t)blockIdx.z * 65535 + blockIdx.y;
  if (r >= rows_pad) return;
  // 2^6 x 2^-E in two factors: 2^(6 - E) itself may lie outside FP32
  const int k = 6 - E[r], k1 = k >> 1;
  const float s1 = __int_as_float((127 + k1) << 23), s2 = __int_as_float((127 + k - k1) << 23);
  const int64_t c0 = (int64_t)blockIdx.x * (256 * SPLIT_CU) + threadIdx.x, plane = rows_pad * kp;
  float x[SPLIT_CU];
#pragma unroll
  for (int u = 0; u < SPLIT_CU; ++u) {
    const int64_t c = c0 + u * 256;
    x[u] = (r < rows && c < K) ? X[r * ldx + c] : 0.f;
  }
  __nv_bfloat16* p = P + r * kp;
#pragma unroll
  for (int u = 0; u < SPLIT_CU; ++u) {
    const int64_t c = c0 + u * 256;
    if (c >= kp) return;
    const float y = x[u] * s1 * s2;            // |y| < 64
    const float a0 = rintf(y);
    const float r1 = (y - a0) * 128.f;         // |r1| <= 64
    const float a1 = rintf(r1);
    const float a2 = rintf((r1 - a1) * 128.f);
    p[c] = __float2bfloat16_rn(a0 * 0x1p-6f);
    p[plane + c] = __float2bfloat16_rn(a1 * 0x1p-13f);
    p[2 * plane + c] = __float2bfloat16_rn(a2 * 0x1p-20f);
  }
}

struct GramArgs {
  double* T;
  int64_t ldt;
  const double* D;   // nullable, ld = ldt
  const int* E;      // row exponents of the split
  double alpha, shift;
  int n;             // rows of X (order of T)
  int prow;          // rows per plane (n rounded up to the tile)
  int n_atoms, accumulate;
};

// tile index -> (bi, bj), bj <= bi, row-major over the lower triangle
__device__ __forceinline__ void tile_of(int t, int& bi, int& bj) {
  int i = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
  while ((i + 1) * (i + 2) / 2 <= t) ++i;
  while (i * (i + 1) / 2 > t) --i;
  bi = i;
  bj = t - i * (i + 1) / 2;
}

// t 2^e in the exponent field: t is 0, not finite, or of an exponent between
// FP32's least and 2^31, and |e| < 300
__device__ __forceinline__ double scale2(double t, int e) {
  const int h = __double2hiint(t), f = (h >> 20) & 0x7ff;
  return f == 0 || f == 0x7ff ? t : __hiloint2double(h + (e << 20), __double2loint(t));
}

__global__ void __launch_bounds__(GR_THREADS, 1)
    k_gram_bf16x3(const __grid_constant__ CUtensorMap tmX, GramArgs ga, int* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bar = (uint64_t*)(sm + NSTAGE * STAGE);
  uint64_t* full = bar;          // [NSTAGE]
  uint64_t* empty = bar + 2;     // [NSTAGE]
  uint64_t* tfull = bar + 4;     // [2]
  uint64_t* tempty = bar + 6;    // [2]
  uint32_t* tslot = (uint32_t*)(bar + 8);
  volatile int* abort_flag = (volatile int*)(bar + 9);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int bi, bj;
  tile_of(blockIdx.x, bi, bj);
  const int n_chunks = (ga.n_atoms + CHUNK_ATOMS - 1) / CHUNK_ATOMS;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { tc::mbar_init(&tfull[b], 1); tc::mbar_init(&tempty[b], 8); }
    *abort_flag = 0;
    tc::fence_mbar_init();
    tc::prefetch_tmap(&tmX);
  }
  if (warp == 0) tc::tmem_alloc(tslot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *tslot;
  if (warp == 0) {
    if (lane == 0) {  // ---- TMA producer: atom a -> stage a % NSTAGE ----
      for (int a = 0; a < ga.n_atoms && !*abort_flag; ++a) {
        const int s = a % NSTAGE;
        if (a >= NSTAGE && !tc::mbar_wait(&empty[s], ((a / NSTAGE) - 1) & 1)) {
          *abort_flag = 1;
          atomicExch(err, VMC_ERR_TIMEOUT);
          break;
        }
        tc::mbar_arrive_expect_tx(&full[s], STAGE);
        uint8_t* st = sm + s * STAGE;
#pragma unroll
        for (int p = 0; p < 3; ++p) {   // plane p of the rows of tile bi (A) and of tile bj (B)
          tc::tma_load_2d(st + p * PLANE, &tmX, &full[s], a * KA, p * ga.prow + bi * GT);
          tc::tma_load_2d(st + (3 + p) * PLANE, &tmX, &full[s], a * KA, p * ga.prow + bj * GT);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // ---- MMA issuer ----
      constexpr uint32_t idesc = tc::idesc_bf16_f32(GT, GT);
      // (A plane, B plane) of the nine products: the leading one, then the rest
      constexpr int pa[9] = {0, 0, 1, 0, 2, 1, 1, 2, 2};
      constexpr int pb[9] = {0, 1, 0, 2, 0, 1, 2, 1, 2};
      for (int c = 0; c < n_chunks && !*abort_flag; ++c) {
        const int buf = c & 1;
        if (c >= 2 && !tc::mbar_wait(&tempty[buf], ((c >> 1) - 1) & 1)) {
          *abort_flag = 1;
          atomicExch(err, VMC_ERR_TIMEOUT);
          break;
        }
        tc::fence_after_sync();
        const uint32_t dt = tbase + (uint32_t)(buf * 2 * GT);   // leading products; small ones at + GT
        const int a0 = c * CHUNK_ATOMS, a1 = min(ga.n_atoms, a0 + CHUNK_ATOMS);
        bool ok = true;
        for (int a = a0; a < a1; ++a) {
          const int s = a % NSTAGE;
          if (!tc::mbar_wait(&full[s], (a / NSTAGE) & 1)) { ok = false; break; }
          tc::fence_after_sync();
          const uint8_t* st = sm + s * STAGE;
#pragma unroll
          for (int q = 0; q < 9; ++q) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const uint64_t ad = tc::sdesc_sw128(tc::smem_u32(st + pa[q] * PLANE) + kk * 32);
              const uint64_t bd = tc::sdesc_sw128(tc::smem_u32(st + (3 + pb[q]) * PLANE) + kk * 32);
              if (q == 0) tc::mma_bf16(dt, ad, bd, idesc, (a > a0 || kk) ? 1u : 0u);
              else tc::mma_bf16(dt + GT, ad, bd, idesc, (a > a0 || q > 1 || kk) ? 1u : 0u);
            }
          }
          tc::mma_commit(&empty[s]);   // the stage is free once these MMAs have read it
        }
        if (!ok) { *abort_flag = 1; atomicExch(err, VMC_ERR_TIMEOUT); break; }
        tc::mma_commit(&tfull[buf]);
      }
    }
  } else {  // ---- epilogue: warps 2..9, TMEM lane quadrant warp % 4, half of the columns each ----
    const int quad = warp & 3, half = (warp - 2) >> 2;
    float hi[EC], lo[EC];
#pragma unroll
    for (int q = 0; q < EC; ++q) hi[q] = lo[q] = 0.f;
    bool ok = true;
    for (int c = 0; c < n_chunks; ++c) {
      const int buf = c & 1;
      ok = tc::mbar_wait(&tfull[buf], (c >> 1) & 1);
      ok = __all_sync(VMC_FULL_MASK, ok);
      if (!ok) { if (lane == 0) { *abort_flag = 1; atomicExch(err, VMC_ERR_TIMEOUT); } break; }
      tc::fence_after_sync();
      const uint32_t ta = tbase + (uint32_t)(buf * 2 * GT + half * EC) + ((uint32_t)(quad * 32) << 16);
#pragma unroll
      for (int g = 0; g < EC / 8; ++g) {
        float v[8], w[8];
        tc::tmem_ld8x2(ta + (uint32_t)(g * 8), GT, v, w);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          float h = hi[g * 8 + q];
          const float e = vmc::two_sum(h, v[q]), f = vmc::two_sum(h, w[q]);
          hi[g * 8 + q] = h;
          lo[g * 8 + q] += e + f;
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(&tempty[buf])) : "memory");
    }
    if (ok) {
      // the loads and MMAs of the tile are complete: their stages become the
      // warps' transpose buffers
      double* tb = reinterpret_cast<double*>(sm) + (warp - 2) * (32 * (EC + 1));
      const int r0 = bi * GT + quad * 32, c0 = bj * GT + half * EC;
      const int gi = r0 + lane;
      const int ej[2] = {ga.E[c0 + lane], ga.E[c0 + 32 + lane]};   // padding rows have one too
#pragma unroll
      for (int q = 0; q < EC; ++q) reinterpret_cast<float2*>(tb)[lane * (EC + 1) + q] = make_float2(hi[q], lo[q]);
      __syncwarp();
#pragma unroll 1
      for (int rb = 0; rb < 32; rb += 4) {   // four rows of T and D in flight at a time
        double t[4][2], d[4][2];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int64_t row = r0 + rb + u, col = c0 + 32 * h + lane;
            const bool in = row < ga.n && col <= row;
            t[u][h] = in && ga.accumulate ? ga.T[row * ga.ldt + col] : 0.0;
            d[u][h] = in && ga.D ? ga.D[row * ga.ldt + col] : 1.0;
          }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int64_t row = r0 + rb + u, col = c0 + 32 * h + lane;
            double* b = &tb[(rb + u) * (EC + 1) + 32 * h + lane];
            const float2 x = *reinterpret_cast<const float2*>(b);
            double val = ga.alpha * scale2((double)x.x + (double)x.y, ga.E[row] + ej[h]);
            if (ga.D) val *= d[u][h];
            if (ga.accumulate) val += t[u][h];
            if (row == col) val += ga.shift;
            if (row < ga.n && col <= row) ga.T[row * ga.ldt + col] = val;
            *b = val;
          }
      }
      __syncwarp();
      for (int q = 0; q < EC; ++q) {     // along the rows of the mirror image
        const int64_t gj = c0 + q;
        if (gi < ga.n && gj < gi) ga.T[gj * ga.ldt + gi] = tb[lane * (EC + 1) + q];
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tbase, 512);
}

PFN_cuTensorMapEncodeTiled_v12000 g_enc = nullptr;

// The three planes stacked as one (3 rows, kp) bf16 matrix: box {64, 128}, SWIZZLE_128B.
bool tmap_planes(CUtensorMap* m, const void* base, uint64_t rows3, uint64_t kp) {
  if (!g_enc) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return false;
    g_enc = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  }
  if (((uintptr_t)base & 15) != 0 || (kp * 2) % 16 != 0) return false;
  cuuint64_t gdim[2] = {(cuuint64_t)kp, (cuuint64_t)rows3};
  cuuint64_t gstr[1] = {(cuuint64_t)kp * 2};
  cuuint32_t box[2] = {KA, GT};
  cuuint32_t es[2] = {1, 1};
  return g_enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), gdim, gstr, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr int kMaxDev = 64;
bool g_gram_attr[kMaxDev] = {};

}  // namespace

extern "C" {

// planes: 3 * rows_pad * kp bf16 workspace, rows_pad = rows rounded up to 128,
// kp = K rounded up to 64.  Rows beyond `rows` are zeroed.
int vmc_split_bf16x3(const float* X, int64_t rows, int64_t K, int64_t ldx, void* planes, int64_t rows_pad,
                     int64_t kp, int* row_exp, void* stream) {
  if (rows < 0 || K < 0 || ldx < K || rows_pad < rows || rows_pad % GT != 0 || kp < K || kp % KA != 0 ||
      (rows > 0 && (!X || !planes)) || (rows_pad > 0 && !row_exp))
    return VMC_ERR_ARGS;
  if (rows_pad == 0) return VMC_OK;
  const dim3 egrid((unsigned)(rows_pad < INT32_MAX ? rows_pad : INT32_MAX), (unsigned)((rows_pad + INT32_MAX - 1) / INT32_MAX));
  k_row_exp<<<egrid, 256, 0, (cudaStream_t)stream>>>(X, rows, rows_pad, K, ldx, row_exp);
  VMC_CUDA_CHECK_LAUNCH();
  if (kp == 0) return VMC_OK;
  const dim3 grid((unsigned)((kp + 256 * SPLIT_CU - 1) / (256 * SPLIT_CU)), (unsigned)(rows_pad < 65535 ? rows_pad : 65535),
                  (unsigned)((rows_pad + 65534) / 65535));
  k_split3<<<grid, 256, 0, (cudaStream_t)stream>>>(X, rows, rows_pad, K, ldx, kp, row_exp, (__nv_bfloat16*)planes);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

int vmc_sr_gram_tc(const void* planes, const int* row_exp, int64_t ns, int64_t rows_pad, int64_t kp, double alpha,
                   double* T, int64_t ldt, const double* D, double diag_shift, int accumulate, int* d_err,
                   void* stream) {
  if (ns <= 0 || rows_pad < ns || rows_pad % GT != 0 || kp <= 0 || kp % KA != 0 || ldt < ns || !planes || !T ||
      !d_err || !row_exp || ns > (1 << 30))
    return VMC_ERR_ARGS;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return VMC_ERR_CUDA;
  if (!g_gram_attr[dev]) {
    if (cudaFuncSetAttribute(k_gram_bf16x3, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM) != cudaSuccess)
      return VMC_ERR_CUDA;
    g_gram_attr[dev] = true;
  }
  CUtensorMap tm;
  if (!tmap_planes(&tm, planes, (uint64_t)(3 * rows_pad), (uint64_t)kp)) return VMC_ERR_UNSUPPORTED;
  const int nt = (int)(rows_pad / GT);
  GramArgs ga{T, ldt, D, row_exp, alpha, diag_shift, (int)ns, (int)rows_pad, (int)(kp / KA), accumulate};
  const int n_tiles = nt * (nt + 1) / 2;
  k_gram_bf16x3<<<(unsigned)n_tiles, GR_THREADS, GR_SMEM, (cudaStream_t)stream>>>(tm, ga, d_err);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

}  // extern "C"
