// FP64 symmetric products on the tensor cores, for the minSR step:
//   gram     C (n, n) [+]= X X^T (+ shift I), the full symmetric matrix
//   update   C -= L L^T on the lower triangle of a trailing matrix (Cholesky)
//
// Fixed-point digits (the Ozaki scheme): each row i gets a power-of-two
// exponent E_i above its largest entry, and x 2^(55 - E_i), rounded to an
// integer (56 bits and sign: the row to 2^-56 of its largest entry, finer than
// FP64's own 2^-53 for entries within a factor 8 of it), is written as seven
// balanced base-256 digits d_0 .. d_6 in [-128, 128], each exact in BF16.  A
// product x_i x_j is the sum of the digit products d_p d_q of level p + q with
// weight 2^(-14 - 8 (p + q)); the 28 products of levels 0..6 are formed.  What is
// left out is at most 6 x 2^-56 of 2^(E_i + E_j) per term (level 7), and the
// operands' rounding 2 x 2^-56 of it: with 2^E at most twice the largest entry,
// 36 x 2^-56 of the two rows' largest entries' product.  The error thus scales
// with those, not with the sum of |x_ik x_jk| as that of FP64 multiply-adds
// does: below theirs where the rows' entries are of one size, above where the
// large entries of two rows stand in different columns (vmc_sr_gram is the
// choice there); relative to sqrt(T_ii T_jj) it is below K 36 x 2^-56 always,
// like the error that a Cholesky factorisation of T commits by itself.
//
// All products of one level share a TMEM accumulator: integers of at most 2^14,
// so 256 columns of K sum to at most 2^22 times the level's products.  Levels 0
// to 3 (one to four products) stay within FP32's 2^24 exact integers, level 4
// (five) has two accumulators of three and two, and is exact as well.  Levels 5
// and 6 (six and seven) pass 2^24 where digits share a sign, and lose a unit or
// two in the additions beyond it, which is 2^-54 and 2^-62 of 2^(E_i + E_j).
// (Level 4 in one accumulator lost units of 2^-46 there.)  Every 256 columns
// the levels are combined as one 64-bit integer (unit 2^-54) and added in FP64.
//
// On GB300 FP64 arithmetic runs at 2 multiply-adds a clock per SM (1.25
// TFLOP/s), BF16 tcgen05 at 1.9 PFLOP/s measured: 28 products leave 34
// TFLOP/s per executed multiply-add pair of the FP64 result, 54x.
//
// Tile: 128 x 64 outputs per CTA (8 accumulators x 64 columns: all 512 TMEM
// columns).  K atoms of 32 (SWIZZLE_64B) so that two
// stages of all seven planes of both operands (84 KB each) fit shared memory;
// one 3-D TMA load per operand and stage brings the seven planes.  Warp 0
// issues the copies, warp 1 (one thread) the MMAs, warps 2..5 combine.
#include <mutex>
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include "common.cuh"
#include "tc.cuh"

namespace {

constexpr int ND = 7;                          // digits per entry, levels per product
constexpr int SPLIT_LV = 4, SPLIT_P = 3;       // products p >= SPLIT_P of level SPLIT_LV: an accumulator of their own
constexpr int NACC = ND + 1;
constexpr int OM = 128, ON = 64;               // tile
constexpr int OK = 32;                         // K atom (64 bytes of BF16)
constexpr int APLANE = OM * OK * 2, BPLANE = ON * OK * 2;
constexpr int OSTAGE = ND * (APLANE + BPLANE);
constexpr int ONST = 2;
constexpr int CHUNK = 256 / OK;                // atoms per drain
constexpr int OZ_THREADS = 192;
constexpr int OZ_SMEM = ONST * OSTAGE + 1024 + 256;
constexpr int BAD_ROW = INT32_MIN;             // exponent of a row holding a NaN or Inf

// TPR threads per row (a warp for short rows, the CTA for long ones): exponent,
// then digits.  Integer arithmetic on the FP64 bit patterns throughout (the
// FP64 pipe is the scarce one).  Rows >= `rows` and columns >= K of the planes
// are zero.
template <int TPR>
__global__ void __launch_bounds__(128) k_split_f64(const double* __restrict__ X, int64_t rows, int64_t rows_pad,
                                                   int64_t K, int64_t ldx, int64_t kp, int* __restrict__ E,
                                                   __nv_bfloat16* __restrict__ P) {
  __shared__ int wmax[4];
  const int t = threadIdx.x % TPR;
  const int64_t r = (int64_t)blockIdx.x * (128 / TPR) + threadIdx.x / TPR;   // rows_pad is a multiple of 128
  const bool live = r < rows;
  const long long* x = reinterpret_cast<const long long*>(X + (live ? r : 0) * ldx);
  int m = 0;
  if (live)
    for (int64_t c = t; c < K; c += TPR) m = max(m, (int)((unsigned long long)(x[c] << 1) >> 53));
  m = __reduce_max_sync(VMC_FULL_MASK, m);
  if (TPR > 32) {
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
    __syncthreads();
    m = max(max(wmax[0], wmax[1]), max(wmax[2], wmax[3]));
  }
  const bool bad = m == 0x7ff;
  if (t == 0) E[r] = bad ? BAD_ROW : (m ? m - 1022 : 0);
  const int64_t plane = rows_pad * kp;
  for (int64_t c0 = (int64_t)t * 4; c0 < kp; c0 += TPR * 4) {
    __nv_bfloat16 d[ND][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long long b = (live && !bad && c0 + q < K) ? x[c0 + q] : 0;
      const int e = (int)((unsigned long long)(b << 1) >> 53);
      const long long mant = e ? ((b & 0xFFFFFFFFFFFFFll) | 0x10000000000000ll) : 0;   // subnormals count as zero
      const int down = m - e - 2;      // right shift that leaves units of 2^(E - 55)
      long long v = down <= 0 ? mant << -down : (down > 54 ? 0 : (mant + (1ll << (down - 1))) >> down);
      if (b < 0) v = -v;
#pragma unroll
      for (int p = ND - 1; p > 0; --p) {
        const int dg = (int)((v + 128) & 255) - 128;
        d[p][q] = __int2bfloat16_rn(dg);
        v = (v - dg) >> 8;
      }
      d[0][q] = __int2bfloat16_rn((int)v);
    }
#pragma unroll
    for (int p = 0; p < ND; ++p) {
      const __nv_bfloat162 lo = __halves2bfloat162(d[p][0], d[p][1]), hi = __halves2bfloat162(d[p][2], d[p][3]);
      *reinterpret_cast<uint2*>(P + p * plane + r * kp + c0) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  }
}

struct OzArgs {
  double* C;
  int64_t ldc;
  const int* E;
  double shift;
  int neg;          // 1: subtract the product
  int n;            // order of C (rows of X)
  int ncols;        // columns of C that are wanted (n for the whole lower triangle)
  int n_atoms;
  int beta;         // 1: add to C, 0: overwrite
  int mirror;       // 1: write the upper triangle too
};

// tile index -> (bi, bj) with bj <= 2 bi + 1 (64-column tiles that touch the
// lower triangle of the 128-row tile bi): bi (bi + 1) tiles precede row bi
__device__ __forceinline__ void oz_tile(int t, int& bi, int& bj) {
  int i = (int)((sqrtf(4.f * (float)t + 1.f) - 1.f) * 0.5f);
  while ((i + 1) * (i + 2) <= t) ++i;
  while (i * (i + 1) > t) --i;
  bi = i;
  bj = t - i * (i + 1);
}

// t (units 2^(ei + ej - 54)) as FP64, negated if neg; NaN for a bad row or
// column.  The power of two goes into the exponent field (t is 0 or at least
// 1 in magnitude): an FP64 multiplication costs a warp 64 clocks here.
__device__ __forceinline__ double oz_scale(double t, int ei, int ej, int neg) {
  if (ei == BAD_ROW || ej == BAD_ROW) return __longlong_as_double(0x7ff8000000000000ll);
  const int e = ei + ej - 54;
  const int h = __double2hiint(t), f = (h >> 20) & 0x7ff;
  if (f == 0) return 0.0;
  if (f + e > 0 && f + e < 0x7ff)
    return __hiloint2double((h + (e << 20)) ^ (neg ? 0x80000000 : 0), __double2loint(t));
  return ldexp(neg ? -t : t, e);
}

__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_syrk_f64tc(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, OzArgs oa,
                 int* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bar = (uint64_t*)(sm + ONST * OSTAGE);
  uint64_t* full = bar;          // [ONST]
  uint64_t* empty = bar + 2;     // [ONST]
  uint64_t* tfull = bar + 4;
  uint64_t* tempty = bar + 5;
  uint32_t* tslot = (uint32_t*)(bar + 6);
  volatile int* abort_flag = (volatile int*)(bar + 7);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int bi, bj;
  if (oa.ncols < oa.n) {   // the leading columns of a panel: row-major over (row tile, column tile)
    const int nct = (oa.ncols + ON - 1) / ON;
    bi = blockIdx.x / nct;
    bj = blockIdx.x - bi * nct;
    if (bj > 2 * bi + 1) return;
  } else {
    oz_tile(blockIdx.x, bi, bj);
  }
  if (bj * ON >= oa.ncols) return;
  const int n_chunks = (oa.n_atoms + CHUNK - 1) / CHUNK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ONST; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
    tc::mbar_init(tfull, 1);
    tc::mbar_init(tempty, 4);
    *abort_flag = 0;
    tc::fence_mbar_init();
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
  }
  if (warp == 0) tc::tmem_alloc(tslot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *tslot;
  if (warp == 0) {
    if (lane == 0) {  // ---- TMA producer: atom a -> stage a % ONST ----
      for (int a = 0; a < oa.n_atoms && !*abort_flag; ++a) {
        const int s = a % ONST;
        if (a >= ONST && !tc::mbar_wait(&empty[s], ((a / ONST) - 1) & 1)) {
          *abort_flag = 1;
          atomicExch(err, VMC_ERR_TIMEOUT);
          break;
        }
        tc::mbar_arrive_expect_tx(&full[s], OSTAGE);
        uint8_t* st = sm + s * OSTAGE;
        tc::tma_load_3d(st, &tmA, &full[s], a * OK, bi * OM, 0);
        tc::tma_load_3d(st + ND * APLANE, &tmB, &full[s], a * OK, bj * ON, 0);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // ---- MMA issuer ----
      constexpr uint32_t idesc = tc::idesc_bf16_f32(OM, ON);
      bool ok = true;
      for (int c = 0; c < n_chunks && ok && !*abort_flag; ++c) {
        if (c > 0 && !tc::mbar_wait(tempty, (c - 1) & 1)) { ok = false; break; }
        tc::fence_after_sync();
        const int a0 = c * CHUNK, a1 = min(oa.n_atoms, a0 + CHUNK);
        for (int a = a0; a < a1; ++a) {
          const int s = a % ONST;
          if (!tc::mbar_wait(&full[s], (a / ONST) & 1)) { ok = false; break; }
          tc::fence_after_sync();
          const uint32_t sa = tc::smem_u32(sm + s * OSTAGE), sb = sa + ND * APLANE;
#pragma unroll
          for (int lv = 0; lv < ND; ++lv)
#pragma unroll
            for (int p = 0; p <= lv; ++p)
#pragma unroll
              for (int kk = 0; kk < OK / 16; ++kk) {
                const bool own = lv == SPLIT_LV && p >= SPLIT_P;
                tc::mma_bf16(tbase + (uint32_t)((own ? ND : lv) * ON), tc::sdesc_sw64(sa + p * APLANE + kk * 32),
                             tc::sdesc_sw64(sb + (lv - p) * BPLANE + kk * 32), idesc,
                             (a > a0 || p != (own ? SPLIT_P : 0) || kk) ? 1u : 0u);
              }
          tc::mma_commit(&empty[s]);   // the stage is free once these MMAs have read it
        }
        if (ok) tc::mma_commit(tfull);
      }
      if (!ok) { *abort_flag = 1; atomicExch(err, VMC_ERR_TIMEOUT); }
    }
  } else {  // ---- warps 2..5: TMEM lane quadrant warp % 4, one output row per lane ----
    const int quad = warp & 3;
    const int64_t gi = (int64_t)bi * OM + quad * 32 + lane;
    double acc[ON];
#pragma unroll
    for (int q = 0; q < ON; ++q) acc[q] = 0.0;
    bool ok = true;
    for (int c = 0; c < n_chunks; ++c) {
      ok = tc::mbar_wait(tfull, c & 1);
      ok = __all_sync(VMC_FULL_MASK, ok);
      if (!ok) { if (lane == 0) { *abort_flag = 1; atomicExch(err, VMC_ERR_TIMEOUT); } break; }
      tc::fence_after_sync();
#pragma unroll
      for (int g = 0; g < ON / 8; ++g) {
        uint32_t v[NACC][8];
        tc::tmem_ld8x8(tbase + ((uint32_t)(quad * 32) << 16) + (uint32_t)(g * 8), ON, v);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          int lv[ND];
#pragma unroll
          for (int p = 0; p < ND; ++p) lv[p] = __float2int_rn(__uint_as_float(v[p][q]));
          lv[SPLIT_LV] += __float2int_rn(__uint_as_float(v[ND][q]));
          // levels 0..3 in units of 2^-38, 4..6 in units of 2^-62; together in 2^-54
          const long long hi = ((((long long)lv[0] * 256 + lv[1]) * 256 + lv[2]) * 256) + lv[3];
          const long long lo = (((long long)lv[4] * 256 + lv[5]) * 256) + lv[6];
          const double t = (double)(hi * 65536 + ((lo + 128) >> 8));
          acc[g * 8 + q] = c == 0 ? t : acc[g * 8 + q] + t;
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(tempty)) : "memory");
    }
    if (ok) {
      const int ei = gi < oa.n ? oa.E[gi] : 0;
      // the loads and MMAs of the tile are complete: their stages become the
      // warp's transpose buffer, so that C is read and written along its rows
      double* buf = reinterpret_cast<double*>(sm) + warp * (32 * (ON + 1));
#pragma unroll
      for (int q = 0; q < ON; ++q) {
        const int gj = bj * ON + q;
        const int ej = gj < oa.n ? oa.E[gj] : 0;
        buf[lane * (ON + 1) + q] = oz_scale(acc[q], ei, ej, oa.neg);
      }
      __syncwarp();
      const int64_t r0 = (int64_t)bi * OM + quad * 32;
      const int64_t c0 = (int64_t)bj * ON + lane, c1 = c0 + 32;
#pragma unroll 1
      for (int rb = 0; rb < 32; rb += 8) {   // eight rows of C in flight at a time
        double o0[8], o1[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int64_t row = r0 + rb + u;
          const bool in = oa.beta && row < oa.n;
          o0[u] = in && c0 <= row && c0 < oa.ncols ? oa.C[row * oa.ldc + c0] : 0.0;
          o1[u] = in && c1 <= row && c1 < oa.ncols ? oa.C[row * oa.ldc + c1] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int64_t row = r0 + rb + u;
          double* b0 = &buf[(rb + u) * (ON + 1) + lane];
          double v0 = b0[0], v1 = b0[32];
          if (oa.beta) { v0 += o0[u]; v1 += o1[u]; }
          if (oa.shift != 0.0 && row - (int64_t)bj * ON < ON) {   // rows that cross the diagonal in this tile
            if (c0 == row) v0 += oa.shift;
            if (c1 == row) v1 += oa.shift;
          }
          if (row < oa.n) {
            if (c0 <= row && c0 < oa.ncols) oa.C[row * oa.ldc + c0] = v0;
            if (c1 <= row && c1 < oa.ncols) oa.C[row * oa.ldc + c1] = v1;
          }
          if (oa.mirror) { b0[0] = v0; b0[32] = v1; }
        }
      }
      __syncwarp();   // every lane: rows past n have lanes too
      if (oa.mirror) {
        for (int q = 0; q < ON; ++q) {     // along the columns of the mirror image's rows
          const int64_t gj = (int64_t)bj * ON + q;
          if (gi < oa.n && gj < gi) oa.C[gj * oa.ldc + gi] = buf[lane * (ON + 1) + q];
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tbase, 512);
}

PFN_cuTensorMapEncodeTiled_v12000 g_enc = nullptr;

// `rows` rows of planes (7, rows_pad, kp) bf16 as a 3-D tensor, box {32, box_rows, 7}, SWIZZLE_64B
bool tmap_digits(CUtensorMap* m, const void* base, uint64_t rows, uint64_t rows_pad, uint64_t kp, uint32_t box_rows) {
  if (!g_enc) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return false;
    g_enc = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  }
  if (((uintptr_t)base & 15) != 0 || kp % OK != 0) return false;
  cuuint64_t gdim[3] = {(cuuint64_t)kp, (cuuint64_t)rows, (cuuint64_t)ND};
  cuuint64_t gstr[2] = {(cuuint64_t)kp * 2, (cuuint64_t)rows_pad * kp * 2};
  cuuint32_t box[3] = {OK, box_rows, ND};
  cuuint32_t es[3] = {1, 1, 1};
  return g_enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), gdim, gstr, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr int kMaxDev = 64;
bool g_oz_attr[kMaxDev] = {};

// row0: first row of the planes that takes part (a multiple of the tile; C and
// E begin there)
int oz_launch(const void* planes, int64_t rows_pad, int64_t kp, const OzArgs& oa, int* d_err, cudaStream_t st,
              int64_t row0 = 0) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return VMC_ERR_CUDA;
  if (!g_oz_attr[dev]) {
    if (cudaFuncSetAttribute(k_syrk_f64tc, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM) != cudaSuccess)
      return VMC_ERR_CUDA;
    g_oz_attr[dev] = true;
  }
  CUtensorMap ta, tb;
  const char* base = (const char*)planes + row0 * kp * 2;
  const int64_t rows = rows_pad - row0;
  if (!tmap_digits(&ta, base, (uint64_t)rows, (uint64_t)rows_pad, (uint64_t)kp, OM) ||
      !tmap_digits(&tb, base, (uint64_t)rows, (uint64_t)rows_pad, (uint64_t)kp, ON))
    return VMC_ERR_UNSUPPORTED;
  const int64_t nt = rows / OM;
  const int64_t tiles = oa.ncols < oa.n ? nt * ((oa.ncols + ON - 1) / ON) : nt * (nt + 1);
  if (tiles > INT32_MAX) return VMC_ERR_ARGS;
  k_syrk_f64tc<<<(unsigned)tiles, OZ_THREADS, OZ_SMEM, st>>>(ta, tb, oa, d_err);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

int64_t pad_to(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

// ---- blocked Cholesky pieces ---------------------------------------------------

constexpr int NB = 64;
constexpr int TB = 64, TK = 16;   // k_syrk_df: output tile, K step

// The Cholesky's trailing update C -= A A^T for FP64 A in double-float
// arithmetic on the FP32 pipes (GB300's FP64 rate is 1/64 of FP32): each
// operand is split into FP32 x = hi + lo (to 2^-48), the leading product
// hi*hi is captured exactly (p and its FMA error term), p is summed with
// Knuth's TwoSum into a (s, c) pair and the small terms (the error term,
// hi*lo + lo*hi) into a third FP32 accumulator; lo*lo (2^-48) is dropped.
// ~12 FP32 instructions per multiply-add, relative accuracy ~2^-45 over the
// tile, far below the Gram matrix's own input rounding.  Same tiling and
// lower-triangle semantics as k_syrk.
__global__ void k_syrk_df(const double* __restrict__ A, int64_t lda, int64_t n, int64_t K, double* __restrict__ C,
                          int64_t ldc, int64_t off, double sgn) {
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (bj > bi) return;
  __shared__ float Ah[TK][TB + 1], Al[TK][TB + 1], Bh[TK][TB + 1], Bl[TK][TB + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t i0 = off + (int64_t)bi * TB, j0 = off + (int64_t)bj * TB;
  float hs[4][4], hc[4][4], sm[4][4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int r = 0; r < 4; ++r) { hs[q][r] = 0.f; hc[q][r] = 0.f; sm[q][r] = 0.f; }
  for (int64_t k0 = 0; k0 < K; k0 += TK) {
    for (int idx = threadIdx.x; idx < TB * TK; idx += 256) {
      const int r = idx / TK, kk = idx - r * TK;
      const int64_t gk = k0 + kk, gi = i0 + r, gj = j0 + r;
      const double a = (gi < off + n && gk < K) ? A[gi * lda + gk] : 0.0;
      const double b = (gj < off + n && gk < K) ? A[gj * lda + gk] : 0.0;
      const float ah = (float)a, bh = (float)b;
      Ah[kk][r] = ah;
      Al[kk][r] = (float)(a - (double)ah);
      Bh[kk][r] = bh;
      Bl[kk][r] = (float)(b - (double)bh);
    }
    __syncthreads();
#pragma unroll 4
    for (int kk = 0; kk < TK; ++kk) {
      float ah[4], al[4], bh[4], bl[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        ah[q] = Ah[kk][ty * 4 + q]; al[q] = Al[kk][ty * 4 + q];
        bh[q] = Bh[kk][tx * 4 + q]; bl[q] = Bl[kk][tx * 4 + q];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float p = __fmul_rn(ah[q], bh[r]);
          const float e = fmaf(ah[q], bh[r], -p);
          sm[q][r] += e + fmaf(ah[q], bl[r], al[q] * bh[r]);
          hc[q][r] += vmc::two_sum(hs[q][r], p);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t gi = i0 + ty * 4 + q, gj = j0 + tx * 4 + r;
      if (gi < off + n && gj < off + n && gj <= gi)
        C[gi * ldc + gj] += sgn * ((double)hs[q][r] + (double)hc[q][r] + (double)sm[q][r]);
    }
}

// An FP64 instruction of a warp occupies its SM quarter for 64 clocks on GB300
// (measured: dependent or not, one lane or 32), so the kernels below spread
// every step over four warps, one a quarter, and count FP64 instructions per
// warp, not latencies.

// Cholesky of one 64 x 64 diagonal tile, one CTA of four warps, as L D L^T
// (a reciprocal per column on the critical chain: three FP64 instructions;
// the square roots are taken for all columns at the end).  Thread (ty, tx) of
// 8 x 16 holds the elements (ty + 8 i, tx + 16 j) in registers.  Step k: the
// column k goes through shared memory (two buffers, one barrier a step), then
// a_ij -= u_i (u_j / d_k).  Eight steps are a phase with the register groups
// left of or above them left out at compile time: ~15 FP64 instructions a warp
// and step (with 16 lanes a row in k_trsm64: minSR of 2049 x 8192 7.98 -> 7.31 ms).
//
// Near the ends of FP64's range 1 / d is subnormal or overflows.  The steps do
// not test for it (a scaled reciprocal in the loop: minSR of 2049 x 8192 7.33 ->
// 7.66 ms); a tile that met such a pivot is factored again from C, with r =
// 1 / (d sc) and a product with sc.
__device__ __forceinline__ bool far_exponent(double d) {
  const int e = (__double2hiint(d) >> 20) - 1023;
  return e < -1000 || e > 1000;
}
template <int KP, bool FAR>
__device__ __forceinline__ void potrf_phase(double (&a)[8][4], double (*uc)[NB], double* dk, double* rk, int tx, int ty,
                                            bool& bad) {
#pragma unroll 1
  for (int kk = 0; kk < 8; ++kk) {
    const int k = 8 * KP + kk;
    __syncthreads();
    const double* u = uc[k & 1];
    double d = u[k];
    if (!(d > 0.0) || (__double2hiint(d) & 0x7ff00000) == 0x7ff00000) {
      bad = true;
      d = 1e-300;
    }
    const double sc = FAR && far_exponent(d) ? (d < 1.0 ? 0x1p300 : 0x1p-300) : 1.0;
    const double r = FAR ? 1.0 / (d * sc) : vmc::rcp_pos(d);
    if (threadIdx.x == 0) { dk[k] = d; rk[k] = r; }
    double ui[8];
#pragma unroll
    for (int i = KP; i < 8; ++i) ui[i] = u[ty + 8 * i];
    const int jn = (k + 1) >> 4;
#pragma unroll
    for (int jj = KP / 2; jj < 4; ++jj) {   // the group of the next column comes first
      const int c = tx + 16 * jj;
      double v = c > k ? u[c] * r : 0.0;
      if (FAR) v *= sc;
#pragma unroll
      for (int i = 2 * jj > KP ? 2 * jj : KP; i < 8; ++i) a[i][jj] = fma(-ui[i], v, a[i][jj]);
      if (jj == jn && c == k + 1)
#pragma unroll
        for (int i = 2 * jj > KP ? 2 * jj : KP; i < 8; ++i) uc[(k + 1) & 1][ty + 8 * i] = a[i][jj];
    }
  }
}
template <bool FAR>
__device__ __forceinline__ void potrf_tile(const double* C, int64_t ldc, int nb, double (&a)[8][4], double (*uc)[NB],
                                           double* dk, double* rk, int tx, int ty, bool& bad) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = ty + 8 * i, c = tx + 16 * j;
      a[i][j] = (r < nb && c <= r) ? C[(int64_t)r * ldc + c] : (r == c ? 1.0 : 0.0);
    }
  if (tx == 0)
#pragma unroll
    for (int i = 0; i < 8; ++i) uc[0][ty + 8 * i] = a[i][0];
  bad = false;
  potrf_phase<0, FAR>(a, uc, dk, rk, tx, ty, bad);
  potrf_phase<1, FAR>(a, uc, dk, rk, tx, ty, bad);
  potrf_phase<2, FAR>(a, uc, dk, rk, tx, ty, bad);
  potrf_phase<3, FAR>(a, uc, dk, rk, tx, ty, bad);
  potrf_phase<4, FAR>(a, uc, dk, rk, tx, ty, bad);
  potrf_phase<5, FAR>(a, uc, dk, rk, tx, ty, bad);
  potrf_phase<6, FAR>(a, uc, dk, rk, tx, ty, bad);
  potrf_phase<7, FAR>(a, uc, dk, rk, tx, ty, bad);
  __syncthreads();
}
__global__ void __launch_bounds__(128) k_potrf64(double* __restrict__ C, int64_t ldc, int nb, int* __restrict__ info) {
  __shared__ double uc[2][NB];
  __shared__ double dk[NB], rk[NB];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double a[8][4];
  bool bad;
  potrf_tile<false>(C, ldc, nb, a, uc, dk, rk, tx, ty, bad);
  const bool far = __syncthreads_or(threadIdx.x < NB && far_exponent(dk[threadIdx.x]));
  if (far) potrf_tile<true>(C, ldc, nb, a, uc, dk, rk, tx, ty, bad);
  if (bad && threadIdx.x == 0) atomicExch(info, 1);
  if (threadIdx.x < NB) {
    const double d = dk[threadIdx.x], sq = sqrt(d);
    dk[threadIdx.x] = sq;
    rk[threadIdx.x] = far ? 1.0 / sq : rk[threadIdx.x] * sq;    // 1 / sqrt(d)
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = ty + 8 * i, c = tx + 16 * j;
      if (r < nb && c < nb) C[(int64_t)r * ldc + c] = c < r ? a[i][j] * rk[c] : (c == r ? dk[c] : 0.0);
    }
}

// Panel below a full 64-column diagonal tile: X = A21 L11^-T.  LPR lanes a row
// (lane q holds the columns q + LPR t), 128 / LPR rows a CTA of four warps: a
// row's 2016 multiply-adds take 528 (LPR 4) to 160 (LPR 16) FP64 instructions of
// its warp.  The unit factor L11 D^-1 is solved with, so that the divisions by
// the diagonal are one product per entry at the end.
template <int LPR>
__global__ void __launch_bounds__(128) k_trsm64(double* __restrict__ C, int64_t ldc, int64_t rows) {
  extern __shared__ double tsm[];
  double* Lu = tsm;                  // Lu[k][c] = L11[c][k] / L11[k][k] for c > k, else 0
  double* rd = Lu + NB * NB;         // 1 / L11[k][k]
  constexpr int NT = NB / LPR;       // entries a lane
  const int lane = threadIdx.x & 31, q = lane % LPR;
  const int64_t row = (int64_t)blockIdx.x * (128 / LPR) + threadIdx.x / LPR;
  double* A = C + (NB + (row < rows ? row : 0)) * ldc + q;
  double x[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) x[t] = A[LPR * t];
  if (threadIdx.x < NB) rd[threadIdx.x] = 1.0 / C[(int64_t)threadIdx.x * ldc + threadIdx.x];
  __syncthreads();
#pragma unroll 16
  for (int m = 0; m < NB * NB / 128; ++m) {
    const int c = m * 2 + (threadIdx.x >> 6), k = threadIdx.x & 63;   // along the rows of L11
    Lu[k * NB + c] = c > k ? C[(int64_t)c * ldc + k] * rd[k] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NB - 1; ++k) {
    const double xk = __shfl_sync(VMC_FULL_MASK, x[k / LPR], lane - q + k % LPR);
#pragma unroll
    for (int t = (k + 1) / LPR; t < NT; ++t) x[t] = fma(-xk, Lu[k * NB + LPR * t + q], x[t]);
  }
  if (row < rows) {
#pragma unroll
    for (int t = 0; t < NT; ++t) A[LPR * t] = x[t] * rd[LPR * t + q];
  }
}
constexpr int TRSM_SMEM = (NB * NB + NB) * 8;
bool g_trsm_attr[kMaxDev] = {};

int factor_step(double* T, int64_t ldt, int64_t n, int64_t k0, int* d_info, cudaStream_t st) {
  const int nb = (int)(n - k0 < NB ? n - k0 : NB);
  double* D = T + k0 * ldt + k0;
  k_potrf64<<<1, 128, 0, st>>>(D, ldt, nb, d_info);
  const int64_t rest = n - k0 - nb;
  if (rest > 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return VMC_ERR_CUDA;
    if (!g_trsm_attr[dev]) {
      if (cudaFuncSetAttribute(k_trsm64<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, TRSM_SMEM) != cudaSuccess ||
          cudaFuncSetAttribute(k_trsm64<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, TRSM_SMEM) != cudaSuccess)
        return VMC_ERR_CUDA;
      g_trsm_attr[dev] = true;
    }
    // a row's chain is the shorter the more lanes share it, while the CTAs fit
    // the GPU at once: 16 lanes to two CTAs of 8 rows on each of 152 SMs
    if (rest <= 2432) k_trsm64<16><<<(unsigned)((rest + 7) / 8), 128, TRSM_SMEM, st>>>(D, ldt, rest);
    else k_trsm64<4><<<(unsigned)((rest + 31) / 32), 128, TRSM_SMEM, st>>>(D, ldt, rest);
  }
  return VMC_OK;
}

int split_f64(const double* X, int64_t rows, int64_t K, int64_t ldx, void* planes, int64_t rows_pad, int64_t kp,
              int* E, cudaStream_t st) {
  __nv_bfloat16* P = (__nv_bfloat16*)planes;
  if (K <= 1024) k_split_f64<32><<<(unsigned)(rows_pad / 4), 128, 0, st>>>(X, rows, rows_pad, K, ldx, kp, E, P);
  else k_split_f64<128><<<(unsigned)rows_pad, 128, 0, st>>>(X, rows, rows_pad, K, ldx, kp, E, P);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

// Columns factored between two updates of the whole trailing matrix.
constexpr int64_t OUTER = 256;

// Workspace of vmc_sr_cholesky_tc: digits and row exponents of two panels (the
// trailing update of one may still read its own while the next is split) and
// of a 64-column tile's rows.
struct CholWork {
  char* planes[2];
  int* E[2];
  char* tplanes;
  int* tE;
  int64_t bytes;
};
CholWork chol_work(int64_t n, void* base) {
  const int64_t rp = pad_to(n, OM), pl = rp * OUTER * 2 * ND, tp = rp * NB * 2 * ND;
  const int64_t eb = pad_to(rp * (int64_t)sizeof(int), 256);
  CholWork w;
  char* p = (char*)base;
  for (int b = 0; b < 2; ++b) { w.planes[b] = p; p += pl; }
  w.tplanes = p; p += tp;
  for (int b = 0; b < 2; ++b) { w.E[b] = (int*)p; p += eb; }
  w.tE = (int*)p; p += eb;
  w.bytes = p - (char*)base;
  return w;
}

// Lookahead: a panel's tiles are a chain of small kernels (a tile 57 us, its
// panel solve 5 to 40) and the trailing update behind it fills the GPU.  The
// chain runs on a stream of high priority: of a panel's update it waits for the
// next panel's 256 columns only, and factors those while the caller's stream
// updates the rest.  Order 8192: 28.2 -> 24.4 ms, 4096: 8.72 -> 8.45, 3000:
// 5.78 -> 5.58, 2049: no difference.  Not under stream capture: the stream and
// events are shared by the calls of all threads, one at a time under g_look_mu,
// and a capture would hold them beyond the call.
constexpr int64_t LOOK_MIN = 2560;
struct Lookahead {
  cudaStream_t chain = nullptr;
  cudaEvent_t ready = nullptr, bulk = nullptr;
  int state = 0;   // 1: usable, -1: creation failed
};
Lookahead g_look[kMaxDev];
std::mutex g_look_mu;

Lookahead* lookahead() {   // under g_look_mu
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return nullptr;
  Lookahead& l = g_look[dev];
  if (l.state == 0) {
    int lo = 0, hi = 0;
    cudaDeviceGetStreamPriorityRange(&lo, &hi);
    const bool ok = cudaStreamCreateWithPriority(&l.chain, cudaStreamNonBlocking, hi) == cudaSuccess &&
                    cudaEventCreateWithFlags(&l.ready, cudaEventDisableTiming) == cudaSuccess &&
                    cudaEventCreateWithFlags(&l.bulk, cudaEventDisableTiming) == cudaSuccess;
    l.state = ok ? 1 : -1;
  }
  return l.state == 1 ? &l : nullptr;
}

// Panels of OUTER columns: their tiles on stream `c`, the trailing update on
// `st` but for the next panel's columns (la), or all on one stream (c == st).
int chol_tc(double* T, int64_t n, int64_t ldt, int* d_info, const CholWork& w, int* d_err, cudaStream_t st,
            cudaStream_t c, Lookahead* la) {
  bool pending = false;   // a trailing update on st that the chain has not waited for
  for (int64_t k0 = 0, k = 0; k0 < n; k0 += OUTER, ++k) {
    const int64_t kend = n < k0 + OUTER ? n : k0 + OUTER;
    for (int64_t j0 = k0; j0 < kend; j0 += NB) {
      int rc = factor_step(T, ldt, n, j0, d_info, c);
      if (rc) return rc;
      const int64_t j1 = j0 + NB, rest = n - j1;
      if (j1 < kend) {   // the panel's remaining columns, K = 64
        const int64_t rp = pad_to(rest, OM);
        rc = split_f64(T + j1 * ldt + j0, rest, NB, ldt, w.tplanes, rp, NB, w.tE, c);
        if (rc) return rc;
        OzArgs oa{T + j1 * (ldt + 1), ldt, w.tE, 0.0, 1, (int)rest, (int)(kend - j1), NB / OK, 1, 0};
        rc = oz_launch(w.tplanes, rp, NB, oa, d_err, c);
        if (rc) return rc;
      }
    }
    const int64_t rest = n - kend;
    if (rest <= 0) break;
    char* planes = w.planes[k & 1];
    int* E = w.E[k & 1];
    const int64_t rp = pad_to(rest, OM);
    int rc = split_f64(T + kend * ldt + k0, rest, OUTER, ldt, planes, rp, OUTER, E, c);
    if (rc) return rc;
    const int64_t head = la && rest > OUTER ? OUTER : rest;   // columns updated on the chain
    // the previous panel's update of these columns, and its reads of the
    // buffers that the next panel's split takes
    if (pending && cudaStreamWaitEvent(c, la->bulk, 0) != cudaSuccess) return VMC_ERR_CUDA;
    pending = false;
    if (head < rest) {
      if (cudaEventRecord(la->ready, c) != cudaSuccess || cudaStreamWaitEvent(st, la->ready, 0) != cudaSuccess)
        return VMC_ERR_CUDA;
      OzArgs oa{T + (kend + head) * (ldt + 1), ldt, E + head, 0.0, 1, (int)(rest - head), (int)(rest - head),
                (int)(OUTER / OK), 1, 0};
      rc = oz_launch(planes, rp, OUTER, oa, d_err, st, head);
      if (rc) return rc;
      if (cudaEventRecord(la->bulk, st) != cudaSuccess) return VMC_ERR_CUDA;
      pending = true;
    }
    OzArgs oa{T + kend * (ldt + 1), ldt, E, 0.0, 1, (int)rest, (int)head, (int)(OUTER / OK), 1, 0};
    rc = oz_launch(planes, rp, OUTER, oa, d_err, c);
    if (rc) return rc;
  }
  return VMC_OK;
}

}  // namespace

extern "C" {

int vmc_split_f64(const double* X, int64_t rows, int64_t K, int64_t ldx, void* planes, int64_t rows_pad, int64_t kp,
                  int* row_exp, void* stream) {
  if (rows <= 0 || K <= 0 || ldx < K || rows_pad < rows || rows_pad % OM != 0 || rows_pad > INT32_MAX || kp < K ||
      kp % OK != 0 || !X || !planes || ((uintptr_t)planes & 15) != 0 || !row_exp)
    return VMC_ERR_ARGS;
  return split_f64(X, rows, K, ldx, planes, rows_pad, kp, row_exp, (cudaStream_t)stream);
}

int vmc_sr_gram_f64_tc(const void* planes, const int* row_exp, int64_t ns, int64_t rows_pad, int64_t kp, double* T,
                       int64_t ldt, double diag_shift, int accumulate, int* d_err, void* stream) {
  if (ns <= 0 || rows_pad < ns || rows_pad % OM != 0 || rows_pad > INT32_MAX / 2 || kp <= 0 || kp % OK != 0 ||
      kp / OK > INT32_MAX || ldt < ns || !planes || !row_exp || !T || !d_err)
    return VMC_ERR_ARGS;
  OzArgs oa{T, ldt, row_exp, diag_shift, 0, (int)ns, (int)ns, (int)(kp / OK), accumulate ? 1 : 0, 1};
  return oz_launch(planes, rows_pad, kp, oa, d_err, (cudaStream_t)stream);
}

// In-place lower Cholesky of T: FP64 tiles and panels, double-float trailing
// updates.  d_info set to 1 on a non-positive pivot.
int vmc_sr_cholesky(double* T, int64_t n, int64_t ldt, int* d_info, void* stream) {
  if (n <= 0 || ldt < n || !T || !d_info) return VMC_ERR_ARGS;
  cudaStream_t s = (cudaStream_t)stream;
  for (int64_t k0 = 0; k0 < n; k0 += NB) {
    const int rc = factor_step(T, ldt, n, k0, d_info, s);
    if (rc) return rc;
    const int64_t rest = n - k0 - NB;
    if (rest > 0) {
      const int64_t nt = (rest + TB - 1) / TB;
      dim3 grid((unsigned)nt, (unsigned)nt);
      k_syrk_df<<<grid, 256, 0, s>>>(T + k0, ldt, rest, NB, T, ldt, k0 + NB, -1.0);
    }
  }
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

int vmc_sr_cholesky_tc_work_bytes(int64_t n, int64_t* bytes) {
  if (n <= 0 || !bytes) return VMC_ERR_ARGS;
  *bytes = chol_work(n, nullptr).bytes;
  return VMC_OK;
}

int vmc_sr_cholesky_tc(double* T, int64_t n, int64_t ldt, int* d_info, void* work, int* d_err, void* stream) {
  if (n <= 0 || n > INT32_MAX / 2 || ldt < n || !T || !d_info || !work || ((uintptr_t)work & 255) != 0 || !d_err)
    return VMC_ERR_ARGS;
  cudaStream_t st = (cudaStream_t)stream;
  const CholWork w = chol_work(n, work);
  Lookahead* la = nullptr;
  std::unique_lock<std::mutex> lock(g_look_mu, std::defer_lock);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (n >= LOOK_MIN && cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
    lock.lock();
    la = lookahead();
  }
  if (!la) {
    const int rc = chol_tc(T, n, ldt, d_info, w, d_err, st, st, nullptr);
    if (rc) return rc;
  } else {
    if (cudaEventRecord(la->ready, st) != cudaSuccess || cudaStreamWaitEvent(la->chain, la->ready, 0) != cudaSuccess)
      return VMC_ERR_CUDA;
    const int rc = chol_tc(T, n, ldt, d_info, w, d_err, st, la->chain, la);
    // the caller's stream waits for what is queued, after an error too
    if (cudaEventRecord(la->ready, la->chain) != cudaSuccess || cudaStreamWaitEvent(st, la->ready, 0) != cudaSuccess)
      return VMC_ERR_CUDA;
    if (rc) return rc;
  }
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

}  // extern "C"
