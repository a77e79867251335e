// Hand-written adjoint of the NNBF log-amplitude: per-sample
// O_k(x) = d log|psi(x)| / d theta_k for every parameter, in the reference's
// parameter order [M_base, W0, b0, W1, b1, out_w, out_b].
//
//   A = M(x)[occ] (nf x nf),  G = A^-T = d log|det A| / dA,
//   Gbar (2N x nf): G scattered into the occupied rows (zero elsewhere)
//   dM_base = Gbar;  d out_b = s Gbar;  d out_w = (s Gbar) (x) h2   (outer product)
//   dh2 = s out_w^T vec(Gbar);  dz1 = dh2 * gelu'(z1);  db1 = dz1;  dW1 = dz1 (x) h1
//   dh1 = W1^T dz1;  dz0 = dh1 * gelu'(z0);  db0 = dz0;  dW0 = dz0 (x) n
//
// One block of 256 threads per configuration; the forward activations and the
// orbital matrix are recomputed (not stored between sampling and gradient
// evaluation), A^-1 comes from a Gauss-Jordan elimination with partial pivoting
// in shared memory.  The out_w block is either written in full (reference row
// layout) or as its two Kronecker factors s*Gbar (2N*nf) and h2 (256), which is
// what the sample-space SR solver consumes at scale.
//
// FP32 in bulk (vmc_nnbf_logpsi_grad_ws): the same adjoint as batched stages
// over work_rows configurations, see "batched FP32 stages" below.
#include <type_traits>

#include "common.cuh"
#include "sgemm.cuh"

using namespace vmc;

namespace {

constexpr int HID = 256;

template <typename T> __device__ __forceinline__ T erf_t(T x);
template <> __device__ __forceinline__ float erf_t<float>(float x) { return erff(x); }
template <> __device__ __forceinline__ double erf_t<double>(double x) { return erf(x); }
template <typename T> __device__ __forceinline__ T exp_t(T x);
template <> __device__ __forceinline__ float exp_t<float>(float x) { return expf(x); }
template <> __device__ __forceinline__ double exp_t<double>(double x) { return exp(x); }

template <typename T>
__device__ __forceinline__ T gelu_v(T x) { return T(0.5) * x * (T(1) + erf_t<T>(x * T(0.70710678118654752440))); }
// d/dx [x Phi(x)] = Phi(x) + x phi(x)
template <typename T>
__device__ __forceinline__ T gelu_d(T x) {
  return T(0.5) * (T(1) + erf_t<T>(x * T(0.70710678118654752440))) +
         x * exp_t<T>(T(-0.5) * x * x) * T(0.39894228040143267794);
}

template <typename T>
struct GradNet {
  const T* w0t;    // (2N, 256)   W0^T
  const T* b0;     // (256)
  const T* w1;     // (256, 256)  W1 [out][in]
  const T* w1t;    // (256, 256)  W1^T [in][out]
  const T* b1;     // (256)
  const T* outw;   // (2N*nf, 256)
  const T* outwt;  // (256, 2N*nf)
  const T* outb;   // (2N*nf)
  const T* mbase;  // (2N, nf)
};

template <typename T>
__global__ void __launch_bounds__(256) k_nnbf_grad(GradNet<T> net, int N, int nf, T s, const uint64_t* __restrict__ occ,
                                                   T* __restrict__ Ofull, int64_t ldf, T* __restrict__ Odense,
                                                   int64_t ldd, T* __restrict__ kg, T* __restrict__ kh,
                                                   double* __restrict__ logabs_out, double* __restrict__ sign_out) {
  extern __shared__ __align__(16) uint8_t gsm[];
  const int tid = threadIdx.x;
  const int64_t w = blockIdx.x;
  const int n_orb = 2 * N;
  const int ldA = nf + 1;
  T* A = reinterpret_cast<T*>(gsm);           // nf x (nf+1)
  T* Ai = A + nf * ldA;                        // nf x (nf+1)
  T* z0 = Ai + nf * ldA;                       // 256
  T* h1 = z0 + HID;                            // 256
  T* z1 = h1 + HID;                            // 256
  T* h2 = z1 + HID;                            // 256
  T* dz1 = h2 + HID;                           // 256
  T* fac = dz1 + HID;                          // 64
  int* orbs = reinterpret_cast<int*>(fac + 64);   // 64
  int* piv = orbs + 64;                            // [0]=pivot row, [1]=ok

  const uint64_t up = occ[2 * w], dn = occ[2 * w + 1];
  const bool count_ok = (__popcll(up) + __popcll(dn)) == nf;
  if (tid < n_orb && orb_occupied(up, dn, N, tid)) {
    const int p = orb_prefix(up, dn, N, tid);
    if (p < 64) orbs[p] = tid;
  }
  if (tid == 0) piv[1] = count_ok ? 1 : 0;
  __syncthreads();
  // ---- forward recompute ----
  {
    T acc = net.b0[tid];
    if (count_ok)
      for (int k = 0; k < nf; ++k) acc += net.w0t[(size_t)orbs[k] * HID + tid];
    z0[tid] = acc;
    h1[tid] = gelu_v<T>(acc);
  }
  __syncthreads();
  {
    T acc = net.b1[tid];
    for (int k = 0; k < HID; ++k) acc += net.w1t[(size_t)k * HID + tid] * h1[k];
    z1[tid] = acc;
    h2[tid] = gelu_v<T>(acc);
  }
  __syncthreads();
  const int nout = n_orb * nf;
  for (int idx = tid; idx < nf * nf; idx += 256) {
    const int pos = idx / nf, c = idx - pos * nf;
    T v = 0;
    if (count_ok) {
      const int j = orbs[pos] * nf + c;
      T acc = net.outb[j];
      for (int k = 0; k < HID; ++k) acc += net.outwt[(size_t)k * nout + j] * h2[k];
      v = net.mbase[j] + s * acc;
    }
    A[pos * ldA + c] = v;
    Ai[pos * ldA + c] = (pos == c) ? T(1) : T(0);
  }
  __syncthreads();
  // ---- Gauss-Jordan inverse with partial pivoting ----
  double la = 0.0;
  int neg = 0;
  for (int k = 0; k < nf && piv[1] == 1; ++k) {
    if (tid < 32) {
      double best = -1.0;
      int bi = k;
      for (int r = k + tid; r < nf; r += 32) {
        double v = fabs((double)A[r * ldA + k]);
        if (v != v) v = INFINITY;   // NaN ranks first, so that it is detected
        if (v > best) { best = v; bi = r; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(VMC_FULL_MASK, best, o);
        const int oi = __shfl_xor_sync(VMC_FULL_MASK, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      if (tid == 0) {
        piv[0] = bi;
        if (!(best > 0.0) || !isfinite(best)) piv[1] = isfinite(best) ? 0 : -1;
      }
    }
    __syncthreads();
    if (piv[1] != 1) break;
    const int p = piv[0];
    if (p != k) {
      for (int c = tid; c < 2 * nf; c += 256) {
        T* M = c < nf ? A : Ai;
        const int cc = c < nf ? c : c - nf;
        const T t0 = M[k * ldA + cc];
        M[k * ldA + cc] = M[p * ldA + cc];
        M[p * ldA + cc] = t0;
      }
      neg ^= 1;
    }
    __syncthreads();
    const T pv = A[k * ldA + k];
    la += log(fabs((double)pv));
    neg ^= (pv < T(0));
    __syncthreads();
    const T ipv = T(1) / pv;
    for (int c = tid; c < 2 * nf; c += 256) {
      if (c < nf) A[k * ldA + c] *= ipv; else Ai[k * ldA + c - nf] *= ipv;
    }
    for (int r = tid; r < nf; r += 256) fac[r] = (r == k) ? T(0) : A[r * ldA + k];
    __syncthreads();
    for (int idx = tid; idx < nf * 2 * nf; idx += 256) {
      const int r = idx / (2 * nf), c = idx - r * 2 * nf;
      if (r == k) continue;
      if (c < nf) A[r * ldA + c] -= fac[r] * A[k * ldA + c];
      else Ai[r * ldA + c - nf] -= fac[r] * Ai[k * ldA + c - nf];
    }
    __syncthreads();
  }
  // piv[1]: 1 regular, 0 singular (or wrong electron count), -1 non-finite entry
  const bool ok = piv[1] == 1;
  if (tid == 0) {
    const double qnan = __longlong_as_double(0x7ff8000000000000ll);
    if (logabs_out) logabs_out[w] = ok ? la : (piv[1] < 0 ? qnan : -INFINITY);
    if (sign_out) sign_out[w] = ok ? (neg ? -1.0 : 1.0) : (piv[1] < 0 ? qnan : 0.0);
  }
  // Gbar[orbs[pos]][c] = Ainv[c][pos]; stored as G[pos][c] in A (reuse)
  for (int idx = tid; idx < nf * nf; idx += 256) {
    const int pos = idx / nf, c = idx - pos * nf;
    A[pos * ldA + c] = ok ? Ai[c * ldA + pos] : T(0);
  }
  __syncthreads();
  // ---- backward through the MLP ----
  {
    // dh2[k] = s * sum_{pos,c} G[pos][c] * out_w[orbs[pos]*nf + c][k]
    T acc = 0;
    if (ok)
      for (int pos = 0; pos < nf; ++pos) {
        const T* wr = net.outw + (size_t)orbs[pos] * nf * HID + tid;
        const T* g = A + pos * ldA;
        for (int c = 0; c < nf; ++c) acc += g[c] * wr[(size_t)c * HID];
      }
    dz1[tid] = s * acc * gelu_d<T>(z1[tid]);
  }
  __syncthreads();
  T dz0;
  {
    T acc = 0;
    for (int j = 0; j < HID; ++j) acc += net.w1[(size_t)j * HID + tid] * dz1[j];
    dz0 = acc * gelu_d<T>(z0[tid]);
  }
  __syncthreads();
  // stash dz0 in z0 (z0 no longer needed)
  z0[tid] = dz0;
  __syncthreads();
  // ---- write O ----
  // offsets in the reference order
  const int64_t oM = 0, oW0 = (int64_t)n_orb * nf, ob0 = oW0 + (int64_t)HID * n_orb, oW1 = ob0 + HID,
                ob1 = oW1 + (int64_t)HID * HID, oOW = ob1 + HID, oOB = oOW + (int64_t)nout * HID;
  // the dense row omits the out_w block: same order with out_b following b1
  for (int pass = 0; pass < 2; ++pass) {
    T* row = pass == 0 ? (Ofull ? Ofull + w * ldf : nullptr) : (Odense ? Odense + w * ldd : nullptr);
    if (!row) continue;
    const int64_t obB = pass == 0 ? oOB : oOW;
    for (int idx = tid; idx < nout; idx += 256) {
      const int o = idx / nf, c = idx - o * nf;
      T g = 0;
      if (ok && orb_occupied(up, dn, N, o)) g = A[orb_prefix(up, dn, N, o) * ldA + c];
      row[oM + idx] = g;
      row[obB + idx] = s * g;
    }
    for (int idx = tid; idx < HID * n_orb; idx += 256) {
      const int j = idx / n_orb, i = idx - j * n_orb;
      row[oW0 + idx] = orb_occupied(up, dn, N, i) ? z0[j] : T(0);
    }
    row[ob0 + tid] = z0[tid];
    for (int idx = tid; idx < HID * HID; idx += 256) {
      const int j = idx / HID, k = idx - j * HID;
      row[oW1 + idx] = dz1[j] * h1[k];
    }
    row[ob1 + tid] = dz1[tid];
    if (pass == 0) {
      for (int64_t idx = tid; idx < (int64_t)nout * HID; idx += 256) {
        const int j = (int)(idx / HID), k = (int)(idx - (int64_t)j * HID);
        const int o = j / nf, c = j - o * nf;
        T g = 0;
        if (ok && orb_occupied(up, dn, N, o)) g = A[orb_prefix(up, dn, N, o) * ldA + c];
        row[oOW + idx] = s * g * h2[k];
      }
    }
  }
  if (kg) {
    for (int idx = tid; idx < nout; idx += 256) {
      const int o = idx / nf, c = idx - o * nf;
      T g = 0;
      if (ok && orb_occupied(up, dn, N, o)) g = A[orb_prefix(up, dn, N, o) * ldA + c];
      kg[w * (int64_t)nout + idx] = s * g;
    }
  }
  if (kh) kh[w * HID + tid] = h2[tid];
}

template <typename T>
size_t grad_smem(int nf) {
  return (size_t)(2 * nf * (nf + 1) + 5 * HID + 64) * sizeof(T) + 2 * 64 * sizeof(int) + 16;
}


// ---------------------------------------------------------------------------
// Batched FP32 stages.  k_nnbf_grad reads the 8 MB of output-layer weights
// (out_w twice) through L2 for every configuration: 12.8 ms for 8192
// configurations of the 8x8 model, whose outputs are 4 GB (0.6 ms of HBM
// writes).  Here the dense layers run as tiled FP32 products over a block of
// configurations (sgemm.cuh), and the inverse in registers:
//   k_g_first     z0, h1 = gelu(z0)                            a CTA per row
//   k_g_hidden    z1 = W1 h1 + b1, h2                          product
//   k_g_backflow  A[pos] = M_base[r] + s (out_w[r] h2 + out_b[r])  product over all
//                 orbitals, the occupied ones kept
//   k_g_invert    A^-1 and the blocks of O that hold it
//   k_g_dh2       out_w^T vec(Gbar), K split over the grid       product
//   k_g_dz1       dz1 = s dh2 gelu'(z1)
//   k_g_dz0       dz0 = (W1^T dz1) gelu'(z0)                     product
//   k_g_write     the W0, b0, W1, b1 (and out_w) blocks of O
// Every sum but dh2's runs in k_nnbf_grad's order (one multiply-add chain per
// value, ascending), so A, its inverse and what is formed from them alone are
// the same to the bit; dh2's chain of 2N nf terms is split in up to 16.
// ---------------------------------------------------------------------------
struct GradWork {       // per work row: floats
  float *z0, *h1, *z1, *h2, *dz1, *dz0, *dh, *gbar, *A;
  int splits;
};

__device__ __forceinline__ bool g_count_ok(uint64_t up, uint64_t dn, int nf) {
  return __popcll(up) + __popcll(dn) == nf;
}

__global__ void __launch_bounds__(256) k_g_first(GradNet<float> net, int N, int nf, const uint64_t* __restrict__ occ,
                                                 GradWork w) {
  __shared__ int orbs[64];
  const int tid = threadIdx.x;
  const int64_t b = blockIdx.x;
  const uint64_t up = occ[2 * b], dn = occ[2 * b + 1];
  const bool ok = g_count_ok(up, dn, nf);
  if (tid < 2 * N && orb_occupied(up, dn, N, tid)) {
    const int p = orb_prefix(up, dn, N, tid);
    if (p < 64) orbs[p] = tid;
  }
  __syncthreads();
  float acc = net.b0[tid];
  if (ok) {
#pragma unroll 8
    for (int k = 0; k < nf; ++k) acc += net.w0t[(size_t)orbs[k] * HID + tid];
  }
  w.z0[b * HID + tid] = acc;
  w.h1[b * HID + tid] = gelu_v<float>(acc);
}

__global__ void __launch_bounds__(sg::NTHR, 2) k_g_hidden(GradNet<float> net, int R, GradWork w, float* __restrict__ kh) {
  __shared__ sg::Smem sm;
  const int m0 = blockIdx.y * sg::BM, n0 = blockIdx.x * sg::BN;
  float2 acc[8][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = n0 + sg::col_of(j);
    const float2 b = make_float2(net.b1[n], net.b1[n + 1]);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][j] = b;
  }
  sg::tile<true, false>(w.h1, HID, net.w1t, HID, R, HID, 0, HID, m0, n0, sm, acc);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t m = m0 + sg::row_of(i);
    if (m >= R) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + sg::col_of(j);
      const float2 z = acc[i][j];
      const float2 h = make_float2(gelu_v<float>(z.x), gelu_v<float>(z.y));
      *reinterpret_cast<float2*>(&w.z1[m * HID + n]) = z;
      *reinterpret_cast<float2*>(&w.h2[m * HID + n]) = h;
      if (kh) { kh[m * HID + n] = h.x; kh[m * HID + n + 1] = h.y; }
    }
  }
}

__global__ void __launch_bounds__(sg::NTHR, 2) k_g_backflow(GradNet<float> net, int N, int nf, float s, int R,
                                                         const uint64_t* __restrict__ occ, GradWork w) {
  __shared__ sg::Smem sm;
  const int nout = 2 * N * nf;
  const int m0 = blockIdx.y * sg::BM, n0 = blockIdx.x * sg::BN;
  float2 acc[8][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = n0 + sg::col_of(j);
    const float2 b = make_float2(n < nout ? net.outb[n] : 0.f, n + 1 < nout ? net.outb[n + 1] : 0.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][j] = b;
  }
  sg::tile<true, false>(w.h2, HID, net.outwt, nout, R, nout, 0, HID, m0, n0, sm, acc);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t m = m0 + sg::row_of(i);
    if (m >= R) continue;
    const uint64_t up = occ[2 * m], dn = occ[2 * m + 1];
    if (!g_count_ok(up, dn, nf)) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int n = n0 + sg::col_of(j) + e;
        if (n >= nout) continue;
        const int o = n / nf, c = n - o * nf;
        if (!orb_occupied(up, dn, N, o)) continue;
        const int pos = orb_prefix(up, dn, N, o);
        w.A[(size_t)m * nf * nf + pos * nf + c] = fmaf(s, e ? acc[i][j].y : acc[i][j].x, net.mbase[n]);
      }
    }
  }
}

// f(I) for the compile-time I equal to the warp-uniform idx: register arrays
// stay in registers, and only that I's instructions run
template <int N, int I = 0, typename F>
__device__ __forceinline__ void at_index(int idx, F f) {
  if constexpr (I < N) {
    if (idx == I) f(std::integral_constant<int, I>{});
    else at_index<N, I + 1>(idx, f);
  }
}

// A^-1 by in-place Gauss-Jordan steps in registers, NW warps a matrix (layout
// and index algebra of k_slater_refresh).  The pivot is the largest |a| of the
// column, on a tie the row that the elimination with row exchanges would have
// at the smaller position; values are those of that elimination on [A | I].
template <int NT, int NW>
__global__ void __launch_bounds__(128) k_g_invert(int N, int nf, float s, int R, const uint64_t* __restrict__ occ,
                                                  GradWork wk, float* __restrict__ Ofull, int64_t ldf,
                                                  float* __restrict__ Odense, int64_t ldd, float* __restrict__ kg,
                                                  double* __restrict__ logabs_out, double* __restrict__ sign_out) {
  constexpr int TX = NW == 4 ? 16 : 8, TY = 32 * NW / TX, NI = NT / TY, NJ = NT / TX;
  constexpr int WPC = NW == 4 ? 1 : 4;
  __shared__ float gst[WPC][NT][NT + 1];
  __shared__ float colw[WPC][NT], prow_[WPC][NT], dpiv_[WPC][NT];
  __shared__ uint8_t pof_[WPC][NT], kof_[WPC][NT];
  const int sub = NW == 4 ? 0 : (threadIdx.x >> 5);
  const int tid = NW == 4 ? threadIdx.x : (threadIdx.x & 31), lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * WPC + sub;
  if (w >= R) return;
  auto sync = [] { if (NW == 4) __syncthreads(); else __syncwarp(); };
  float *col = colw[sub], *prow = prow_[sub], *dpiv = dpiv_[sub];
  uint8_t *pof = pof_[sub], *kof = kof_[sub];
  const uint64_t up = occ[2 * w], dn = occ[2 * w + 1];
  const int tx = tid % TX, ty = tid / TX;
  int state = g_count_ok(up, dn, nf) ? 1 : 0;   // 1 regular, 0 singular or wrong count, -1 non-finite
  const float* Aw = wk.A + (size_t)w * nf * nf;
  float a[NI][NJ];
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int r = ty + TY * i, c = tx + TX * j;
      a[i][j] = (state && r < nf && c < nf) ? Aw[r * nf + c] : (r == c ? 1.f : 0.f);
    }
  if (tx == 0)
#pragma unroll
    for (int i = 0; i < NI; ++i) col[ty + TY * i] = a[i][0];
  uint64_t live = nf == 64 ? ~0ull : ((1ull << nf) - 1ull);
  const int r0 = lane % NT, r1 = lane + 32;
  int pos0 = r0, pos1 = r1;      // positions of the lane's rows
  int neg = 0;
#pragma unroll 1
  for (int k = 0; k < nf && state == 1; ++k) {
    sync();   // column k complete
    const bool l0 = (live >> r0) & 1ull, l1 = NT > 32 && r1 < NT && ((live >> (r1 & 63)) & 1ull);
    const unsigned h0 = l0 ? (__float_as_uint(fabsf(col[r0])) + 1u) : 0u;
    const unsigned h1 = l1 ? (__float_as_uint(fabsf(col[r1 < NT ? r1 : 0])) + 1u) : 0u;
    const unsigned mh = __reduce_max_sync(VMC_FULL_MASK, max(h0, h1));
    const unsigned pp = __reduce_min_sync(VMC_FULL_MASK, min(h0 == mh ? (unsigned)pos0 : 255u,
                                                             h1 == mh ? (unsigned)pos1 : 255u));
    if (mh <= 1u || mh >= 0x7f800001u) {   // zero, or Inf / NaN
      state = mh <= 1u ? 0 : -1;
      break;
    }
    const unsigned b0 = __ballot_sync(VMC_FULL_MASK, h0 == mh && (unsigned)pos0 == pp);
    const unsigned b1 = __ballot_sync(VMC_FULL_MASK, h1 == mh && (unsigned)pos1 == pp);
    const int p = b0 ? (__ffs(b0) - 1) % NT : 31 + __ffs(b1);
    if (pos0 == k) pos0 = (int)pp;
    if (pos1 == k) pos1 = (int)pp;
    if (r0 == p) pos0 = k;
    if (r1 == p) pos1 = k;
    const float pv = col[p];
    neg ^= ((int)pp != k) ^ (pv < 0.f);
    const float ipv = 1.0f / pv;
    live &= ~(1ull << p);
    if (tid == 0) { dpiv[k] = pv; pof[k] = (uint8_t)p; kof[p] = (uint8_t)k; }
    const int pi = p / TY;
    const bool mine = ty == p % TY;    // the warp's lanes that hold row p (register row pi)
    at_index<NI>(pi, [&](auto I) {
      if (mine)
#pragma unroll
        for (int j = 0; j < NJ; ++j) prow[tx + TX * j] = a[I][j];
    });
    float u[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) u[i] = col[ty + TY * i];
    sync();   // pivot row complete, column k read
    float v[NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) v[j] = prow[tx + TX * j] * ipv;
    at_index<NJ>(k / TX, [&](auto J) {   // column k: -a_ik / d
      if (tx == k % TX) {
        v[J] = ipv;
#pragma unroll
        for (int i = 0; i < NI; ++i) a[i][J] = 0.f;
      }
    });
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int i = 0; i < NI; ++i) a[i][j] = fmaf(-u[i], v[j], a[i][j]);
    at_index<NI>(pi, [&](auto I) {
      if (mine)
#pragma unroll
        for (int j = 0; j < NJ; ++j) a[I][j] = v[j];
    });
    at_index<NJ>((k + 1) / TX, [&](auto J) {
      if (tx == (k + 1) % TX)
#pragma unroll
        for (int i = 0; i < NI; ++i) col[ty + TY * i] = a[i][J];
    });
  }
  const bool ok = state == 1;
  sync();
  if (ok) {   // G[p_j][c] = A^-1[c][p_j] = a[p_c][j]
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int rr = ty + TY * i, c = tx + TX * j;
        if (rr < nf && c < nf) gst[sub][(int)pof[c]][(int)kof[rr]] = a[i][j];
      }
  }
  sync();
  if (tid == 0 && (logabs_out || sign_out)) {
    const double qnan = __longlong_as_double(0x7ff8000000000000ll);
    double la = 0.0;
    if (ok)
      for (int k = 0; k < nf; ++k) la += log(fabs((double)dpiv[k]));
    if (logabs_out) logabs_out[w] = ok ? la : (state < 0 ? qnan : -INFINITY);
    if (sign_out) sign_out[w] = ok ? (neg ? -1.0 : 1.0) : (state < 0 ? qnan : 0.0);
  }
  // Gbar and the blocks of O that hold it, an orbital a warp
  const int n_orb = 2 * N, nout = n_orb * nf;
  float* gb = wk.gbar + (size_t)w * nout;
  const int64_t oOW = (int64_t)nout + (int64_t)HID * n_orb + HID + (int64_t)HID * HID + HID;
  for (int o = NW == 4 ? (threadIdx.x >> 5) : 0; o < n_orb; o += NW) {
    const bool occd = ok && orb_occupied(up, dn, N, o);
    const int pos = occd ? orb_prefix(up, dn, N, o) : 0;
    for (int c = lane; c < nf; c += 32) {
      const float g = occd ? gst[sub][pos][c] : 0.f;
      const int idx = o * nf + c;
      gb[idx] = g;
      if (Ofull) { Ofull[w * ldf + idx] = g; Ofull[w * ldf + oOW + (int64_t)nout * HID + idx] = s * g; }
      if (Odense) { Odense[w * ldd + idx] = g; Odense[w * ldd + oOW + idx] = s * g; }
      if (kg) kg[w * (int64_t)nout + idx] = s * g;
    }
  }
}

// partial sums of dh2 over the output slice blockIdx.z
__global__ void __launch_bounds__(sg::NTHR, 2) k_g_dh2(GradNet<float> net, int nout, int R, int kchunk, GradWork w) {
  __shared__ sg::Smem sm;
  const int m0 = blockIdx.y * sg::BM, n0 = blockIdx.x * sg::BN;
  const int kb = blockIdx.z * kchunk, ke = min(nout, kb + kchunk);
  float2 acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  sg::tile<true, false>(w.gbar, nout, net.outw, HID, R, HID, kb, ke, m0, n0, sm, acc);
  float* out = w.dh + (size_t)blockIdx.z * R * HID;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t m = m0 + sg::row_of(i);
    if (m >= R) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(&out[m * HID + n0 + sg::col_of(j)]) = acc[i][j];
  }
}

// The product runs over all orbitals, Gbar being zero at the empty ones and in
// rows without an inverse; where an output weight there is not finite, 0 times
// it is NaN, and the sum over the row's own orbitals is taken instead.
__global__ void k_g_dz1(GradNet<float> net, int N, int nf, int64_t n, float s, const uint64_t* __restrict__ occ,
                        GradWork w) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float acc = w.dh[i];
  for (int z = 1; z < w.splits; ++z) acc += w.dh[z * n + i];
  if (!isfinite(acc)) {
    const int64_t b = i / HID, nout = (int64_t)2 * N * nf;
    const uint64_t up = occ[2 * b], dn = occ[2 * b + 1];
    bool inverse = false;     // A^-1 has a non-zero entry
    acc = 0.f;
    for (int o = 0; o < 2 * N; ++o) {
      if (!orb_occupied(up, dn, N, o)) continue;
      for (int64_t j = (int64_t)o * nf; j < (int64_t)(o + 1) * nf; ++j) {
        const float g = w.gbar[b * nout + j];
        inverse |= g != 0.f;
        acc += g * net.outw[j * HID + (i - b * HID)];
      }
    }
    if (!inverse) acc = 0.f;
  }
  w.dz1[i] = s * acc * gelu_d<float>(w.z1[i]);
}

__global__ void __launch_bounds__(sg::NTHR, 2) k_g_dz0(GradNet<float> net, int R, GradWork w) {
  __shared__ sg::Smem sm;
  const int m0 = blockIdx.y * sg::BM, n0 = blockIdx.x * sg::BN;
  float2 acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  sg::tile<true, false>(w.dz1, HID, net.w1, HID, R, HID, 0, HID, m0, n0, sm, acc);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t m = m0 + sg::row_of(i);
    if (m >= R) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t o = m * HID + n0 + sg::col_of(j);
      w.dz0[o] = acc[i][j].x * gelu_d<float>(w.z0[o]);
      w.dz0[o + 1] = acc[i][j].y * gelu_d<float>(w.z0[o + 1]);
    }
  }
}

// 256-wide or n_orb-wide rows of O, a row a warp: W0 (256 rows, dz0_j at the
// occupied orbitals), W1 (256 rows, dz1_j h1) and, for the full rows, out_w
// (nout rows, s g_j h2).  Bound by the HBM writes (4 GB for 8192 dense rows of
// the 8x8 model); 16-byte stores where the rows are aligned.
__global__ void __launch_bounds__(256) k_g_write(int N, int nf, float s, const uint64_t* __restrict__ occ, GradWork w,
                                                 float* __restrict__ O, int64_t ld, int full) {
  __shared__ alignas(16) float h1[HID], h2[HID], oc[128];
  const int64_t b = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31;
  const int n_orb = 2 * N, nout = n_orb * nf;
  const uint64_t up = occ[2 * b], dn = occ[2 * b + 1];
  h1[tid] = w.h1[b * HID + tid];
  if (full) h2[tid] = w.h2[b * HID + tid];
  if (tid < n_orb) oc[tid] = orb_occupied(up, dn, N, tid) ? 1.f : 0.f;
  __syncthreads();
  float* row = O + b * ld;
  float* pW0 = row + nout;
  float* pb0 = pW0 + (int64_t)HID * n_orb;
  float* pW1 = pb0 + HID;
  float* pb1 = pW1 + (int64_t)HID * HID;
  float* pOW = pb1 + HID;
  const float *dz0 = w.dz0 + b * HID, *dz1 = w.dz1 + b * HID, *gb = w.gbar + (size_t)b * nout;
  if (blockIdx.y == 0) { pb0[tid] = dz0[tid]; pb1[tid] = dz1[tid]; }
  const bool v4 = ((uintptr_t)pW0 & 15) == 0 && (n_orb & 3) == 0;
  const int nrows = 2 * HID + (full ? nout : 0);
  for (int t = blockIdx.y * 8 + (tid >> 5); t < nrows; t += gridDim.y * 8) {
    float* dst;
    const float* src;
    float f;
    int len = HID;
    if (t < HID) { dst = pW0 + (int64_t)t * n_orb; src = oc; f = dz0[t]; len = n_orb; }
    else if (t < 2 * HID) { dst = pW1 + (int64_t)(t - HID) * HID; src = h1; f = dz1[t - HID]; }
    else { dst = pOW + (int64_t)(t - 2 * HID) * HID; src = h2; f = s * gb[t - 2 * HID]; }
    const bool sel = t < HID;   // W0: a copy or a zero, not a product
    if (v4) {
      for (int c = lane * 4; c < len; c += 128) {
        const float4 x = *reinterpret_cast<const float4*>(src + c);
        float4 o;
        if (sel) o = make_float4(x.x != 0.f ? f : 0.f, x.y != 0.f ? f : 0.f, x.z != 0.f ? f : 0.f, x.w != 0.f ? f : 0.f);
        else o = make_float4(f * x.x, f * x.y, f * x.z, f * x.w);
        __stcs(reinterpret_cast<float4*>(dst + c), o);
      }
    } else {
      for (int c = lane; c < len; c += 32) dst[c] = sel ? (src[c] != 0.f ? f : 0.f) : f * src[c];
    }
  }
}

// Slices of dh2's K: enough CTAs for two on each of 152 SMs, at most 16.
int g_splits(int64_t R) {
  const int64_t tiles = (R + sg::BM - 1) / sg::BM * (HID / sg::BN);
  int64_t z = 304 / tiles;
  return (int)(z < 1 ? 1 : (z > 16 ? 16 : z));
}

// floats of workspace for R rows
int64_t g_floats(int64_t R, int64_t nout, int nf) {
  return R * (6 * HID + (int64_t)g_splits(R) * HID + nout + (int64_t)nf * nf);
}

}  // namespace

extern "C" int vmc_nnbf_logpsi_grad(int prec, const void* const* gnet, int n_sites, int nf, int hidden, double bf_scale,
                                    const uint64_t* occ, int64_t B, void* O_full, int64_t ld_full, void* O_dense,
                                    int64_t ld_dense, void* kron_g, void* kron_h, double* logabs, double* sign,
                                    void* stream) {
  if (n_sites < 1 || n_sites > 64 || nf < 1 || nf > 64 || hidden != HID || B < 0 || (prec != 0 && prec != 1))
    return VMC_ERR_ARGS;
  if (B == 0) return VMC_OK;
  if (!gnet || !occ) return VMC_ERR_ARGS;
  const int64_t n_orb = 2 * n_sites, nout = n_orb * nf;
  const int64_t Np = nout + HID * n_orb + HID + HID * HID + HID + nout * HID + nout;
  const int64_t Nd = Np - nout * HID;
  if (O_full && ld_full < Np) return VMC_ERR_ARGS;
  if (O_dense && ld_dense < Nd) return VMC_ERR_ARGS;
  cudaStream_t st = (cudaStream_t)stream;
  if (prec == 0) {
    GradNet<float> g{(const float*)gnet[0], (const float*)gnet[1], (const float*)gnet[2], (const float*)gnet[3],
                     (const float*)gnet[4], (const float*)gnet[5], (const float*)gnet[6], (const float*)gnet[7],
                     (const float*)gnet[8]};
    const size_t sm = grad_smem<float>(nf);
    cudaFuncSetAttribute(k_nnbf_grad<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_nnbf_grad<float><<<(unsigned)B, 256, sm, st>>>(g, n_sites, nf, (float)bf_scale, occ, (float*)O_full, ld_full,
                                                     (float*)O_dense, ld_dense, (float*)kron_g, (float*)kron_h, logabs,
                                                     sign);
  } else {
    GradNet<double> g{(const double*)gnet[0], (const double*)gnet[1], (const double*)gnet[2], (const double*)gnet[3],
                      (const double*)gnet[4], (const double*)gnet[5], (const double*)gnet[6], (const double*)gnet[7],
                      (const double*)gnet[8]};
    const size_t sm = grad_smem<double>(nf);
    cudaFuncSetAttribute(k_nnbf_grad<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_nnbf_grad<double><<<(unsigned)B, 256, sm, st>>>(g, n_sites, nf, bf_scale, occ, (double*)O_full, ld_full,
                                                      (double*)O_dense, ld_dense, (double*)kron_g, (double*)kron_h,
                                                      logabs, sign);
  }
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

extern "C" int vmc_nnbf_grad_work_bytes(int n_sites, int nf, int64_t work_rows, int64_t* bytes) {
  if (n_sites < 1 || n_sites > 64 || nf < 1 || nf > 64 || work_rows <= 0 || !bytes) return VMC_ERR_ARGS;
  *bytes = g_floats(work_rows, (int64_t)2 * n_sites * nf, nf) * (int64_t)sizeof(float);
  return VMC_OK;
}

extern "C" int vmc_nnbf_logpsi_grad_ws(const void* const* gnet, int n_sites, int nf, int hidden, double bf_scale,
                                       const uint64_t* occ, int64_t B, float* O_full, int64_t ld_full, float* O_dense,
                                       int64_t ld_dense, float* kron_g, float* kron_h, double* logabs, double* sign,
                                       void* work, int64_t work_rows, void* stream) {
  if (n_sites < 1 || n_sites > 64 || nf < 1 || nf > 64 || hidden != HID || B < 0 || work_rows <= 0 ||
      work_rows > INT32_MAX / 2)
    return VMC_ERR_ARGS;
  if (B == 0) return VMC_OK;
  if (!gnet || !occ || !work || ((uintptr_t)work & 15) != 0) return VMC_ERR_ARGS;
  const int64_t n_orb = 2 * n_sites, nout = n_orb * nf;
  const int64_t Np = nout + HID * n_orb + HID + HID * HID + HID + nout * HID + nout;
  const int64_t Nd = Np - nout * HID;
  if (O_full && ld_full < Np) return VMC_ERR_ARGS;
  if (O_dense && ld_dense < Nd) return VMC_ERR_ARGS;
  cudaStream_t st = (cudaStream_t)stream;
  GradNet<float> g{(const float*)gnet[0], (const float*)gnet[1], (const float*)gnet[2], (const float*)gnet[3],
                   (const float*)gnet[4], (const float*)gnet[5], (const float*)gnet[6], (const float*)gnet[7],
                   (const float*)gnet[8]};
  const float s = (float)bf_scale;
  const int N = n_sites;
  for (int64_t w0 = 0; w0 < B; w0 += work_rows) {
    const int64_t R = B - w0 < work_rows ? B - w0 : work_rows;
    const int splits = g_splits(work_rows);   // of the workspace's size, also for the last block
    GradWork w;
    w.splits = splits;
    float* p = (float*)work;
    for (float** q : {&w.z0, &w.h1, &w.z1, &w.h2, &w.dz1, &w.dz0}) { *q = p; p += R * HID; }
    w.dh = p; p += (int64_t)splits * R * HID;
    w.gbar = p; p += R * nout;
    w.A = p;
    const uint64_t* oc = occ + 2 * w0;
    float* of = O_full ? O_full + w0 * ld_full : nullptr;
    float* od = O_dense ? O_dense + w0 * ld_dense : nullptr;
    float* kg = kron_g ? kron_g + w0 * nout : nullptr;
    float* kh = kron_h ? kron_h + w0 * HID : nullptr;
    double* la = logabs ? logabs + w0 : nullptr;
    double* sg_ = sign ? sign + w0 : nullptr;
    const unsigned mt = (unsigned)((R + sg::BM - 1) / sg::BM);
    k_g_first<<<(unsigned)R, 256, 0, st>>>(g, N, nf, oc, w);
    k_g_hidden<<<dim3(HID / sg::BN, mt), sg::NTHR, 0, st>>>(g, (int)R, w, kh);
    k_g_backflow<<<dim3((unsigned)((nout + sg::BN - 1) / sg::BN), mt), sg::NTHR, 0, st>>>(g, N, nf, s, (int)R, oc, w);
    const unsigned one = (unsigned)R, four = (unsigned)((R + 3) / 4);
    if (nf <= 16)
      k_g_invert<16, 1><<<four, 128, 0, st>>>(N, nf, s, (int)R, oc, w, of, ld_full, od, ld_dense, kg, la, sg_);
    else if (nf <= 32)
      k_g_invert<32, 1><<<four, 128, 0, st>>>(N, nf, s, (int)R, oc, w, of, ld_full, od, ld_dense, kg, la, sg_);
    else if (nf <= 48)
      k_g_invert<48, 4><<<one, 128, 0, st>>>(N, nf, s, (int)R, oc, w, of, ld_full, od, ld_dense, kg, la, sg_);
    else
      k_g_invert<64, 4><<<one, 128, 0, st>>>(N, nf, s, (int)R, oc, w, of, ld_full, od, ld_dense, kg, la, sg_);
    const int kchunk = (int)(((nout + splits - 1) / splits + sg::BK - 1) / sg::BK * sg::BK);
    k_g_dh2<<<dim3(HID / sg::BN, mt, (unsigned)splits), sg::NTHR, 0, st>>>(g, (int)nout, (int)R, kchunk, w);
    k_g_dz1<<<(unsigned)((R * HID + 255) / 256), 256, 0, st>>>(g, N, nf, R * HID, s, oc, w);
    k_g_dz0<<<dim3(HID / sg::BN, mt), sg::NTHR, 0, st>>>(g, (int)R, w);
    if (od) k_g_write<<<dim3((unsigned)R, 4), 256, 0, st>>>(N, nf, s, oc, w, od, ld_dense, 0);
    if (of) k_g_write<<<dim3((unsigned)R, 32), 256, 0, st>>>(N, nf, s, oc, w, of, ld_full, 1);
  }
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}
