// Slater-determinant walkers: one or two warps per walker.
//
// Per-walker state (global memory, owned by the caller):
//   occ[2]          packed up / down bits
//   slot_orb[nf]    orbital held by each row slot of A (A[k] = M[slot_orb[k]])
//   G[nf][nf]       G[k][c] = (A^-1)[c][k]  (column k of the inverse, contiguous)
//   sign, logabs    psi(x) = sign * exp(logabs), with psi = det(M[ascending occupied rows])
//   n_acc           accepted moves since the last full re-inversion
//
// The slot order drifts away from the ascending row order as moves are
// accepted; the reordering sign is tracked combinatorially (parity of the
// occupied orbitals passed over) so that sign always refers to the ascending
// (reference) row order.  A full re-inversion resets the slots to ascending
// order.
#include "common.cuh"

using namespace vmc;

namespace {

constexpr int kMaxNf = 64;

__device__ __forceinline__ int gstride(int nf) { return nf + 1; }

// 1/|d| for finite d != 0 (rcp_pos, common.cuh) with d's sign.
__device__ __forceinline__ double rcp_signed(double d) { return copysign(rcp_pos(fabs(d)), d); }

__device__ __forceinline__ double dot_row(const double* __restrict__ Mrow, const double* Grow, int nf) {
  double acc = 0.0;
  for (int c = 0; c < nf; ++c) acc = fma(Mrow[c], Grow[c], acc);
  return acc;
}

__device__ __forceinline__ int find_slot(const uint8_t* slot, int nf, int orb) {
  const int lane = threadIdx.x & 31;
  unsigned b0 = __ballot_sync(VMC_FULL_MASK, lane < nf && slot[lane] == orb);
  if (b0) return __ffs(b0) - 1;
  unsigned b1 = __ballot_sync(VMC_FULL_MASK, lane + 32 < nf && slot[lane + 32] == orb);
  return b1 ? 31 + __ffs(b1) : -1;
}

// ---------------------------------------------------------------------------
// Full re-inversion: in-place Gauss-Jordan exchange steps with partial
// pivoting on the nf x nf matrix in registers (NT = nf rounded up to a tile).
// An FP64 instruction takes a warp 64 clocks of its SM quarter on GB300, so the
// nf^3 multiply-adds are the limit: the matrix is inverted in place (the
// augmented [A | I] form takes twice as many), and a walker's matrix is spread
// over NW warps so that all four quarters work on it (NT > 32: 4 warps of a
// CTA, NT / 8 x NT / 16 elements a thread; smaller: one warp, NT / 4 x NT / 8).
// Thread (ty, tx) holds the elements (ty + TY i, tx + TX j).  Step k exchanges
// row variable p (the pivot row, searched over the rows not used yet) with
// column variable k:
//   a_ij -= a_ik v_j,  a_ik = a_ik / d,  a_pj = -v_j,  a_pk = 1 / d,
//   v_j = a_pj / d, d = a_pk,
// one multiply-add per element with the operands of row p and column k
// replaced.  No rows move: with p_k the pivot row of step k the inverse is
// A^-1[k][p_j] = a[p_k][j], and the parity of the permutation k -> p_k is
// counted from the unused rows above each pivot row.  Resets slots to
// ascending occupied order.  A singular matrix gives sign 0, logabs -inf and G = 0; a
// non-finite entry (NaN or Inf parameters) NaN sign and log-amplitude.
template <int NT, int NW>
__global__ void __launch_bounds__(128) k_slater_refresh(
    const double* __restrict__ M, int nf, int N, const uint64_t* __restrict__ occ, int64_t B, double* __restrict__ G,
    uint8_t* __restrict__ slot_orb, double* __restrict__ sign, double* __restrict__ logabs, int32_t* __restrict__ n_acc,
    int threshold, int* __restrict__ n_singular) {
  constexpr int TX = NW == 4 ? 16 : 8, TY = 32 * NW / TX, NI = NT / TY, NJ = NT / TX;
  constexpr int PER = NT * (NT + 1) + 4 * NT;     // doubles per walker
  extern __shared__ __align__(16) double sm[];
  const int tid = NW == 4 ? threadIdx.x : (threadIdx.x & 31), lane = threadIdx.x & 31;
  const int64_t w = NW == 4 ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (w >= B) return;
  if (threshold > 0 && n_acc && n_acc[w] < threshold) return;
  auto sync = [] { if (NW == 4) __syncthreads(); else __syncwarp(); };
  double* base = sm + (NW == 4 ? 0 : (size_t)(threadIdx.x >> 5) * PER);
  double* gst = base;                       // staged G, NT x (NT + 1)
  double* col = gst + NT * (NT + 1);        // column k
  double* prow = col + NT;                  // pivot row
  double* dpiv = prow + NT;                 // pivots
  uint8_t* pof = reinterpret_cast<uint8_t*>(dpiv + NT);   // p_k
  uint8_t *kof = pof + NT, *sl = kof + NT;                // its inverse; the slots' orbitals
  const uint64_t up = occ[2 * w], dn = occ[2 * w + 1];
  const int tx = tid % TX, ty = tid / TX;
  const double qnan = __longlong_as_double(0x7ff8000000000000ll);
  if (__popcll(up) + __popcll(dn) != nf) {
    // wrong electron count for this orbital matrix: report singular, leave a
    // well-formed (all-zero) state so later kernels never index with garbage
    for (int k = tid; k < nf; k += 32 * NW) slot_orb[w * nf + k] = 0;
    for (int idx = tid; idx < nf * nf; idx += 32 * NW) G[w * nf * nf + idx] = 0.0;
    if (tid == 0) {
      sign[w] = 0.0;
      logabs[w] = -INFINITY;
      if (n_acc) n_acc[w] = 0;
      if (n_singular) atomicAdd(n_singular, 1);
    }
    return;
  }
  for (int o = tid; o < 2 * N; o += 32 * NW)   // ascending occupied orbitals -> slots
    if (orb_occupied(up, dn, N, o)) sl[orb_prefix(up, dn, N, o)] = (uint8_t)o;
  sync();
  double a[NI][NJ];
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int r = ty + TY * i, c = tx + TX * j;
      a[i][j] = (r < nf && c < nf) ? M[(int)sl[r] * nf + c] : (r == c ? 1.0 : 0.0);
    }
  if (tx == 0)
#pragma unroll
    for (int i = 0; i < NI; ++i) col[ty + TY * i] = a[i][0];
  uint64_t live = nf == 64 ? ~0ull : ((1ull << nf) - 1ull);   // rows not used as pivots yet
  int par = 0;
  bool ok = true, nonfinite = false;
#pragma unroll 1
  for (int k = 0; k < nf; ++k) {
    sync();   // column k complete
    // pivot: largest |a_ik| over the live rows, smallest row on a tie, from the
    // bit patterns (a NaN ranks above every number)
    unsigned h0 = 0, l0 = 0, h1 = 0, l1 = 0;
    const int r0 = lane % NT, r1 = lane + 32;
    if ((live >> r0) & 1ull) { const double v = fabs(col[r0]); h0 = (unsigned)__double2hiint(v) + 1u; l0 = (unsigned)__double2loint(v); }
    if (NT > 32 && r1 < NT && ((live >> (r1 & 63)) & 1ull)) {
      const double v = fabs(col[r1 < NT ? r1 : 0]);
      h1 = (unsigned)__double2hiint(v) + 1u;
      l1 = (unsigned)__double2loint(v);
    }
    const unsigned mh = __reduce_max_sync(VMC_FULL_MASK, max(h0, h1));
    const unsigned ml = __reduce_max_sync(VMC_FULL_MASK, max(h0 == mh ? l0 : 0u, h1 == mh ? l1 : 0u));
    const unsigned b0 = __ballot_sync(VMC_FULL_MASK, h0 == mh && l0 == ml);
    const unsigned b1 = __ballot_sync(VMC_FULL_MASK, h1 == mh && l1 == ml);
    const int p = b0 ? (__ffs(b0) - 1) % NT : 31 + __ffs(b1);
    if ((mh == 1u && ml == 0u) || mh >= 0x7ff00001u) {   // zero, or NaN / Inf
      nonfinite = mh >= 0x7ff00001u;
      ok = false;
      break;
    }
    const double d = col[p];
    const double r = rcp_signed(d);
    par ^= __popcll(live & ((1ull << p) - 1ull)) & 1;
    live &= ~(1ull << p);
    if (tid == 0) { dpiv[k] = d; pof[k] = (uint8_t)p; kof[p] = (uint8_t)k; }
    {
      const int pi = p / TY;
      const bool mine = ty == p % TY;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {   // selects: a branch per i would index the registers through local memory
        double v = a[0][j];
#pragma unroll
        for (int i = 1; i < NI; ++i) v = i == pi ? a[i][j] : v;
        if (mine) prow[tx + TX * j] = v;
      }
    }
    double u[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) u[i] = (ty + TY * i == p) ? -1.0 : -col[ty + TY * i];
    sync();   // pivot row complete, column k read
    const int jn = (k + 1) / TX;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = tx + TX * j;
      const double v = c == k ? -r : prow[c] * r;
#pragma unroll
      for (int i = 0; i < NI; ++i)
        a[i][j] = fma(u[i], v, (c == k || ty + TY * i == p) ? 0.0 : a[i][j]);
      if (j == jn && c == k + 1)
#pragma unroll
        for (int i = 0; i < NI; ++i) col[ty + TY * i] = a[i][j];
    }
  }
  sync();
  if (ok) {   // G[p_j][c] = A^-1[c][p_j] = a[p_c][j]
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int rr = ty + TY * i, c = tx + TX * j;
        if (rr < nf && c < nf) gst[(int)pof[c] * (NT + 1) + (int)kof[rr]] = a[i][j];
      }
  }
  sync();
  for (int idx = tid; idx < nf * nf; idx += 32 * NW) {
    const int k = idx / nf, c = idx - k * nf;
    G[w * nf * nf + idx] = ok ? gst[k * (NT + 1) + c] : 0.0;
  }
  for (int k = tid; k < nf; k += 32 * NW) slot_orb[w * nf + k] = sl[k];
  if (tid < 32) {
    double la = 0.0;
    int neg = 0;
    if (ok)
      for (int k = lane; k < nf; k += 32) { la += log(fabs(dpiv[k])); neg ^= dpiv[k] < 0.0; }
    la = warp_sum(la);
    neg = (__popc(__ballot_sync(VMC_FULL_MASK, neg)) & 1) ^ par;
    if (lane == 0) {
      sign[w] = ok ? (neg ? -1.0 : 1.0) : (nonfinite ? qnan : 0.0);
      logabs[w] = ok ? la : (nonfinite ? qnan : -INFINITY);
      if (n_acc) n_acc[w] = 0;
      if (!ok && !nonfinite && n_singular) atomicAdd(n_singular, 1);
    }
  }
}

// ---------------------------------------------------------------------------
// Metropolis sweep, WPW = ceil(nf / 32) warps a walker, a row of G a lane.  The
// FP64 pipe is the limit (64 clocks a warp instruction and SM quarter) and
// shared memory holds six 64-orbital walkers an SM: with two warps each they
// load the four quarters evenly.  Both warps of a walker decide every proposal
// for themselves (the acceptance ratio needs two to four products of length
// nf) and meet only when one is accepted.  4096 walkers, nf = 64, a step of
// the 8x8 lattice with its refreshes: 4.84 ms with one warp a walker, 4.43 with two.
template <int WPW>
__global__ void k_slater_sweep(const double* __restrict__ M, int nf, int N, uint64_t* __restrict__ occ, int64_t B,
                               const int32_t* __restrict__ edges, int E, int n_sweeps, float hopping_rate,
                               uint64_t seed, uint64_t sweep_offset, const float* __restrict__ r_move,
                               const uint8_t* __restrict__ r_bit, const float* __restrict__ r_acc,
                               double* __restrict__ G, uint8_t* __restrict__ slot_orb, double* __restrict__ sign,
                               double* __restrict__ logabs, int32_t* __restrict__ n_acc) {
  extern __shared__ double sm[];
  const int wib = threadIdx.x / (32 * WPW), lane = threadIdx.x & 31;   // walker in the block
  const int64_t w = (int64_t)blockIdx.x * (blockDim.x / (32 * WPW)) + wib;
  if (w >= B) return;
  const int t = threadIdx.x % (32 * WPW);                              // thread of the walker: its row
  auto meet = [wib] {
    if (WPW == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + wib), "r"(32 * WPW) : "memory");
  };
  const int gsd = gstride(nf);
  const int per = nf * gsd + 2 * nf + 8 + 4;
  double* g = sm + (size_t)wib * per;
  double* tmp = g + nf * gsd;
  double* Rs = tmp + 2 * nf;
  uint8_t* sl = (uint8_t*)(Rs + 4);
  for (int idx = t; idx < nf * nf; idx += 32 * WPW) {
    int k = idx / nf, c = idx - k * nf;
    g[k * gsd + c] = G[w * nf * nf + idx];
  }
  for (int k = t; k < nf; k += 32 * WPW) sl[k] = slot_orb[w * nf + k];
  uint64_t up = occ[2 * w], dn = occ[2 * w + 1];
  double sg = sign[w], la = logabs[w];
  int nacc = n_acc[w];
  meet();
  double* row = g + (t < nf ? t : 0) * gsd;   // threads past nf compute row 0's products, unused
  double rm = 1.0;
  int re = 0;
  for (int s = 0; s < n_sweeps; ++s) {
    for (int e = 0; e < E; ++e) {
      const int i = edges[2 * e], j = edges[2 * e + 1];
      const int xi = site_state(up, dn, i), xj = site_state(up, dn, j);
      if (xi == xj) continue;
      float u_move, u_acc;
      int bit;
      if (r_move) {
        size_t ridx = ((size_t)s * E + e) * (size_t)B + (size_t)w;
        u_move = r_move[ridx]; bit = r_bit[ridx] & 1; u_acc = r_acc[ridx];
      } else {
        EdgeDraw d = draw_edge(seed, (uint64_t)w, sweep_offset + (uint64_t)s, (uint32_t)e);
        u_move = d.u_move; bit = d.bit; u_acc = d.u_acc;
      }
      int ni, nj;
      propose_pair(xi, xj, u_move, bit, hopping_rate, ni, nj);
      Moves mv = pair_moves(i, j, xi, ni, N);
      const int k1 = find_slot(sl, nf, mv.a[0]);
      const int k2 = (mv.n == 2) ? find_slot(sl, nf, mv.a[1]) : -1;
      if (k1 < 0 || (mv.n == 2 && k2 < 0)) continue;  // inconsistent slot table: never index with it
      int par = reorder_parity(up, dn, N, mv.a[0], mv.b[0]);
      uint64_t up1 = up, dn1 = dn;
      apply_move(up1, dn1, N, mv.a[0], mv.b[0]);
      if (mv.n == 2) {
        par ^= reorder_parity(up1, dn1, N, mv.a[1], mv.b[1]);
        apply_move(up1, dn1, N, mv.a[1], mv.b[1]);
      }
      const double* m1 = M + (size_t)mv.b[0] * nf;
      const double* m2 = (mv.n == 2) ? M + (size_t)mv.b[1] * nf : m1;
      // acceptance ratio: the products of the new orbital rows with the
      // replaced rows of G only (lane = column); the products with every row
      // follow on acceptance
      double r;
      {
        const double* g1 = g + k1 * gsd;
        double q0 = 0.0, q1 = 0.0, q2 = 0.0, q3 = 0.0;
        if (mv.n == 2) {
          const double* g2 = g + k2 * gsd;
          for (int c = lane; c < nf; c += 32) {
            const double x1 = m1[c], x2 = m2[c], y1 = g1[c], y2 = g2[c];
            q0 = fma(x1, y1, q0); q1 = fma(x1, y2, q1); q2 = fma(x2, y1, q2); q3 = fma(x2, y2, q3);
          }
          // four sums at once: each exchange halves the values a lane carries
          const bool hi16 = lane & 16, hi8 = lane & 8;
          double s0 = hi16 ? q2 : q0, s1 = hi16 ? q3 : q1;
          s0 += __shfl_xor_sync(VMC_FULL_MASK, hi16 ? q0 : q2, 16);
          s1 += __shfl_xor_sync(VMC_FULL_MASK, hi16 ? q1 : q3, 16);
          double t = hi8 ? s1 : s0;
          t += __shfl_xor_sync(VMC_FULL_MASK, hi8 ? s0 : s1, 8);
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(VMC_FULL_MASK, t, o);
          const double R00 = __shfl_sync(VMC_FULL_MASK, t, 0), R01 = __shfl_sync(VMC_FULL_MASK, t, 8);
          const double R10 = __shfl_sync(VMC_FULL_MASK, t, 16), R11 = __shfl_sync(VMC_FULL_MASK, t, 24);
          r = R00 * R11 - R01 * R10;
        } else {
          for (int c = lane; c < nf; c += 32) q0 = fma(m1[c], g1[c], q0);
          r = warp_sum(q0);
        }
      }
      if (!((double)u_acc < r * r)) continue;
      // accept: rank-1 / rank-2 inverse update; the new rows' products with this thread's row first
      double w1 = 0.0, w2 = 0.0;
      if (mv.n == 2) {
#pragma unroll 4
        for (int c = 0; c < nf; ++c) {
          const double y = row[c];
          w1 = fma(m1[c], y, w1);
          w2 = fma(m2[c], y, w2);
        }
      } else {
#pragma unroll 4
        for (int c = 0; c < nf; ++c) w1 = fma(m1[c], row[c], w1);
      }
      if (t == k1) { Rs[0] = w1; Rs[2] = w2; }
      if (t == k2) { Rs[1] = w1; Rs[3] = w2; }
      for (int c = t; c < nf; c += 32 * WPW) {
        tmp[c] = g[k1 * gsd + c];
        if (mv.n == 2) tmp[nf + c] = g[k2 * gsd + c];
      }
      meet();
      const double R00 = Rs[0];
      double R01 = 0.0, R10 = 0.0, R11 = 0.0;
      if (mv.n == 2) {
        R01 = Rs[1];
        R10 = Rs[2];
        R11 = Rs[3];
        r = R00 * R11 - R01 * R10;
      } else {
        r = R00;
      }
      const double ir = rcp_signed(r);
      if (t < nf) {
        const double v1 = w1 - (t == k1 ? 1.0 : 0.0);
        if (mv.n == 2) {
          const double v2 = w2 - (t == k2 ? 1.0 : 0.0);
          const double alpha = (R11 * v1 - R01 * v2) * ir, beta = (-R10 * v1 + R00 * v2) * ir;
#pragma unroll 4
          for (int c = 0; c < nf; ++c) row[c] = fma(-beta, tmp[nf + c], fma(-alpha, tmp[c], row[c]));
        } else {
          const double alpha = v1 * ir;
#pragma unroll 4
          for (int c = 0; c < nf; ++c) row[c] = fma(-alpha, tmp[c], row[c]);
        }
      }
      if (t == 0) {
        sl[k1] = (uint8_t)mv.b[0];
        if (mv.n == 2) sl[k2] = (uint8_t)mv.b[1];
      }
      meet();
      up = up1; dn = dn1;
      sg *= ((r < 0) != (par != 0)) ? -1.0 : 1.0;
      // log|psi| as a running product of the ratios, renormalised to a mantissa
      // in [1, 2) and an exponent (one logarithm per launch; r is finite and
      // not zero here, |r| > sqrt(u))
      rm *= fabs(r);
      const int hi = __double2hiint(rm);
      if ((unsigned)((hi >> 20) - 1) < 0x7feu) {
        re += (hi >> 20) - 1023;
        rm = __hiloint2double((hi & 0xfffff) | (1023 << 20), __double2loint(rm));
      } else {           // subnormal or overflowed product
        la += log(rm);
        rm = 1.0;
      }
      ++nacc;
    }
  }
  la += log(rm) + (double)re * 0.69314718055994530942;
  for (int idx = t; idx < nf * nf; idx += 32 * WPW) {
    int k = idx / nf, c = idx - k * nf;
    G[w * nf * nf + idx] = g[k * gsd + c];
  }
  for (int k = t; k < nf; k += 32 * WPW) slot_orb[w * nf + k] = sl[k];
  if (t == 0) {
    occ[2 * w] = up; occ[2 * w + 1] = dn;
    sign[w] = sg; logabs[w] = la; n_acc[w] = nacc;
  }
}

// ---------------------------------------------------------------------------
// E_loc(x) = U * #doublons + sum_hops (-t) (-1)^{symmray parity} psi(eta)/psi(x),
// with psi(eta)/psi(x) = (-1)^{reorder parity} * M[b] . A^-1[:, slot(a)].
__global__ void k_slater_eloc(const double* __restrict__ M, int nf, int N, const uint64_t* __restrict__ occ,
                              int64_t B, const int32_t* __restrict__ edges, int E, double t, double U,
                              const double* __restrict__ G, const uint8_t* __restrict__ slot_orb,
                              double* __restrict__ eloc) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  __shared__ int8_t orb2slot_all[8][128];
  if (w >= B) return;
  int8_t* o2s = orb2slot_all[warp];
  for (int o = lane; o < 128; o += 32) o2s[o] = -1;
  __syncwarp();
  for (int k = lane; k < nf; k += 32) {
    const int o = slot_orb[w * nf + k];
    if (o < 2 * N) o2s[o] = (int8_t)k;
  }
  __syncwarp();
  const uint64_t up = occ[2 * w], dn = occ[2 * w + 1];
  const double* g = G + (size_t)w * nf * nf;
  double acc = 0.0;
  for (int term = lane; term < 2 * E; term += 32) {
    const int e = term >> 1, s = (term & 1) ? 0 : 1;
    int i = edges[2 * e], j = edges[2 * e + 1];
    if (i > j) { int tt = i; i = j; j = tt; }
    const uint64_t m = s ? up : dn;
    const int oi = (int)((m >> i) & 1ull), oj = (int)((m >> j) & 1ull);
    if (oi == oj) continue;
    const int base = s ? 0 : N;
    const int a = base + (oi ? i : j), b = base + (oi ? j : i);
    const int k = o2s[a];
    if (k < 0) continue;  // inconsistent state (zero amplitude walker)
    double r = dot_row(M + (size_t)b * nf, g + (size_t)k * nf, nf);
    if (reorder_parity(up, dn, N, a, b)) r = -r;
    const double c = symmray_parity(up, dn, i, j, s) ? t : -t;
    acc = fma(c, r, acc);
  }
  acc = warp_sum(acc);
  if (lane == 0) eloc[w] = acc + U * (double)__popcll(up & dn);
}

// O[w][o*nf + c] = G[slot(o)][c] for occupied o, else 0.
__global__ void k_slater_grad(const double* __restrict__ G, const uint8_t* __restrict__ slot_orb, int64_t B,
                              int n_orb, int nf, double* __restrict__ O, int64_t ldo) {
  __shared__ int8_t o2s[128];
  const int64_t w = blockIdx.x;
  for (int o = threadIdx.x; o < 128; o += blockDim.x) o2s[o] = -1;
  __syncthreads();
  for (int k = threadIdx.x; k < nf; k += blockDim.x) {
    const int o = slot_orb[w * nf + k];
    if (o < n_orb) o2s[o] = (int8_t)k;
  }
  __syncthreads();
  const double* g = G + (size_t)w * nf * nf;
  for (int idx = threadIdx.x; idx < n_orb * nf; idx += blockDim.x) {
    const int o = idx / nf, c = idx - o * nf;
    const int k = o2s[o];
    O[w * ldo + idx] = (k >= 0) ? g[k * nf + c] : 0.0;
  }
}

template <int NT, int NW>
int launch_refresh(const double* M, int nf, int N, const uint64_t* occ, int64_t B, double* G, uint8_t* slot_orb,
                   double* sign, double* logabs, int32_t* n_acc, int threshold, int* n_singular, cudaStream_t st) {
  constexpr int wpc = NW == 4 ? 1 : 4;   // walkers per CTA
  const size_t smem = (size_t)wpc * (NT * (NT + 1) + 4 * NT) * sizeof(double);
  cudaFuncSetAttribute(k_slater_refresh<NT, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_slater_refresh<NT, NW><<<(unsigned)((B + wpc - 1) / wpc), 128, smem, st>>>(M, nf, N, occ, B, G, slot_orb, sign,
                                                                              logabs, n_acc, threshold, n_singular);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}
size_t sweep_smem_per_walker(int nf) { return ((size_t)nf * (nf + 1) + 2 * nf + 8 + 4) * sizeof(double); }

int walkers_per_block(size_t per_walker) {
  size_t budget = 96 * 1024;
  int wpb = (int)(budget / per_walker);
  if (wpb < 1) wpb = 1;
  if (wpb > 8) wpb = 8;
  return wpb;
}

}  // namespace

extern "C" {

int vmc_slater_refresh(const double* M, int n_orb, int nf, const uint64_t* occ, int64_t B, int n_sites, double* G,
                       uint8_t* slot_orb, double* sign, double* logabs, int32_t* n_acc, int threshold,
                       int* d_n_singular, void* stream) {
  if (B < 0 || nf < 1 || nf > kMaxNf || n_sites < 1 || n_sites > 64 || n_orb != 2 * n_sites) return VMC_ERR_ARGS;
  if (B == 0) return VMC_OK;
  if (!M || !occ || !G || !slot_orb || !sign || !logabs) return VMC_ERR_ARGS;
  cudaStream_t st = (cudaStream_t)stream;
  // one warp a walker up to 32 (a barrier a step costs more than the idle
  // quarters there), four above, the tile no wider than nf asks for
  if (nf <= 16)
    return launch_refresh<16, 1>(M, nf, n_sites, occ, B, G, slot_orb, sign, logabs, n_acc, threshold, d_n_singular, st);
  if (nf <= 32)
    return launch_refresh<32, 1>(M, nf, n_sites, occ, B, G, slot_orb, sign, logabs, n_acc, threshold, d_n_singular, st);
  if (nf <= 48)
    return launch_refresh<48, 4>(M, nf, n_sites, occ, B, G, slot_orb, sign, logabs, n_acc, threshold, d_n_singular, st);
  return launch_refresh<64, 4>(M, nf, n_sites, occ, B, G, slot_orb, sign, logabs, n_acc, threshold, d_n_singular, st);
}

int vmc_slater_sweep(const double* M, int n_orb, int nf, uint64_t* occ, int64_t B, int n_sites, const int32_t* edges,
                     int n_edges, int n_sweeps, float hopping_rate, uint64_t seed, uint64_t sweep_offset,
                     const float* r_move, const uint8_t* r_bit, const float* r_acc, double* G, uint8_t* slot_orb,
                     double* sign, double* logabs, int32_t* n_acc, void* stream) {
  if (B < 0 || nf < 1 || nf > kMaxNf || n_sites < 1 || n_sites > 64 || n_orb != 2 * n_sites || n_edges < 0 ||
      n_sweeps < 0)
    return VMC_ERR_ARGS;
  if ((r_move != nullptr) != (r_acc != nullptr) || (r_move != nullptr) != (r_bit != nullptr)) return VMC_ERR_ARGS;
  if (B == 0 || n_sweeps == 0 || n_edges == 0) return VMC_OK;
  if (!M || !occ || !edges || !G || !slot_orb || !sign || !logabs || !n_acc) return VMC_ERR_ARGS;
  const size_t per = sweep_smem_per_walker(nf);
  const int wpb = walkers_per_block(per);
  const size_t smem = per * wpb;
  const unsigned grid = (unsigned)((B + wpb - 1) / wpb);
  cudaStream_t st = (cudaStream_t)stream;
  auto launch = [&](auto kernel, int warps) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kernel<<<grid, 32 * warps * wpb, smem, st>>>(M, nf, n_sites, occ, B, edges, n_edges, n_sweeps, hopping_rate, seed,
                                                 sweep_offset, r_move, r_bit, r_acc, G, slot_orb, sign, logabs, n_acc);
  };
  if (nf <= 32) launch(k_slater_sweep<1>, 1);
  else launch(k_slater_sweep<2>, 2);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

int vmc_slater_local_energy(const double* M, int n_orb, int nf, const uint64_t* occ, int64_t B, int n_sites,
                            const int32_t* edges, int n_edges, double t, double U, const double* G,
                            const uint8_t* slot_orb, double* eloc, void* stream) {
  if (B < 0 || nf < 1 || nf > kMaxNf || n_sites < 1 || n_sites > 64 || n_orb != 2 * n_sites || n_edges < 0)
    return VMC_ERR_ARGS;
  if (B == 0) return VMC_OK;
  if (!M || !occ || !G || !slot_orb || !eloc || (n_edges > 0 && !edges)) return VMC_ERR_ARGS;
  const int wpb = 8;
  k_slater_eloc<<<(unsigned)((B + wpb - 1) / wpb), 32 * wpb, 0, (cudaStream_t)stream>>>(
      M, nf, n_sites, occ, B, edges, n_edges, t, U, G, slot_orb, eloc);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

int vmc_slater_logpsi_grad(const double* G, const uint8_t* slot_orb, int64_t B, int n_orb, int nf, double* O,
                           int64_t ldo, void* stream) {
  if (B < 0 || nf < 1 || nf > kMaxNf || n_orb < nf || n_orb > 128 || ldo < (int64_t)n_orb * nf) return VMC_ERR_ARGS;
  if (B == 0) return VMC_OK;
  if (!G || !slot_orb || !O) return VMC_ERR_ARGS;
  k_slater_grad<<<(unsigned)B, 128, 0, (cudaStream_t)stream>>>(G, slot_orb, B, n_orb, nf, O, ldo);
  VMC_CUDA_CHECK_LAUNCH();
  return VMC_OK;
}

}  // extern "C"
