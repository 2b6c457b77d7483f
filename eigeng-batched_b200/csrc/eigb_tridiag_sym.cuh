// Phase 1, symmetric on-chip form: Householder tridiagonalization with the
// upper triangle of the matrix in 32 x 32 blocks held in registers and
// shared memory, on one CTA or on a cluster of CTAs.
//
// The method is that of eigb_tridiag.cuh (bottom-up reduction,
// tred1_tiled.hpp:42-205).  Only blocks (R, C) with R <= C are kept.  Block
// g = C(C+1)/2 + R belongs to CTA g % CN and there, as local block
// l = g / CN, to warp l % NW, slot l / NW: the first RS slots of a warp are
// in its registers, the others in shared memory.  The numbering goes column
// by column, so the blocks still active at any step are a prefix and stay
// spread evenly over the CTAs and warps, and the blocks in shared memory are
// the ones that are finished first.
//
// A lane (lr, lc) = (lane & 3, lane >> 2) holds, of every block, rows
// 2 lr + 8 (j ^ (lane >> 3)) + {0, 1}, j < 4, and columns
// 2 lc + 16 (h ^ (lane >> 1 & 1)) + {0, 1}, h < 2.  One pass over a block
// applies the rank-2 update of the step before, and forms both products that
// a symmetric block takes part in (rows times v_C, columns times v_R): a
// lane sums 8 rows and 4 columns itself, and a reduce-scatter of 7 + 3
// exchanges leaves each lane one row's and one column's sum.  The exclusive
// ors make all but the last exchange of either free of selects: the values
// a lane sends are always those of the same registers.
#pragma once
#include <cooperative_groups.h>

#include "eigb_common.cuh"

namespace eigb {

namespace cg = cooperative_groups;

// Reflectors, their factors and the block factors of the formation of Q, per
// matrix, in the workspace: beta[n], S[nJ][16][16] (double), V[n][ldv] with
// reflector k in column k, rows 0 .. k-1.
constexpr int FQ_B = 16;  // reflectors per block of the formation of Q
__host__ __device__ inline int fq_blocks(int n) { return (n - 1 + FQ_B - 1) / FQ_B; }
__host__ __device__ inline int fq_ldv(int n) { return (n + 7) & ~7; }
__host__ __device__ inline size_t fq_off_s(int n) { return sizeof(double) * (size_t)((n + 1) & ~1); }
__host__ __device__ inline size_t fq_off_v(int n)
{
  return fq_off_s(n) + sizeof(double) * FQ_B * FQ_B * (size_t)fq_blocks(n);
}
template <class T> __host__ __device__ inline size_t fq_bytes(int n)
{
  return (fq_off_v(n) + sizeof(T) * (size_t)n * fq_ldv(n) + 15) & ~(size_t)15;
}

__host__ __device__ inline int sym_nbk(int n) { return (n + 31) / 32; }
__host__ __device__ inline int sym_nblk(int n) { return sym_nbk(n) * (sym_nbk(n) + 1) / 2; }
__host__ __device__ inline int sym_local(int n, int cn) { return (sym_nblk(n) + cn - 1) / cn; }
// CTAs exchange their sums whole (each gets all of all) for CN < 8; from 8
// on they go to the row block's home CTA first, which sends the total out.
__host__ __device__ constexpr bool sym_homes(int cn) { return cn >= 8; }
// Shared-memory elements: the blocks beyond the register slots, the row and
// column sums of every local block, (u, w, v), two buffers of the next
// column, the posted warp sums and scalars, and for CN > 1 the sums of the
// CTAs.
__host__ __device__ inline size_t sym_smem_elems(int n, int nw, int rs, int cn)
{
  const int nl = sym_local(n, cn), nr = 32 * sym_nbk(n);
  const int nsm = nl > nw * rs ? nl - nw * rs : 0;
  const int home = (sym_nbk(n) + cn - 1) / cn;
  return (size_t)nsm * 1024 + (size_t)nl * 64 + 5 * (size_t)nr + 2 * 32 + 8 +
         (cn > 1 ? (sym_homes(cn) ? (size_t)home * cn * 32 + nr : 2 * (size_t)cn * nr) + 2 * (size_t)cn : 0);
}

template <class T> struct SymPair;
template <> struct SymPair<double> { using V = double2; };
template <> struct SymPair<float> { using V = float2; };
template <class T> __device__ __forceinline__ void sld2(const T *p, T &a, T &b)
{
  const typename SymPair<T>::V v = *reinterpret_cast<const typename SymPair<T>::V *>(p);
  a = v.x;
  b = v.y;
}
template <class T> __device__ __forceinline__ void sst2(T *p, const T a, const T b)
{
  typename SymPair<T>::V v;
  v.x = a;
  v.y = b;
  *reinterpret_cast<typename SymPair<T>::V *>(p) = v;
}

// The pass over a block: S(j, e, h, f) (row pair j, row e of it, column pair
// h, column f of it) through `get`/`put`.  Adds the update of the step before
// (u, w), returns the sums with v of row 2 lr + 8 (lane >> 3) + (lane >> 2 & 1)
// and of column 2 lc + 16 (lane >> 1 & 1) + (lane & 1), and where cc >= 0
// hands column cc of the updated block to `col`.  xR, xC: (u, w, v) of the
// block's rows and columns, 32 each.
template <class T, class Get, class Put, class Col>
__device__ __forceinline__ void sym_block(const int lane, const T *__restrict__ xR, const T *__restrict__ xC, Get get,
                                          Put put, const int cc, Col col, T &rs, T &cs)
{
  const int lr = lane & 3, lc = lane >> 2, xj = lane >> 3, xh = (lane >> 1) & 1;
  T uc[2][2], wc[2][2], vc[2][2], yr[4][2], yc[2][2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const T *p = xC + 2 * lc + 16 * (h ^ xh);
    sld2(p, uc[h][0], uc[h][1]);
    sld2(p + 32, wc[h][0], wc[h][1]);
    sld2(p + 64, vc[h][0], vc[h][1]);
    yc[h][0] = yc[h][1] = T(0);
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const T *p = xR + 2 * lr + 8 * (j ^ xj);
    T ur[2], wr[2], vr[2];
    sld2(p, ur[0], ur[1]);
    sld2(p + 32, wr[0], wr[1]);
    sld2(p + 64, vr[0], vr[1]);
    T s[2][2][2];
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
      for (int h = 0; h < 2; h++) get(j, e, h, s[e][h][0], s[e][h][1]);
#pragma unroll
    for (int e = 0; e < 2; e++) {
      T y[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
#pragma unroll
        for (int f = 0; f < 2; f++) {
          s[e][h][f] = fma(wr[e], uc[h][f], fma(ur[e], wc[h][f], s[e][h][f]));
          yc[h][f] = fma(s[e][h][f], vr[e], yc[h][f]);
        }
        y[h] = fma(s[e][h][1], vc[h][1], s[e][h][0] * vc[h][0]);
      }
      yr[j][e] = y[0] + y[1];
    }
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
      for (int h = 0; h < 2; h++) put(j, e, h, s[e][h][0], s[e][h][1]);
    if (cc >= 0 && lc == ((cc >> 1) & 7)) {
      const bool h1 = (cc >> 4) ^ xh, f1 = cc & 1;
      const T a0 = f1 ? s[0][0][1] : s[0][0][0], a1 = f1 ? s[0][1][1] : s[0][1][0];
      const T b0 = f1 ? s[1][0][1] : s[1][0][0], b1 = f1 ? s[1][1][1] : s[1][1][0];
      col(2 * lr + 8 * (j ^ xj), h1 ? a1 : a0, h1 ? b1 : b0);
    }
  }
  // rows: lanes 16 and 8 apart hold the other row pairs, lanes 4 apart split
  // the pair; columns: lanes 2 and 1 apart
  T k4[2][2], k2[2], c2[2];
#pragma unroll
  for (int e = 0; e < 2; e++) {
#pragma unroll
    for (int j = 0; j < 2; j++) k4[j][e] = yr[j][e] + __shfl_xor_sync(0xffffffffu, yr[j + 2][e], 16);
    c2[e] = yc[0][e] + __shfl_xor_sync(0xffffffffu, yc[1][e], 2);
  }
#pragma unroll
  for (int e = 0; e < 2; e++) k2[e] = k4[0][e] + __shfl_xor_sync(0xffffffffu, k4[1][e], 8);
  const bool he = lane & 4, hf = lane & 1;
  const T sr = he ? k2[0] : k2[1], sc = hf ? c2[0] : c2[1];
  rs = (he ? k2[1] : k2[0]) + __shfl_xor_sync(0xffffffffu, sr, 4);
  cs = (hf ? c2[1] : c2[0]) + __shfl_xor_sync(0xffffffffu, sc, 1);
}

// Range.  The recurrences form u.Au, of third degree in the matrix, and
// beta = 1 / (l anorm) of degree -2 in a column, so both ends of the exponent
// range limit them.  Powers of two, which are exact, keep them inside:
//  - the matrix is scaled so that its largest magnitude mx lies in
//    [2^K, 2^(K+1)), K as large as the third-degree sums of n <= 1024 allow:
//    they stay below 2^7 |A|^3 with |A| <= 2^10 mx, so 40 + 3 K < 1023 (127);
//  - a column whose squares sum to less than sym_tiny, far below the rest of
//    the matrix, has to be scaled to entries below 2 by itself.  From sym_tiny
//    on |v|^3 is a normal number with all its bits (640 * 3/2 < 1022 - 53;
//    66 * 3/2 < 126 - 24).  A reflector does not change with the length of
//    its u; only the subdiagonal entry is scaled back.
// So blocks of a matrix may differ by more than the square root of the range.
// Scaled columns are rare and the test for them must precede the pass over
// the matrix (1 to 3 % of the solve: n=12 70.6 -> 72.7 us, n=256 FP64 32.50 ->
// 32.69 ms), so a first run only notes beside the pass whether it met one (70.0
// us, 32.50 ms); a second run (SCALED) then starts from the input, which the
// first has left alone.
template <class T> __device__ __forceinline__ T sym_tiny() { return sizeof(T) == 8 ? (T)0x1p-640 : (T)0x1p-66; }
// to: the power of two for a largest magnitude mx > 0 to reach [2^K, 2^(K+1)); back: its inverse
template <class T> __device__ __forceinline__ void sym_pow2(const T mx, const int K, T &to, T &back)
{
  const int lim = sizeof(T) == 8 ? 1000 : 120;
  int k = 0;
  if (mx > T(0) && mx < (T)INFINITY) k = max(-lim, min(lim, ilogb(mx) - K));
  to = (T)ldexp(1.0, -k);
  back = (T)ldexp(1.0, k);
}
template <class T> __device__ __forceinline__ void sym_scale(const T mx, T &to, T &back)
{
  sym_pow2(mx, sizeof(T) == 8 ? 300 : 28, to, back);
}
template <class T> __device__ __forceinline__ T warp_max(T x)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmax_t(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// Sums of the one-CTA forms in an order that does not depend on the form (NW,
// RS), so that batches of any size, whose launches hand over at other orders
// (sym_next), give the same bits: |v|^2 by row blocks of 32, v.Av by blocks l %
// 8, those of a group from the last to the first.  The form of a cluster
// is fixed by the order instead, the two-warp forms of FP32 are in no chain, and
// orders up to 64 have but one form (ORD false).  Costs up to 1.6 % of a solve
// (FP64 n=128 L=4096 8.96 -> 9.11 ms, n=256 L=2048 32.48 -> 32.57); hand-overs at
// fixed orders instead would cost small batches 2 to 6 %, none at all large ones
// 2 to 4 %.
template <class T> __host__ __device__ constexpr bool sym_ord(int nw, int cn)
{
  return cn == 1 && (sizeof(T) == 8 || nw > 2);
}
// Two and four sums over a warp at once, with the additions of warp_sum: the
// one that sym_slot2 or sym_slot4 names.
template <class T> __device__ __forceinline__ T sym_half(const T a, const T b, const bool hi, const int o)
{
  T mine = a, other = b;
  if (hi) mine = b;
  if (hi) other = a;
  return mine + __shfl_xor_sync(0xffffffffu, other, o);
}
template <class T> __device__ __forceinline__ T sym_sum8(T s)
{
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
__device__ __forceinline__ int sym_slot2(const int lane) { return lane >> 4; }
template <class T> __device__ __forceinline__ T sym_sum2(const T a, const T b, const int lane)
{
  const T s = sym_half(a, b, lane & 16, 16);
  return sym_sum8(s + __shfl_xor_sync(0xffffffffu, s, 8));
}
__device__ __forceinline__ int sym_slot4(const int lane) { return lane >> 3; }
template <class T> __device__ __forceinline__ T sym_sum4(const T a, const T b, const T c, const T d, const int lane)
{
  const T x = sym_half(a, c, lane & 16, 16), y = sym_half(b, d, lane & 16, 16);
  return sym_sum8(sym_half(x, y, lane & 8, 8));
}

// One step i (i = n-1 .. 1) removes column i with the reflector u whose raw
// entries v are the rows < i of that column: u = v - anorm e_{i-1}, so
//   A u = A v - anorm A e_{i-1},   u.A u = v.Av - 2 anorm (A v)_{i-1} + anorm^2 A_{i-1,i-1},
// and the pass over the blocks needs v alone; the square root and the
// reciprocal that give anorm and beta run beside it in one warp.  Per step:
//   tail     every thread for its rows: y = A v from the posted block sums,
//            p = beta (y - anorm a_{i-1}), w = p + alpha u; column i-1
//            of the updated matrix, which is the next v; its norm posted
//   barrier  (CTA)
//   pass     every block: rank-2 update with (u, w), products with v, the
//            column after the next handed over
//   barrier  (CTA), and for CN > 1 the CTAs' sums exchanged: every CTA
//            gets all of them (or their totals, sym_homes) and computes the
//            tail for all rows itself
//   barrier  (cluster)
//
// Reduces the leading n x n block of A down to order `stop` (0: to the end),
// where it leaves the updated leading block in A's blocks (R <= C) for a call
// with fewer warps or CTAs; `first` is the call on the whole matrix.  Returns
// true if it has to be run again with SCALED; A is as it was then.
template <class T, int NW, int RS, int CN, bool SCALED, bool ORD = sym_ord<T>(NW, CN)>
__device__ __forceinline__ bool tridiag_sym(T *A, const int nm, const int n, const int stop, const bool first,
                                            const T *Ap, T *d_out, T *e_out, T *V, const int ldv, double *beta_out,
                                            T *sm)
{
  constexpr int NT = 32 * NW;
  // a warp's groups of blocks, and the posted sums that can differ from 0
  constexpr int NG = !ORD ? 1 : (NW < 2 ? 4 : 8 / NW);
  constexpr int NSG = !ORD ? NW : (2 * NW < (sizeof(T) == 8 ? 8 : 12) ? 2 * NW : (sizeof(T) == 8 ? 8 : 12));
  constexpr int NDT = !ORD ? NW : (NW < 2 ? 4 : 8);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int rank = CN > 1 ? (int)(blockIdx.x % CN) : 0;
  const int nbk = sym_nbk(n), nr = 32 * nbk, nblk = sym_nblk(n), nl = sym_local(n, CN);
  const int nsm = nl > NW * RS ? nl - NW * RS : 0;
  T *blk = sm;
  T *prow = blk + (size_t)nsm * 1024;
  T *pcol = prow + (size_t)nl * 32;
  T *uwv = pcol + (size_t)nl * 32;  // [nbk][3][32]
  T *cb = uwv + 3 * nr;  // 2 * nr
  T *dotp = cb + 2 * nr; // 32
  T *sg = dotp + 32;     // 32
  T *sc = sg + 32;       // 8: anorm, beta, ul, whether a column was tiny, the factor of a scaled column's e
  T *dg = sc + 8;        // 2 * CN
  T *yg = dg + (CN > 1 ? 2 * CN : 0);  // the CTAs' sums: 2 * CN * nr, or nr totals and home * CN * 32
  T *yh = yg + nr;

  const int lr = lane & 3, lc = lane >> 2, xj = lane >> 3, xh = (lane >> 1) & 1;
  auto elem = [&](int r, int c) -> T {  // element (r, c) of the input, 0 outside
    // the blocks on the diagonal are kept in full, their halves rounded apart, and handed over so
    const int a = first ? min(r, c) : r, b = first ? max(r, c) : c;
    if (!first && r >= n) return T(0);
    if (b >= n) return T(0);
    return Ap ? Ap[a + (size_t)b * (b + 1) / 2] : A[a + (size_t)b * nm];
  };

  // ---- blocks of this warp ----
  T mx = T(0);  // largest magnitude
  T S[RS][32];
  int bR[RS], bC[RS];  // block rows and columns of the register slots
#pragma unroll
  for (int s = 0; s < RS; s++) {
    const int g = (s * NW + warp) * CN + rank;
    bR[s] = 0;
    bC[s] = 1 << 20;  // never active
    if (g < nblk) {
      int c = 0;
      while ((c + 1) * (c + 2) / 2 <= g) c++;
      bC[s] = c;
      bR[s] = g - c * (c + 1) / 2;
    }
#pragma unroll
    for (int x = 0; x < 32; x++)  // x = ((j * 2 + e) * 2 + h) * 2 + f
      S[s][x] = g < nblk ? elem(32 * bR[s] + 2 * lr + 8 * ((x >> 3) ^ xj) + ((x >> 2) & 1),
                                32 * bC[s] + 2 * lc + 16 * (((x >> 1) & 1) ^ xh) + (x & 1))
                         : T(0);
#pragma unroll
    for (int x = 0; x < 32; x++) mx = fmax_t(mx, fabs_t(S[s][x]));
  }
  for (int l = RS * NW + warp; l < nl; l += NW) {
    const int g = l * CN + rank;
    if (g >= nblk) break;
    int c = 0;
    while ((c + 1) * (c + 2) / 2 <= g) c++;
    const int r = g - c * (c + 1) / 2;
    T *B = blk + (size_t)(l - RS * NW) * 1024;
#pragma unroll
    for (int x = 0; x < 16; x++) {
      const int rr = 32 * r + 2 * lr + 8 * ((x >> 2) ^ xj) + ((x >> 1) & 1), cl = 32 * c + 2 * lc + 16 * ((x & 1) ^ xh);
      const T a0 = elem(rr, cl), a1 = elem(rr, cl + 1);
      sst2(B + (x * 32 + lane) * 2, a0, a1);
      mx = fmax_t(mx, fmax_t(fabs_t(a0), fabs_t(a1)));
    }
  }
  for (int r = t; r < nr; r += NT) {
    T *x = uwv + 96 * (r >> 5) + (r & 31);
    x[0] = x[32] = x[64] = T(0);
    cb[((n - 1) & 1) * nr + r] = elem(r, n - 1);
  }
  if (first && rank == 0 && t == 0) e_out[n - 1] = T(0);
  if (t < 8) sc[t] = T(0);
  for (int q = t; q < 64; q += NT) dotp[q] = T(0);  // and sg
  // scale: the largest magnitude of the CTA, then of the cluster's CTAs
  mx = warp_max(mx);
  if (lane == 0) prow[warp] = mx;  // prow is free until the first pass
  // A CTA's shared memory may be written by another only once it runs: the
  // cluster meets before the first such store.
  if (CN > 1) cg::this_cluster().sync();
  else __syncthreads();
  mx = T(0);
  for (int q = 0; q < NW; q++) mx = fmax_t(mx, prow[q]);
  if (CN > 1) {
    if (t < CN) *cg::this_cluster().map_shared_rank(dg + rank, t) = mx;
    cg::this_cluster().sync();
    mx = T(0);
    for (int q = 0; q < CN; q++) mx = fmax_t(mx, dg[q]);
  }
  T to, back;
  sym_scale(mx, to, back);
#pragma unroll
  for (int s = 0; s < RS; s++)
#pragma unroll
    for (int x = 0; x < 32; x++) S[s][x] *= to;
  for (int l = RS * NW + warp; l < nl && l * CN + rank < nblk; l += NW) {
    T *B = blk + (size_t)(l - RS * NW) * 1024 + 2 * lane;
#pragma unroll
    for (int x = 0; x < 16; x++) {
      T a0, a1;
      sld2(B + x * 64, a0, a1);
      sst2(B + x * 64, a0 * to, a1 * to);
    }
  }
  for (int r = t; r < nr; r += NT) cb[((n - 1) & 1) * nr + r] *= to;
  if (CN > 1) cg::this_cluster().sync();  // also: dg is free for the first step's sums
  else __syncthreads();

  for (int i = n - 1;; --i) {
    // ---- tail of step i+1: column i of the updated matrix ----
    const T *cbi = cb + (i & 1) * nr;
    const T anorm = sc[0], beta = sc[1], ul = sc[2];
    T dsum = T(0), yi = T(0);
    const int nact = (i >> 5) + 1;  // block columns that step i+1 touched
    if (i < n - 1) {
      if (CN > 1) {
        const T *y0 = yg + (sym_homes(CN) ? 0 : (size_t)(i & 1) * CN * nr);
        const T *d0 = dg + (i & 1) * CN;
#pragma unroll
        for (int q = 0; q < CN; q++) dsum += d0[q];
#pragma unroll
        for (int q = 0; q < (sym_homes(CN) ? 1 : CN); q++) yi += y0[(size_t)q * nr + i];
      } else {
        T a1 = T(0);
#pragma unroll
        for (int q = 0; q < NDT; q += 2) {
          T x0, x1;
          sld2(dotp + q, x0, x1);
          dsum += x0;
          a1 += x1;
        }
        dsum += a1;
        const int R = i >> 5, ri = i & 31;
        const T *pc = pcol + (size_t)(R * (R + 1) / 2) * 32 + ri;
        yi = prow[(size_t)(R * (R + 1) / 2 + R) * 32 + ri];
        T y1 = T(0);
#pragma unroll 4
        for (int j = 0; j < R; j++) y1 += pc[32 * j];
        yi += y1;
      }
    }
    const T ci = cbi[i];
    const T pi = beta * fma(-anorm, ci, yi);
    const T uau = fma(anorm * anorm, ci, fma(T(-2) * anorm, yi, dsum));
    const T alpha = T(0.5) * beta * (beta * uau);
    const T wi = fma(alpha, ul, pi);
    T sig = T(0), sig1 = T(0);  // of the warp's first row block, and its second
    for (int r = t; r < nr; r += NT) {
      T *xr = uwv + 96 * (r >> 5) + (r & 31);
      T u = T(0), w = T(0), v = T(0);
      if (r <= i) {
        T y = T(0);
        if (i < n - 1) {
          if (CN > 1) {
            const T *y0 = yg + (sym_homes(CN) ? 0 : (size_t)(i & 1) * CN * nr) + r;
#pragma unroll
            for (int q = 0; q < (sym_homes(CN) ? 1 : CN); q++) y += y0[(size_t)q * nr];
          } else {
            const int R = r >> 5, ri = r & 31;
            const T *pc = pcol + (size_t)(R * (R + 1) / 2) * 32 + ri;
            T y1 = T(0);
#pragma unroll 4
            for (int j = 0; j < R; j++) y += pc[32 * j];
            int g = R * (R + 1) / 2 + R;
#pragma unroll 4
            for (int c = R; c < nact; c++) {
              y1 += prow[(size_t)g * 32 + ri];
              g += c + 1;
            }
            y += y1;
          }
        }
        const T c = cbi[r];
        u = r == i ? ul : xr[64];
        w = fma(alpha, u, beta * fma(-anorm, c, y));
        const T x = fma(w, ul, fma(u, wi, c));
        if (r == i) {
          if (rank == 0 && i >= stop) d_out[i] = x * back;
        } else {
          v = x;
        }
        if (rank == 0 && i < n - 1) V[(size_t)(i + 1) * ldv + r] = u;
      }
      xr[0] = u;
      xr[32] = w;
      xr[64] = v;
      const bool second = ORD && r != t;
      sig1 = second ? v * v : sig1;
      sig = second ? sig : fma(v, v, sig);
    }
    if (i == 0) break;
    if (i < stop) {  // i = stop - 1: the pending update alone, and the block goes out
      const bool again = sc[3] != T(0);
      __syncthreads();
      if (again) return true;
      auto out = [&](const int l, auto get) {
        const int g = l * CN + rank;
        int C = 0;
        while ((C + 1) * (C + 2) / 2 <= g) C++;
        const int R = g - C * (C + 1) / 2;
        const T *xR = uwv + 96 * R, *xC = uwv + 96 * C;
#pragma unroll
        for (int x = 0; x < 32; x++) {
          const int r = 2 * lr + 8 * ((x >> 3) ^ xj) + ((x >> 2) & 1), c = 2 * lc + 16 * (((x >> 1) & 1) ^ xh) + (x & 1);
          const T v = fma(xR[32 + r], xC[c], fma(xR[r], xC[32 + c], get(x)));
          A[32 * R + r + (size_t)(32 * C + c) * nm] = v * back;
        }
      };
      const int nout = (stop / 32) * (stop / 32 + 1) / 2;
      for (int l = RS * NW + warp; l * CN + rank < nout; l += NW) {
        const T *B = blk + (size_t)(l - RS * NW) * 1024 + 2 * lane;
        out(l, [&](const int x) { return B[(x >> 1) * 64 + (x & 1)]; });
      }
#pragma unroll
      for (int s = 0; s < RS; s++)
        if ((s * NW + warp) * CN + rank < nout) out(s * NW + warp, [&](const int x) { return S[s][x]; });
      return false;
    }
    if (!ORD) {
      sig = warp_sum(sig);
      if (lane == 0) sg[warp] = sig;
    } else {
      sig = sym_sum2(sig, sig1, lane);
      if ((lane & 15) == 0) sg[warp + NW * sym_slot2(lane)] = sig;
    }
    __syncthreads();
    if constexpr (SCALED) {
      T s = T(0), eb = T(1);
      for (int q = 0; q < NSG; q++) s += sg[q];
      if (s < sym_tiny<T>()) {
        T mv = T(0), up;
        for (int r = t; r < nr; r += NT) mv = fmax_t(mv, fabs_t(uwv[96 * (r >> 5) + 64 + (r & 31)]));
        mv = warp_max(mv);
        if (lane == 0) dotp[warp] = mv;  // free until the end of the pass
        __syncthreads();
        for (int q = 0; q < NW; q++) mv = fmax_t(mv, dotp[q]);
        sym_pow2(mv, 0, up, eb);
        sig = sig1 = T(0);
        for (int r = t; r < nr; r += NT) {
          T *x = uwv + 96 * (r >> 5) + 64 + (r & 31);
          const T v = *x * up;
          *x = v;
          const bool second = ORD && r != t;
          sig1 = second ? v * v : sig1;
          sig = second ? sig : fma(v, v, sig);
        }
        if (!ORD) {
          sig = warp_sum(sig);
          if (lane == 0) sg[warp] = sig;
        } else {
          sig = sym_sum2(sig, sig1, lane);
          if ((lane & 15) == 0) sg[warp + NW * sym_slot2(lane)] = sig;
        }
      }
      if (t == 0) sc[4] = eb;
      __syncthreads();
    }

    // ---- the reflector's scalars, in the last warp ----
    if (warp == NW - 1) {
      T s0 = T(0), s1 = T(0);
#pragma unroll
      for (int q = 0; q < NSG; q += 2) {
        T x0, x1;
        sld2(sg + q, x0, x1);
        s0 += x0;
        s1 += x1;
      }
      const T last = uwv[96 * ((i - 1) >> 5) + 64 + ((i - 1) & 31)];
      const T an = -copysign_t(sqr_t(s0 + s1), last);
      const T l = last - an;
      const T b = T(1) / flip0to1(l * an);
      if (lane == 0) {
        sc[0] = an;
        sc[1] = b;
        sc[2] = l;
        if (rank == 0) {
          e_out[i - 1] = (SCALED ? an * sc[4] : an) * back;
          beta_out[i] = (double)b;
        }
      }
      // l an is in [-2, -1] |v|^2; 0 for a v whose squares vanish, or no v
      if (!SCALED && (b <= T(-1) / sym_tiny<T>() || b > T(0))) {
        bool any = b < T(0);
        for (int r = lane; r < i; r += 32) any |= uwv[3 * (r - lane) + 64 + lane] != T(0);
        if (__any_sync(0xffffffffu, any) && lane == 0) sc[3] = T(1);
      }
    }

    // ---- pass over the blocks ----
    const int ca = (i - 1) >> 5;  // last active block column, which holds column i-1
    const int par = (i - 1) & 1;
    T dot[NG];
#pragma unroll
    for (int a = 0; a < NG; a++) dot[a] = T(0);
    const int myr = 2 * lr + 8 * xj + ((lane >> 2) & 1);
    const int myc = 2 * lc + 16 * xh + (lane & 1);
    auto put_col = [&](const int R) {
      return [=](const int r, const T x0, const T x1) {
        T *dst = cb + par * nr + 32 * R + r;
        if (CN > 1) {
#pragma unroll
          for (int q = 0; q < CN; q++) sst2(cg::this_cluster().map_shared_rank(dst, q), x0, x1);
        } else {
          sst2(dst, x0, x1);
        }
      };
    };
    // blocks in shared memory, from the last active one
    const int nact1 = ((ca + 1) * (ca + 2) / 2 - rank + CN - 1) / CN - 1 - warp;  // local blocks active, less 1 + warp
    for (int l = warp + (nact1 & ~(NW - 1)); l >= RS * NW; l -= NW) {
      const int g = l * CN + rank;
      int C = (int)((sqrtf(8.0f * (float)g + 1.0f) - 1.0f) * 0.5f);
      if ((C + 1) * (C + 2) / 2 <= g) C++;
      if (C * (C + 1) / 2 > g) C--;
      const int R = g - C * (C + 1) / 2;
      T *B = blk + (size_t)(l - RS * NW) * 1024 + 2 * lane;
      T rsum, csum;
      sym_block<T>(
          lane, uwv + 96 * R, uwv + 96 * C,
          [&](int j, int e, int h, T &x0, T &x1) { sld2(B + ((j * 2 + e) * 2 + h) * 64, x0, x1); },
          [&](int j, int e, int h, T x0, T x1) { sst2(B + ((j * 2 + e) * 2 + h) * 64, x0, x1); },
          C == ca ? ((i - 1) & 31) : -1, put_col(R), rsum, csum);
      prow[l * 32 + myr] = rsum;
      pcol[l * 32 + myc] = csum;
      const T z = rsum * (R == C ? T(1) : T(2)), vr = uwv[96 * R + 64 + myr];
#pragma unroll
      for (int a = 0; a < NG; a++) {
        const T x = fma(z, vr, dot[a]);
        dot[a] = NG == 1 || (l & 7) / NW == a ? x : dot[a];
      }
    }
#pragma unroll
    for (int s = RS - 1; s >= 0; s--) {
      if (bC[s] <= ca) {
        const int R = bR[s], C = bC[s], l = s * NW + warp;
        T rsum, csum;
        sym_block<T>(
            lane, uwv + 96 * R, uwv + 96 * C,
            [&](int j, int e, int h, T &x0, T &x1) {
              x0 = S[s][((j * 2 + e) * 2 + h) * 2];
              x1 = S[s][((j * 2 + e) * 2 + h) * 2 + 1];
            },
            [&](int j, int e, int h, T x0, T x1) {
              S[s][((j * 2 + e) * 2 + h) * 2] = x0;
              S[s][((j * 2 + e) * 2 + h) * 2 + 1] = x1;
            },
            C == ca ? ((i - 1) & 31) : -1, put_col(R), rsum, csum);
        prow[l * 32 + myr] = rsum;
        pcol[l * 32 + myc] = csum;
        dot[s % NG] = fma(rsum * (R == C ? T(1) : T(2)), uwv[96 * R + 64 + myr], dot[s % NG]);
      }
    }
    if constexpr (NG == 4) {
      const T x = sym_sum4(dot[0], dot[1], dot[2], dot[3], lane);
      if ((lane & 7) == 0) dotp[warp + NW * sym_slot4(lane)] = x;
    } else if constexpr (NG == 2) {
      const T x = sym_sum2(dot[0], dot[1], lane);
      if ((lane & 15) == 0) dotp[warp + NW * sym_slot2(lane)] = x;
    } else {
      const T x = warp_sum(dot[0]);
      if (lane == 0) dotp[warp] = x;
    }
    __syncthreads();

    if (CN > 1) {
      // this CTA's sums, to every CTA
      for (int r = t; r < i; r += NT) {
        const int R = r >> 5, ri = r & 31;
        T y = T(0);
        for (int j = 0; j <= ca; j++) {
          const int g = j < R ? R * (R + 1) / 2 + j : j * (j + 1) / 2 + R;
          if (g % CN == rank) y += (j < R ? pcol : prow)[(size_t)(g / CN) * 32 + ri];
        }
        if (sym_homes(CN)) {
          *cg::this_cluster().map_shared_rank(yh + ((R / CN) * CN + rank) * 32 + ri, R % CN) = y;
        } else {
          T *dst = yg + (size_t)(par * CN + rank) * nr + r;
#pragma unroll
          for (int q = 0; q < CN; q++) *cg::this_cluster().map_shared_rank(dst, q) = y;
        }
      }
      if (warp == NW - 1) {
        T x = lane < NW ? dotp[lane] : T(0);
        x = warp_sum(x);
        if (lane < CN) *cg::this_cluster().map_shared_rank(dg + par * CN + rank, lane) = x;
      }
      if (sym_homes(CN)) {
        cg::this_cluster().sync();
        for (int s = warp; s * CN + rank <= ca; s += NW) {  // row block s * CN + rank: its total, to every CTA
          const int R = s * CN + rank;
          T y0 = T(0), y1 = T(0);
#pragma unroll
          for (int q = 0; q < CN; q += 2) {
            y0 += yh[(s * CN + q) * 32 + lane];
            y1 += yh[(s * CN + q + 1) * 32 + lane];
          }
          y0 += y1;
          T *dst = yg + 32 * R + lane;
#pragma unroll
          for (int q = 0; q < CN; q++) *cg::this_cluster().map_shared_rank(dst, q) = y0;
        }
      }
      cg::this_cluster().sync();
    }
  }
  if (t == 0 && rank == 0) beta_out[0] = 0.0;
  const bool again = sc[3] != T(0);
  __syncthreads();  // a second run begins with its shared memory
  return again;
}

}  // namespace eigb
