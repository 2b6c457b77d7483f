// Phase 1 for n <= 32: one warp per matrix, the matrix in registers.
//
// The reduction is that of eigb_tridiag_sym.cuh (same recurrences: products
// with the raw column, the norm's correction afterwards) on a single 32 x 32
// block held in full: lane (lr, lc) = (lane & 3, lane >> 2) has rows 2 lr +
// 8 (j ^ (lane >> 3)) + {0, 1}, j < 4, and columns 2 lc + 16 h + {0, 1}, so a
// step's update and product are 96 multiply-adds a lane and three exchanges
// sum the rows.  Lane r also owns row r of the vectors.  Then M = H_1 ...
// H_{n-1} with row r of M in lane r and the reflectors broadcast from shared
// memory, and Q = M^T goes out through shared memory.
#pragma once
#include "eigb_common.cuh"
#include "eigb_tridiag_sym.cuh"

namespace eigb {

constexpr int TW_LD = 34;  // pitch of the reflectors and of the staged matrix: even, for paired loads
// shared-memory elements per warp: reflectors / staging, (u, w, v), column and product, beta
__host__ __device__ constexpr int tw_smem_elems() { return 32 * TW_LD + 96 + 64 + 32; }

// Returns true, with A as it was, if it has to be run again with SCALED
// (see eigb_tridiag_sym.cuh).
template <class T, bool SCALED>
__device__ __forceinline__ bool tridiag_warp(T *A, const int nm, const int n, const T *Ap, T *d_out, T *e_out,
                                             T *sm)
{
  const int lane = threadIdx.x & 31;
  const int lr = lane & 3, lc = lane >> 2, xj = lane >> 3;
  T *V = sm;  // reflector k in V[k * TW_LD ..]
  T *uwv = V + 32 * TW_LD;
  T *cb = uwv + 96, *yb = cb + 32, *beta_s = yb + 32;

  // upper triangle through shared memory, then the block
  if (Ap) {
    for (int c = 0; c < n; c++)
      if (lane <= c) V[c * TW_LD + lane] = Ap[lane + c * (c + 1) / 2];
  } else {
#pragma unroll 8
    for (int c = 0; c < n; c++)
      if (lane <= c) V[c * TW_LD + lane] = A[lane + (size_t)c * nm];
  }
  __syncwarp();
  T S[4][2][2][2];  // row pair j, row e, column pair h, column f
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int f = 0; f < 2; f++) {
          const int r = 2 * lr + 8 * (j ^ xj) + e, c = 2 * lc + 16 * h + f;
          const int a = min(r, c), b = max(r, c);
          S[j][e][h][f] = b < n ? V[b * TW_LD + a] : T(0);
        }
  T mx = T(0);
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int f = 0; f < 2; f++) mx = fmax_t(mx, fabs_t(S[j][e][h][f]));
  T to, back;
  sym_scale(warp_max(mx), to, back);
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int f = 0; f < 2; f++) S[j][e][h][f] *= to;
  T col = lane < n ? V[(n - 1) * TW_LD + lane] * to : T(0);  // raw column i of the matrix before the pending update
  __syncwarp();
  uwv[lane] = uwv[32 + lane] = uwv[64 + lane] = T(0);

  const int myr = 2 * lr + 8 * xj + ((lane >> 2) & 1);  // the row whose sum this lane ends up with
  T anorm = T(0), beta = T(0), ul = T(0), dsum = T(0), y = T(0), v = T(0);
  for (int i = n - 1;; --i) {
    // tail of step i+1: column i of the updated matrix
    const T ci = __shfl_sync(0xffffffffu, col, i), yi = __shfl_sync(0xffffffffu, y, i);
    const T pi = beta * fma(-anorm, ci, yi);
    const T uau = fma(anorm * anorm, ci, fma(T(-2) * anorm, yi, dsum));
    const T alpha = T(0.5) * beta * (beta * uau);
    const T wi = fma(alpha, ul, pi);
    const T u = lane == i ? ul : (lane < i ? v : T(0));
    const T w = lane <= i ? fma(alpha, u, beta * fma(-anorm, col, y)) : T(0);
    const T x = fma(w, ul, fma(u, wi, col));
    if (lane == i) d_out[i] = x * back;
    if (i < n - 1) V[(i + 1) * TW_LD + lane] = u;
    v = lane < i ? x : T(0);
    if (i == 0) break;
    uwv[lane] = u;
    uwv[32 + lane] = w;
    uwv[64 + lane] = v;
    __syncwarp();
    // the reflector's scalars
    T sig = warp_sum(v * v), eb = T(1);  // eb: scales a scaled column's e back
    if constexpr (SCALED) {
      if (sig < sym_tiny<T>()) {
        T up;
        sym_pow2(warp_max(fabs_t(v)), 0, up, eb);
        v *= up;
        uwv[64 + lane] = v;
        __syncwarp();
        sig = warp_sum(v * v);
      }
    }
    const T last = __shfl_sync(0xffffffffu, v, i - 1);
    anorm = -copysign_t(sqr_t(sig), last);
    ul = last - anorm;
    beta = T(1) / flip0to1(ul * anorm);
    if (lane == 0) {
      e_out[i - 1] = anorm * eb * back;
      beta_s[i] = beta;
    }
    // update with (u, w), product with v, column i-1
    T uc[2][2], wc[2][2], vc[2][2], yr[4][2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const T *p = uwv + 2 * lc + 16 * h;
      sld2(p, uc[h][0], uc[h][1]);
      sld2(p + 32, wc[h][0], wc[h][1]);
      sld2(p + 64, vc[h][0], vc[h][1]);
    }
    const bool mine = lc == (((i - 1) >> 1) & 7), h1 = (i - 1) >> 4, f1 = (i - 1) & 1;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int rj = 2 * lr + 8 * (j ^ xj);
      T ur[2], wr[2];
      sld2(uwv + rj, ur[0], ur[1]);
      sld2(uwv + 32 + rj, wr[0], wr[1]);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        T s[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
#pragma unroll
          for (int f = 0; f < 2; f++)
            S[j][e][h][f] = fma(wr[e], uc[h][f], fma(ur[e], wc[h][f], S[j][e][h][f]));
          s[h] = fma(S[j][e][h][1], vc[h][1], S[j][e][h][0] * vc[h][0]);
        }
        yr[j][e] = s[0] + s[1];
      }
      if (mine) {
        const T a0 = f1 ? S[j][0][0][1] : S[j][0][0][0], a1 = f1 ? S[j][0][1][1] : S[j][0][1][0];
        const T b0 = f1 ? S[j][1][0][1] : S[j][1][0][0], b1 = f1 ? S[j][1][1][1] : S[j][1][1][0];
        sst2(cb + rj, h1 ? a1 : a0, h1 ? b1 : b0);
      }
    }
    T k4[2][2], k2[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
#pragma unroll
      for (int j = 0; j < 2; j++) k4[j][e] = yr[j][e] + __shfl_xor_sync(0xffffffffu, yr[j + 2][e], 16);
      k2[e] = k4[0][e] + __shfl_xor_sync(0xffffffffu, k4[1][e], 8);
    }
    const bool he = lane & 4;
    const T sr = he ? k2[0] : k2[1];
    yb[myr] = (he ? k2[1] : k2[0]) + __shfl_xor_sync(0xffffffffu, sr, 4);
    __syncwarp();
    col = cb[lane];
    y = yb[lane];
    dsum = warp_sum(v * y);
    __syncwarp();  // cb, yb and uwv are rewritten in the next step
  }
  if (lane == 0) e_out[n - 1] = T(0);
  __syncwarp();
  if (!SCALED) {  // a tiny column, by its beta = 1 / (l an) as in tridiag_sym
    const T b = lane > 0 && lane < n ? beta_s[lane] : T(-1);
    bool tiny = b <= T(-1) / sym_tiny<T>();
    if (b > T(0))
      for (int r = 0; r < lane; r++) tiny |= V[lane * TW_LD + r] != T(0);
    if (__any_sync(0xffffffffu, tiny)) return true;
  }

  // M <- M + beta_k (M u_k) u_k^T, row r in lane r
  T M[32];
#pragma unroll
  for (int c = 0; c < 32; c++) M[c] = c == lane ? T(1) : T(0);
  for (int k = 1; k < n; k++) {
    const T *uk = V + k * TW_LD;
    const T bk = beta_s[k];
    T a[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
    for (int c = 0; c < 32; c += 8) {
      if (c < k) {  // entries from k on are zero
        T q[8];
#pragma unroll
        for (int x = 0; x < 8; x += 2) sld2(uk + c + x, q[x], q[x + 1]);
#pragma unroll
        for (int x = 0; x < 8; x++) a[x & 3] = fma(M[c + x], q[x], a[x & 3]);
      }
    }
    const T g = bk * ((a[0] + a[1]) + (a[2] + a[3]));
#pragma unroll
    for (int c = 0; c < 32; c += 8) {
      if (c < k) {
        T q[8];
#pragma unroll
        for (int x = 0; x < 8; x += 2) sld2(uk + c + x, q[x], q[x + 1]);
#pragma unroll
        for (int x = 0; x < 8; x++) M[c + x] = fma(g, q[x], M[c + x]);
      }
    }
  }
  __syncwarp();
  // Q(c, r) = M(r, c): column r of Q from lane r's row
#pragma unroll
  for (int c = 0; c < 32; c += 2) sst2(V + lane * TW_LD + c, M[c], M[c + 1]);
  __syncwarp();
  if (lane < n)
    for (int c = 0; c < n; c++) A[lane + (size_t)c * nm] = V[c * TW_LD + lane];
  return false;
}

}  // namespace eigb
