// Phase 1, formation of Q from stored reflectors on the FP64 tensor cores.
//
// M = Q^T = H_1 H_2 ... H_{n-1}, H_k = I + beta_k v_k v_k^T with v_k in rows
// 0 .. k-1.  Blocks of 16 reflectors are applied at once in compact form,
// M <- M + (M V) S V^T, S upper triangular (Schreiber and Van Loan 1989):
// S_jj = beta_j, S(0:j, j) = beta_j S(0:j, 0:j) (V(:, 0:j)^T v_j).
// Rows of M are independent, and row r (column r of Q) first changes at
// reflector r+1.
//
// A warp holds 8 rows of M in the accumulator layout of mma.sync m8n8k4: in
// tile t lane (g, q) = (lane / 4, lane % 4) has M(g, 8t + 2q + {0, 1}).  The
// same registers serve as the A operand of M V when the contraction index
// runs 0, 2, 4, 6 in one product and 1, 3, 5, 7 in the next, which costs
// nothing: the reflector panel in shared memory is read in that order.  So
// M stays in registers from the identity to the end, FP64 for both types.
#pragma once
#include "eigb_common.cuh"
#include "eigb_tridiag_sym.cuh"

namespace eigb {

// D = A B + D for one 8 x 8 tile, k = 4: this lane's A(g, q), B(q, g) and
// D(g, 2q), D(g, 2q + 1)
__device__ __forceinline__ void fq_dmma(double &d0, double &d1, const double a, const double b)
{
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// Block factors S for block J of one matrix, one warp: the Gram matrix of the
// block's 16 reflectors by mma, then S row by row (lane i < 16 row i).
// gs: 16 x 17 doubles of shared memory of this warp.
template <class T>
__device__ void fq_factor(const int n, const int J, const T *__restrict__ V, const int ldv,
                          const double *__restrict__ beta, double *__restrict__ S, double *gs)
{
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int ka = FQ_B * J + 1 + g, kb = ka + 8;  // this lane's reflectors
  const int rows = min(FQ_B * (J + 1), n - 1);
  const T *va = V + (size_t)ka * ldv, *vb = V + (size_t)kb * ldv;
  double c[3][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 4
  for (int r0 = 0; r0 < rows; r0 += 4) {
    const int r = r0 + q;
    const double a = (ka < n && r < ka) ? (double)va[r] : 0.0;
    const double b = (kb < n && r < kb) ? (double)vb[r] : 0.0;
    fq_dmma(c[0][0], c[0][1], a, a);
    fq_dmma(c[1][0], c[1][1], a, b);
    fq_dmma(c[2][0], c[2][1], b, b);
  }
#pragma unroll
  for (int x = 0; x < 2; x++) {
    gs[g * 17 + 2 * q + x] = c[0][x];
    gs[g * 17 + 8 + 2 * q + x] = c[1][x];
    gs[(8 + g) * 17 + 8 + 2 * q + x] = c[2][x];
  }
  __syncwarp();
  if (lane < FQ_B) {
    double s[FQ_B];
#pragma unroll
    for (int j = 0; j < FQ_B; j++) {
      const int k = FQ_B * J + 1 + j;
      const double b = k < n ? beta[k] : 0.0;
      double x = 0.0;
#pragma unroll
      for (int l = 0; l < j; l++) x = fma(s[l], gs[l * 17 + j], x);
      s[j] = j < lane ? 0.0 : (j == lane ? b : b * x);
    }
#pragma unroll
    for (int j = 0; j < FQ_B; j++) S[lane * FQ_B + j] = s[j];
  }
}

// pitch of a reflector in the panel (doubles) and panels that fit
__host__ __device__ inline int fq_lds(int n) { return (n + 15) & ~15; }
constexpr int FQ_LDT = 18;  // pitch of S in shared memory: the reads of its rows 2q conflict-free
__host__ __device__ inline size_t fq_smem_bytes(int n, int nbuf)
{
  return sizeof(double) * ((size_t)nbuf * (FQ_B * (size_t)fq_lds(n) + FQ_B * FQ_LDT) + 8 * 8 * FQ_B);
}

// Panel layout: entry (r, f) of reflector f at f * lds + 2 ((r / 2) ^ x(f)) +
// r % 2.  With this x both reads are free of bank conflicts: pairs of rows
// of two neighbouring reflectors (M V), and four rows of the reflectors
// 2q + s (X V^T).
__device__ __forceinline__ int fq_swz(const int f) { return (((f ^ (f >> 1)) & 1) << 2) | (((f >> 2) & 1) << 1); }

// Rows of M for NCG warps per 8 rows: warp (rg, cg) holds the NTL column
// tiles from cg * NTL on.  One CTA of 8 warps does 64 / NCG rows; the NCG
// partial products M V of a row group are exchanged through shared memory.
template <class T, int NTL, int NCG>
__device__ void form_q(T *A, const int nm, const int n, const int row_cta, const T *__restrict__ V, const int ldv,
                       const double *__restrict__ Sg, const int nbuf, double *sm)
{
  constexpr int RG = 8 / NCG;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int cgi = warp % NCG, rg = warp / NCG;
  const int r0 = row_cta + 8 * rg;
  const int lds = fq_lds(n), nJ = fq_blocks(n);
  double *Vs = sm;
  double *Ss = Vs + (size_t)nbuf * FQ_B * lds;
  double *Wx = Ss + (size_t)nbuf * FQ_B * FQ_LDT;

  auto fill = [&](const int J, const int buf) {
    double *D = Vs + (size_t)buf * FQ_B * lds;
    const int npair = 8 * (J + 1);  // row pairs of the panel
#pragma unroll
    for (int ff = 0; ff < 2; ff++) {
      const int f = 2 * warp + ff, k = FQ_B * J + 1 + f, x = fq_swz(f);
      const T *src = V + (size_t)k * ldv;
      for (int p = lane; p < npair; p += 32) {
        double *dst = D + f * lds + 2 * (p ^ x);
        if (k < n && 2 * p + 1 < k) {
          if (sizeof(T) == 8) {
            cp_async<16>(dst, src + 2 * p);
          } else {
            T a, b;
            const typename SymPair<T>::V v = *reinterpret_cast<const typename SymPair<T>::V *>(src + 2 * p);
            a = v.x;
            b = v.y;
            *reinterpret_cast<double2 *>(dst) = make_double2((double)a, (double)b);
          }
        } else {
          *reinterpret_cast<double2 *>(dst) = make_double2((k < n && 2 * p < k) ? (double)src[2 * p] : 0.0, 0.0);
        }
      }
    }
    cp_async<8>(Ss + buf * FQ_B * FQ_LDT + (t >> 4) * FQ_LDT + (t & 15), Sg + (size_t)J * FQ_B * FQ_B + t);
    cp_async_commit();
  };

  double M[NTL][2];
#pragma unroll
  for (int j = 0; j < NTL; j++) {
    const int c = 8 * (cgi * NTL + j) + 2 * q;
    M[j][0] = c == r0 + g ? 1.0 : 0.0;
    M[j][1] = c + 1 == r0 + g ? 1.0 : 0.0;
  }
  const int J0 = row_cta / FQ_B;
  if (J0 < nJ) fill(J0, 0);
  for (int J = J0; J < nJ; J++) {
    const int buf = nbuf == 2 ? (J - J0) & 1 : 0;
    cp_async_wait_all();
    __syncthreads();
    if (nbuf == 2 && J + 1 < nJ) fill(J + 1, buf ^ 1);
    const double *D = Vs + (size_t)buf * FQ_B * lds;
    const double *St = Ss + buf * FQ_B * FQ_LDT;
    const bool act = r0 < FQ_B * (J + 1) && r0 < n;
    const int nt = 2 * (J + 1) - cgi * NTL;  // this warp's tiles in the panel's rows
    double w[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    if (act && nt > 0) {
      double w1[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
      const int x0 = fq_swz(g), x1 = fq_swz(8 + g);
      const double *d0 = D + g * lds, *d1 = D + (8 + g) * lds;
#pragma unroll
      for (int j = 0; j < NTL; j++) {
        if (j < nt) {
          const int pr = 4 * (cgi * NTL + j) + q;
          const double2 b0 = *reinterpret_cast<const double2 *>(d0 + 2 * (pr ^ x0));
          const double2 b1 = *reinterpret_cast<const double2 *>(d1 + 2 * (pr ^ x1));
          fq_dmma(w[0][0], w[0][1], M[j][0], b0.x);
          fq_dmma(w[1][0], w[1][1], M[j][0], b1.x);
          fq_dmma(w1[0][0], w1[0][1], M[j][1], b0.y);
          fq_dmma(w1[1][0], w1[1][1], M[j][1], b1.y);
        }
      }
#pragma unroll
      for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) w[a][b] += w1[a][b];
    }
    if (NCG > 1) {
      if (act) {
        double *wx = Wx + warp * 8 * FQ_B + 4 * lane;
        *reinterpret_cast<double2 *>(wx) = make_double2(w[0][0], w[0][1]);
        *reinterpret_cast<double2 *>(wx + 2) = make_double2(w[1][0], w[1][1]);
      }
      __syncthreads();
      if (act) {
        w[0][0] = w[0][1] = w[1][0] = w[1][1] = 0.0;
#pragma unroll
        for (int c = 0; c < NCG; c++) {
          const double *wx = Wx + (rg * NCG + c) * 8 * FQ_B + 4 * lane;
          const double2 a = *reinterpret_cast<const double2 *>(wx);
          const double2 b = *reinterpret_cast<const double2 *>(wx + 2);
          w[0][0] += a.x;
          w[0][1] += a.y;
          w[1][0] += b.x;
          w[1][1] += b.y;
        }
      }
    }
    if (act && nt > 0) {
      double x[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int s = 0; s < 2; s++)
#pragma unroll
          for (int c = j; c < 2; c++)  // S(8..15, 0..7) = 0
            fq_dmma(x[c][0], x[c][1], w[j][s], St[(8 * j + 2 * q + s) * FQ_LDT + 8 * c + g]);
#pragma unroll
      for (int j = 0; j < NTL; j++) {
        if (j < nt) {
          const int r = 8 * (cgi * NTL + j) + g;
#pragma unroll
          for (int a = 0; a < 2; a++)
#pragma unroll
            for (int s = 0; s < 2; s++) {
              const int f = 8 * a + 2 * q + s;
              fq_dmma(M[j][0], M[j][1], x[a][s], D[f * lds + 2 * ((r >> 1) ^ fq_swz(f)) + (r & 1)]);
            }
        }
      }
    }
    if (nbuf == 1 && J + 1 < nJ) {
      __syncthreads();
      fill(J + 1, 0);
    }
  }
  // row r of M is column r of Q
  const int r = r0 + g;
  if (r < n) {
    T *Ar = A + (size_t)r * nm;
    const bool pairs = !(nm & 1) && (reinterpret_cast<uintptr_t>(A) % sizeof(typename SymPair<T>::V)) == 0;
#pragma unroll
    for (int j = 0; j < NTL; j++) {
      const int c = 8 * (cgi * NTL + j) + 2 * q;
      if (pairs && c + 1 < n) {
        typename SymPair<T>::V v;
        v.x = (T)M[j][0];
        v.y = (T)M[j][1];
        *reinterpret_cast<typename SymPair<T>::V *>(Ar + c) = v;
      } else {
        if (c < n) Ar[c] = (T)M[j][0];
        if (c + 1 < n) Ar[c + 1] = (T)M[j][1];
      }
    }
  }
}

}  // namespace eigb
