// Symmetric matrix function of a solved batch: Z = V diag(f(w)) V^T.
//
// The reference ships this as a prototype, symdmt.cu:5-80 (z(i,j) =
// sum_k a(i,k) d(k) a(j,k), one warp per matrix, d supplied by the
// caller); its README:171 names the use: powers such as the square root or
// the inverse of a matrix right after its eigendecomposition (LETKF
// transforms, main.cpp:68-167).  Here f is applied on the fly:
//   SYMF_DIAG: f(x) = x         (d given by the caller in w, as symdmt)
//   SYMF_POW:  f(x) = pow(x, p) (p = 1/2 square root, -1 inverse, ...)
//   SYMF_EXP:  f(x) = exp(p x)
//
// The products run on the FP64 tensor cores (mma.sync m8n8k4) for both
// types.  A warp computes one 32 x 32 tile of Z on or above the diagonal (the
// 8 x 8 mma tiles below it are left out) and stores it to both triangles, so
// Z is exactly symmetric.  With lane (g, q) = (lane / 4, lane % 4), the A
// fragment V(i, k) and the B fragment V(j, k) of 8 rows and 4 columns are the
// same picture, row g, column q, so one panel of V serves both; f(w_k) scales
// B as it is loaded.
//   n <= 32   one warp per matrix, fragments straight from global memory
//   n <= 128  one CTA per matrix, a warp per tile: V is read once
//   above     one CTA of 8 warps per 128 x 64 block of Z, two CTAs an SM
// Panels keep the input's type; FP32 is widened as a fragment is loaded.
#pragma once
#include "eigb_common.cuh"

namespace eigb {

enum { SYMF_DIAG = 0, SYMF_POW = 1, SYMF_EXP = 2 };

constexpr int SF_KC = 16;     // columns of V per panel
// Pitch of a panel: 4 mod 16 doubles or 8 mod 32 floats, so that the fragment
// loads (four columns, rows of 8) are free of bank conflicts.
template <class T> __host__ __device__ constexpr int sf_ld() { return sizeof(T) == 8 ? 132 : 136; }

template <class T> __device__ __forceinline__ T symf_apply(const int func, const T x, const T p)
{
  if (func == SYMF_POW) return pow(x, p);
  if (func == SYMF_EXP) return exp(p * x);
  return x;
}

// upper-triangular tile index t -> (ti, tj), ti <= tj, row by row over the
// upper triangle of an nt x nt tile grid
__host__ __device__ __forceinline__ void symf_tile(int t, const int nt, int &ti, int &tj)
{
  ti = 0;
  while (t >= nt - ti) {
    t -= nt - ti;
    ti++;
  }
  tj = ti + t;
}
// the same, column by column
__host__ __device__ __forceinline__ void sf_tile(int t, int &ti, int &tj)
{
  tj = 0;
  while (t > tj) {
    t -= tj + 1;
    tj++;
  }
  ti = t;
}

__device__ __forceinline__ void sf_dmma(double (&d)[2], const double a, const double b)
{
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// the 32 x 32 tile at (i0, j0), i0 <= j0, to both triangles of Z
template <class T>
__device__ __forceinline__ void sf_store(T *Z, const int nm, const int n, const int i0, const int j0,
                                         const double (&acc)[4][4][2])
{
  const int g = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll
  for (int x = 0; x < 4; x++)
#pragma unroll
    for (int y = 0; y < 4; y++) {
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int i = i0 + 8 * x + g, j = j0 + 8 * y + 2 * q + e;
        if (i <= j && j < n) {
          const T v = (T)acc[x][y][e];
          Z[i + (size_t)j * nm] = v;
          Z[j + (size_t)i * nm] = v;
        }
      }
    }
}

// n <= 32, SFW_WARPS matrices per CTA
constexpr int SFW_WARPS = 4;
template <class T>
__global__ void __launch_bounds__(32 * SFW_WARPS) k_symfunc_w(const long L, const int nm, const int n,
                                                              const T *__restrict__ v, const T *__restrict__ w,
                                                              T *__restrict__ z, const int func, const T p)
{
  const long k = (long)blockIdx.x * SFW_WARPS + (threadIdx.x >> 5);
  if (k >= L) return;  // uniform per warp; no CTA barrier below
  const int g = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
  const T *V = v + (size_t)k * nm * n;
  const T *W = w + (size_t)k * n;
  double acc[4][4][2];
#pragma unroll
  for (int x = 0; x < 4; x++)
#pragma unroll
    for (int y = 0; y < 4; y++) acc[x][y][0] = acc[x][y][1] = 0.0;
  T a[8][4], f[8];  // all of V first: its loads overlap
#pragma unroll
  for (int s = 0; s < 8; s++) {
    const int c = 4 * s + q;
    f[s] = c < n ? W[c] : T(0);
#pragma unroll
    for (int x = 0; x < 4; x++) {
      const int i = 8 * x + g;
      a[s][x] = (c < n && i < n) ? V[i + (size_t)c * nm] : T(0);
    }
  }
#pragma unroll
  for (int s = 0; s < 8; s++) {
    if (4 * s >= n) break;
    const double fs = 4 * s + q < n ? (double)symf_apply(func, f[s], p) : 0.0;
#pragma unroll
    for (int y = 0; y < 4; y++) {
      const double b = fs * (double)a[s][y];
#pragma unroll
      for (int x = 0; x <= y; x++) sf_dmma(acc[x][y], (double)a[s][x], b);
    }
  }
  sf_store<T>(z + (size_t)k * nm * n, nm, n, 0, 0, acc);
}

// n > 32.  ONE (n <= 128): one CTA per matrix, a warp per tile on or above the
// diagonal.  Else a CTA of 8 warps per block of 128 rows (bi) and 64 columns
// (cj) that reaches the diagonal or lies above it, a warp per tile, those
// below the diagonal idle.  Two panels of SF_KC columns in flight; one panel
// holds the block's 128 rows and, unless they are among them, the rows of V
// that its 64 columns take.
// Nine loads from shared memory feed 16 mma, and each panel costs a barrier, so
// warps in flight count; above 128 also the idle tiles of the blocks at the
// diagonal and at the end (n=256: 18 TFLOP/s of the upper half).  Blocks of 128 x 64 with two CTAs an SM against
// 128 x 128 with 16 warps and one, both types as doubles in the panel, B200,
// ms: FP64 n=256 L=2048 2.18 / 1.87, n=512 L=256 1.85 / 1.59, n=1000 L=32
// 1.66 / 1.43; FP32 n=128 L=4096 0.47 / 0.42, n=201 L=1000 0.87 / 0.68.
template <class T> __host__ __device__ inline size_t symf_smem_bytes(int n)
{
  return sizeof(T) * 2 * (size_t)(n <= 128 ? 1 : 2) * SF_KC * sf_ld<T>() + sizeof(double) * (size_t)((n + 15) & ~15);
}
// column blocks of 64 of the row blocks before bi: those with 64 cj + 63 >= 128 b
__host__ __device__ inline int symf_blocks(int n)
{
  const int nc = (n + 63) / 64, nb = (n + 127) / 128;
  int t = 0;
  for (int b = 0; b < nb; b++) t += nc - 2 * b;
  return t;
}
template <class T, bool ONE>
__global__ void __launch_bounds__(ONE ? 320 : 256, 2) k_symfunc_tc(const int nm, const int n, const T *__restrict__ v,
                                                                   const T *__restrict__ w, T *__restrict__ z,
                                                                   const int func, const T p, const int per)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LD = sf_ld<T>();
  const long k = blockIdx.x / per;
  int bi = 0, cj = 0;
  if (!ONE) {
    int t = (int)(blockIdx.x % per);
    const int nc = (n + 63) / 64;
    while (t >= nc - 2 * bi) t -= nc - 2 * bi++;
    cj = 2 * bi + t;
  }
  const bool two = !ONE && cj >= 2 * bi + 2;  // the columns' rows are not among the block's
  const T *V = v + (size_t)k * nm * n;
  const T *W = w + (size_t)k * n;
  constexpr int PS = (ONE ? 1 : 2) * SF_KC * LD;
  double *fw = reinterpret_cast<double *>(smem_raw);
  T *panel = reinterpret_cast<T *>(fw + ((n + 15) & ~15));
  const int t = threadIdx.x, nt = blockDim.x, lane = t & 31, warp = t >> 5, g = lane >> 2, q = lane & 3;
  int ti, tj;  // tile in 32s
  if (ONE) {
    sf_tile(warp, ti, tj);
  } else {
    ti = 4 * bi + (warp & 3);
    tj = 2 * cj + (warp >> 2);
  }
  const int i0 = 32 * ti, j0 = 32 * tj;
  const bool act = i0 <= j0 && j0 < n;

  for (int c = t; c < ((n + 15) & ~15); c += nt) fw[c] = c < n ? (double)symf_apply(func, W[c], p) : 0.0;
  // panel of columns c0 .. c0+15: the block's rows (and its columns')
  auto fill = [&](const int c0, T *P) {
    for (int h = 0; h < (two ? 2 : 1); h++) {
      const int r0 = h == 0 ? 128 * bi : 64 * cj;
      const int rows = min(h == 0 ? 128 : 64, ((n - r0 + 31) & ~31));
      for (int c = warp; c < SF_KC; c += nt >> 5) {
        T *D = P + (h * SF_KC + c) * LD;
        const T *src = V + r0 + (size_t)(c0 + c) * nm;
        for (int r = lane; r < rows; r += 32) {
          if (c0 + c < n && r0 + r < n) cp_async<sizeof(T)>(D + r, src + r);
          else D[r] = T(0);
        }
      }
    }
    cp_async_commit();
  };
  double acc[4][4][2];
#pragma unroll
  for (int x = 0; x < 4; x++)
#pragma unroll
    for (int y = 0; y < 4; y++) acc[x][y][0] = acc[x][y][1] = 0.0;
  fill(0, panel);
  int cur = 0;
  for (int c0 = 0; c0 < n; c0 += SF_KC, cur ^= 1) {
    cp_async_wait_all();
    __syncthreads();
    if (c0 + SF_KC < n) fill(c0 + SF_KC, panel + (cur ^ 1) * PS);
    if (act) {
      const T *PA = panel + cur * PS + q * LD + i0 - 128 * bi + g;
      const T *PB = panel + cur * PS + q * LD + g + (two ? SF_KC * LD + j0 - 64 * cj : j0 - 128 * bi);
      const bool diag = i0 == j0;
#pragma unroll
      for (int s = 0; s < SF_KC / 4; s++) {
        double a[4], b[4];
        const double f = fw[c0 + 4 * s + q];
#pragma unroll
        for (int x = 0; x < 4; x++) {
          a[x] = (double)PA[4 * s * LD + 8 * x];
          b[x] = f * (double)PB[4 * s * LD + 8 * x];
        }
#pragma unroll
        for (int y = 0; y < 4; y++)
#pragma unroll
          for (int x = 0; x < 4; x++)
            if (x <= y || !diag) sf_dmma(acc[x][y], a[x], b[y]);
      }
    }
  }
  if (act) sf_store<T>(z + (size_t)k * nm * n, nm, n, i0, j0, acc);
}

}  // namespace eigb
