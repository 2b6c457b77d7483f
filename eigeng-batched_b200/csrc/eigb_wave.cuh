// Phase 3, wave form: K sweeps at a time pass over rows of Z in memory.
//
// The sweeps of the QL phase (segments of rotations, eigb_common.cuh) are
// taken K at a time, whatever their ranges, and run as a K-stage pipeline
// over the columns from the highest to the lowest: at step s column x =
// xtop - s enters, sweep j does its rotation x + j on the value that sweep
// j-1 hands it and on its carried value h[j], and column x + K leaves.  A
// sweep outside its range does the identity rotation, so the pipeline fills
// and drains without branches.  Every element receives the operations of the
// sweeps one after another, in that order.
//
// A thread has R rows.  A column is read and written once for K rotations
// (4 K arithmetic instructions a row), coalesced over the rows, so Z stays
// where it is, in a, and mostly in L2; what a row needs on chip is its K
// carried values.  The rotations of K sweeps are laid out step by step in
// shared memory by one more warp (two buffers of WV_S steps), which also
// walks the segment headers of the next group: every thread then reads them
// at consecutive addresses, as broadcasts.
#pragma once
#include "eigb_common.cuh"

namespace eigb {

constexpr int WV_S = 32;  // steps per record buffer

// records per step in shared memory: K and a pad that spreads the staging
// stores of consecutive steps over the banks
template <class T> __host__ __device__ constexpr int wv_pitch(int K) { return sizeof(T) == 8 ? K + 1 : K + 2; }

template <int K> struct WaveGroup {
  int pos[K], top[K], bot[K];  // first record and rotation range of each sweep (top < bot: none)
  int xtop, steps;
};

// rows staged at a time by the sorted write-back: 32 KB at most, so that the
// stage does not cost CTAs an SM (64 KB: n=512 FP64 two instead of three)
template <class T> __host__ __device__ inline int wv_perm_rows(int n)
{
  const int r = (int)(32768 / (sizeof(T) * (size_t)n));
  return r >= 32 ? 32 : (r >= 16 ? 16 : (r >= 8 ? 8 : 4));
}
template <class T> __host__ __device__ inline size_t wv_smem_bytes(int n, int K)
{
  const size_t recs = sizeof(Rec<T>) * 2 * WV_S * (size_t)wv_pitch<T>(K);
  const size_t perm = sizeof(T) * (size_t)n * wv_perm_rows<T>(n);
  const size_t sort = 2 * sizeof(T) * (size_t)n + 2 * sizeof(int) * (size_t)n;
  return (((recs > perm ? recs : perm) + 15) & ~(size_t)15) + sort;
}

// Two rotations of neighbouring sweeps from shared memory
__device__ __forceinline__ void wv_rec2(const Rec<double> *p, Rec<double> &a, Rec<double> &b)
{
  const double2 x = *reinterpret_cast<const double2 *>(p), y = *reinterpret_cast<const double2 *>(p + 1);
  a.c = x.x;
  a.s = x.y;
  b.c = y.x;
  b.s = y.y;
}
__device__ __forceinline__ void wv_rec2(const Rec<float> *p, Rec<float> &a, Rec<float> &b)
{
  const float4 x = *reinterpret_cast<const float4 *>(p);
  a.c = x.x;
  a.s = x.y;
  b.c = x.z;
  b.s = x.w;
}

// Rows row0 .. row0+nrow-1 of the matrix A; blockDim.x = 32 (warps of rows)
// + 32.  src/nrec: the records; ev: the unsorted eigenvalues.
// U columns are loaded ahead of the ones at work.
template <class T, int K, int R, int U>
__device__ void wave_apply(T *A, const int nm, const int n, const int row0, const int nrow, const Rec<T> *src,
                           const int nrec, const T *ev, const int sort, T *w_out, unsigned char *smem)
{
  constexpr int P = wv_pitch<T>(K);
  __shared__ WaveGroup<K> grp[2];
  __shared__ int more[2];  // whether the group in grp[.] exists
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nt = blockDim.x;
  const bool producer = warp == (nt >> 5) - 1;
  Rec<T> *rb = reinterpret_cast<Rec<T> *>(smem);

  // ---- the producer's part ----
  int wp = 0, wk = 0;                     // walk: next header, sweeps of the next group found
  int wtop = -1, wbot = n;                // their range
  auto walk = [&](WaveGroup<K> &g, const int upto) {  // lane 0: headers until sweep `upto` of the group
    while (wk < upto && wp < nrec) {
      const Rec<T> hd = src[wp];
      const int i0 = hdr_i0(hd), cnt = hdr_cnt(hd);
      g.pos[wk] = wp + 1;
      g.top[wk] = i0;
      g.bot[wk] = i0 - cnt + 1;
      wtop = max(wtop, i0);
      wbot = min(wbot, i0 - cnt + 1);
      wp += 1 + cnt;
      wk++;
    }
  };
  auto close = [&](WaveGroup<K> &g) -> int {  // lane 0: completes the group; 0 if it has no sweep
    walk(g, K);
    const int any = wk;
    for (int j = wk; j < K; j++) {
      g.pos[j] = 0;
      g.top[j] = -1;
      g.bot[j] = 0;
    }
    g.xtop = wtop + 1;
    g.steps = wtop + 2 - wbot + K;
    wk = 0;
    wtop = -1;
    wbot = n;
    return any;
  };
  auto stage = [&](const WaveGroup<K> &g, const int s0, Rec<T> *dst) {
    const int i0 = g.xtop - (s0 + lane);
#pragma unroll
    for (int j = 0; j < K; j++) {
      const int i = i0 + j;
      Rec<T> *d = dst + lane * P + j;
      if (i >= g.bot[j] && i <= g.top[j]) {
        cp_async<sizeof(Rec<T>)>(d, src + g.pos[j] + (g.top[j] - i));
      } else {
        Rec<T> id;
        id.c = T(1);
        id.s = T(0);
        *d = id;
      }
    }
    cp_async_commit();
  };

  if (producer) {
    if (lane == 0) more[0] = close(grp[0]);
    __syncwarp();
    if (more[0]) stage(grp[0], 0, rb);
    cp_async_wait_all();
  }
  __syncthreads();

  T *zr[R];
  bool own[R];
#pragma unroll
  for (int q = 0; q < R; q++) {
    const int r = (warp * R + q) * 32 + lane;
    own[q] = !producer && r < nrow;
    zr[q] = A + row0 + (own[q] ? r : 0);
  }
  int cur = 0, buf = 0;
  bool go = more[0] != 0;
  while (go) {
    const WaveGroup<K> &g = grp[cur];
    const int steps = g.steps, xtop = g.xtop, xbot = xtop - (steps - K) + 1;  // columns xbot .. xtop
    T h[K][R];
    T v[U][R];
#pragma unroll
    for (int j = 0; j < K; j++)
#pragma unroll
      for (int q = 0; q < R; q++) h[j][q] = T(0);
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int q = 0; q < R; q++)
        v[u][q] = (own[q] && xtop - u >= xbot) ? zr[q][(size_t)(xtop - u) * nm] : T(0);
    for (int s0 = 0; s0 < steps; s0 += WV_S) {
      const bool last = s0 + WV_S >= steps;
      if (producer) {
        Rec<T> *dst = rb + (buf ^ 1) * WV_S * P;
        if (!last) {
          stage(g, s0 + WV_S, dst);
          if (lane == 0) walk(grp[cur ^ 1], min(K, wk + 4));
        } else {
          if (lane == 0) more[cur ^ 1] = close(grp[cur ^ 1]);
          __syncwarp();
          if (more[cur ^ 1]) stage(grp[cur ^ 1], 0, dst);
        }
        cp_async_wait_all();
      } else {
        const Rec<T> *rs = rb + buf * WV_S * P;
        const int se = min(WV_S, steps - s0);
        for (int s = 0; s < se; s += U) {  // steps past the last are identities on zeros that are not stored
          const int x = xtop - s0 - s;
          T nv[U][R];
#pragma unroll
          for (int u = 0; u < U; u++)
#pragma unroll
            for (int q = 0; q < R; q++)
              nv[u][q] = (own[q] && x - U - u >= xbot) ? zr[q][(size_t)(x - U - u) * nm] : T(0);
#pragma unroll
          for (int u = 0; u < U; u++) {
#pragma unroll
            for (int j = 0; j < K; j += 2) {
              Rec<T> a, b;
              wv_rec2(rs + (s + u) * P + j, a, b);
#pragma unroll
              for (int q = 0; q < R; q++) {
                const T y = fma(a.c, h[j][q], a.s * v[u][q]);
                h[j][q] = fma(-a.s, h[j][q], a.c * v[u][q]);
                v[u][q] = fma(b.c, h[j + 1][q], b.s * y);
                h[j + 1][q] = fma(-b.s, h[j + 1][q], b.c * y);
              }
            }
            const int xo = x - u + K;
            if (xo <= xtop && xo >= xbot) {
#pragma unroll
              for (int q = 0; q < R; q++)
                if (own[q]) zr[q][(size_t)xo * nm] = v[u][q];
            }
          }
#pragma unroll
          for (int u = 0; u < U; u++)
#pragma unroll
            for (int q = 0; q < R; q++) v[u][q] = nv[u][q];
        }
      }
      __syncthreads();
      buf ^= 1;
    }
    cur ^= 1;
    go = more[cur] != 0;
  }

  // ---- DO_SORT: eigenvalues, and the columns of these rows, in order ----
  const size_t recs = sizeof(Rec<T>) * 2 * WV_S * (size_t)P, perm = sizeof(T) * (size_t)n * wv_perm_rows<T>(n);
  T *sd = reinterpret_cast<T *>(smem + (((recs > perm ? recs : perm) + 15) & ~(size_t)15));
  T *sdd = sd + n;
  int *inv = reinterpret_cast<int *>(sdd + n);
  int *pos = inv + n;
  for (int c = t; c < n; c += nt) sd[c] = ev[c];
  __syncthreads();
  bool bad = false, moved = false;
  for (int c = t; c < n; c += nt) {
    int cnt = c;
    if (sort) {
      const T dc = sd[c];
      cnt = 0;
      bad |= (dc != dc);
      for (int q = 0; q < n; q++) {
        const T dq = sd[q];
        cnt += (dq < dc) ? 1 : 0;
        bad |= (q != c) && (dq == dc);
      }
    }
    inv[c] = cnt;
    moved |= cnt != c;
  }
  if (__syncthreads_or(bad)) {
    if (t == 0) {
      for (int c = 0; c < n; c++) sdd[c] = sd[c];
      select_sort_serial(n, sdd, pos);
      for (int j = 0; j < n; j++) inv[pos[j]] = j;
    }
    moved = true;
    __syncthreads();
  }
  if (w_out)
    for (int c = t; c < n; c += nt) w_out[inv[c]] = sd[c];
  if (!__syncthreads_or(moved)) return;
  const int pr = wv_perm_rows<T>(n);  // a power of two
  T *tile = reinterpret_cast<T *>(smem);
  const int sh = 31 - __clz(pr);
  for (int q0 = 0; q0 < nrow; q0 += pr) {
    const int rows = min(pr, nrow - q0);
    T *Ar = A + row0 + q0;
#pragma unroll 4
    for (int idx = t; idx < n * pr; idx += nt) {
      const int rr = idx & (pr - 1), c = idx >> sh;
      if (rr < rows) tile[idx] = Ar[rr + (size_t)c * nm];
    }
    __syncthreads();
#pragma unroll 4
    for (int idx = t; idx < n * pr; idx += nt) {
      const int rr = idx & (pr - 1), c = idx >> sh;
      if (rr < rows) Ar[rr + (size_t)inv[c] * nm] = tile[idx];
    }
    __syncthreads();
  }
}

}  // namespace eigb
