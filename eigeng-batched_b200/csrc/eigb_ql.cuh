// Phase 2: QL iteration on the tridiagonal (d, e), emitting plane rotations.
//
// The eigenvalue recurrence of QL is a serial chain per matrix; it does not
// depend on the eigenvectors.  It therefore runs one matrix per thread
// (a warp advances 32 independent chains at once) and writes the rotations
// as a stream of records that phase 3 applies to Q with a whole team per
// matrix.  The same generator also runs inside phase 3 (one thread, small
// chunks) for the rare matrix whose stream exceeded its capacity.
//
// The generator is resumable: it returns when the output buffer is full,
// keeping every loop variable in QLGen, and continues from the same
// rotation on the next call.
//
// tql2: explicit-shift QL, tql2_tiled.hpp:3-192 / tql2.hpp:3-213.
// imtql2: implicit Wilkinson-shift QL, imtql2_tiled.hpp:3-176 / imtql2.hpp.
// Deflation tolerances, the sweep limit and the e(n) = 0 convention follow
// the reference; the rotation (c, s, r) is formed with one reciprocal
// square root (givens()) rather than hypot + two divisions.
#pragma once
#include "eigb_common.cuh"

namespace eigb {

enum { QL_TQL2 = 0, QL_IMTQL2 = 1 };
enum { PC_START = 0, PC_ROT = 1, PC_DONE = 2 };

template <class T> struct QLGen {
  int pc, l, m, i, itr, ierr;
  int seg_pos, seg_cnt, seg_i0;
  T shift, tst1, c, c2, c3, s, s2, p, el1, dl1, ei, di1, r, delta;
};

// Strided view of one chain's d and e (interleaved across the threads of a
// block so that divergent indices stay bank-conflict free).
template <class T> struct DEView {
  T *d, *e;
  int st;
  __host__ __device__ __forceinline__ T &D(int i) const { return d[i * st]; }
  __host__ __device__ __forceinline__ T &E(int i) const { return e[i * st]; }
};

// One tql2 chase step at index i (tql2_tiled.hpp:94-115): from the
// previous (c, s, p) and (e_i, d_i) to the new rotation (cn, sn), the new p
// and the values stored at i+1.  Shared by both generators.
//
// The next step waits for pn alone, so that is formed as y q with q = p d_i
// - c e_i^2 ready before y = 1/sqrt(p^2 + e_i^2).
template <class T> struct Tql2Step {
  T cn, sn, r, pn, gg, h;
};
template <class T> struct Tql2Pre {
  T sig, y, q, gg, h;
};
// what the step needs before its rotation, y on its way ...
template <class T>
__host__ __device__ __forceinline__ Tql2Pre<T> tql2_begin(const T c, const T p, const T ei, const T di)
{
  Tql2Pre<T> a;
  a.sig = fma(p, p, mul_rn(ei, ei));
  a.gg = mul_rn(c, ei);
  a.h = mul_rn(c, p);
  a.q = fma(p, di, -mul_rn(ei, a.gg));
  a.y = rsq_fast(a.sig);
  return a;
}
// ... and the rotation
template <class T>
__host__ __device__ __forceinline__ Tql2Step<T> tql2_end(const Tql2Pre<T> &a, const T p, const T ei, const T di)
{
  Tql2Step<T> k;
  k.gg = a.gg;
  k.h = a.h;
  k.cn = mul_rn(p, a.y);
  k.sn = mul_rn(ei, a.y);
  k.r = mul_rn(a.sig, a.y);
  k.pn = mul_rn(a.y, a.q);
  return k;
}
// the whole step, for p and e of any size
template <class T>
__host__ __device__ __forceinline__ Tql2Step<T> tql2_any(const T c, const T p, const T ei, const T di)
{
  const Tql2Pre<T> a = tql2_begin(c, p, ei, di);
  Tql2Step<T> k = tql2_end(a, p, ei, di);
  if (!rsq_plain(a.sig)) {
    givens_any(p, ei, k.cn, k.sn, k.r);
    k.pn = fma(k.cn, di, -mul_rn(k.sn, k.gg));
  }
  return k;
}
// the values stored at i+1, from the step's rotation and the s before it
template <class T> __host__ __device__ __forceinline__ T tql2_e1(const Tql2Step<T> &k, const T s) { return mul_rn(s, k.r); }
template <class T> __host__ __device__ __forceinline__ T tql2_d1(const Tql2Step<T> &k, const T di)
{
  return fma(k.sn, fma(k.cn, k.gg, mul_rn(k.sn, di)), k.h);
}

// Explicit shift of tql2 (tql2_tiled.hpp:64-75): new d(l), d(l+1).
template <class T>
__host__ __device__ __forceinline__ void tql2_shift(const T dl_old, const T dl1_old, const T el, T &dl, T &dl1)
{
  const T p = (dl1_old - dl_old) / (el + el);
  const T r = hypot1(p);
  const T psr = p + copysign_t(r, p);
  dl = el / psr;
  dl1 = mul_rn(el, psr);
}

// End of a tql2 sweep (tql2_tiled.hpp:126-130): new e(l), d(l).
template <class T>
__host__ __device__ __forceinline__ void tql2_close(const T c, const T s, const T s2, const T c3, const T el1,
                                                    const T ei, const T dl1, T &el, T &dl)
{
  const T r = mul_rn(mul_rn(mul_rn(mul_rn(-s, s2), c3), el1), ei) / dl1;
  el = mul_rn(s, r);
  dl = mul_rn(c, r);
}

// One imtql2 chase step (imtql2_tiled.hpp:86-115) after the rotation
// (cn, sn) has been formed: returns the new d(i+1) and updates di1, delta,
// r.
template <class T>
__host__ __device__ __forceinline__ T imtql2_step(const T cn, const T sn, const T c_old, const T ei, const T di,
                                                  T &di1, T &delta, T &r)
{
  const T b = mul_rn(c_old, ei);
  const T dix = di1 - delta;
  di1 = di;
  const T q = fma(di - dix, sn, mul_rn(T(2) * cn, b));
  const T dx1 = fma(sn, q, dix);
  delta = dx1 - dix;
  r = fma(cn, q, -b);
  return dx1;
}

// Wilkinson-type shift of imtql2 (imtql2_tiled.hpp:67-75).
template <class T>
__host__ __device__ __forceinline__ T imtql2_shift(const T dl, const T dl1, const T el, const T dm)
{
  const T f = (dl1 - dl) / (el + el);
  const T g = hypot1(f);
  return (dm - dl) + el / (f + copysign_t(g, f));
}

template <class T>
__host__ __device__ __forceinline__ void ql_close_seg(QLGen<T> &g, Rec<T> *buf)
{
  if (g.seg_pos >= 0) {
    buf[g.seg_pos] = make_hdr(g.seg_i0, g.seg_cnt, T(0));
    g.seg_pos = -1;
  }
}

// Runs until done or until `cap` records are in buf; returns the number of
// records written.  g.pc == PC_DONE when the iteration has finished; then
// g.ierr is 0 or the failing index l (1-based, tql2_tiled.hpp:138).
template <class T>
__host__ __device__ int ql_tql2(QLGen<T> &g, const DEView<T> v, const int n, Rec<T> *buf, const int cap,
                       const int max_sweep)
{
  const T tol = Num<T>::eps() * Num<T>::tolmul();
  int nrec = 0;
  if (g.pc == PC_DONE) return 0;
  if (g.pc == PC_ROT) goto resume_rot;
  g.ierr = 0;
  g.shift = T(0);
  g.tst1 = T(0);
  g.seg_pos = -1;
  if (n <= 1) goto finish;
  for (g.l = 0; g.l < n; g.l++) {
    {
      const T t = (fabs_t(v.D(g.l)) + fabs_t(v.E(g.l))) * tol;
      g.tst1 = fmax_t(g.tst1, t);
      int m = g.l;
      while (m < n && !(fabs_t(v.E(m)) <= g.tst1)) m++;
      if (m >= n) {  // only with NaN data
        g.ierr = g.l + 1;
        goto finish;
      }
      g.m = m;
    }
    if (g.m != g.l) {
      for (g.itr = 0; g.itr < max_sweep; g.itr++) {
        {  // explicit shift, tql2_tiled.hpp:64-80
          const int l = g.l;
          const T dl_old = v.D(l);
          T dl;
          tql2_shift(dl_old, v.D(l + 1), v.E(l), dl, g.dl1);
          v.D(l) = dl;
          v.D(l + 1) = g.dl1;
          g.delta = dl_old - dl;
          // d(j) -= delta for j >= l+2 (tql2_tiled.hpp:77-80): the sweep below
          // reads d(l+2..m) exactly once, before overwriting them, and
          // subtracts delta on that read; only d(m+1..n-1) are updated here.
          for (int j = g.m + 1; j < n; j++) v.D(j) -= g.delta;
          g.shift += g.delta;
        }
        g.c = T(1); g.c2 = T(1); g.c3 = T(1);
        g.s = T(0); g.s2 = T(0);
        g.p = (g.m >= g.l + 2) ? v.D(g.m) - g.delta : v.D(g.m);
        g.el1 = v.E(g.l + 1);
        g.ei = T(0);
        for (g.i = g.m - 1; g.i >= g.l; g.i--) {
          if (nrec + (g.seg_pos < 0 ? 2 : 1) > cap) {
            ql_close_seg(g, buf);
            g.pc = PC_ROT;
            return nrec;
          }
        resume_rot:
          if (g.seg_pos < 0) {
            g.seg_pos = nrec++;
            g.seg_cnt = 0;
            g.seg_i0 = g.i;
          }
          {  // QL step, tql2_tiled.hpp:94-115
            const int i = g.i;
            g.c3 = g.c2;
            g.c2 = g.c;
            g.s2 = g.s;
            const T ei = v.E(i);
            const T di = (i >= g.l + 2) ? v.D(i) - g.delta : v.D(i);
            const Tql2Step<T> k = tql2_any(g.c, g.p, ei, di);
            g.p = k.pn;
            v.E(i + 1) = tql2_e1(k, g.s);
            v.D(i + 1) = tql2_d1(k, di);
            g.c = k.cn;
            g.s = k.sn;
            g.ei = ei;
            Rec<T> rec;
            rec.c = k.cn;
            rec.s = k.sn;
            buf[nrec++] = rec;
            g.seg_cnt++;
          }
        }
        ql_close_seg(g, buf);
        {  // tql2_tiled.hpp:126-135
          T el, dl;
          tql2_close(g.c, g.s, g.s2, g.c3, g.el1, g.ei, g.dl1, el, dl);
          v.E(g.l) = el;
          v.D(g.l) = dl;
        }
        if (fabs_t(v.E(g.l)) <= g.tst1) break;
      }
      if (g.itr >= max_sweep) {
        g.ierr = g.l + 1;
        goto finish;
      }
    }
    v.D(g.l) += g.shift;
  }
finish:
  ql_close_seg(g, buf);
  g.pc = PC_DONE;
  return nrec;
}

template <class T>
__host__ __device__ int ql_imtql2(QLGen<T> &g, const DEView<T> v, const int n, Rec<T> *buf, const int cap,
                         const int max_sweep)
{
  const T tol = Num<T>::eps() * Num<T>::tolmul();
  int nrec = 0;
  if (g.pc == PC_DONE) return 0;
  if (g.pc == PC_ROT) goto resume_rot;
  g.ierr = 0;
  g.seg_pos = -1;
  if (n <= 1) goto finish;
  for (g.l = 0; g.l < n; g.l++) {
    for (g.itr = 0; g.itr <= max_sweep; g.itr++) {
      {  // deflation test, imtql2_tiled.hpp:56-61
        int m = n - 1;
        for (int mm = g.l; mm < n - 1; mm++) {
          const T t1 = (fabs_t(v.D(mm)) + fabs_t(v.D(mm + 1))) * tol;
          const T t2 = fabs_t(v.E(mm));
          if (!(t2 > t1)) {
            m = mm;
            break;
          }
        }
        g.m = m;
      }
      if (g.m == g.l) break;
      // Wilkinson-type shift, imtql2_tiled.hpp:67-75
      g.di1 = v.D(g.m);
      g.r = imtql2_shift(v.D(g.l), v.D(g.l + 1), v.E(g.l), g.di1);
      g.s = T(1);
      g.c = T(1);
      g.delta = T(0);
      for (g.i = g.m - 1; g.i >= g.l; g.i--) {
        if (nrec + (g.seg_pos < 0 ? 2 : 1) > cap) {
          ql_close_seg(g, buf);
          g.pc = PC_ROT;
          return nrec;
        }
      resume_rot:
        {  // imtql2_tiled.hpp:86-115
          const int i = g.i;
          const T ei = v.E(i);
          const T f = mul_rn(g.s, ei);
          T c, s, r;
          givens(g.r, f, c, s, r);
          if (r == T(0)) {
            g.r = T(0);
            break;
          }
          if (g.seg_pos < 0) {
            g.seg_pos = nrec++;
            g.seg_cnt = 0;
            g.seg_i0 = i;
          }
          const T dx1 = imtql2_step(c, s, g.c, ei, v.D(i), g.di1, g.delta, g.r);
          v.E(i + 1) = r;
          v.D(i + 1) = dx1;
          g.c = c;
          g.s = s;
          Rec<T> rec;
          rec.c = c;
          rec.s = s;
          buf[nrec++] = rec;
          g.seg_cnt++;
        }
      }
      ql_close_seg(g, buf);
      {
        const int j = (g.i + 1 > g.l) ? g.i + 1 : g.l;
        v.D(j) -= g.delta;
        v.E(j) = g.r;
        v.E(g.m) = T(0);
      }
    }
    if (g.itr > max_sweep) {
      g.ierr = g.l + 1;
      goto finish;
    }
  }
finish:
  ql_close_seg(g, buf);
  g.pc = PC_DONE;
  return nrec;
}

// ---------------------------------------------------------------------------
// Fast single-call forms used by phase 2: the whole iteration in one call
// with a fixed record capacity, no resume points, and the capacity checked
// once per sweep.  Same arithmetic as ql_tql2 / ql_imtql2 (identical
// rotations and eigenvalues).  Returns the record count, or -1 when the
// capacity would be exceeded (phase 3 then regenerates with the resumable
// form).  *ierr receives 0 or the failing 1-based index.
//
// Storage of a chain: element i of d and e at stride st, in two arrays
// (DESep) or, on the GPU, as pairs, one load and one store for both (DEPair).
template <class T> struct DESep {
  T *dp, *ep;
  int st;
  struct Cur {
    T *d, *e;
  };
  __host__ __device__ __forceinline__ Cur at(int i) const { return Cur{dp + i * st, ep + i * st}; }
  __host__ __device__ __forceinline__ void move(Cur &c, int k) const
  {
    c.d += k * st;
    c.e += k * st;
  }
  __host__ __device__ __forceinline__ T d(const Cur &c, int k) const { return c.d[k * st]; }
  __host__ __device__ __forceinline__ T e(const Cur &c, int k) const { return c.e[k * st]; }
  __host__ __device__ __forceinline__ void get(const Cur &c, int k, T &x, T &y) const
  {
    x = c.d[k * st];
    y = c.e[k * st];
  }
  __host__ __device__ __forceinline__ void put(const Cur &c, int k, T x, T y) const
  {
    c.d[k * st] = x;
    c.e[k * st] = y;
  }
  __host__ __device__ __forceinline__ void put_d(const Cur &c, int k, T x) const { c.d[k * st] = x; }
  __host__ __device__ __forceinline__ void put_e(const Cur &c, int k, T y) const { c.e[k * st] = y; }
};
template <class T> struct DEVec;
template <> struct DEVec<double> { using V = double2; };
template <> struct DEVec<float> { using V = float2; };
template <class T> struct DEPair {
  using V = typename DEVec<T>::V;
  V *q;
  int st;
  using Cur = V *;
  __host__ __device__ __forceinline__ Cur at(int i) const { return q + i * st; }
  __host__ __device__ __forceinline__ void move(Cur &c, int k) const { c += k * st; }
  __host__ __device__ __forceinline__ T d(const Cur &c, int k) const { return c[k * st].x; }
  __host__ __device__ __forceinline__ T e(const Cur &c, int k) const { return c[k * st].y; }
  __host__ __device__ __forceinline__ void get(const Cur &c, int k, T &x, T &y) const
  {
    const V v = c[k * st];
    x = v.x;
    y = v.y;
  }
  __host__ __device__ __forceinline__ void put(const Cur &c, int k, T x, T y) const
  {
    V v;
    v.x = x;
    v.y = y;
    c[k * st] = v;
  }
  __host__ __device__ __forceinline__ void put_d(const Cur &c, int k, T x) const { c[k * st].x = x; }
  __host__ __device__ __forceinline__ void put_e(const Cur &c, int k, T y) const { c[k * st].y = y; }
};

// Magnitude as an integer that orders as the magnitude does (the upper word
// of a double), and bounds that keep p^2 + e^2 plain (rsq_plain) for every p:
// |e| >= QL_LOW, and d, e of the whole matrix at most ql_high.
__host__ __device__ __forceinline__ int ql_mag(double x)
{
#ifdef __CUDA_ARCH__
  return __double2hiint(x) & 0x7fffffff;
#else
  long long b;
  memcpy(&b, &x, 8);
  return (int)(b >> 32) & 0x7fffffff;
#endif
}
__host__ __device__ __forceinline__ int ql_mag(float x)
{
#ifdef __CUDA_ARCH__
  return __float_as_int(x) & 0x7fffffff;
#else
  int b;
  memcpy(&b, &x, 4);
  return b & 0x7fffffff;
#endif
}
template <class T> __host__ __device__ constexpr int ql_low() { return sizeof(T) == 8 ? 0x23000000 : 0x27000000; }  // 2^-463, 2^-49
template <class T> __host__ __device__ constexpr int ql_high() { return sizeof(T) == 8 ? 0x5b700000 : 0x53000000; } // 2^440, 2^39

// The rotation loop is bound by the latency of its recurrence (p -> y -> p)
// and, with several chains a scheduler, by instruction issue.  What a
// rotation leaves behind (its record, d and e of i+1) is therefore formed and
// stored one step later, while that step's y is on its way, and four steps
// are unrolled into one block without branches: whether every rotation of a
// sweep will be plain is known before it, from the smallest |e| that the sweep
// before left and the largest entry of the matrix.  (A test in each rotation
// cost a quarter: it cut the block.)  Measured on B200 against the loop that
// finished each rotation in place with the library's rsqrt (phase 2, ms; with
// a test per rotation in brackets): FP64 n=128 L=4096 2.44 -> 1.30 (1.59),
// n=256 L=2048 10.7 -> 5.1 (6.4), n=512 L=256 30.0 -> 14.6 (18.4), n=1000 L=32
// 109 -> 53 (67); FP32 n=128 2.36 -> 0.87 (1.05), n=256 9.2 -> 3.2 (4.3).
template <class T, class S>
__host__ __device__ int ql_tql2_fast_s(const S v, const int n, Rec<T> *__restrict__ out, const int cap,
                                       const int max_sweep, int *ierr)
{
  using Cur = typename S::Cur;
  const T tol = Num<T>::eps() * Num<T>::tolmul();
  int nrec = 0;
  *ierr = 0;
  if (n <= 1) return 0;
  T shift = T(0), tst1 = T(0);
  bool small = true;  // no entry above ql_high (none is a NaN)
  {
    Cur q = v.at(0);
    for (int i = 0; i < n; i++, v.move(q, 1)) {
      T d0, e0;
      v.get(q, 0, d0, e0);
      small = small && ql_mag(d0) <= ql_high<T>() && ql_mag(e0) <= ql_high<T>();
    }
  }
  for (int l = 0; l < n; l++) {
    const Cur lp = v.at(l);
    {
      T d0, e0;
      v.get(lp, 0, d0, e0);
      tst1 = fmax_t(tst1, (fabs_t(d0) + fabs_t(e0)) * tol);
    }
    int m = l;
    {  // first m >= l with |e(m)| <= tst1, four at a time
      Cur ep = lp;
      bool found = false;
      for (; m + 4 <= n; m += 4, v.move(ep, 4)) {
        const T a0 = v.e(ep, 0), a1 = v.e(ep, 1), a2 = v.e(ep, 2), a3 = v.e(ep, 3);
        const bool b0 = fabs_t(a0) <= tst1, b1 = fabs_t(a1) <= tst1, b2 = fabs_t(a2) <= tst1, b3 = fabs_t(a3) <= tst1;
        if (b0 || b1 || b2 || b3) {
          m += b0 ? 0 : (b1 ? 1 : (b2 ? 2 : 3));
          found = true;
          break;
        }
      }
      if (!found)
        for (; m < n && !(fabs_t(v.e(ep, 0)) <= tst1); m++) v.move(ep, 1);
    }
    if (m >= n) {
      *ierr = l + 1;
      return nrec;
    }
    if (m != l) {
      const int len = m - l;
      // smallest |e| of the block: those found by the search are above tst1
      int emin = ql_mag(tst1);
      const bool above = small && emin >= ql_low<T>();
      int itr;
      for (itr = 0; itr < max_sweep; itr++) {
        if (nrec + 1 + len > cap) return -1;
        T dl_old, el, dl1_old, el1, dl, dl1;
        v.get(lp, 0, dl_old, el);
        v.get(lp, 1, dl1_old, el1);
        tql2_shift(dl_old, dl1_old, el, dl, dl1);
        v.put_d(lp, 0, dl);
        v.put_d(lp, 1, dl1);
        const T delta = dl_old - dl;
        {  // d(l+2..m) are shifted on read
          Cur jp = v.at(m + 1);
          for (int j = m + 1; j < n; j++, v.move(jp, 1)) v.put_d(jp, 0, v.d(jp, 0) - delta);
        }
        shift += delta;
        T c = T(1), c2 = T(1), c3 = T(1), s = T(0), s2 = T(0);
        Cur qp = v.at(m);  // i+1
        T p = (m >= l + 2) ? v.d(qp, 0) - delta : v.d(qp, 0);
        T ei = T(0), di = T(0), so = T(0);
        // the step whose outputs are pending; its record goes to *o, the
        // segment's header slot (written last) while there is none
        Tql2Step<T> k;
        k.cn = k.sn = k.r = k.pn = k.gg = k.h = T(0);
        Rec<T> *o = out + nrec;
        T d_n, e_n;  // the next step's d(i), e(i), loaded a step ahead
        v.get(qp, -1, d_n, e_n);
        // With every |e| of the block at least ql_low no rotation needs
        // checking; e(l+1) .. e(m-1) of the next sweep are measured here, e(l)
        // stays above tst1.
        const bool fast = above && emin >= ql_low<T>();
        emin = 0x7fffffff;
        if (fast) {
          auto step = [&](const bool first, const T sub, const bool more, const bool meas) {
            c3 = c2;
            c2 = c;
            s2 = s;
            ei = e_n;
            const T dn = d_n - sub;
            if (more) v.get(qp, -2, d_n, e_n);
            const Tql2Pre<T> a = tql2_begin(c, p, ei, dn);
            const T e1 = tql2_e1(k, so), d1 = tql2_d1(k, di);
            Rec<T> rec;
            rec.c = c;
            rec.s = s;
            *o++ = rec;
            if (!first) v.put(qp, 1, d1, e1);
            if (meas) emin = min(emin, ql_mag(e1));
            k = tql2_end(a, p, ei, dn);
            di = dn;
            so = s;
            p = k.pn;
            c = k.cn;
            s = k.sn;
            v.move(qp, -1);
          };
          int i = m - 1;
          step(true, i >= l + 2 ? delta : T(0), i > l, false);
          i--;
          if (i >= l) {
            step(false, i >= l + 2 ? delta : T(0), i > l, false);
            i--;
          }
#pragma unroll 4
          for (; i >= l + 2; i--) step(false, delta, true, true);
          for (; i >= l; i--) step(false, T(0), i > l, true);
        } else {
#pragma unroll 1
          for (int i = m - 1; i >= l; i--) {
            c3 = c2;
            c2 = c;
            s2 = s;
            ei = e_n;
            const T dn = (i >= l + 2) ? d_n - delta : d_n;
            v.get(qp, i > l ? -2 : -1, d_n, e_n);
            const T e1 = tql2_e1(k, so), d1 = tql2_d1(k, di);
            Rec<T> rec;
            rec.c = c;
            rec.s = s;
            *o++ = rec;
            if (i < m - 1) v.put(qp, 1, d1, e1);
            emin = min(emin, i < m - 2 ? ql_mag(e1) : 0x7fffffff);
            k = tql2_any(c, p, ei, dn);
            di = dn;
            so = s;
            p = k.pn;
            c = k.cn;
            s = k.sn;
            v.move(qp, -1);
          }
        }
        if (len > 1) emin = min(emin, ql_mag(tql2_e1(k, so)));
        v.put(qp, 1, tql2_d1(k, di), tql2_e1(k, so));
        {
          Rec<T> rec;
          rec.c = c;
          rec.s = s;
          *o = rec;
        }
        out[nrec] = make_hdr(m - 1, len, T(0));
        nrec += 1 + len;
        T eln, dln;
        tql2_close(c, s, s2, c3, el1, ei, dl1, eln, dln);
        v.put(lp, 0, dln, eln);
        if (fabs_t(eln) <= tst1) break;
      }
      if (itr >= max_sweep) {
        *ierr = l + 1;
        return nrec;
      }
    }
    v.put_d(lp, 0, v.d(lp, 0) + shift);
  }
  return nrec;
}

template <class T, class S>
__host__ __device__ int ql_imtql2_fast_s(const S v, const int n, Rec<T> *__restrict__ out, const int cap,
                                         const int max_sweep, int *ierr)
{
  using Cur = typename S::Cur;
  const T tol = Num<T>::eps() * Num<T>::tolmul();
  int nrec = 0;
  *ierr = 0;
  if (n <= 1) return 0;
  for (int l = 0; l < n; l++) {
    int itr;
    for (itr = 0; itr <= max_sweep; itr++) {
      int m = n - 1;
      {
        Cur mp = v.at(l);
        T d0, e0;
        for (int mm = l; mm < n - 1; mm++, v.move(mp, 1)) {
          v.get(mp, 0, d0, e0);
          const T t1 = (fabs_t(d0) + fabs_t(v.d(mp, 1))) * tol;
          if (!(fabs_t(e0) > t1)) {
            m = mm;
            break;
          }
        }
      }
      if (m == l) break;
      if (nrec + 1 + (m - l) > cap) return -1;
      const Cur lp = v.at(l);
      Cur ip = v.at(m);  // i+1
      T di1 = v.d(ip, 0);
      T r = imtql2_shift(v.d(lp, 0), v.d(lp, 1), v.e(lp, 0), di1);
      T s = T(1), c = T(1), delta = T(0);
      Rec<T> *o = out + nrec + 1;
      int i;
      int cnt = 0;
      for (i = m - 1; i >= l; i--) {
        T di, ei;
        v.get(ip, -1, di, ei);
        const T f = mul_rn(s, ei);
        T cn, sn, rn;
        givens(r, f, cn, sn, rn);
        if (rn == T(0)) {
          r = T(0);
          break;
        }
        const T dx1 = imtql2_step(cn, sn, c, ei, di, di1, delta, r);
        v.put(ip, 0, dx1, rn);
        c = cn;
        s = sn;
        Rec<T> rec;
        rec.c = cn;
        rec.s = sn;
        *o++ = rec;
        cnt++;
        v.move(ip, -1);
      }
      if (cnt > 0) {
        out[nrec] = make_hdr(m - 1, cnt, T(0));
        nrec += 1 + cnt;
      }
      const Cur jp = v.at((i + 1 > l) ? i + 1 : l);
      v.put(jp, 0, v.d(jp, 0) - delta, r);
      v.put_e(v.at(m), 0, T(0));
    }
    if (itr > max_sweep) {
      *ierr = l + 1;
      return nrec;
    }
  }
  return nrec;
}

template <class T>
__host__ __device__ int ql_tql2_fast(T *__restrict__ d, T *__restrict__ e, const int st, const int n,
                                     Rec<T> *__restrict__ out, const int cap, const int max_sweep, int *ierr)
{
  return ql_tql2_fast_s<T>(DESep<T>{d, e, st}, n, out, cap, max_sweep, ierr);
}
template <class T>
__host__ __device__ int ql_imtql2_fast(T *__restrict__ d, T *__restrict__ e, const int st, const int n,
                                       Rec<T> *__restrict__ out, const int cap, const int max_sweep, int *ierr)
{
  return ql_imtql2_fast_s<T>(DESep<T>{d, e, st}, n, out, cap, max_sweep, ierr);
}

// Not inlined: it runs for the rare matrix whose records overflowed, and its
// state would cost the apply kernels registers (k3_warp n=32 L=16384: 0.60 ms,
// inlined 0.80).
template <class T>
__host__ __device__ __noinline__ int ql_run(int method, QLGen<T> &g, const DEView<T> v, const int n,
                                      Rec<T> *buf, const int cap, const int max_sweep)
{
  return method == QL_IMTQL2 ? ql_imtql2(g, v, n, buf, cap, max_sweep)
                             : ql_tql2(g, v, n, buf, cap, max_sweep);
}

}  // namespace eigb
