// Host build of the reductions of phase 1 on chip (csrc/eigb_tridiag_sym.cuh,
// eigb_tridiag_warp.cuh), run by tests/host/simt.hpp.
#include "simt.hpp"

#include "../../eigeng-batched_b200/csrc/eigb_sym_cfg.cuh"
#include "../../eigeng-batched_b200/csrc/eigb_tridiag_sym.cuh"
#include "../../eigeng-batched_b200/csrc/eigb_tridiag_warp.cuh"

// One launch of k1_sym<T, NW, RS, CN> for one matrix: leading m x m block
// down to `stop`.  V: n x ldv, beta: n.
template <class T, int NW, int RS, int CN>
static long sym(T *A, int nm, int m, int stop, bool first, const T *Ap, T *d, T *e, T *V, int ldv, double *beta,
                int high_first)
{
  const size_t bytes = sizeof(T) * eigb::sym_smem_elems(m, NW, RS, CN);
  return simt::run(CN, 32 * NW, bytes, high_first != 0, [&] {
    if (eigb::tridiag_sym<T, NW, RS, CN, false>(A, nm, m, stop, first, Ap, d, e, V, ldv, beta, simt::shared<T>()))
      eigb::tridiag_sym<T, NW, RS, CN, true>(A, nm, m, stop, first, Ap, d, e, V, ldv, beta, simt::shared<T>());
  });
}
template <class T>
static long sym_any(int nw, int rs, int cn, T *A, int nm, int m, int stop, int first, const T *Ap, T *d, T *e, T *V,
                    int ldv, double *beta, int hf)
{
#define FORM(NW, RS, CN) \
  if (nw == NW && rs == RS && cn == CN) return sym<T, NW, RS, CN>(A, nm, m, stop, first != 0, Ap, d, e, V, ldv, beta, hf)
  if constexpr (sizeof(T) == 8) {
    FORM(1, 2, 1);
    FORM(2, 1, 1);
    FORM(4, 1, 1);
    FORM(4, 2, 1);
    FORM(8, 2, 1);
    FORM(8, 2, 2);
    FORM(8, 2, 4);
    FORM(8, 2, 8);
    FORM(8, 2, 16);
  } else {
    FORM(2, 1, 1);
    FORM(2, 2, 1);
    FORM(4, 1, 1);
    FORM(4, 4, 1);
    FORM(8, 1, 1);
    FORM(8, 4, 1);
    FORM(8, 4, 2);
    FORM(8, 4, 4);
    FORM(8, 4, 8);
  }
#undef FORM
  return -2;
}

// k1_warp for one matrix, n <= 32: Q (A = Q T Q^T) in A's place
template <class T> static long warp(T *A, int nm, int n, const T *Ap, T *d, T *e)
{
  return simt::run(1, 32, sizeof(T) * eigb::tw_smem_elems(), false, [&] {
    if (eigb::tridiag_warp<T, false>(A, nm, n, Ap, d, e, simt::shared<T>()))
      eigb::tridiag_warp<T, true>(A, nm, n, Ap, d, e, simt::shared<T>());
  });
}

// The launches of the reduction of order n for cnt matrices on 148 SMs, as the
// library chooses them: four ints each (order, warps, blocks in registers,
// CTAs); returns their number.
template <class T> static int chain(int n, long cnt, int *out)
{
  int k = 0;
  for (int m = n; m > 0; m = eigb::sym_next<T>(m, cnt, 148), k++) {
    const eigb::SymCfg c = eigb::sym_cfg<T>(m);
    out[4 * k] = m;
    out[4 * k + 1] = c.nw;
    out[4 * k + 2] = c.rs;
    out[4 * k + 3] = c.cn;
  }
  return k;
}

extern "C" {
int host_sym_chain(int esize, int n, long cnt, int *out)
{
  return esize == 8 ? chain<double>(n, cnt, out) : chain<float>(n, cnt, out);
}
long host_warp_d(double *A, int nm, int n, const double *Ap, double *d, double *e) { return warp(A, nm, n, Ap, d, e); }
long host_warp_f(float *A, int nm, int n, const float *Ap, float *d, float *e) { return warp(A, nm, n, Ap, d, e); }
long host_sym_d(int nw, int rs, int cn, double *A, int nm, int m, int stop, int first, const double *Ap, double *d,
                double *e, double *V, int ldv, double *beta, int hf)
{
  return sym_any<double>(nw, rs, cn, A, nm, m, stop, first, Ap, d, e, V, ldv, beta, hf);
}
long host_sym_f(int nw, int rs, int cn, float *A, int nm, int m, int stop, int first, const float *Ap, float *d,
                float *e, float *V, int ldv, double *beta, int hf)
{
  return sym_any<float>(nw, rs, cn, A, nm, m, stop, first, Ap, d, e, V, ldv, beta, hf);
}
}
