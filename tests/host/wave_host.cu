// Host build of phase 3's wave form (csrc/eigb_wave.cuh), run by
// tests/host/simt.hpp: nrow rows of the column-major n x n matrix A, one CTA.
#include "simt.hpp"

#include "../../eigeng-batched_b200/csrc/eigb_wave.cuh"

template <class T, int R, int U>
static long run(T *A, int nm, int n, int row0, int nrow, const T *recs, int nrec, const T *ev, int sort, T *w)
{
  const int warps = (nrow + 32 * R - 1) / (32 * R) + 1;
  return simt::run(1, 32 * warps, eigb::wv_smem_bytes<T>(n, 16), false, [&] {
    eigb::wave_apply<T, 16, R, U>(A, nm, n, row0, nrow, reinterpret_cast<const eigb::Rec<T> *>(recs), nrec, ev, sort, w,
                                  simt::shared<unsigned char>());
  });
}

extern "C" long host_wave_d(int r, double *A, int nm, int n, int row0, int nrow, const double *recs, int nrec,
                            const double *ev, int sort, double *w)
{
  return r == 2 ? run<double, 2, 2>(A, nm, n, row0, nrow, recs, nrec, ev, sort, w)
                : run<double, 1, 4>(A, nm, n, row0, nrow, recs, nrec, ev, sort, w);
}
extern "C" long host_wave_f(int r, float *A, int nm, int n, int row0, int nrow, const float *recs, int nrec,
                            const float *ev, int sort, float *w)
{
  return r == 2 ? run<float, 2, 4>(A, nm, n, row0, nrow, recs, nrec, ev, sort, w)
                : run<float, 1, 4>(A, nm, n, row0, nrow, recs, nrec, ev, sort, w);
}
