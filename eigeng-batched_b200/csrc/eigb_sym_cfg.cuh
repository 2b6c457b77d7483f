// Launch configurations of k1_sym (host code; the kernel is in
// eigb_tridiag_sym.cuh).  A matrix has the same eigenpairs, bit for bit,
// whatever the batch, the part of it or the chunk that it is solved in: the
// number of CTAs, which changes the order of sums, depends on the order of the
// matrix alone; the other choices do not change it.
#pragma once

namespace eigb {

// k1_sym: warps, blocks per warp in registers and CTAs per matrix
struct SymCfg {
  int nw, rs, cn, mb;  // mb: CTAs an SM the registers are bounded for
};
// Measured on B200 (the reduction alone, ms).  Where several matrices fit an
// SM, small CTAs with few blocks in registers win, their step chains hiding
// one another: FP64 n=64 L=20000 one warp x 2 blocks 2.85, two x 1 3.26, four
// x 1 4.43; n=96 L=8000 two x 1, six CTAs 3.07, four x 1 3.40; n=128 L=4096 4 warps x 1 block, three CTAs 3.04, x 2
// blocks, two CTAs 3.48, 8 x 2, one CTA 5.62; n=160 L=3000 4.65 / 4.05 /
// 5.69.  From n = 161 on 4 warps no longer have two CTAs an SM (n=192 L=2048
// 6.58 against 5.20 with 8).  Above 256 the fewest CTAs that hold the
// triangle: n=512 L=256 4 CTAs 13.4, 8 CTAs 28.8; n=384 L=512 15.3 / 36.8;
// n=736 L=64 8 CTAs 15.6, 16 CTAs 29.2.  FP32: n=96 L=8000 2 x 1,
// eight CTAs 1.67, 4 x 1 2.07; n=128 L=4096 2 x 2 1.66, 4 x 1 1.76; n=160 L=3000 4 x 1 2.14, 8 x 1
// 2.80; n=224 L=2048 4.33 / 3.53; n=256 8 x 1 7.06, 4 x 4 5.04, 8 x 4 6.28;
// n=288 L=1024 4 x 4 5.79, 8 x 4 4.03; n=1000 L=32 8 CTAs 14.2, 16 21.1.
template <class T> SymCfg sym_cfg(int n)
{
  if (sizeof(T) == 8) {
    if (n <= 64) return {1, 2, 1, 8};
    if (n <= 96) return {2, 1, 1, 6};
    if (n <= 128) return {4, 1, 1, 3};
    if (n <= 160) return {4, 2, 1, 2};
    if (n <= 256) return {8, 2, 1, 1};
    if (n <= 352) return {8, 2, 2, 1};
    if (n <= 512) return {8, 2, 4, 1};
    if (n <= 736) return {8, 2, 8, 1};
    return {8, 2, 16, 1};
  }
  if (n <= 96) return {2, 1, 1, 8};
  if (n <= 128) return {2, 2, 1, 6};
  if (n <= 160) return {4, 1, 1, 4};
  if (n <= 224) return {8, 1, 1, 2};
  if (n <= 256) return {4, 4, 1, 2};
  if (n <= 384) return {8, 4, 1, 1};
  if (n <= 512) return {8, 4, 2, 1};
  if (n <= 736) return {8, 4, 4, 1};
  return {8, 4, 8, 1};
}
// Order at which a reduction of order n, for cnt matrices, hands the leading
// block over to a launch with fewer CTAs or warps (0: none).  A matrix keeps
// its SMs to the last step otherwise, and the last steps have little to do.
//  - One CTA a matrix: where the batch takes more than one wave of CTAs,
//    another launch packs the small blocks closer.  Measured on B200 (the
//    reduction with the formation of Q, ms, without / with): FP64 n=96 L=8000
//    4.14 / 3.99, n=128 L=4096 3.98 / 3.76, n=160 L=3000 5.65 / 5.31, n=256
//    L=2048 12.5 / 11.2; FP32 n=200 L=1000 2.60 / 2.39.  In a single wave it
//    costs: FP64 n=128 L=8 0.30 / 0.37, n=256 L=8 0.78 / 0.90.
//  - A cluster: always, at the orders that cost a small batch least.  (ms,
//    without / at the order given:) FP64 n=400 256: L=500 21.4 / 15.6, L=4 1.27 /
//    1.42; n=512 256: L=256 17.6 / 14.6, L=4 1.98 / 2.14; n=736 512, 256: L=64
//    19.4 / 14.3, L=4 3.53 / 3.78; n=1000 736, 512, 256: L=32 30.1 / 21.5, L=4
//    5.97 / 6.42.  Also 352: n=512 L=256 14.0, but L=4 2.38.  FP32 n=400 384:
//    L=500 12.6 / 10.7, L=4 1.26 / 1.49; n=512 384: L=256 11.5 / 10.1, L=4 2.00 /
//    2.22; n=736 384: L=100 18.5 / 16.5, L=4 3.22 / 3.57; n=1000 736: L=32 19.7 /
//    14.8, L=4 5.78 / 5.98.  At 256 or 160 instead the solve of n=400 L=400 takes
//    4 or 5 % longer than with 384 (19.3 ms), that of L=4 1 or 3 % less.
template <class T> int sym_next(int n, long cnt, int sms)
{
  const SymCfg c = sym_cfg<T>(n);
  const bool wave = cnt * c.cn > (long)sms * c.mb;
  if (sizeof(T) == 8) {
    if (c.cn > 1) return n > 736 ? 736 : (n > 512 ? 512 : 256);
    return wave ? (n > 128 ? 128 : (n > 64 ? 64 : 0)) : 0;
  }
  if (c.cn > 1) return n > 736 ? 736 : 384;
  return wave && n > 160 ? 160 : 0;
}

}  // namespace eigb
