// Largest error in ulp of rsq_fast (csrc/eigb_common.cuh) over its plain range,
// and CUDA's rsqrt beside it, for tests/test_gpu_rsq.py.
#include "../../eigeng-batched_b200/csrc/eigb_common.cuh"

// |y sqrt(x) - 1| in ulps of y for y near 1/sqrt(x): (x y^2 - 1) / 2 with
// x y^2 to twice the precision
__device__ double err_ulp(const double x, const double y)
{
  const double p = y * y, pe = fma(y, y, -p), t = x * p, te = fma(x, p, -t);
  const double e = 0.5 * ((t - 1.0) + te + x * pe);
  return fabs(e * y) / (__longlong_as_double(__double_as_longlong(y) + 1) - y);
}
__device__ double err_ulp(const float x, const float y)
{
  const double r = 1.0 / sqrt((double)x);  // far closer than half a float ulp
  return fabs((double)y - r) / ((double)__int_as_float(__float_as_int(y) + 1) - (double)y);
}
__device__ void post(double *out, const double e)
{
  atomicMax(reinterpret_cast<unsigned long long *>(out), (unsigned long long)__double_as_longlong(e));
}
// doubles: hash of the index as the mantissa and the exponent's parity, the
// exponent over the plain range; the range's two ends for the first indices
__global__ void k_double(const long n, double *out)
{
  double a = 0.0, b = 0.0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    unsigned long long z = (unsigned long long)i * 0x9e3779b97f4a7c15ull + 0x632be59bd9b4e019ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    const int ex = -928 + (int)(z >> 52) % 1856;  // 2^-928 .. 2^928
    double x = ldexp(1.0 + (double)(z & 0xfffffffffffffull) * 0x1p-52, ex);
    if (i == 0) x = 0x1p-928;
    if (i == 1) x = __longlong_as_double(__double_as_longlong(0x1p928) - 1);
    if (!eigb::rsq_plain(x)) post(out + 2, 1.0);
    a = fmax(a, err_ulp(x, eigb::rsq_fast(x)));
    b = fmax(b, err_ulp(x, rsqrt(x)));
  }
  post(out, a);
  post(out + 1, b);
}
// floats: every mantissa at both parities of the exponent, at the middle and
// at both ends of the range
__global__ void k_float(double *out)
{
  double a = 0.0, b = 0.0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < 6l << 23; i += (long)gridDim.x * blockDim.x) {
    const int ex[6] = {0, 1, -100, -99, 98, 99};
    const float x = ldexpf(1.0f + (float)(i & 0x7fffff) * 0x1p-23f, ex[i >> 23]);
    if (!eigb::rsq_plain(x)) post(out + 2, 1.0);
    a = fmax(a, err_ulp(x, eigb::rsq_fast(x)));
    b = fmax(b, err_ulp(x, __frsqrt_rn(x)));
  }
  post(out, a);
  post(out + 1, b);
}
// just outside the plain range: not taken
__global__ void k_outside(double *out)
{
  const double d[6] = {0.0, __longlong_as_double(__double_as_longlong(0x1p-928) - 1), 0x1p928, INFINITY, nan(""), 1e-320};
  const float f[6] = {0.0f, __int_as_float(__float_as_int(0x1p-100f) - 1), 0x1p100f, INFINITY, nanf(""), 1e-44f};
  for (int i = 0; i < 6; i++)
    if (eigb::rsq_plain(d[i]) || eigb::rsq_plain(f[i])) post(out + 3, 1.0);
}

// out: 8 doubles on the device, zeroed; [0..2] double, [4..6] float, [3] and [7]
extern "C" int rsq_errors(const long n, double *out)
{
  k_double<<<1184, 256>>>(n, out);
  k_float<<<1184, 256>>>(out + 4);
  k_outside<<<1, 1>>>(out);
  return (int)cudaDeviceSynchronize();
}
