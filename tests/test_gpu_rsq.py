"""rsq_fast, the QL phase's reciprocal square root, on the device.  Its last
operation rounds y + y e (1/2 + 3 e / 8), with e = 1 - x y^2 formed without the
rounding of y^2.  Double: y is the hardware's approximation cut to 20 bits, so y
in [1, 2) is off by at most 2^-20 plus the approximation's own error, taken as
2^-22; the remainder of the series, 5/16 e^3 with e twice the relative error, is
then at most 1.25^3 * 2.5 / 256 < 0.02 ulp, and the roundings of the small term
are below 2^-15 ulp.  Float: with the approximation off by 2^-22 the remainder
3/8 e^2 is below 2^-17 ulp.  The bounds: 0.52 and 0.501 ulp."""
import ctypes
import os
import subprocess

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_error_over_the_plain_range(tmp_path):
    so = os.path.join(str(tmp_path), "librsq.so")
    subprocess.check_call(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                           "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-o", so,
                           os.path.join(ROOT, "tests", "device", "rsq_dev.cu")])
    f = ctypes.CDLL(so).rsq_errors
    f.argtypes = [ctypes.c_long, ctypes.c_void_p]
    out = torch.zeros(8, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert f(1 << 28, out.data_ptr()) == 0
    d, dlib, dbad, dout, s, slib, sbad, _ = out.tolist()
    print("double %.5f (rsqrt %.5f), float %.7f (__frsqrt_rn %.7f) ulp" % (d, dlib, s, slib))
    assert dbad == sbad == dout == 0.0  # the range holds these arguments and no other
    assert 0.49 < dlib < 1.01 and 0.49 < slib <= 0.5 + 1e-6  # the yardstick itself
    assert d <= 0.52 and s <= 0.501
