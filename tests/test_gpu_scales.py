"""Entries near both ends of what the solver takes: its squares must neither
overflow nor underflow (QL forms p^2 + e^2), so magnitudes of 2^+-470 in FP64
and 2^+-52 in FP32 are inside, while third-degree terms (u.Au in the
reduction) are not representable there.  The solve is homogeneous: against the
same matrix unscaled, which differs by a power of two, the eigenvalues agree
within the parity bound and the gate's residual (relative) raises no flag."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("n", [7, 32, 130, 200, 300, 600])
@pytest.mark.parametrize("sign", [1, -1])
def test_extreme_scales(oracle_mod, dtype, n, sign):
    import eigeng_b200 as E
    dt = torch.float64 if dtype == "f64" else torch.float32
    k = sign * (470 if dtype == "f64" else 52)
    eps = torch.finfo(dt).eps
    a0 = torch.from_numpy(oracle_mod.sym_uniform(3, n, seed=n)).cuda().to(dt)
    b0 = (a0.double() * 2.0 ** k).to(dt)  # exact
    a, b = a0.clone(), b0.clone()
    w, ia = E.solve(a, n)
    ws, ib = E.solve(b, n)
    torch.cuda.synchronize()
    assert (ia == 0).all() and (ib == 0).all()
    back = ws.double() * 2.0 ** -k
    scale = w.double().abs().amax(dim=1, keepdim=True)
    assert ((back - w.double()).abs() <= 64 * n * eps * scale).all()
    e1, e2, fl = E.check(a0, back.to(dt), b, n)
    assert (fl == 0).all(), (e1, e2)
