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


@pytest.mark.parametrize("small_first", [True, False])
@pytest.mark.parametrize("dtype,big,small", [
    ("f32", 1e10, 1e-5), ("f32", 1e10, 1e-10), ("f32", 1e10, 1e-12), ("f32", 1e8, 1e-13), ("f32", 1e15, 1e-14),
    ("f64", 1e75, 1e-75), ("f64", 1e100, 1e-60), ("f64", 1e90, 1e-80), ("f64", 1e140, 1e-135)])
@pytest.mark.parametrize("n", [32, 130, 400])
def test_graded_blocks(oracle_mod, n, dtype, big, small, small_first):
    """Block-diagonal matrices whose blocks differ by 1e-15 to 1e-29 (FP32)
    and 1e-150 to 1e-275 (FP64): finite, converged, no flag of the gate; and
    with the small block first, where QL's deflation threshold is still its
    own, its eigenvalues to rounding of its own norm."""
    import eigeng_b200 as E
    dt = torch.float64 if dtype == "f64" else torch.float32
    eps = torch.finfo(dt).eps
    k = n // 2
    x = torch.from_numpy(oracle_mod.sym_uniform(2, n, seed=n))
    a0 = torch.zeros((2, n, n), dtype=torch.float64)
    lo, hi = (small, big) if small_first else (big, small)
    a0[:, :k, :k] = lo * x[:, :k, :k]
    a0[:, k:, k:] = hi * x[:, k:, k:]
    a0 = a0.to(dt).cuda()
    a = a0.clone()
    w, info = E.solve(a, n)
    e1, e2, fl = E.check(a0, w, a, n)
    torch.cuda.synchronize()
    assert torch.isfinite(a).all() and torch.isfinite(w).all() and (info == 0).all()
    assert (fl == 0).all(), (e1, e2)
    if small_first:
        # the deflation threshold is 512 eps (FP64) or 16 eps (FP32) of |d| + |e|
        ref = torch.linalg.eigvalsh(a0[:, :k, :k].double() / small)
        got = torch.stack([v[v.abs().argsort()[:k]].sort().values for v in w.double()]) / small
        assert ((got - ref).abs() <= (64 * n + 1024) * eps * ref.abs().amax(dim=1, keepdim=True)).all()
