"""Phase 3 in its wave form (n >= 128: 16 sweeps per pass over rows in
memory) against the shared-memory form, which applies the same rotations to
every element in the same order: equal bits, at the edges of its rows per
thread and per CTA and of its column and sweep groups, for one and two rows
per thread (the batch decides), with decoupled blocks (sweeps of many tops
and lengths in one group), ties and sort off."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _both(E, a0, n, nm, sort=True, method=0):
    a, b = a0.clone(), a0.clone()
    wa, ia = E.solve(a, n, nm, sort=sort, method=method)
    wb, ib = E.solve(b, n, nm, sort=sort, method=method, zmem=E.ZMEM_SHARED)
    torch.cuda.synchronize()
    assert torch.equal(ia, ib) and torch.equal(wa, wb) and torch.equal(a[:, :, :n], b[:, :, :n])
    assert (ia == 0).all()
    return a


@pytest.mark.parametrize("dtype,n,nm,L", [
    ("f64", 128, 128, 3), ("f64", 128, 131, 300), ("f64", 129, 129, 200), ("f64", 191, 192, 7), ("f64", 200, 200, 160),
    ("f64", 256, 256, 150), ("f64", 257, 257, 2), ("f64", 513, 513, 2), ("f64", 600, 601, 70), ("f64", 1024, 1024, 1),
    ("f32", 128, 128, 300), ("f32", 145, 145, 3), ("f32", 256, 256, 150), ("f32", 300, 303, 130), ("f32", 1000, 1000, 1)])
def test_wave_form_equals_shared_memory_form(oracle_mod, dtype, n, nm, L):
    import eigeng_b200 as E
    dt = torch.float64 if dtype == "f64" else torch.float32
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = torch.rand((L, n, n), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    a0 = torch.zeros((L, n, nm), dtype=dt, device="cuda")
    a0[:, :, :n] = x + x.mT
    if n < 513:
        # blocks of different orders, the last one diagonal: many short sweeps
        for k, cut in ((0, n // 3), (1, n - 5)):
            a0[k % L, :cut, cut:n] = 0
            a0[k % L, cut:, :cut] = 0
        a0[-1, :, :n] *= torch.eye(n, dtype=dt, device="cuda")
        if L > 2:
            a0[2, :, :n] = torch.eye(n, dtype=dt, device="cuda")
    _both(E, a0, n, nm)


@pytest.mark.parametrize("sort,method", [(False, 0), (True, 1), (False, 1)])
def test_wave_form_options(sort, method):
    import eigeng_b200 as E
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    x = torch.rand((4, 150, 150), generator=g, device="cuda", dtype=torch.float64)
    _both(E, x + x.mT, 150, 150, sort, method)
