"""n <= 32, the register forms of phase 1 (k1_warp) and of the rotation apply
(k3_warp): every order, against the oracle's eigenvalues and with the
reference's gate; packed input, padding, blocks of many tops
and lengths, and records regenerated chunk by chunk give the same bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", list(range(2, 33)))
def test_every_small_order(oracle_mod, n, dtype):
    import eigeng_b200 as E
    O = oracle_mod
    L, nm = 9, n + (n % 3)
    a0 = np.zeros((L, n, nm))
    a0[:, :, :n] = O.sym_uniform(L, n, seed=n)
    if n > 4:  # decoupled blocks
        a0[1, :2, 2:n] = a0[1, 2:, :2] = 0
        a0[2, :n - 2, n - 2:n] = a0[2, n - 2:, :n - 2] = 0
    a0[3, :, :n] = np.diag(np.arange(n))
    a0[4, :, :n] = np.eye(n)
    a0 = a0.astype(dtype)
    ao = np.ascontiguousarray(a0[:, :, :n])
    wo, _, _ = O.eigen_batch(ao.copy(), n)
    t0 = torch.from_numpy(a0).cuda()
    a = t0.clone()
    w, info = E.solve(a, n, nm)
    b = t0.clone()
    wb, ib = E.solve(b, n, nm, rec_cap=4)
    zp, wp, ip = E.solve_packed(E.pack_upper(t0, n, nm), n)
    torch.cuda.synchronize()
    assert (info == 0).all() and torch.equal(ib, info) and torch.equal(ip, info)
    assert torch.equal(wb, w) and torch.equal(b, a) and torch.equal(wp, w) and torch.equal(zp, a[:, :, :n])
    assert torch.equal(a[:, :, n:], t0[:, :, n:])
    eps = np.finfo(dtype).eps
    scale = np.maximum(np.abs(wo).max(axis=1, keepdims=True), 1e-30)
    assert (np.abs(w.cpu().numpy() - wo) <= 64 * n * eps * scale).all()
    e1, e2, fl = E.check(t0, w, a, n, nm)
    torch.cuda.synchronize()
    assert (fl == 0).all(), (e1, e2)
