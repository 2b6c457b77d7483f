"""Phase 1 for n > 32: the reduction on the upper triangle in registers and
shared memory (k1_sym) and the formation of Q from its reflectors
(k1_factor, k1_formq), at the edges of their 32 x 32 blocks, of the 16
reflectors of a block factor and of the orders from which a matrix takes
more warps or a larger cluster.

The reduction alone: A = Q T Q^T with the Q that the phase leaves in a and
the T in the workspace.  Householder tridiagonalization is backward stable
(the error in A of n - 1 two-sided reflections is below a small multiple of
n eps ||A||_F, and Q's distance from orthogonality below one of n eps
sqrt(n)); the bounds are 8 n eps of the Frobenius norms, which random
roundings undercut by far."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

F64 = [33, 34, 47, 48, 49, 63, 64, 65, 66, 80, 81, 96, 97, 127, 128, 129, 160, 161, 191, 256, 257, 288, 352, 353, 512, 513, 736, 737, 1024]
F32 = [65, 97, 128, 129, 160, 161, 193, 224, 225, 256, 257, 384, 385, 512, 513, 736, 737, 1024]


def _reduce(E, a, n, nm, rec_cap=0):
    L = a.shape[0]
    wk = E.workspace(L, nm, n, a.dtype, rec_cap=rec_cap, chunk=L)
    wk.fill_(255)
    w = torch.empty((L, n), dtype=a.dtype, device="cuda")
    assert E.stage(a, w, wk, n, E.STAGE_REDUCE, nm=nm, rec_cap=rec_cap) == 0
    es, row = a.element_size(), L * n * a.element_size()
    d = wk[:row].view(a.dtype).view(L, n)
    o = (row + 255) // 256 * 256
    e = wk[o:o + row].view(a.dtype).view(L, n)
    torch.cuda.synchronize()
    return d.double(), e.double()


@pytest.mark.parametrize("dtype,n", [("f64", n) for n in F64] + [("f32", n) for n in F32])
def test_reduction_reproduces_the_matrix(oracle_mod, dtype, n):
    import eigeng_b200 as E
    dt = torch.float64 if dtype == "f64" else torch.float32
    L, nm = (2 if n > 300 else 5), n + (n % 3)
    a0 = np.zeros((L, n, nm))
    a0[:, :, :n] = oracle_mod.sym_uniform(L, n, seed=7000 + n)
    full = torch.from_numpy(a0[:, :, :n].copy()).cuda().to(dt).double()
    A = full.tril() + full.tril(-1).mT  # storage [column][row]: rows <= column are the upper triangle
    a = torch.full((L, n, nm), float("nan"), dtype=dt, device="cuda")  # the strict lower triangle is not read
    low = torch.ones((n, n), dtype=torch.bool, device="cuda").tril()
    a[:, :, :n] = torch.where(low, full.to(dt), a[:, :, :n])
    for rec_cap in (0, 16):  # the reflectors in the records' place, and in their own
        b = a.clone()
        d, e = _reduce(E, b, n, nm, rec_cap)
        Qt = b[:, :, :n].double()
        T = torch.diag_embed(d) + torch.diag_embed(e[:, :n - 1], 1) + torch.diag_embed(e[:, :n - 1], -1)
        eps = torch.finfo(dt).eps
        res = torch.linalg.matrix_norm(Qt.mT @ T @ Qt - A) / torch.linalg.matrix_norm(A)
        orth = torch.linalg.matrix_norm(Qt @ Qt.mT - torch.eye(n, dtype=torch.float64, device="cuda")) / n ** 0.5
        assert res.max().item() <= 8 * n * eps and orth.max().item() <= 8 * n * eps, (res, orth)
        assert torch.isnan(b[:, :, n:]).all()  # padding untouched


@pytest.mark.parametrize("dtype,n", [("f64", 65), ("f64", 161), ("f64", 300), ("f32", 129), ("f32", 400)])
def test_packed_input_and_special_matrices(oracle_mod, dtype, n):
    """Packed input gives the bits of the full one; zero, identity, diagonal
    and tridiagonal matrices (reflectors of norm zero) come out exactly
    orthogonal enough, and one NaN stays in its own matrix."""
    import eigeng_b200 as E
    dt = torch.float64 if dtype == "f64" else torch.float32
    eye = torch.eye(n, dtype=dt, device="cuda")
    tri = 2 * eye - torch.diag(torch.ones(n - 1, dtype=dt, device="cuda"), 1) \
        - torch.diag(torch.ones(n - 1, dtype=dt, device="cuda"), -1)
    rnd = torch.from_numpy(oracle_mod.sym_uniform(2, n, seed=n)).cuda().to(dt)
    a0 = torch.stack([torch.zeros_like(eye), eye, torch.diag(torch.arange(n, device="cuda").to(dt)), tri, rnd[0],
                      rnd[1], rnd[0]])
    a0[5, 3, 2] = float("nan")  # row 2 of column 3: in the upper triangle
    a = a0.clone()
    w, info = E.solve(a, n)
    zp, wp, ip = E.solve_packed(E.pack_upper(a0, n), n)
    torch.cuda.synchronize()
    assert torch.equal(ip, info) and info[5].item() != 0 and (info[[0, 1, 2, 3, 4, 6]] == 0).all()
    ok = [0, 1, 2, 3, 4, 6]
    assert torch.equal(zp[ok], a[ok]) and torch.equal(wp[ok], w[ok])
    assert torch.equal(a[6], a[4]) and torch.equal(w[6], w[4])
    V = a[ok].double()
    eps = torch.finfo(dt).eps
    orth = torch.linalg.matrix_norm(V @ V.mT - eye.double()) / n ** 0.5
    R = a0[ok].double() @ V.mT - V.mT * w[ok].double()[:, None, :]
    scale = torch.linalg.matrix_norm(a0[ok].double()).clamp(min=1e-30)
    # n - 1 reflections and about n rotations per row and column
    assert (orth <= 32 * n * eps).all() and (torch.linalg.matrix_norm(R) / scale <= 32 * n * eps).all()


@pytest.mark.parametrize("dtype,n,L", [("f64", 65, 900), ("f64", 96, 900), ("f64", 128, 460), ("f64", 129, 300),
                                       ("f64", 353, 60), ("f32", 161, 310), ("f32", 385, 80)])
def test_more_than_a_wave_of_matrices(dtype, n, L):
    """Batches of more than one wave of CTAs; every matrix comes back as Q T Q^T."""
    import eigeng_b200 as E
    dt = torch.float64 if dtype == "f64" else torch.float32
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = (torch.rand((L, n, n), generator=g, device="cuda", dtype=torch.float64) * 2 - 1).to(dt)
    A = (x.tril() + x.tril(-1).mT).double()
    a = x.tril() + torch.full_like(x, float("nan")).triu(1)
    d, e = _reduce(E, a, n, n)
    T = torch.diag_embed(d) + torch.diag_embed(e[:, :n - 1], 1) + torch.diag_embed(e[:, :n - 1], -1)
    Qt = a.double()
    eps = torch.finfo(dt).eps
    res = torch.linalg.matrix_norm(Qt.mT @ T @ Qt - A) / torch.linalg.matrix_norm(A)
    orth = torch.linalg.matrix_norm(Qt @ Qt.mT - torch.eye(n, dtype=torch.float64, device="cuda")) / n ** 0.5
    assert res.max().item() <= 8 * n * eps and orth.max().item() <= 8 * n * eps, (res.max(), orth.max())


@pytest.mark.parametrize("dtype,n,L", [("f64", 72, 900), ("f64", 128, 460), ("f64", 200, 160), ("f64", 400, 40),
                                       ("f32", 200, 310), ("f32", 600, 40)])
def test_parts_of_a_batch_give_the_same_bits(dtype, n, L):
    """A batch of more than one wave of CTAs, and parts of it that are less: in
    internal chunks, through the stages in two parts, packed, and as a mixed
    batch, every matrix has the eigenpairs of the one call, bit for bit."""
    import eigeng_b200 as E
    dt = torch.float64 if dtype == "f64" else torch.float32
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = (torch.rand((L, n, n), generator=g, device="cuda", dtype=torch.float64) * 2 - 1).to(dt)
    a0 = x.tril() + x.tril(-1).mT
    a = a0.clone()
    w, info = E.solve(a, n)
    b = a0.clone()
    wb, _ = E.solve(b, n, chunk=L // 3)
    s = a0.clone()
    ws, infos = torch.empty_like(w), torch.empty_like(info)
    wk = E.workspace(L, n, n, dt, chunk=L)
    for first, count in ((0, L // 2), (L // 2, L - L // 2)):
        assert E.stage(s, ws, wk, n, E.STAGE_ALL, first, count, info=infos) == 0
    zp, wp, _ = E.solve_packed(E.pack_upper(a0[:7], n), n)
    k = 5
    u = torch.cat([a0[:k].reshape(-1), a0[0, :40, :40].reshape(-1)])
    wu, _ = E.solve_uneven(u, [n] * k + [40])
    torch.cuda.synchronize()
    assert (info == 0).all() and (infos == 0).all()
    assert torch.equal(b, a) and torch.equal(wb, w)
    assert torch.equal(s, a) and torch.equal(ws, w)
    assert torch.equal(zp, a[:7]) and torch.equal(wp, w[:7])
    assert torch.equal(u[:k * n * n].view(k, n, n), a[:k]) and torch.equal(wu[:k * n].view(k, n), w[:k])
