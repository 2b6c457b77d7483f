"""V f(w) V^T at the edges of its forms: one warp per matrix up to n = 32, a
warp per 32 x 32 tile up to n = 128, 128 x 64 blocks above; orders that are
no multiple of the mma tiles or of the 16-column panels.

Against the product in FP64: a term is rounded once when f(w_k) scales it and
once in its multiply-add, so an entry is within (n + 2) eps sum_k |v_ik f_k
v_jk| of it, with eps of FP64 for both types plus the rounding of the result
(and, in FP32, of f itself, 4 eps32 of the same sum)."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("n,nm,L", [(1, 1, 9), (2, 3, 5), (31, 31, 6), (32, 33, 3), (33, 33, 2), (47, 48, 3), (63, 63, 2),
                                    (96, 96, 2), (97, 99, 2), (127, 127, 2), (129, 129, 2), (160, 161, 2), (191, 191, 2), (193, 193, 2), (255, 255, 2),
                                    (257, 257, 1), (1024, 1024, 1)])
def test_tiles(dtype, n, nm, L):
    import eigeng_b200 as E
    dt = torch.float64 if dtype == "f64" else torch.float32
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    v = torch.randn((L, n, nm), generator=g, device="cuda", dtype=torch.float64).to(dt)
    w = torch.rand((L, n), generator=g, device="cuda", dtype=torch.float64).to(dt) + 0.25
    for func, p in ((E.FUNC_DIAG, 0.0), (E.FUNC_POW, -0.5), (E.FUNC_EXP, 0.7)):
        z = torch.full((L, n, nm), float("nan"), dtype=dt, device="cuda")
        E.symfunc(v, w, n, func, p, nm, z)
        V, W = v[:, :, :n].double(), w.double()
        f = W if func == E.FUNC_DIAG else (W ** p if func == E.FUNC_POW else torch.exp(p * W))
        ref = (V.mT * f[:, None, :]) @ V
        mag = (V.mT.abs() * f[:, None, :]) @ V.abs()
        got = z[:, :, :n].double()
        e64, e = torch.finfo(torch.float64).eps, torch.finfo(dt).eps
        tol = 2 * (n + 2) * e64 * mag + (4 * e * mag if dtype == "f32" else 8 * e64 * mag) + e * ref.abs()
        assert ((got - ref).abs() <= tol).all()
        assert torch.equal(got, got.mT) and torch.isnan(z[:, :, n:]).all()


@pytest.mark.parametrize("orders", [(200, 250), (227, 200), (380, 300)])
def test_threads_of_different_orders(orders):
    """Two host threads that launch the same kernels at different orders, each
    on its own stream: every call succeeds and gives the bits of a lone one.
    One kernel in each phase, other sizes of shared memory; 227 and 380 take all
    but 2 KB of what a block can have."""
    import threading
    import eigeng_b200 as E
    out, errors = {}, []

    def work(n, reps):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                g = torch.Generator(device="cuda")
                g.manual_seed(n)
                v = torch.randn((2, n, n), generator=g, device="cuda", dtype=torch.float64)
                w = torch.rand((2, n), generator=g, device="cuda", dtype=torch.float64)
                a0 = v + v.mT
                for _ in range(reps):
                    z = torch.empty_like(v)
                    E.symfunc(v, w, n, E.FUNC_DIAG, 0.0, n, z)
                    a = a0.clone()
                    ev, info = E.solve(a, n)
                torch.cuda.current_stream().synchronize()
                out[n, reps] = (z, a, ev)
        except Exception as e:  # noqa: BLE001
            errors.append((n, repr(e)))

    for n in orders:
        work(n, 1)
    threads = [threading.Thread(target=work, args=(n, 150)) for n in orders]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for n in orders:
        assert all(torch.equal(x, y) for x, y in zip(out[n, 1], out[n, 150]))
