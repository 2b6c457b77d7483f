"""The reductions of phase 1 on chip (k1_sym, k1_warp), run on the CPU from
the library's source: fibers for the GPU threads, barriers and shuffles of
warps, CTAs and clusters (tests/host/simt.hpp).  Its schedule lets one CTA of a
cluster go as far as it can before the next one starts."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HOST = os.path.join(ROOT, "tests", "host")
CUDA = "/usr/local/cuda/include"

F64, F32 = np.float64, np.float32


@pytest.fixture(scope="module")
def lib():
    if not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("CUDA headers not available")
    out = os.path.join(tempfile.mkdtemp(prefix="eigb_sym_"), "libsym_host.so")
    subprocess.check_call(["g++", "-x", "c++", "-std=c++20", "-O1", "-ffp-contract=off", "-Wno-unknown-pragmas", "-fPIC",
                           "-U_FORTIFY_SOURCE",  # it takes jumps between stacks for an error
                           "-shared", "-I" + CUDA, "-o", out, os.path.join(HOST, "sym_host.cu")])
    so = ctypes.CDLL(out)
    P, I = ctypes.c_void_p, ctypes.c_int
    for s in ("d", "f"):
        f = getattr(so, "host_sym_" + s)
        f.restype, f.argtypes = ctypes.c_long, [I, I, I, P, I, I, I, I, P, P, P, P, I, P, I]
        f = getattr(so, "host_warp_" + s)
        f.restype, f.argtypes = ctypes.c_long, [P, I, I, P, P, P]
    return so


def _p(x):
    return None if x is None else ctypes.c_void_p(x.ctypes.data)


def uniform(n, dtype, seed):
    b = np.random.default_rng(seed).uniform(-1, 1, (n, n))
    return ((b + b.T) / 2).astype(dtype)


def launch(lib, form, A, m, stop, first, d, e, V, beta, high_first=0):
    """One launch; the number of accesses to CTAs that were not running."""
    f = lib.host_sym_d if A.dtype == F64 else lib.host_sym_f
    r = f(*form, _p(A), A.shape[1], m, stop, first, None, _p(d), _p(e), _p(V), V.shape[1], _p(beta), high_first)
    assert r >= 0, "a thread waits for good" if r == -1 else "form not built"
    return r


def reflectors(V, beta):
    """Q = (H_1 ... H_{n-1})^T from reflector k in V[k, :k]."""
    n = V.shape[0]
    Q = np.eye(n)
    for k in range(1, n):
        v = np.zeros(n)
        v[:k] = V[k, :k]
        Q = Q + beta[k] * np.outer(Q @ v, v)
    return Q.T


def tridiagonal(d, e):
    e = e.astype(F64)
    return np.diag(d.astype(F64)) + np.diag(e[:-1], 1) + np.diag(e[:-1], -1)


def reduce(lib, form, a0, high_first=0):
    n, dt = a0.shape[0], a0.dtype
    A, V = a0.copy(), np.full((n, (n + 7) & ~7), np.nan, dt)
    d, e, beta = np.full(n, np.nan, dt), np.full(n, np.nan, dt), np.full(n, np.nan)
    early = launch(lib, form, A, n, 0, 1, d, e, V, beta, high_first)
    return early, d, e, reflectors(V, beta)


@pytest.mark.parametrize("high_first", [0, 1])
@pytest.mark.parametrize("dtype,form,n", [(F64, (8, 2, 2), 70), (F64, (8, 2, 4), 70), (F64, (8, 2, 8), 40),
                                          (F64, (8, 2, 16), 40), (F32, (8, 4, 2), 70), (F32, (8, 4, 4), 40),
                                          (F32, (8, 4, 8), 40)])
def test_cluster_touches_only_running_ctas(lib, dtype, form, n, high_first):
    """Shared memory of another CTA may be accessed only once all CTAs of the
    cluster run, and until they end; and A = Q T Q^T."""
    a0 = uniform(n, dtype, n)
    early, d, e, Q = reduce(lib, form, a0, high_first)
    assert early == 0
    eps = np.finfo(dtype).eps
    a = a0.astype(F64)
    assert np.linalg.norm(Q @ tridiagonal(d, e) @ Q.T - a) <= 8 * n * eps * np.linalg.norm(a)
    assert np.linalg.norm(Q.T @ Q - np.eye(n)) <= 8 * n * eps * n ** 0.5


def reduce_warp(lib, a0):
    n, dt = a0.shape[0], a0.dtype
    A, d, e = a0.copy(), np.full(n, np.nan, dt), np.full(n, np.nan, dt)
    f = lib.host_warp_d if dt == F64 else lib.host_warp_f
    assert f(_p(A), n, n, None, _p(d), _p(e)) == 0
    return d, e, A.T.astype(F64)


@pytest.mark.parametrize("small_first", [False, True])
@pytest.mark.parametrize("dtype,big,small", [
    (F32, 1e10, 1e-5), (F32, 1e10, 1e-10), (F32, 1e10, 1e-12), (F32, 1e8, 1e-13), (F32, 1e16, 1e-14), (F32, 1, 1e-18),
    (F64, 1e75, 1e-75), (F64, 1e100, 1e-60), (F64, 1e90, 1e-80), (F64, 1e145, 1e-140), (F64, 1, 1e-150)])
@pytest.mark.parametrize("form,n", [("warp", 32), ("small", 50), ("cluster", 70)])
def test_graded_blocks(lib, form, n, dtype, big, small, small_first):
    """Block-diagonal matrices whose blocks differ by up to nearly the range
    of the type: each block is reduced as if it were alone, A_b = Q_b T_b
    Q_b^T to rounding of its own norm.  The reduction is backward stable block
    by block because no reflector of one block has an entry in another."""
    k = n // 2
    lo, hi = (small, big) if small_first else (big, small)
    a0 = np.zeros((n, n))
    a0[:k, :k] = lo * uniform(k, F64, 1)
    a0[k:, k:] = hi * uniform(n - k, F64, 2)
    a0 = a0.astype(dtype)
    if form == "warp":
        d, e, Q = reduce_warp(lib, a0)
    else:
        f = {"small": {F64: (1, 2, 1), F32: (2, 1, 1)}, "cluster": {F64: (8, 2, 2), F32: (8, 4, 2)}}[form][dtype]
        _, d, e, Q = reduce(lib, f, a0)
    assert np.isfinite(d).all() and np.isfinite(e).all() and np.isfinite(Q).all()
    eps = np.finfo(dtype).eps
    T, a = tridiagonal(d, e), a0.astype(F64)
    assert np.linalg.norm(Q.T @ Q - np.eye(n)) <= 8 * n * eps * n ** 0.5
    for b in (slice(0, k), slice(k, n)):
        s = np.abs(a[b, b]).max()
        R = Q[b, b] @ (T[b, b] / s) @ Q[b, b].T - a[b, b] / s
        assert np.linalg.norm(R) <= 8 * n * eps * np.linalg.norm(a[b, b] / s)


def chain(lib, dtype, n, cnt):
    """[(order, form)]: the launches that the library's rule gives cnt matrices of order n."""
    out = np.zeros(64, np.int32)
    k = lib.host_sym_chain(np.dtype(dtype).itemsize, n, ctypes.c_long(cnt), _p(out))
    return [(int(x[0]), tuple(int(y) for y in x[1:])) for x in out.reshape(-1, 4)[:k]]


def run_chain(lib, launches, a0):
    n, dt = a0.shape[0], a0.dtype
    A, V = a0.copy(), np.full((n, (n + 7) & ~7), np.nan, dt)
    d, e, beta = np.full(n, np.nan, dt), np.full(n, np.nan, dt), np.full(n, np.nan)
    for q, (m, form) in enumerate(launches):
        stop = launches[q + 1][0] if q + 1 < len(launches) else 0
        assert launch(lib, form, A, m, stop, int(q == 0), d, e, V, beta) == 0
    return d, e, reflectors(V, beta)


MANY = [(F64, 72, [72, 64]), (F64, 96, [96, 64]), (F64, 128, [128, 64]), (F64, 130, [130, 128, 64]),
        (F64, 161, [161, 128, 64]), (F64, 256, [256, 128, 64]), (F32, 170, [170, 160]), (F32, 230, [230, 160]),
        (F32, 290, [290, 160])]


@pytest.mark.parametrize("dtype,n,orders", MANY)
def test_small_and_large_batches_give_the_same_bits(lib, dtype, n, orders):
    """A batch of more than one wave of CTAs hands its leading blocks over to
    smaller ones, a single matrix does not: the same d, e and Q, bit for bit,
    and A = Q T Q^T."""
    many, one = chain(lib, dtype, n, 100000), chain(lib, dtype, n, 1)
    assert [m for m, _ in many] == orders and [m for m, _ in one] == [n]
    a0 = uniform(n, dtype, n)
    d, e, Q = run_chain(lib, many, a0)
    d1, e1, Q1 = run_chain(lib, one, a0)
    assert np.array_equal(d, d1) and np.array_equal(e, e1) and np.array_equal(Q, Q1)
    eps, a = np.finfo(dtype).eps, a0.astype(F64)
    assert np.linalg.norm(Q @ tridiagonal(d, e) @ Q.T - a) <= 8 * n * eps * np.linalg.norm(a)
    assert np.linalg.norm(Q.T @ Q - np.eye(n)) <= 8 * n * eps * n ** 0.5


@pytest.mark.parametrize("dtype,n", [(F64, 130), (F64, 260), (F32, 170)])
def test_graded_blocks_across_a_hand_over(lib, dtype, n):
    """Blocks of very different magnitude, block by block as if alone, with the
    border between them at another order than the hand-overs."""
    launches = chain(lib, dtype, n, 100000)
    assert len(launches) > 1
    k = n // 2
    a0 = uniform(n, dtype, n)
    a0[:k, k:] = a0[k:, :k] = 0
    a0[:k, :k] *= dtype(1e-20 if dtype == F32 else 1e-200)
    d, e, Q = run_chain(lib, launches, a0)
    T, eps, a = tridiagonal(d, e), np.finfo(dtype).eps, a0.astype(F64)
    assert np.linalg.norm(Q.T @ Q - np.eye(n)) <= 8 * n * eps * n ** 0.5
    for b in (slice(0, k), slice(k, n)):
        s = np.abs(a[b, b]).max()
        R = Q[b, b] @ (T[b, b] / s) @ Q[b, b].T - a[b, b] / s
        assert np.linalg.norm(R) <= 8 * n * eps * np.linalg.norm(a[b, b] / s)


def test_chain_of_every_order(lib):
    """The launches shrink to the end; those of more than one CTA a matrix,
    which sum in another order, are the same for every batch."""
    for dtype in (F64, F32):
        for n in range(33, 1025):
            few, many = chain(lib, dtype, n, 1), chain(lib, dtype, n, 100000)
            for c in (few, many):
                assert c[0][0] == n and all(x[0] > y[0] for x, y in zip(c, c[1:]))
            assert [x for x in few if x[1][2] > 1] == [x for x in many if x[1][2] > 1]
    for n, few, many in ((1000, [736, 512, 256], [736, 512, 256, 128, 64]), (513, [512, 256], [512, 256, 128, 64]),
                         (300, [256], [256, 128, 64])):
        assert [m for m, _ in chain(lib, F64, n, 1)] == [n] + few
        assert [m for m, _ in chain(lib, F64, n, 100000)] == [n] + many
