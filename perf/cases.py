"""The calls whose speed is followed: what programs do with this library.

A program decomposes a batch of symmetric matrices in place with a workspace
that it keeps, and then forms the matrix function it wants from the pairs.
Each case is that whole step, solve plus `symfunc`: in ensemble filters the
transform A^(-1/2) of covariance-like matrices, elsewhere the propagator
exp(A) of normalised symmetric operators.  The eigenvectors' content comes
back through the function: alone, each of them is determined up to its sign
only.

The in-place calls work on a copy of the batch, which the program keeps.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "eigeng-batched_b200"))
import eigeng_b200 as E  # noqa: E402

DT = {"f64": torch.float64, "f32": torch.float32}


def listed():
    return [
        # the smallest calls, where launches and latency count: the local
        # analysis of a 12-member ensemble over a few grid points
        dict(name="small_f64_n12", form="dropin", dtype="f64", family="letkf", n=12, nm=12, L=100),
        # many tiny matrices, the largest order that one warp takes
        dict(name="f64_n32", form="dropin", dtype="f64", family="uniform", n=32, nm=32, L=16384),
        # packed upper triangles, as covariance codes store them; an odd order
        dict(name="packed_f64_n45", form="packed", dtype="f64", family="uniform", n=45, nm=45, L=6000),
        dict(name="f32_n64", form="dropin", dtype="f32", family="uniform", n=64, nm=64, L=20000),
        # the ensemble-transform batch that the benchmark names, both types
        dict(name="f64_n128", form="dropin", dtype="f64", family="letkf", n=128, nm=128, L=4096),
        dict(name="f32_n128", form="dropin", dtype="f32", family="letkf", n=128, nm=128, L=4096),
        # an odd order in a padded array
        dict(name="f32_n201_nm208", form="dropin", dtype="f32", family="uniform", n=201, nm=208, L=1000),
        dict(name="f64_n256", form="dropin", dtype="f64", family="uniform", n=256, nm=256, L=2048),
        # tight clusters through the FP32 solve refined to FP64
        dict(name="refined_f64_n256", form="refined", dtype="f64", family="clustered", n=256, nm=256, L=512),
        # few large matrices: under two a multiprocessor, then a quarter of one
        dict(name="f64_n512", form="dropin", dtype="f64", family="uniform", n=512, nm=512, L=256),
        dict(name="f64_n1000", form="dropin", dtype="f64", family="uniform", n=1000, nm=1000, L=32),
        # blocks of many orders in one call, as a block-diagonal operator has them
        dict(name="uneven_f64", form="uneven", dtype="f64", family="uniform",
             orders="9x60 17x60 32x60 47x60 64x40 90x40 120x40 128x30 161x30 200x20 255x20 300x16 384x12 500x8"),
    ]


def draw(rng):
    dtype = rng.choice(["f64", "f64", "f32"])
    form = rng.choice(["dropin", "dropin", "dropin", "packed", "uneven"])
    if form == "uneven":
        orders = sorted({_log(rng, 8, 512) for _ in range(rng.randint(3, 14))})
        return dict(form=form, dtype=dtype, family="uniform",
                    orders=" ".join("%dx%d" % (n, _log(rng, 1, min(60, max(2, 6.4e8 // n**3)))) for n in orders))
    n = _log(rng, 3, 1024)
    return dict(form=form, dtype=dtype, family=rng.choice(["uniform", "letkf"]), n=n,
                nm=n if form == "packed" else n + rng.choice([0, 0, 0, 1, 3, 8]),
                L=_log(rng, 4, max(5, min(20000, 2.6e10 // n**3))))


def _log(rng, lo, hi):
    """A whole number from lo to hi, its logarithm spread evenly."""
    return max(lo, min(int(hi), int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _orders(case):
    if case["form"] != "uneven":
        return [(case["n"], case["L"])]
    return [tuple(int(x) for x in o.split("x")) for o in case["orders"].split()]


def _pieces(family, n, L, seed):
    """What the matrices are made of: (L, n, n) float64 on the GPU, and the
    spectrum where the family has a given one."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + n)
    if family == "letkf":  # (n-1) I + Y^T Y, Y iid N(0,1)/sqrt(n)
        y = torch.randn((L, n, n), generator=g, device="cuda", dtype=torch.float64).div_(math.sqrt(n))
        a = torch.bmm(y.mT, y)
        a.diagonal(dim1=1, dim2=2).add_(n - 1.0)
        return a, None
    b = torch.rand((L, n, n), generator=g, device="cuda", dtype=torch.float64).mul_(2).sub_(1)
    if family == "uniform":  # (B + B^T)/2, B iid U[-1,1], scaled to a norm near 0.82 at any order
        return b.add_(b.mT.clone()).div_(2 * math.sqrt(n)), None
    # eigenvalues in clusters of eight 1e-8 apart, 0.1 between clusters, in
    # the basis exp(K) of a skew-symmetric K
    q = torch.linalg.matrix_exp(b.sub_(b.mT.clone()).div_(math.sqrt(n)))
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    lam = 0.1 * torch.floor(k / 8) + 1e-8 * torch.remainder(k, 8)
    lam = (lam - lam.mean()).expand(L, n)
    a = torch.bmm(q * lam[:, None, :], q.mT)
    return a.add_(a.mT.clone()).div_(2), (q, lam)


def _matrices(case, seed):
    """[(n, batch)]: the float64 batches of each order."""
    return [(n, _pieces(case["family"], n, L, seed)[0]) for n, L in _orders(case)]


def _func(case):
    return (E.FUNC_POW, -0.5) if case["family"] == "letkf" else (E.FUNC_EXP, 1.0)


def prepare(case, seed):
    dt, form = DT[case["dtype"]], case["form"]
    func, p = _func(case)
    s = dict(form=form, func=func, p=p)
    if form == "uneven":
        mats = [(n, a.to(dt)) for n, a in _matrices(case, seed)]
        s["a0"] = torch.cat([a.reshape(-1) for _, a in mats])
        s["orders"] = [(n, a.shape[0]) for n, a in mats]
        s["ns"] = [n for n, L in s["orders"] for _ in range(L)]
        s["a"], s["z"] = torch.empty_like(s["a0"]), torch.empty_like(s["a0"])
        return s
    n, nm, L = case["n"], case["nm"], case["L"]
    a = _matrices(case, seed)[0][1].to(dt)
    s.update(n=n, nm=nm)
    if form == "packed":
        s["ap"] = E.pack_upper(a, n)
        s["z"] = torch.empty_like(a)
        return s
    a0 = torch.zeros((L, n, nm), dtype=dt, device="cuda")
    a0[:, :, :n] = a
    s["a0"], s["a"], s["z"] = a0, torch.empty_like(a0), torch.zeros_like(a0)
    if form == "refined":
        s["wk"] = E.refine_workspace(L, nm, n)
    else:
        s["w"] = torch.empty((L, n), dtype=dt, device="cuda")
        s["wk"] = E.workspace(L, nm, n, dt)
    return s


def run(s):
    func, p = s["func"], s["p"]
    if s["form"] == "packed":
        v, w, info = E.solve_packed(s["ap"], s["n"])
        return {"w": w, "z": E.symfunc(v, w, s["n"], func, p, z=s["z"]), "info": info}
    a = s["a"].copy_(s["a0"])
    if s["form"] == "uneven":
        w, info = E.solve_uneven(a, s["ns"])
        oa = ow = 0
        for n, L in s["orders"]:
            E.symfunc(a[oa:oa + L * n * n], w[ow:ow + L * n], n, func, p, z=s["z"][oa:oa + L * n * n])
            oa, ow = oa + L * n * n, ow + L * n
        return {"w": w, "z": s["z"], "info": info}
    if s["form"] == "refined":
        w, info, iters = E.solve_refined(a, s["n"], s["nm"], wk=s["wk"])
        return {"w": w, "z": E.symfunc(a, w, s["n"], func, p, s["nm"], s["z"]), "info": info, "iters": iters}
    E.eigen_GPU_batch(a, s["w"], s["wk"], s["n"], s["nm"])
    return {"w": s["w"], "z": E.symfunc(a, s["w"], s["n"], func, p, s["nm"], s["z"])}


def work(case):
    """Bytes: the input and the function once, eigenvalues written.  Flops:
    9 n^3 for a symmetric QR decomposition with vectors (Golub and Van Loan),
    n^3 for one triangle of V f(w) V^T."""
    s = 8 if case["dtype"] == "f64" else 4
    by = fl = 0.0
    for n, L in _orders(case):
        read = n * (n + 1) // 2 if case["form"] == "packed" else n * n
        by += L * s * (read + n * n + n)
        fl += L * 10.0 * n**3
    return {"bytes": by, "flops": fl}


def _inverse_root(a):
    """A^(-1/2) of a well-conditioned positive definite batch: the coupled
    Newton-Schulz iteration on A / c."""
    c = torch.linalg.matrix_norm(a)[:, None, None]
    eye = torch.eye(a.shape[-1], dtype=a.dtype, device=a.device)
    y, z = a / c, eye.expand_as(a).clone()
    for _ in range(40):
        t = 1.5 * eye - 0.5 * torch.bmm(z, y)
        y, z = torch.bmm(y, t), torch.bmm(t, z)
    return z / torch.sqrt(c)


def exact(case, seed):
    dt = DT[case["dtype"]]
    ws, zs = [], []
    for n, L in _orders(case):
        a, known = _pieces(case["family"], n, L, seed)
        if known is not None:
            q, lam = known
            ws.append(torch.sort(lam, dim=1).values)
            zs.append(torch.bmm(q * torch.exp(lam)[:, None, :], q.mT))
            continue
        a = a.to(dt).to(torch.float64)
        zs.append(_inverse_root(a) if case["family"] == "letkf" else torch.linalg.matrix_exp(a))
        # the 64-bit eigenvalues where they come in a few seconds
        if ws is not None and (n <= 32 or L * n <= 600000):
            ws.append(torch.linalg.eigvalsh(a))
        else:
            ws = None
    if case["form"] == "uneven":
        w = None if ws is None else torch.cat([x.reshape(-1) for x in ws])
        return {"w": w, "z": torch.cat([x.reshape(-1) for x in zs])}
    z = torch.zeros((case["L"], case["n"], case["nm"]), dtype=torch.float64, device="cuda")
    z[:, :, :case["n"]] = zs[0]
    return {"w": None if ws is None else ws[0], "z": z}
