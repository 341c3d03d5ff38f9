"""The calls whose speed is tracked: what a user of the library has it do, from one small host call to the largest SVD.

Every case goes through the package's public entry points (``vecjac_gb300.api``, ``.batch``,
``.autodiff``). ``listed()`` gives the named cases, ``draw(rng)`` one more from the ranges they stand
for, ``prepare(case, seed)`` the inputs on the GPU (or in host memory where the call takes host
pointers), ``run(state)`` one pass, ``work(case)`` what the pass cannot do without, and
``exact(case, seed)`` the same outputs from plain 64-bit arithmetic.

The families (``case["op"]``):

* ``bjac2_host`` / ``bjac2``: the batched 2x2 Hermitian EVD on host arrays (the drop-in call of the
  reference's callers) and on device arrays; kinds d, z, s, c; inputs of ``workloads.pairs2x2``.
* ``svd_host`` / ``svd``: the one-sided Jacobi SVD on host arrays and on device arrays.
* ``mixed``: the mixed-precision SVD of FP64 data.
* ``batch``: many real matrices of uneven shapes in one launch.
* ``diff``: the differentiable batched SVD, forward and backward.
"""
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import vecjac_gb300 as vj
from vecjac_gb300 import autodiff, workloads
from vecjac_gb300.batch import Batch, padded_shape

STRATEGY = 4  # the modulus ordering, the one every benchmark of the package uses


def listed():
    return [
        # a caller of the reference's dbjac2_ with a few thousand pairs in host memory: one sweep step's
        # worth of 2x2 problems, where the copies and the launch count
        {"name": "bjac2_host_d_4096", "op": "bjac2_host", "kind": "d", "n": 4096, "sines": True},
        # large device-resident batches: FP64 real at a power of two, FP32 complex at an odd number of
        # vectors (the package's headline workload is these batches at 2^28 and 2^27)
        {"name": "bjac2_d_2e26", "op": "bjac2", "kind": "d", "n": 1 << 26, "sines": False},
        {"name": "bjac2_c_odd", "op": "bjac2", "kind": "c", "n": 16 * 2500007, "sines": True},
        # the smallest SVD: dvjsvd_ on host arrays
        {"name": "svd_host_d_64x32", "op": "svd_host", "kind": "d", "m": 64, "n": 32, "decades": 3},
        # the plain SVD of every data type: the 1024 x 1024 FP64 benchmark matrix, a medium FP64 complex
        # one, an FP32 one whose sizes are odd multiples of the vector length
        {"name": "svd_d_1024x1024", "op": "svd", "kind": "d", "m": 1024, "n": 1024, "decades": 6},
        {"name": "svd_z_512x256", "op": "svd", "kind": "z", "m": 512, "n": 256, "decades": 4},
        {"name": "svd_s_656x608", "op": "svd", "kind": "s", "m": 656, "n": 608, "decades": 2},
        # the mixed-precision SVD: real square, and the 4096 x 2048 complex benchmark shape
        {"name": "mixed_d_1024x1024", "op": "mixed", "kind": "d", "m": 1024, "n": 1024, "decades": 2},
        {"name": "mixed_z_4096x2048", "op": "mixed", "kind": "z", "m": 4096, "n": 2048, "decades": 2},
        # thousands of small matrices of uneven shapes (the package's 20,000-matrix workload, fewer and
        # smaller), FP32 and FP64
        {"name": "batch_s_4000", "op": "batch", "kind": "s", "count": 4000, "mmax": 256},
        {"name": "batch_d_1500", "op": "batch", "kind": "d", "count": 1500, "mmax": 128},
        # a training step through the SVD layer: forward and gradient of 128 x 64 matrices, k = 16
        {"name": "diff_2048x128x64", "op": "diff", "count": 2048, "m": 128, "n": 64, "k": 16},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi // step, max(-(-lo // step), round(v / step)))) * step


def draw(rng):
    op = rng.choice(["bjac2_host", "bjac2", "bjac2", "svd_host", "svd", "svd", "mixed", "mixed", "batch", "batch", "diff"])
    if op == "bjac2_host":
        return {"op": op, "kind": rng.choice("dzsc"), "n": _log(rng, 16, 1 << 18, 16), "sines": rng.random() < 0.5}
    if op == "bjac2":
        return {"op": op, "kind": rng.choice("dzsc"), "n": _log(rng, 1 << 10, 1 << 26, 16), "sines": rng.random() < 0.5}
    if op in ("svd_host", "svd"):
        kind = rng.choice("dzsc")
        lanes = 8 if kind in "dz" else 16
        top = 64 if op == "svd_host" else 384
        n = _log(rng, 2 * lanes, top, 2 * lanes)
        return {"op": op, "kind": kind, "m": _log(rng, n, 2 * top, lanes), "n": n, "decades": 2 if kind in "sc" else 4}
    if op == "mixed":
        kind = rng.choice("dz")
        n = _log(rng, 64, 768, 16)
        return {"op": op, "kind": kind, "m": _log(rng, n, 1536, 8), "n": n, "decades": rng.choice([1, 2])}
    if op == "batch":
        kind = rng.choice("ds")
        return {"op": op, "kind": kind, "count": _log(rng, 20, 2000), "mmax": _log(rng, 32, 128 if kind == "d" else 256)}
    n = _log(rng, 32, 64, 32)
    return {"op": op, "count": _log(rng, 64, 2048), "m": _log(rng, n, 128, 16), "n": n, "k": _log(rng, 1, 16)}


# ---------------- inputs ----------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _ortho(x):
    """Orthonormal columns of a Gaussian x (..., m, n): Cholesky QR, repeated to full accuracy."""
    for _ in range(3):
        r = torch.linalg.cholesky(x.mH @ x, upper=True)
        x = torch.linalg.solve_triangular(r, x, upper=True, left=False)
    return x


def _factors(kind, m, n, decades, seed):
    """U (m, n), sigma (n, descending), V (n, n) in 64 bits: Haar factors, sigma log-uniform over the decades,
    one in each n-th of the range, away from its ends, so that the singular vectors are determined."""
    g = _gen(seed)
    dt = torch.complex128 if kind in "zc" else torch.float64
    U = _ortho(torch.randn((m, n), generator=g, device="cuda", dtype=dt))
    V = _ortho(torch.randn((n, n), generator=g, device="cuda", dtype=dt))
    at = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.25 + 0.5 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)) / n
    return U, 10.0 ** (-decades * at), V


def _real(kind):
    return torch.float64 if kind in "dz" else torch.float32


def _columns(A, kind):
    """(re, im) planes of A in column-major storage: tensors (n, m) of the kind's real type; im is None for real data."""
    At = A.mT
    if A.is_complex():
        return At.real.to(_real(kind)).contiguous(), At.imag.to(_real(kind)).contiguous()
    return At.to(_real(kind)).contiguous(), None


def _uneven(case, seed):
    """The batch's matrices: Gaussian, columns scaled over two decades, shapes of workloads.uneven_shapes (the case's own)."""
    m, n = workloads.uneven_shapes(case["count"], 1, mmax=case["mmax"])
    rng = np.random.default_rng(seed)
    dt = np.float64 if case["kind"] == "d" else np.float32
    return [rng.standard_normal((int(a), int(b)), dtype=dt) * (10.0 ** rng.uniform(-2.0, 0.0, int(b))).astype(dt) for a, b in zip(m, n)]


def _spaced(case, seed):
    """A (count, m, n) in 64 bits with its factors and the cotangents of sigma, U_k and V_k."""
    c, m, n, k = case["count"], case["m"], case["n"], case["k"]
    g = _gen(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    U, V = _ortho(rnd(c, m, n)), _ortho(rnd(c, n, n))
    at = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.25 + 0.5 * torch.rand((c, n), generator=g, device="cuda", dtype=torch.float64)) / n
    return U, 10.0 ** (1.0 - 2.0 * at), V, rnd(c, n), rnd(c, m, k), rnd(c, n, k)


def prepare(case, seed):
    op = case["op"]
    st = {"case": case}
    if op == "bjac2_host":
        st["ins"] = workloads.pairs2x2(case["kind"], case["n"], seed)
    elif op == "bjac2":
        n, kind = case["n"], case["kind"]
        st["ins"] = workloads.pairs2x2_torch(kind, n, seed)
        st["outs"] = [torch.empty(n, dtype=_real(kind), device="cuda") for _ in range(5 if kind in "zc" else 4)]
        st["p"] = torch.zeros(n // (8 if kind in "dz" else 16), dtype=torch.int32, device="cuda")
    elif op == "svd_host":
        U, s, V = _factors(case["kind"], case["m"], case["n"], case["decades"], seed)
        A = ((U * s) @ V.mH).cpu().numpy()
        st["G"] = np.asfortranarray(A.real)
        st["Gi"] = np.asfortranarray(A.imag) if case["kind"] in "zc" else None
        st["js"], st["stp"] = vj.pjs(STRATEGY, case["n"])
    elif op in ("svd", "mixed"):
        kind, m, n = case["kind"], case["m"], case["n"]
        U, s, V = _factors(kind, m, n, case["decades"], seed)
        st["G0"], st["G0i"] = _columns((U * s) @ V.mH, kind)
        new = lambda *s_: torch.empty(s_, dtype=_real(kind), device="cuda")  # noqa: E731
        cplx = kind in "zc"
        st["G"], st["Gi"] = new(n, m), new(n, m) if cplx else None
        st["V"], st["Vi"] = new(n, n), new(n, n) if cplx else None
        st["eS"], st["fS"] = new(n), new(n)
        js, st["stp"] = vj.pjs(STRATEGY, n)
        st["js"] = torch.from_numpy(js.astype(np.int32)).cuda()
    elif op == "batch":
        st["batch"] = Batch(_uneven(case, seed), case["kind"])
    else:
        U, s, V, dS, dU, dV = _spaced(case, seed)
        st["A"] = ((U * s[:, None, :]) @ V.mT).float().requires_grad_()
        st["cot"] = [dS.float(), dU.float(), dV.float()]
    return st


# ---------------- one pass ----------------

def _fixed(G, Gi, V, Vi):
    """The columns of U and V (rows of the tensors) with the sign or phase that makes the largest entry of v_j positive."""
    if Gi is None:
        s = torch.sign(V.gather(1, V.abs().argmax(1, keepdim=True)))
        return [G * s, V * s]
    v = torch.complex(V, Vi)
    p = v.gather(1, (V * V + Vi * Vi).argmax(1, keepdim=True))
    p = p.conj() / p.abs()
    return [torch.complex(G, Gi) * p, v * p]


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "bjac2_host":
        return list(vj.bjac2(case["kind"], -case["n"] if case["sines"] else case["n"], *st["ins"]))
    if op == "bjac2":
        n, kind, ins, outs = case["n"], case["kind"], st["ins"], st["outs"]
        c, at, sat = outs[0], outs[1], outs[2] if kind in "zc" else None
        r = vj.bjac2_dev(kind, -n if case["sines"] else n, ins[0], ins[1], ins[2], ins[3] if kind in "zc" else None, c,
                         at, sat, outs[-2], outs[-1], st["p"])
        return [r] + outs + [st["p"]]
    if op == "svd_host":
        return list(vj.vjsvd(case["kind"], st["G"], st["js"], st["stp"], Gi=st["Gi"]))
    if op in ("svd", "mixed"):
        kind, m, n, cplx = case["kind"], case["m"], case["n"], case["kind"] in "zc"
        st["G"].copy_(st["G0"])  # the call overwrites its matrix
        if cplx:
            st["Gi"].copy_(st["G0i"])
        kw = dict(Gi=st["Gi"], ldGi=m, Vi=st["Vi"], ldVi=n) if cplx else {}
        if op == "svd":
            r = vj.vjsvd_dev(kind, m, n, st["G"], m, st["V"], n, st["eS"], st["fS"], st["js"], st["stp"], **kw)
            return [r, st["eS"], st["fS"], st["G"], st["V"]] + ([st["Gi"], st["Vi"]] if cplx else [])
        vj.vjsvd_mixed_dev(kind, m, n, st["G"], m, st["V"], n, st["eS"], st["fS"], st["js"], st["stp"], **kw)
        return [st["eS"], st["fS"]] + _fixed(st["G"], st["Gi"], st["V"], st["Vi"])
    if op == "batch":
        b = st["batch"]
        b.run(STRATEGY, block=256)
        return [b.info, b.eS, b.fS, b.G, b.V]
    S, U, V = autodiff.svd_k(st["A"], case["k"])
    (dA,) = torch.autograd.grad([S, U, V], st["A"], st["cot"])
    return [S.detach(), U.detach(), V.detach(), dA]


def work(case):
    op = case["op"]
    if op in ("bjac2_host", "bjac2"):
        w, f = {"d": (56.5, 30), "z": (72.5, 45), "s": (28.25, 30), "c": (36.25, 45)}[case["kind"]]
        return {"bytes": w * case["n"], "flops": f * case["n"]}
    if op == "diff":
        c, m, n, k = case["count"], case["m"], case["n"], case["k"]
        svd = 6 * n * (n - 1) / 2 * (12 * m + 6 * n)
        return {"bytes": c * 4.0 * (2 * m * n + n + 2 * (m + n) * k + n), "flops": c * (svd + 2.0 * (m * n * k + n * n * k + n ** 3 + m * n * (n + k)))}
    if op == "batch":
        m, n = workloads.uneven_shapes(case["count"], 1, mmax=case["mmax"])
        m, n = m.astype(np.float64), n.astype(np.float64)
        b = 8 if case["kind"] == "d" else 4
        return {"bytes": float(b * np.sum(2 * m * n + n * n + 2 * n)), "flops": float(np.sum(6 * n * (n - 1) / 2 * (12 * m + 6 * n)))}
    m, n, planes = case["m"], case["n"], 2 if case["kind"] in "zc" else 1
    b = 8 if case["kind"] in "dz" else 4
    per = (36 * m + 20 * n) if planes == 2 else (12 * m + 6 * n)
    # (six sweeps are what the method takes with quadratic convergence from a good start)
    return {"bytes": b * (planes * (2.0 * m * n + n * n) + 2 * n), "flops": 6 * n * (n - 1) / 2 * per}


# ---------------- 64-bit values ----------------

def _exact2x2(kind, ins, sines):
    """[c, t or s (re[, im]), l1, l2] of every 2x2 from the tangent formula in 64 bits, scaled by the largest entry."""
    a = [torch.as_tensor(x).double() for x in ins]
    e = torch.frexp(torch.stack([x.abs() for x in a]).max(0).values)[1]
    a = [torch.ldexp(x, -e) for x in a]
    mod = a[2].abs() if len(a) == 3 else torch.hypot(a[2], a[3])
    t2 = torch.copysign(torch.clamp(2 * mod / (a[0] - a[1]).abs(), max=1e150), a[0] - a[1])
    t = t2 / (1 + torch.sqrt(1 + t2 * t2))
    s2 = 1 + t * t
    s = t / torch.sqrt(s2) if sines else t
    dirs = [torch.sign(a[2])] if len(a) == 3 else [a[2] / mod, a[3] / mod]
    l1 = (a[0] + t * (2 * mod + a[1] * t)) / s2
    l2 = (a[1] + t * (a[0] * t - 2 * mod)) / s2
    return [1 / torch.sqrt(s2)] + [s * d for d in dirs] + [torch.ldexp(l1, e), torch.ldexp(l2, e)]


def _ef(s):
    """sigma = f 2^e with f in [1, 2); a zero is (-inf, 1)."""
    f, e = torch.frexp(s)
    return [torch.where(s > 0, (e - 1).double(), torch.full_like(s, -math.inf)), torch.where(s > 0, 2 * f, torch.ones_like(s))]


def exact(case, seed):
    op = case["op"]
    if op == "bjac2_host":
        return [None] + _exact2x2(case["kind"], workloads.pairs2x2(case["kind"], case["n"], seed), case["sines"]) + [None]
    if op == "bjac2":
        return [None] + _exact2x2(case["kind"], workloads.pairs2x2_torch(case["kind"], case["n"], seed), case["sines"]) + [None]
    if op in ("svd_host", "svd", "mixed"):
        U, s, V = _factors(case["kind"], case["m"], case["n"], case["decades"], seed)
        cplx = case["kind"] in "zc"
        if op == "mixed":
            Ut, Vt = U.mT, V.mT  # rows are columns; A = U diag(s) V^H
            if cplx:
                return _ef(s) + _fixed(Ut.real, Ut.imag, Vt.real, Vt.imag)
            return _ef(s) + _fixed(Ut, None, Vt, None)
        # (the signs of the singular vectors are the algorithm's own: no value for U and V)
        if op == "svd_host":
            return [None, None, None] + _ef(s) + ([None, None] if cplx else [])
        return [None] + _ef(s) + [None] * (4 if cplx else 2)
    if op == "batch":
        mats = _uneven(case, seed)
        with ThreadPoolExecutor(8) as ex:
            sv = list(ex.map(lambda A: np.linalg.svd(A.astype(np.float64), compute_uv=False), mats))
        s = [np.concatenate([v, np.zeros(padded_shape(*A.shape, case["kind"])[1] - A.shape[1])]) for A, v in zip(mats, sv)]
        return [None] + _ef(torch.from_numpy(np.concatenate(s))) + [None, None]
    U, S, V, dS, dU, dV = _spaced(case, seed)
    k = case["k"]
    sgn = torch.sign(V.gather(1, V.abs().argmax(1, keepdim=True)))
    U, V = U * sgn, V * sgn
    n = S.shape[1]
    J, K = S.new_zeros(len(S), n, n), S.new_zeros(len(S), n, n)
    J[:, :, :k], K[:, :, :k] = U.mT @ dU, V.mT @ dV
    si, sj = S[:, :, None], S[:, None, :]
    d = (sj - si) * (sj + si)
    F = torch.where(d != 0, 1 / torch.where(d != 0, d, torch.ones_like(d)), torch.zeros_like(d))
    N = torch.diag_embed(dS) + F * ((J - J.mT) * sj + si * (K - K.mT)) - J / sj
    dA = U @ (N @ V.mT) + dU @ (V[:, :, :k] / S[:, None, :k]).mT
    return [S, U[:, :, :k], V[:, :, :k], dA]
