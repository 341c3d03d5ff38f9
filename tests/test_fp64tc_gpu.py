"""The FP64 products of the mixed SVD on the tensor cores (csrc/fp64tc.cu) through the SVD
itself, at the edges of their tiles (64 columns, 128 rows, 32 elements of K) and where the
refinement hands over to the plain sweeps: pairs of equal singular values, graded columns over
12 decades, a rank-deficient matrix. V and U orthogonal and the residual within the bounds of
the other mixed tests (32 n eps), singular values within 32 n eps of the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["d", "z"])
@pytest.mark.parametrize("m,n,case", [(16, 16, "spread"), (72, 48, "spread"), (136, 64, "spread"), (200, 80, "spread"),
                                      (136, 128, "equal"), (264, 144, "graded"), (160, 96, "deficient"),
                                      (520, 272, "spread")])
def test_mixed_at_tile_edges(kind, m, n, case):
    import torch
    import vecjac_gb300 as vj
    from vecjac_gb300 import build
    from vecjac_gb300 import workloads as W
    build.build()
    rng = np.random.default_rng(m * 1000 + n)
    U0, V0 = W.haar(m, rng, kind == "z")[:, :n], W.haar(n, rng, kind == "z")
    sig = np.logspace(0, -2, n)
    if case == "equal":
        sig = np.repeat(sig[::4], 4)
    if case == "deficient":
        sig[-n // 4:] = 0
    A = (U0 * sig) @ V0.conj().T
    if case == "graded":
        A = A * np.logspace(0, -12, n)
    ref = np.linalg.svd(A, compute_uv=False)
    js, stp = vj.pjs(4, n)
    t = lambda x: torch.tensor(np.ascontiguousarray(x.T), dtype=torch.float64, device="cuda")
    G, V = t(A.real), torch.empty((n, n), dtype=torch.float64, device="cuda")
    kw = {}
    if kind == "z":
        kw = dict(Gi=t(A.imag), ldGi=m, Vi=torch.empty((n, n), dtype=torch.float64, device="cuda"), ldVi=n)
    e = torch.empty(n, dtype=torch.float64, device="cuda")
    f = torch.empty_like(e)
    r, _, _ = vj.vjsvd_mixed_dev(kind, m, n, G, m, V, n, e, f, torch.tensor(js.astype(np.int32), device="cuda"), stp, **kw)
    torch.cuda.synchronize()
    assert r >= 0, r
    s = f.cpu().numpy() * np.exp2(e.cpu().numpy())
    U, Vm = G.cpu().numpy().T, V.cpu().numpy().T
    if kind == "z":
        U, Vm = U + 1j * kw["Gi"].cpu().numpy().T, Vm + 1j * kw["Vi"].cpu().numpy().T
    eps = np.finfo(np.float64).eps
    assert np.max(np.abs(np.sort(s)[::-1] - ref)) <= 32 * n * eps * ref[0]
    assert np.linalg.norm(Vm.conj().T @ Vm - np.eye(n)) <= 32 * n * eps
    assert np.linalg.norm(A @ Vm - U * s) <= 32 * n * eps * ref[0]
    big = s > 1e3 * n * eps * s.max() if case == "deficient" else s > 0
    Ub = U[:, big]
    assert np.linalg.norm(Ub.conj().T @ Ub - np.eye(Ub.shape[1])) <= 32 * n * eps
