"""The mixed SVD's refinements by a rotation of large norm (csrc/mixed.cu): after a single FP32
stage the singular directions of five decades of singular values are only known to about 1e-2,
and the generator's norm is beyond what the series takes in one application."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


@pytest.mark.parametrize("kind", ["d", "z"])
@pytest.mark.parametrize("m,n", [(512, 256), (768, 512)])
def test_one_stage(kind, m, n):
    import torch
    import vecjac_gb300 as vj
    from vecjac_gb300 import build
    build.build()
    rng = np.random.default_rng(m + n)

    def ortho(r, c):
        x = rng.standard_normal((r, c)) + (1j * rng.standard_normal((r, c)) if kind == "z" else 0)
        return np.linalg.qr(x)[0]

    sig = 10.0 ** (-5.0 * (np.arange(n) + rng.uniform(0.25, 0.75, n)) / n)
    A = (ortho(m, n) * sig) @ ortho(n, n).conj().T
    js, stp = vj.pjs(4, n)
    dev = lambda x: torch.tensor(np.ascontiguousarray(x.T), dtype=torch.float64, device="cuda")
    G, Gi = dev(A.real), dev(A.imag) if kind == "z" else None
    V = torch.empty((n, n), dtype=torch.float64, device="cuda")
    Vi = torch.empty_like(V) if kind == "z" else None
    eS = torch.empty(n, dtype=torch.float64, device="cuda")
    fS = torch.empty_like(eS)
    r, r32, r64 = vj.vjsvd_mixed_dev(kind, m, n, G, m, V, n, eS, fS, torch.tensor(js.astype(np.int32), device="cuda"), stp,
                                     Gi=Gi, ldGi=m, Vi=Vi, ldVi=n, stages=1)
    torch.cuda.synchronize()
    assert r >= 0 and r32 > 0 and r64 > 0
    host = lambda x, y: x.cpu().numpy().T + (1j * y.cpu().numpy().T if kind == "z" else 0)
    U, W = host(G, Gi), host(V, Vi)
    s = fS.cpu().numpy() * np.exp2(eS.cpu().numpy())
    # the bounds of the mixed SVD's other tests: 32 n eps
    tol = 32 * n * EPS
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) <= tol
    assert np.max(np.abs(W.conj().T @ W - np.eye(n))) <= tol
    assert np.max(np.abs(A @ W - U * s)) <= tol * np.max(np.abs(A)) * np.sqrt(n)
    assert np.max(np.abs(np.sort(s)[::-1] - np.sort(sig)[::-1])) <= tol * sig.max()
