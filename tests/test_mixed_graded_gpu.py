"""The mixed SVD of matrices with columns (and rows) over many decades (csrc/mixed.cu): FP32 stages whose
Gram entries leave the FP32 range must not lose the call. The bounds are those of the mixed SVD's other
tests (32 n eps)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def mixed(kind, A):
    import torch
    import vecjac_gb300 as vj
    from vecjac_gb300 import build
    build.build()
    m, n = A.shape
    js, stp = vj.pjs(4, n)
    dev = lambda x: torch.tensor(np.ascontiguousarray(x.T), dtype=torch.float64, device="cuda")
    G, V = dev(A.real), torch.empty((n, n), dtype=torch.float64, device="cuda")
    kw = dict(Gi=dev(A.imag), ldGi=m, Vi=torch.empty_like(V), ldVi=n) if kind == "z" else {}
    eS = torch.empty(n, dtype=torch.float64, device="cuda")
    fS = torch.empty_like(eS)
    r, _, _ = vj.vjsvd_mixed_dev(kind, m, n, G, m, V, n, eS, fS, torch.tensor(js.astype(np.int32), device="cuda"), stp, **kw)
    torch.cuda.synchronize()
    host = lambda x, y: x.cpu().numpy().T + (1j * y.cpu().numpy().T if kind == "z" else 0)
    return r, host(G, kw.get("Gi")), host(V, kw.get("Vi")), fS.cpu().numpy() * np.exp2(eS.cpu().numpy())


def matrix(kind, m, n, cols, rows, seed=1):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if kind == "z" else 0)
    return A * 10.0 ** (-cols * rng.random(n)) * 10.0 ** (-rows * rng.random((m, 1)))


@pytest.mark.parametrize("kind,m,n,cols,rows", [("z", 1024, 1024, 30, 0), ("z", 1024, 1024, 12, 12), ("d", 512, 256, 30, 0),
                                                ("z", 512, 256, 30, 0), ("d", 2048, 2048, 30, 0)])
def test_graded(kind, m, n, cols, rows):
    A = matrix(kind, m, n, cols, rows)
    r, U, V, s = mixed(kind, A)
    assert r >= 0, r
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) <= 32 * n * EPS
    assert np.max(np.abs(V.conj().T @ V - np.eye(n))) <= 32 * n * EPS
    assert np.max(np.abs(A @ V - U * s)) <= 32 * n * EPS * s.max()


@pytest.mark.parametrize("kind", ["d", "z"])
@pytest.mark.parametrize("m,n,cols", [(128, 64, 4), (160, 96, 12), (520, 272, 12), (1032, 1024, 12), (520, 272, 30)])
def test_columns_to_their_own_length(kind, m, n, cols):
    """A v_j - u_j sigma_j within 32 n eps sigma_j, for every j: a short column's v_j needs its small
    entries, where A's columns are long, to their own accuracy. (The terms of A v_j are of the order of
    sigma_j, so that the products here add less than n eps sigma_j.)"""
    A = matrix(kind, m, n, cols, 0, seed=2)
    r, U, V, s = mixed(kind, A)
    assert r >= 0, r
    assert np.max(np.linalg.norm(A @ V - U * s, axis=0) / s) <= 32 * n * EPS
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) <= 32 * n * EPS
    assert np.max(np.abs(V.conj().T @ V - np.eye(n))) <= 32 * n * EPS
