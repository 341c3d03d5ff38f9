"""The mixed SVD of matrices with pairs of nearly equal singular values (csrc/mixed.cu): the
rotation of such a pair is its cosine over the relative gap, so the entries of the factor that
the refinement multiplies G by are far larger than the cosines, and its digits have to follow the
entries. The columns of A V - U S show what they leave out: every one of them is within
32 eps ||A||_2, from at most ten products (two stages, up to six refinements, the last scaling) of
which each adds at most about three roundings of the column."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


@pytest.mark.parametrize("kind", ["d", "z"])
@pytest.mark.parametrize("m,n", [(160, 64), (520, 272)])
@pytest.mark.parametrize("gap", [1e-11, 1e-10, 1e-9, 1e-8, 1e-7, 1e-6])
def test_near_equal_pairs(kind, m, n, gap):
    import torch
    import vecjac_gb300 as vj
    from vecjac_gb300 import build
    build.build()
    rng = np.random.default_rng(m + n)

    def ortho(r, c):
        x = rng.standard_normal((r, c)) + (1j * rng.standard_normal((r, c)) if kind == "z" else 0)
        return np.linalg.qr(x)[0]

    sig = 10.0 ** (-(np.arange(n) + 0.5) / n)
    sig[n // 4:3 * n // 4:n // 8] = sig[n // 4 + 1:3 * n // 4 + 1:n // 8] * (1 + gap)
    A = (ortho(m, n) * sig) @ ortho(n, n).conj().T
    js, stp = vj.pjs(4, n)
    dev = lambda x: torch.tensor(np.ascontiguousarray(x.T), dtype=torch.float64, device="cuda")
    G, Gi = dev(A.real), dev(A.imag) if kind == "z" else None
    V = torch.empty((n, n), dtype=torch.float64, device="cuda")
    Vi = torch.empty_like(V) if kind == "z" else None
    eS = torch.empty(n, dtype=torch.float64, device="cuda")
    fS = torch.empty_like(eS)
    r, _, _ = vj.vjsvd_mixed_dev(kind, m, n, G, m, V, n, eS, fS, torch.tensor(js.astype(np.int32), device="cuda"), stp,
                                 Gi=Gi, ldGi=m, Vi=Vi, ldVi=n)
    torch.cuda.synchronize()
    assert r >= 0
    host = lambda x, y: x.cpu().numpy().T + (1j * y.cpu().numpy().T if kind == "z" else 0)
    U, W = host(G, Gi), host(V, Vi)
    s = fS.cpu().numpy() * np.exp2(eS.cpu().numpy())
    assert np.max(np.linalg.norm(A @ W - U * s, axis=0)) <= 32 * EPS * sig.max()
    # the bounds of the mixed SVD's other tests: 32 n eps
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) <= 32 * n * EPS
    assert np.max(np.abs(W.conj().T @ W - np.eye(n))) <= 32 * n * EPS
