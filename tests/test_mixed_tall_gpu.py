"""The mixed SVD of tall matrices (csrc/mixed.cu), whose digits are cut and multiplied a panel of rows
at a time: more rows than one launch's grid has row blocks (65535 x 64), at a row count that is not a
multiple of the panels'. The bounds are those of the mixed SVD's other tests (32 n eps)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def run(kind, m, n, seed=1):
    import torch
    import vecjac_gb300 as vj
    from vecjac_gb300 import build
    build.build()
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dt = torch.complex128 if kind == "z" else torch.float64
    A = torch.randn((n, m), generator=g, device="cuda", dtype=dt).mT
    A *= 10.0 ** -torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    js, stp = vj.pjs(4, n)
    G = A.mT.real.clone() if kind == "z" else A.mT.clone()
    V = torch.empty((n, n), dtype=torch.float64, device="cuda")
    kw = dict(Gi=A.mT.imag.clone(), ldGi=m, Vi=torch.empty_like(V), ldVi=n) if kind == "z" else {}
    eS = torch.empty(n, dtype=torch.float64, device="cuda")
    fS = torch.empty_like(eS)
    r, _, _ = vj.vjsvd_mixed_dev(kind, m, n, G, m, V, n, eS, fS, torch.tensor(js.astype(np.int32), device="cuda"), stp, **kw)
    torch.cuda.synchronize()
    assert r >= 0, r
    s = fS * torch.exp2(eS)
    U, W = (torch.complex(G, kw["Gi"]).mT, torch.complex(V, kw["Vi"]).mT) if kind == "z" else (G.mT, V.mT)
    I = torch.eye(n, device="cuda", dtype=dt)
    assert torch.linalg.norm(U.mH @ U - I).item() <= 32 * n * EPS
    assert torch.linalg.norm(W.mH @ W - I).item() <= 32 * n * EPS
    assert torch.linalg.norm(A @ W - U * s).item() <= 32 * n * EPS * s.max().item()


@pytest.mark.parametrize("kind", ["d", "z"])
def test_more_rows_than_a_grid(kind):
    run(kind, 65535 * 64 + 72, 16)


@pytest.mark.parametrize("kind", ["d", "z"])
@pytest.mark.parametrize("m,n", [(1000, 16), (1032, 16), (2056, 96), (5000, 80), (33336, 64), (40008, 144)])
def test_split_k(kind, m, n):
    """K split over CTAs: from one slice to many, the last of them shorter than the others."""
    run(kind, m, n)
