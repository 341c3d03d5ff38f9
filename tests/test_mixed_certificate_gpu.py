"""The mixed SVD's certificate from the last Gram matrix (csrc/mixed.cu, csrc/gram_bound.cuh)
against the check that computes every cosine: where the certificate lets the finishing sweep go, the
same columns (U scaled by their norms, V preset) pass the all-pairs check of preset = 2, which
decides pairs near the tolerance by the reference's own dot products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,m,n", [("d", 1032, 512), ("z", 1032, 512), ("d", 4104, 128), ("z", 2056, 96)])
def test_agrees_with_the_cosines(kind, m, n, monkeypatch, capfd):
    import torch
    import vecjac_gb300 as vj
    from vecjac_gb300 import build
    build.build()
    rng = np.random.default_rng(m + n)
    A = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if kind == "z" else 0)
    A = A * 10.0 ** -rng.uniform(0, 2, n)
    js, stp = vj.pjs(4, n)
    js = torch.tensor(js.astype(np.int32), device="cuda")
    dev = lambda x: torch.tensor(np.ascontiguousarray(x.T), dtype=torch.float64, device="cuda")
    G, V = dev(A.real), torch.empty((n, n), dtype=torch.float64, device="cuda")
    kw = dict(Gi=dev(A.imag), ldGi=m, Vi=torch.empty_like(V), ldVi=n) if kind == "z" else {}
    eS = torch.empty(n, dtype=torch.float64, device="cuda")
    fS = torch.empty_like(eS)
    monkeypatch.setenv("VJ_TRACE", "1")
    r, _, _ = vj.vjsvd_mixed_dev(kind, m, n, G, m, V, n, eS, fS, js, stp, **kw)
    torch.cuda.synchronize()
    assert "certified 1" in capfd.readouterr().err
    assert r == 0
    s = (fS * torch.exp2(eS))[:, None]
    for x in [G] + ([kw["Gi"]] if kind == "z" else []):
        x.mul_(s)
    assert vj.vjsvd_dev(kind, m, n, G, m, V, n, eS, fS, js, stp, preset=2, **kw) == 0
