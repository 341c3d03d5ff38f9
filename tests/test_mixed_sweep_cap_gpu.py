"""swp caps every phase of the mixed SVD (include/vecjac_gb300.h): its FP64 phase before the finishing
sweeps makes at most swp refinements and sweeps, also where the FP32 stages left only those to do (a
matrix close to its own U Sigma)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["d", "z"])
@pytest.mark.parametrize("swp", [0, 1, 2, 999])
def test_cap(kind, swp):
    import torch
    import vecjac_gb300 as vj
    from vecjac_gb300 import build
    build.build()
    m, n = 192, 96
    rng = np.random.default_rng(7)

    def gauss(r, c):
        return rng.standard_normal((r, c)) + (1j * rng.standard_normal((r, c)) if kind == "z" else 0)

    V0 = np.linalg.qr(np.eye(n) + 1e-4 * gauss(n, n))[0]
    A = (np.linalg.qr(gauss(m, n))[0] * np.logspace(0, -2, n)) @ V0.conj().T
    js, stp = vj.pjs(4, n)
    dev = lambda x: torch.tensor(np.ascontiguousarray(x.T), dtype=torch.float64, device="cuda")
    G, V = dev(A.real), torch.empty((n, n), dtype=torch.float64, device="cuda")
    kw = dict(Gi=dev(A.imag), ldGi=m, Vi=torch.empty_like(V), ldVi=n) if kind == "z" else {}
    eS = torch.empty(n, dtype=torch.float64, device="cuda")
    r, r32, r64 = vj.vjsvd_mixed_dev(kind, m, n, G, m, V, n, eS, torch.empty_like(eS),
                                     torch.tensor(js.astype(np.int32), device="cuda"), stp, swp, **kw)
    torch.cuda.synchronize()
    assert 0 <= r <= swp and r32 <= 2 * swp and r64 <= swp
    if swp == 999:
        assert r64 >= 2  # (the cap of 1 has something to cut off)
