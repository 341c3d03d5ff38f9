"""The ways through the mixed SVD's FP64 phase (csrc/mixed.cu), each by a matrix that takes it, as the
trace (VJ_TRACE=1) tells: refinement by a rotation applied in parts, pairs of equal singular values
rotated one by one before a refinement, clusters that go to the plain sweeps. The bounds are those of
the mixed SVD's other tests (32 n eps)."""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


@pytest.mark.parametrize("kind", ["d", "z"])
@pytest.mark.parametrize("way", ["parts", "pairs", "sweeps"])
def test_way(kind, way, monkeypatch, capfd):
    import torch
    import vecjac_gb300 as vj
    from vecjac_gb300 import build
    build.build()
    m, n = 768, 512
    rng = np.random.default_rng(m + n)

    def ortho(r, c):
        x = rng.standard_normal((r, c)) + (1j * rng.standard_normal((r, c)) if kind == "z" else 0)
        return np.linalg.qr(x)[0]

    if way == "parts":  # (one FP32 stage leaves cosines of 1e-2 among five decades)
        sig = 10.0 ** (-5.0 * (np.arange(n) + rng.uniform(0.25, 0.75, n)) / n)
    elif way == "pairs":
        sig = 10.0 ** (-(np.arange(n) + 0.5) / n)
        sig[8::32] = sig[9::32]
    else:
        sig = np.repeat(np.logspace(0, -1, n // 8), 8)
    A = (ortho(m, n) * sig) @ ortho(n, n).conj().T
    js, stp = vj.pjs(4, n)
    dev = lambda x: torch.tensor(np.ascontiguousarray(x.T), dtype=torch.float64, device="cuda")
    G, V = dev(A.real), torch.empty((n, n), dtype=torch.float64, device="cuda")
    kw = dict(Gi=dev(A.imag), ldGi=m, Vi=torch.empty_like(V), ldVi=n) if kind == "z" else {}
    eS = torch.empty(n, dtype=torch.float64, device="cuda")
    fS = torch.empty_like(eS)
    monkeypatch.setenv("VJ_TRACE", "1")
    capfd.readouterr()
    r, _, _ = vj.vjsvd_mixed_dev(kind, m, n, G, m, V, n, eS, fS, torch.tensor(js.astype(np.int32), device="cuda"), stp,
                                 stages=1 if way == "parts" else 0, **kw)
    torch.cuda.synchronize()
    err = capfd.readouterr().err
    assert r >= 0
    # (norm of the generator, pairs left out of it) of every Gram matrix
    seen = [(float(a), int(b)) for a, b in re.findall(r"refinement \d+: .*\|K\| <= (\S+), (\d+) left out", err)]
    assert seen and ("FP64 sweep" in err) == (way == "sweeps"), err
    if way == "parts":
        assert any(0.06 < a <= 0.48 and b == 0 for a, b in seen), err
    if way == "pairs":
        assert seen[0][1] > 0 and seen[-1][1] == 0, err
    host = lambda x, y: x.cpu().numpy().T + (1j * y.cpu().numpy().T if kind == "z" else 0)
    U, W = host(G, kw.get("Gi")), host(V, kw.get("Vi"))
    s = fS.cpu().numpy() * np.exp2(eS.cpu().numpy())
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) <= 32 * n * EPS
    assert np.max(np.abs(W.conj().T @ W - np.eye(n))) <= 32 * n * EPS
    assert np.max(np.abs(A @ W - U * s)) <= 32 * n * EPS * np.max(np.abs(A)) * np.sqrt(n)
