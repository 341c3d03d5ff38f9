"""The launch configurations that the batched SVD's callers get (vecjac_gb300/batch.py, autodiff.py):
svd_batch times the library's default, too, and what is kept from the timing is kept for batches with
about as many matrices per SM only. Sizes that no other test tunes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["d", "s"])
def test_default_is_among_the_candidates(kind, monkeypatch):
    from vecjac_gb300 import batch as B
    from vecjac_gb300 import build
    build.build()
    rng = np.random.default_rng(1)
    mats = [rng.standard_normal((64, 32)).astype(np.float64 if kind == "d" else np.float32) for _ in range(5)]
    seen = set()
    run = B.Batch.run
    monkeypatch.setattr(B, "_TUNED", {})
    monkeypatch.setattr(B.Batch, "run", lambda self, *a, **k: (seen.add(k.get("occupancy", 0)), run(self, *a, **k))[1])
    assert all(r[0] > 0 for r in B.svd_batch(mats, kind))
    assert {0, 2, 3, 4} <= seen


def test_kept_by_count(monkeypatch):
    import torch
    from vecjac_gb300 import autodiff as AD
    from vecjac_gb300 import batch as B
    from vecjac_gb300 import build
    build.build()
    monkeypatch.setattr(B, "_TUNED", {})
    monkeypatch.setattr(AD, "_BLOCK", {})
    rng = np.random.default_rng(2)
    for count in (4, 5, 2000):
        A = rng.standard_normal((count, 32, 32)).astype(np.float32)
        B.autotune(B.Batch(list(A), "s"), 4)
        AD.svd_batch_dev(torch.from_numpy(A).cuda())
    assert len(B._TUNED) == 2 and len(AD._BLOCK) == 2
