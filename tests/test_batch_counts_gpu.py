"""Batches of equal matrices (csrc/batch.cu): as many as there are clusters, SMs or CTAs, and one more
or less, so that every launch (clusters, the CTAs that they leave room for, small matrices) has
some or none: bit for bit the results of one launch at another register bound, and a batch of one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,m,n", [("d", 128, 64), ("d", 32, 16), ("s", 128, 64), ("s", 304, 32)])
@pytest.mark.parametrize("count", [1, 37, 74, 75, 148, 149, 152, 153, 296, 297, 304, 305])
def test_equal_matrices(kind, m, n, count):
    import torch
    from vecjac_gb300 import batch as B
    from vecjac_gb300 import build
    build.build()
    rng = np.random.default_rng(count)
    dt = np.float64 if kind == "d" else np.float32
    A = rng.standard_normal((m, n)).astype(dt)
    one = B.Batch([A], kind)
    one.run(4, block=128)
    b = B.Batch([A] * (count // 2) + [-A] * (count - count // 2), kind)
    got = []
    for block, occ in ((256, 0), (128, 0), (256, 3)):
        for t in (b.info, b.eS, b.fS, b.G, b.V):
            t.fill_(-7)
        b.run(4, block=block, occupancy=occ)
        torch.cuda.synchronize()
        got.append([t.clone() for t in (b.info, b.eS, b.fS, b.G, b.V)])
    for g in got[1:]:
        for x, y in zip(got[0], g):
            assert torch.equal(x, y)
    # (a matrix and its negative: the same V, eS and fS)
    for x, y in zip((b.info, b.eS, b.fS, b.V), (one.info, one.eS, one.fS, one.V)):
        assert torch.equal(x.view(count, -1), y.view(1, -1).expand(count, -1))
