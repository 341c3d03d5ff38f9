"""The batched SVD's clusters (csrc/batch.cu, csrc/batch_core.cuh): matrices large enough for a
team of CTAs beside matrices for one, at the edges of the groups of pairs that a warp and a
CTA take, bit for bit what the oracle gives for each."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["d", "s"])
@pytest.mark.parametrize("block", [64, 256])
def test_large_and_small_matrices(kind, block):
    import torch
    from vecjac_gb300 import batch as B
    from vecjac_gb300 import build
    build.build()
    O.build()
    rst = O.Restatement()
    rng = np.random.default_rng(17)
    L = 8 if kind == "d" else 16
    dt = np.float64 if kind == "d" else np.float32
    # (m, n) in multiples of the reference's rules: one group of pairs, a CTA's worth and one
    # more, several groups per warp
    shapes = [(2 * L, 2 * L), (96, 64), (112, 96), (160, 160), (5 * L, 2 * L), (176, 128), (4 * L, 4 * L), (200, 96)]
    mats = [(rng.standard_normal(s) * 10.0 ** rng.uniform(-2, 0, s[1])).astype(dt) for s in shapes]
    mats[3][:, 7] = 0  # a zero column in a large matrix
    bad = np.ones((192, 192), dt)
    bad[3, 100] = np.nan  # a large matrix that is not finite: -80
    mats.append(bad)
    b = B.Batch(mats, kind)
    b.run(4, block=block)
    torch.cuda.synchronize()
    for A, r in zip(mats, b.results()):
        m2, n2 = B.padded_shape(A.shape[0], A.shape[1], kind)
        P = np.zeros((m2, n2), dt)
        P[:A.shape[0], :A.shape[1]] = A
        js, stp = rst.pjs(4, n2)
        o = rst.vjsvd(kind, P, js, stp)
        assert r[0] == o[0], (A.shape, r[0], o[0])
        if o[0] >= 0:
            for x, y in zip(r[1:], o[1:]):
                assert np.array_equal(np.ascontiguousarray(x).view(np.uint8), np.ascontiguousarray(y).view(np.uint8)), A.shape
