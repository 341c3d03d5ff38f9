"""The batched SVD's two launches (csrc/batch.cu) and the FP32 rotations in registers
(csrc/batch_core.cuh, rot_sum_f32): columns at the edges of the register blocks and beyond,
columns whose scale factors are not normal numbers, and batches in which every launch has
matrices, in any order: bit for bit the oracle's results and those of one launch."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint8)


@pytest.mark.parametrize("kind", ["d", "s"])
@pytest.mark.parametrize("m", [32, 112, 128, 144, 240, 256, 272])
def test_column_lengths(kind, m):
    import torch
    from vecjac_gb300 import batch as B
    from vecjac_gb300 import build
    build.build()
    O.build()
    rst = O.Restatement()
    rng = np.random.default_rng(m)
    dt = np.float64 if kind == "d" else np.float32
    far = (900, 1060) if kind == "d" else (100, 140)
    mats = [rng.standard_normal((m, 32)) * 10.0 ** rng.uniform(-2, 0, 32) for _ in range(3)]
    mats[1][:, 3] *= 2.0 ** far[0]
    mats[1][:, 9] *= 2.0 ** -far[1]  # subnormal, also after the scaling of the whole matrix
    mats[2][:, 5] = 0
    mats = [A.astype(dt) for A in mats]
    b = B.Batch(mats, kind)
    b.run(4, block=256)
    torch.cuda.synchronize()
    js, stp = rst.pjs(4, 32)
    for A, r in zip(mats, b.results()):
        o = rst.vjsvd(kind, A, js, stp)
        assert r[0] == o[0]
        if o[0] >= 0:
            for x, y in zip(r[1:], o[1:]):
                assert np.array_equal(bits(x), bits(y))


@pytest.mark.parametrize("kind", ["d", "s"])
@pytest.mark.parametrize("order", ["down", "up"])
def test_parts_agree(kind, order):
    import torch
    from vecjac_gb300 import batch as B
    from vecjac_gb300 import build
    build.build()
    rng = np.random.default_rng(3)
    dt = np.float64 if kind == "d" else np.float32
    shapes = [(192, 160)] * 2 + [(96, 64)] * 40 + [(32, 32)] * 900
    shapes = shapes if order == "down" else shapes[::-1]
    mats = [rng.standard_normal(s).astype(dt) for s in shapes]
    b = B.Batch(mats, kind)
    b.run(4, block=256)
    torch.cuda.synchronize()
    got = [t.clone() for t in (b.info, b.eS, b.fS, b.G, b.V)]
    b.run(4, block=256, occupancy=3)
    torch.cuda.synchronize()
    for x, y in zip(got, (b.info, b.eS, b.fS, b.G, b.V)):
        assert torch.equal(x, y)


def test_parts_in_a_graph():
    import torch
    from vecjac_gb300 import batch as B
    from vecjac_gb300 import build
    build.build()
    rng = np.random.default_rng(4)
    mats = [rng.standard_normal(s).astype(np.float32) for s in [(128, 96)] * 3 + [(32, 32)] * 500]
    b = B.Batch(mats, "s")
    b.run(4, block=128)
    torch.cuda.synchronize()
    want = [t.clone() for t in (b.info, b.eS, b.fS, b.G, b.V)]
    g = B.capture(b, 4, block=128)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    for x, y in zip(want, (b.info, b.eS, b.fS, b.G, b.V)):
        assert torch.equal(x, y)
