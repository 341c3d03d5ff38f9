"""The plain SVD where the columns of a CTA's pairs do not fit in shared memory (csrc/jsvd.cu,
step_launch): FP32 with one pair per CTA, staged and read from L2, FP64 with one, two and four pairs
read from L2, and the sizes on both sides of each limit. The first eight steps of a sweep, bit for bit
the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# dynamic shared memory of P pairs: 8 m P bytes (s), 16 (c), 16 (d), 32 (z) beside the products' buffers
@pytest.mark.parametrize("kind,m,n", [
    ("s", 4096, 608 + 32), ("s", 4112, 608 + 32),     # four pairs staged; one pair staged
    ("s", 22528, 32), ("s", 22544, 32),               # one pair staged; from L2
    ("c", 4096, 320), ("c", 4112, 320),               # two pairs staged; one pair staged
    ("c", 10240, 32), ("c", 10256, 32),               # one pair staged; from L2
    ("d", 12032, 16), ("d", 12040, 16), ("d", 5888, 320), ("d", 5896, 320), ("d", 2824, 640),
    ("z", 5888, 16), ("z", 5896, 16), ("z", 2816, 320), ("z", 2824, 320), ("z", 1288, 624)])
def test_columns_beyond_shared_memory(kind, m, n):
    import vecjac_gb300 as vj
    from vecjac_gb300 import build
    build.build()
    O.build()
    rst = O.Restatement()
    rng = np.random.default_rng(m + n)
    dt = np.float64 if kind in "dz" else np.float32
    G = (rng.standard_normal((m, n)) * 10.0 ** -rng.uniform(0, 2, n)).astype(dt)
    kw = dict(Gi=rng.standard_normal((m, n)).astype(dt)) if kind in "zc" else {}
    js, stp = rst.pjs(4, n)
    stp = min(stp, 8)
    a, b = vj.vjsvd(kind, G, js, stp, 1, **kw), rst.vjsvd(kind, G, js, stp, 1, **kw)
    assert a[0] == b[0]
    for x, y in zip(a[1:], b[1:]):
        assert np.array_equal(np.ascontiguousarray(x).view(np.uint8), np.ascontiguousarray(y).view(np.uint8))
