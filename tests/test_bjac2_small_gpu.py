"""Small ?bjac2_ calls on pageable arrays.

Up to 512 KiB of output arrays the kernel writes into the library's page-locked memory and the
calling thread copies on; above that the copy engine does. Both must give the device entry's
results bit for bit, touch nothing beyond the arrays' ends, and take outputs at any element.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 512 << 10


@pytest.fixture(scope="module")
def vj():
    import vecjac_gb300
    from vecjac_gb300 import build
    build.build()
    return vecjac_gb300


@pytest.mark.parametrize("kind", ["d", "z", "s", "c"])
@pytest.mark.parametrize("size", ["one", "odd", "last", "past"])
def test_small_outputs_match_device_entry(vj, kind, size):
    import torch
    from vecjac_gb300 import workloads as W
    dt = np.float64 if kind in "dz" else np.float32
    lanes = 8 if kind in "dz" else 16
    nout = 5 if kind in "zc" else 4
    last = LIMIT // (nout * dt().itemsize) // lanes * lanes
    n = {"one": lanes, "odd": 37 * lanes, "last": last, "past": last + lanes}[size]
    ins = W.pairs2x2(kind, n, seed=17)
    guard = 3
    names = ["c", "at", "sat", "l1", "l2"] if kind in "zc" else ["c", "at", "l1", "l2"]
    full = {k: np.full(n + 2 * guard, 7, dt) for k in names}
    full["p"] = np.full(n // lanes + 2 * guard, 7, np.uint32)
    got = vj.bjac2(kind, -n, *ins, **{k: v[guard:-guard] for k, v in full.items()})
    assert got[0] == 1
    dins = [torch.from_numpy(np.array(x)).cuda() for x in ins]
    douts = {k: torch.zeros(n, dtype=dins[0].dtype, device="cuda") for k in names}
    dp = torch.zeros(n // lanes, dtype=torch.int32, device="cuda")
    assert vj.bjac2_dev(kind, -n, dins[0], dins[1], dins[2], dins[3] if kind in "zc" else None, douts["c"], douts["at"],
                        douts.get("sat"), douts["l1"], douts["l2"], dp) == 1
    torch.cuda.synchronize()
    for k in names + ["p"]:
        want = (dp if k == "p" else douts[k]).cpu().numpy()
        assert np.array_equal(full[k][guard:-guard].view(np.uint8), want.view(np.uint8)), k
        assert (full[k][:guard] == 7).all() and (full[k][-guard:] == 7).all(), k
