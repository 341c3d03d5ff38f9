"""Captured batched SVDs beside others (csrc/host.cu, batch_plan_take): a replay on one stream while more
eager calls than there are slots go through another, a capture that is the first call of all on its
thread, and graphs that come and go, each with the results of a call by itself."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(seed, shapes, kind="s"):
    from vecjac_gb300 import batch as B
    rng = np.random.default_rng(seed)
    return B.Batch([rng.standard_normal(s).astype(np.float32 if kind == "s" else np.float64) for s in shapes], kind)


def outs(b):
    return [t.clone() for t in (b.info, b.eS, b.fS, b.G, b.V)]


def test_replay_beside_many_calls():
    import torch
    from vecjac_gb300 import batch as B
    from vecjac_gb300 import build
    build.build()
    big = make(1, [(192, 128)] * 120 + [(64, 32)] * 400)
    small = make(2, [(32, 32)] * 3)
    for b in (big, small):
        b.run(4, block=128)
    torch.cuda.synchronize()
    want, wants = outs(big), outs(small)
    g = B.capture(big, 4, block=128)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(30):
            g.replay()
    main = torch.cuda.Stream()
    for _ in range(1200):
        small.run(4, block=128, stream=main.cuda_stream, reset=False)
    torch.cuda.synchronize()
    for x, y in zip(want, outs(big)):
        assert torch.equal(x, y)
    small.run(4, block=128)
    torch.cuda.synchronize()
    for x, y in zip(wants, outs(small)):
        assert torch.equal(x, y)


def test_graphs_come_and_go():
    import torch
    from vecjac_gb300 import batch as B
    from vecjac_gb300 import build
    build.build()
    b = make(3, [(96, 64)] * 5 + [(32, 32)] * 50, "d")
    b.run(4, block=256)
    torch.cuda.synchronize()
    want = outs(b)
    kept = []
    for k in range(100):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(1 + k % 2):
                b.run(4, block=256, stream=torch.cuda.current_stream().cuda_stream)
        if k % 10 == 0:
            kept.append(g)
    for g in kept:
        b.info.fill_(-7)
        g.replay()
        torch.cuda.synchronize()
        for x, y in zip(want, outs(b)):
            assert torch.equal(x, y)


def test_threads():
    import torch
    from vecjac_gb300 import build
    build.build()
    bs = [make(10 + k, [(64, 64)] * 3 + [(32, 32)] * 20) for k in range(4)]
    want = []
    for b in bs:
        b.run(4, block=64)
        torch.cuda.synchronize()
        want.append(outs(b))
    streams = [torch.cuda.Stream() for _ in bs]
    torch.cuda.synchronize()

    def work(b, s):
        with torch.cuda.stream(s):
            for _ in range(100):
                b.run(4, block=64, stream=s.cuda_stream)

    ts = [threading.Thread(target=work, args=x) for x in zip(bs, streams)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    for b, w in zip(bs, want):
        for x, y in zip(w, outs(b)):
            assert torch.equal(x, y)
