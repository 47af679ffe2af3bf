"""GPU test of the dependent launches: a kernel may start while its predecessor in the stream still
runs, so a chain of calls that each read what the one before wrote (in two buffers in turn, the weights
of the next call included) and that nothing waits between must give the bits of the same chain with a
synchronisation after every call. Sizes: both sides of the 1184-block line of the early release, one,
two and three kernels a call, tiny and batched kernels, TMA and plain passes (8-byte aligned buffers).
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2n,batch", [(3, 1), (3, 700001), (6, 100003), (9, 37), (10, 1), (12, 1183), (12, 1185),
                                         (14, 3), (15, 1), (16, 9), (17, 5), (18, 3), (20, 1), (20, 5), (22, 1), (24, 1)])
@pytest.mark.parametrize("shift", [0, 1])  # offset of every buffer in complex values: 1 = not 16-byte aligned
def test_unsynchronised_chain_same_bits(ofb, log2n, batch, shift):
    import torch
    n = 1 << log2n
    values = n * batch
    g = torch.Generator(device="cuda").manual_seed(1000 * log2n + batch)
    x = torch.randn(2 * (values + 1), device="cuda", generator=g) / n ** 0.5
    plan = ofb.Plan(n)
    stream = torch.cuda.current_stream().cuda_stream
    out = []
    for sync in (True, False):
        a, b = x.clone(), torch.zeros_like(x)
        pa, pb = a.data_ptr() + 8 * shift, b.data_ptr() + 8 * shift
        if not sync:
            torch.cuda.synchronize()
        for i in range(6):
            for call in (lambda: plan.dev_forward(pa, pb, batch, stream),
                         lambda: plan.dev_inverse(pb, pa, batch, stream),
                         # one transform, windowed by what the call before wrote last
                         lambda: plan.dev_weighted(pb, pb + 8 * n, 1, pa + 8 * (values - n), None, False, stream)
                         if batch > 2 else None):
                call()
                if sync:
                    torch.cuda.synchronize()
            if log2n > 0:  # keep the magnitudes: the pair multiplies by n
                a.mul_(1.0 / n)
        torch.cuda.synchronize()
        plan.check()
        out.append((a, b))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert bool(torch.isfinite(out[0][0]).all())


@pytest.mark.parametrize("count,lo,hi", [(1, 4, 4), (200, 0, 4), (300, 3, 8), (700, 4, 9), (40, 13, 16), (3000, 4, 12)])
def test_uneven_launches_back_to_back(ofb, count, lo, hi):
    """The last block of an uneven launch zeroes the batch's counters: launches that nothing waits
    between, each reading what the one before wrote (graph replays below 2^16 values, dependent launches
    beyond), give the bits of the same launches with a synchronisation after each."""
    import numpy as np
    import torch
    r = np.random.RandomState(count)
    m = r.randint(lo, hi + 1, count)
    off = np.concatenate([[0], np.cumsum(1 << m)[:-1]])
    batch = ofb.UnevenBatch(m, r.randint(0, 2, count), off)
    x = torch.randn(2 * batch.span, device="cuda", generator=torch.Generator(device="cuda").manual_seed(count))
    stream = torch.cuda.current_stream().cuda_stream
    out = []
    for sync in (True, False):
        a, b = x.clone(), torch.zeros_like(x)
        torch.cuda.synchronize()
        for i in range(4):
            batch.execute(a.data_ptr(), b.data_ptr(), stream)
            if sync:
                torch.cuda.synchronize()
            batch.execute(b.data_ptr(), a.data_ptr(), stream)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        assert batch.status() == 0
        out.append((a, b))
    # 2^16-point transforms grow by up to 2^16 per call pair: compare the bits, whatever they are
    assert torch.equal(out[0][0].view(torch.int32), out[1][0].view(torch.int32))
    assert torch.equal(out[0][1].view(torch.int32), out[1][1].view(torch.int32))


def test_stream_capture_replays(ofb):
    """Two chained calls of each kind recorded in one graph (dependent launches become programmatic
    edges) give, replayed, the bits of the same calls outside it."""
    import torch
    calls = []
    for log2n, batch in ((6, 300), (12, 1200), (13, 400), (14, 5), (15, 2), (15, 400), (18, 3), (20, 1), (24, 1)):
        n = 1 << log2n
        plan = ofb.Plan(n)
        calls.append((2 * n * batch, lambda a, b, s, p=plan, k=batch: p.dev_forward(a, b, k, s), plan))
    c = ofb.Columns(1 << 13, 1 << 8)
    calls.append((2 << 21, lambda a, b, s, c=c: c.execute(a, b, 0, s), c))
    for floats, call, _keep in calls:
        x = torch.randn(floats, device="cuda")
        y, z, y2, z2 = (torch.zeros_like(x) for _ in range(4))
        s = torch.cuda.Stream()
        torch.cuda.synchronize()
        call(x.data_ptr(), y.data_ptr(), s.cuda_stream)
        call(y.data_ptr(), z.data_ptr(), s.cuda_stream)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            call(x.data_ptr(), y2.data_ptr(), s.cuda_stream)
            call(y2.data_ptr(), z2.data_ptr(), s.cuda_stream)
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, y2) and torch.equal(z, z2)
        del graph
