"""GPU tests of calls that nothing waits between and that read, and overwrite, what the calls before
them wrote: they give the bits of the same calls with a synchronisation after each.

A grid of 1184 blocks or more lets the stream's next kernel start early, so the producers here have at
least that many blocks and no other kernel stands between the calls:
  - pairs x -> y -> x, whose third call reads again what the first one read and the second overwrote,
    at grids that are all resident and at larger ones;
  - a ring of adjacent slices of one buffer whose ends share 32-byte sectors;
  - every other kind of kernel as the consumer of a large one-kernel batch or a two-pass batch, writing
    over the producer's input.
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def bits(torch, fill, calls):
    """The buffers of fill() after `calls`, with and without a synchronisation after each call."""
    out = []
    for sync in (True, False):
        state = fill()
        torch.cuda.synchronize()
        for call in calls:
            call(*state)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        out.append(state)
    for a, b in zip(*out):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


def normal(torch, values, seed):
    return torch.randn(2 * values, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


# blocks of 2048 values (2^0 .. 2^9, 2^11), 4096 (2^10, 2^12), passes of 2^16 in 32 tiles a transform
@pytest.mark.parametrize("log2n,batch", [(0, 2048 * 1184), (3, 256 * 1184), (3, 256 * 2368), (4, 128 * 1500), (6, 32 * 1184),
                                         (6, 32 * 2000), (6, 32 * 9000), (9, 4 * 1184), (9, 4 * 2368), (11, 1184),
                                         (12, 1184), (12, 2368), (12, 4096), (16, 37), (16, 74), (16, 256)])
@pytest.mark.parametrize("shift", [0, 1])  # offset of every buffer in complex values: 1 = not 16-byte aligned
def test_there_and_back(ofb, log2n, batch, shift):
    import torch
    values = batch << log2n
    plan = ofb.Plan(1 << log2n)
    s = torch.cuda.current_stream().cuda_stream
    x = normal(torch, values + 1, log2n)
    calls = []
    for i in range(6):
        calls.append(lambda a, b: plan.dev_forward(a.data_ptr() + 8 * shift, b.data_ptr() + 8 * shift, batch, s))
        calls.append(lambda a, b: plan.dev_inverse(b.data_ptr() + 8 * shift, a.data_ptr() + 8 * shift, batch, s))
    bits(torch, lambda: (x.clone(), torch.zeros_like(x)), calls)
    plan.check()


@pytest.mark.parametrize("log2n,batch", [(3, 256 * 1184 + 1), (6, 32 * 1500 + 1), (9, 4 * 2000 + 1), (12, 1300), (13, 160),
                                         (16, 40), (18, 3), (20, 1)])
@pytest.mark.parametrize("shift", [1, 2, 3])  # where the slices' ends lie in a 32-byte sector (complex values)
def test_adjacent_slices(ofb, log2n, batch, shift):
    """a -> b -> c -> a with a, b, c back to back; then b -> c windowed by the first transform of a, which
    the call before wrote and which ends next to other values."""
    import torch
    n, values = 1 << log2n, batch << log2n
    plan = ofb.Plan(n)
    s = torch.cuda.current_stream().cuda_stream
    x = normal(torch, 3 * values + shift, log2n) / n ** 1.5  # the last call's result is about n ** 2

    def ring(i, j, inverse=False, weight=False):
        def call(arena):
            src, dst = (arena.data_ptr() + 8 * (shift + k * values) for k in (i, j))
            if weight:
                plan.dev_weighted(src, dst, batch, arena.data_ptr() + 8 * shift, arena.data_ptr() + 8 * (shift + values - n),
                                  inverse, s)
            else:
                (plan.dev_inverse if inverse else plan.dev_forward)(src, dst, batch, s)
        return call
    calls = [ring(0, 1), ring(1, 2, True), ring(2, 0), ring(1, 2, weight=True), ring(2, 1, True), ring(1, 0),
             ring(1, 2, True, weight=True), ring(2, 0, True)]
    for _ in range(3):
        bits(torch, lambda: (x.clone(),), calls)
    plan.check()


VALUES = 1 << 24
PRODUCERS = [(3, VALUES >> 3), (6, VALUES >> 6), (12, VALUES >> 12), (16, VALUES >> 16)]
CONSUMERS = [(13, None), (14, None), (15, None), (16, None), (18, None), (20, None), (22, None), (24, None), (12, "columns"),
             (20, "columns"), (16, "uneven"), (12, "uneven")]


@pytest.mark.parametrize("producer", PRODUCERS)
@pytest.mark.parametrize("log2n,kind", CONSUMERS)
def test_consumers_of_large_grids(ofb, producer, log2n, kind):
    import numpy as np
    import torch
    s = torch.cuda.current_stream().cuda_stream
    first = ofb.Plan(1 << producer[0])
    x = normal(torch, VALUES, log2n) / 2.0 ** (producer[0] / 2)
    if kind == "columns":
        second = ofb.Columns(1 << log2n, VALUES >> log2n, 4, VALUES)
        consume = [lambda a, b: second.execute(b.data_ptr(), a.data_ptr(), 0, s)]
    elif kind == "uneven":
        r = np.random.RandomState(log2n)
        m = r.randint(4, log2n + 1, 200 << (16 - log2n))
        off = np.concatenate([[0], np.cumsum(1 << m)[:-1]])
        second = ofb.UnevenBatch(m, r.randint(0, 2, len(m)), off)
        assert 1 << 16 < second.span <= VALUES
        consume = [lambda a, b: second.execute(b.data_ptr(), a.data_ptr(), s)]
    else:
        second = ofb.Plan(1 << log2n)
        batch = VALUES >> log2n
        consume = [lambda a, b: second.dev_forward(b.data_ptr(), a.data_ptr(), batch, s)]
        if batch > 1:  # the weights are what the producer wrote, too
            consume.append(lambda a, b: second.dev_weighted(b.data_ptr(), a.data_ptr(), batch,
                                                            b.data_ptr() + 8 * (VALUES - (1 << log2n)), None, True, s))
    calls = []
    for i in range(3):
        calls.append(lambda a, b: first.dev_forward(a.data_ptr(), b.data_ptr(), producer[1], s))
        calls.append(consume[i % len(consume)])
    bits(torch, lambda: (x.clone(), torch.zeros_like(x)), calls)
    first.check()
    assert second.status() == 0


@pytest.mark.parametrize("log2n", [7, 8])
@pytest.mark.parametrize("extra", [-1, 0, 5])  # transforms beyond the 6.3 million values from which on L1 serves
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_large_batches_through_l1(ofb, log2n, extra, shift):
    """2^7 and 2^8 at the line of the ordinary launch with cached loads (csrc/fft_kernels.cu): the bits of
    two calls below it, nothing written past the batch, and chains as above."""
    import torch
    n, batch = 1 << log2n, ((3 << 21) >> log2n) + extra
    values = batch << log2n
    plan = ofb.Plan(n)
    s = torch.cuda.current_stream().cuda_stream
    x = normal(torch, values + shift, log2n)
    a, b = (torch.full((2 * (values + shift + 4),), 7.0, device="cuda") for _ in range(2))
    px, pa, pb = (t.data_ptr() + 8 * shift for t in (x, a, b))
    half = batch // 2
    for call in (plan.dev_forward, plan.dev_inverse):
        call(px, pa, batch, s)
        call(px, pb, half, s)
        call(px + 8 * n * half, pb + 8 * n * half, batch - half, s)
        torch.cuda.synchronize()
        assert torch.equal(a, b)
        assert bool((a[2 * (values + shift):] == 7.0).all())
    calls = []
    for _ in range(4):
        calls.append(lambda u, v: plan.dev_forward(u.data_ptr() + 8 * shift, v.data_ptr() + 8 * shift, batch, s))
        calls.append(lambda u, v: plan.dev_inverse(v.data_ptr() + 8 * shift, u.data_ptr() + 8 * shift, half, s))
    bits(torch, lambda: (x.clone(), torch.zeros_like(x)), calls)
    plan.check()
