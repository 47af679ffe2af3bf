"""GPU tests of the one-trip cluster kernel of 2^15 (csrc/fft_cluster.cu), which default plans use for
aligned batches of at least 360 transforms.

It does the two passes' arithmetic on the same values, so a default plan gives the bits of an explicit
(8, 7) plan: below the line, at it, one above, and for batches that leave clusters idle in the last
round; both directions, either weight; nothing is written past the batch. An expired copy wait makes
the whole cluster leave with nothing written, and is reported.
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

N = 1 << 15


@pytest.mark.parametrize("batch", [359, 360, 361, 433, 719, 1500])
def test_equals_two_passes(ofb, batch):
    import torch
    g = torch.Generator(device="cuda").manual_seed(batch)
    x = torch.randn(2 * N * batch, device="cuda", generator=g)
    pre, post = (torch.randn(2 * N, device="cuda", generator=g) for _ in range(2))
    default, passes = ofb.Plan(N), ofb.Plan(N, split=(8, 7), l2_keep=False)
    for inverse in (False, True):
        for w0, w1 in ((None, None), (pre, None), (None, post), (pre, post)):
            got = []
            for plan in (default, passes):
                out = torch.full((2 * N * batch + 4,), 7.0, device="cuda")
                if w0 is None and w1 is None:
                    (plan.dev_inverse if inverse else plan.dev_forward)(x.data_ptr(), out.data_ptr(), batch)
                else:
                    plan.dev_weighted(x.data_ptr(), out.data_ptr(), batch, None if w0 is None else w0.data_ptr(),
                                      None if w1 is None else w1.data_ptr(), inverse)
                torch.cuda.synchronize()
                plan.check()
                got.append(out)
            assert torch.equal(got[0], got[1])
            assert bool((got[0][2 * N * batch:] == 7.0).all())


def test_expired_wait_is_reported(ofb):
    import torch
    batch = 400
    x = torch.randn(2 * N * batch, device="cuda")
    out = torch.full_like(x, 7.0)
    plan = ofb.Plan(N)
    ofb.lib().onefft_debug_expire_waits(1)
    try:
        plan.dev_forward(x.data_ptr(), out.data_ptr(), batch)
        torch.cuda.synchronize()
    finally:
        ofb.lib().onefft_debug_expire_waits(0)
    assert plan.status() != 0 and plan.status() == 0
    assert bool((out == 7.0).all())
    plan.dev_forward(x.data_ptr(), out.data_ptr(), batch)
    torch.cuda.synchronize()
    plan.check()
    want = torch.fft.fft(torch.view_as_complex(x.view(-1, 2)).view(batch, N)[-1].to(torch.complex128))
    got = torch.view_as_complex(out.view(-1, 2)).view(batch, N)[-1]
    assert float((got - want).abs().norm() / want.abs().norm()) < 1e-6


def test_many_rounds_forward(ofb):
    """Forward without weights, where nothing but the cluster's barriers stands between a block's reads
    of its landing buffer and the peer's stores into it: about 70 transforms a cluster, several launches
    in a row, every one with the passes' bits."""
    import torch
    batch = 5000
    x = torch.randn(2 * N * batch, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    out, want = torch.empty_like(x), torch.empty_like(x)
    default, passes = ofb.Plan(N), ofb.Plan(N, split=(8, 7), l2_keep=False)
    passes.dev_forward(x.data_ptr(), want.data_ptr(), batch)
    for _ in range(8):
        out.fill_(7.0)
        default.dev_forward(x.data_ptr(), out.data_ptr(), batch)
        torch.cuda.synchronize()
        default.check()
        assert torch.equal(out, want)


def test_more_transforms_than_a_launch_takes(ofb):
    """65538 transforms (17 GB a buffer): the ones around the slice's end have the bits of a call of their own."""
    import torch
    batch = 65538
    x = torch.empty(2 * N * batch, device="cuda").normal_(generator=torch.Generator(device="cuda").manual_seed(3))
    out = torch.full_like(x, 7.0)
    plan = ofb.Plan(N)
    plan.dev_forward(x.data_ptr(), out.data_ptr(), batch)
    for first in (0, batch - 6):
        want = torch.empty(2 * N * 6, device="cuda")
        plan.dev_forward(x.data_ptr() + 8 * N * first, want.data_ptr(), 6)
        torch.cuda.synchronize()
        plan.check()
        assert torch.equal(out[2 * N * first:2 * N * (first + 6)], want)
