"""GPU tests of the pipelined one-kernel transforms of 2^13 and 2^14 (csrc/fft_long.cu).

They run the Stockham schedule of k_batched on the same values, so a 16-byte aligned input (bulk
copies, k_batched_long) and the same input at an odd complex offset (k_batched) give the same bits:
forward, inverse, with either weight or both, for batches around the persistent grid (one or two
transforms an SM). An expired copy wait leaves the output alone and is reported.
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("log2n", [13, 14])
@pytest.mark.parametrize("blocks,extra", [(0, 1), (0, 2), (1, -1), (1, 0), (1, 1), (2, -1), (2, 1), (3, 5)])
def test_same_bits_as_the_unaligned_path(ofb, log2n, blocks, extra):
    import torch
    n, batch = 1 << log2n, blocks * sms() + extra
    g = torch.Generator(device="cuda").manual_seed(log2n * 100 + batch)
    x = torch.randn(2 * n * batch, device="cuda", generator=g)
    shifted = torch.empty(2 * n * batch + 2, device="cuda")[2:]
    shifted.copy_(x)
    assert x.data_ptr() % 16 == 0 and shifted.data_ptr() % 16 == 8
    pre, post = (torch.randn(2 * n, device="cuda", generator=g) for _ in range(2))
    plan = ofb.Plan(n)
    for inverse in (False, True):
        for w0, w1 in ((None, None), (pre, None), (None, post), (pre, post)):
            got = []
            for src in (x, shifted):
                out = torch.full((2 * n * batch + 4,), 7.0, device="cuda")
                if w0 is None and w1 is None:
                    (plan.dev_inverse if inverse else plan.dev_forward)(src.data_ptr(), out.data_ptr(), batch)
                else:
                    plan.dev_weighted(src.data_ptr(), out.data_ptr(), batch, None if w0 is None else w0.data_ptr(),
                                      None if w1 is None else w1.data_ptr(), inverse)
                torch.cuda.synchronize()
                plan.check()
                got.append(out)
            assert torch.equal(got[0], got[1])
            assert bool((got[0][2 * n * batch:] == 7.0).all())


@pytest.mark.parametrize("log2n", [13, 14])
def test_expired_wait_is_reported(ofb, log2n):
    import torch
    n, batch = 1 << log2n, 3 * sms()
    x = torch.randn(2 * n * batch, device="cuda")
    out = torch.full_like(x, 7.0)
    plan = ofb.Plan(n)
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
    want = torch.fft.fft(torch.view_as_complex(x.view(-1, 2)).view(batch, n)[-1].to(torch.complex128))
    got = torch.view_as_complex(out.view(-1, 2)).view(batch, n)[-1]
    assert float((got - want).abs().norm() / want.abs().norm()) < 1e-6
