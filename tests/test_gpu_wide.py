"""GPU tests of the wide-tile passes (csrc/fft_wide.cu), which the tuned table uses at 2^18 .. 2^24 and 2^28 .. 2^30.

They do the arithmetic of the per-thread-load passes (k_pass) on the same values, so a default plan
gives the bits of a plan with the same pass lengths and no bulk copies: both directions, with either
weight, for one transform (the last tiles leave blocks idle) and for batches whose tiles straddle the
persistent grid. Buffers at an odd complex offset take the plain passes of their own table: the bits of
that explicit split. An expired copy wait writes nothing and is reported.
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

# size -> (pass lengths of the default plan, pass lengths for unaligned buffers)
SPLITS = {17: ((8, 9), (10, 7)), 18: ((10, 8), (10, 8)), 19: ((11, 8), (8, 11)), 20: ((10, 10), (12, 8)),
          21: ((11, 10), (11, 10)), 22: ((11, 11), (8, 7, 7)), 23: ((12, 11), (8, 8, 7)), 24: ((12, 12), (8, 8, 8)),
          26: ((8, 8, 10), (8, 8, 10)), 27: ((8, 9, 10), (8, 9, 10)), 28: ((9, 9, 10), (10, 10, 8))}
CASES = [(17, 9), (18, 1), (18, 7), (19, 1), (19, 5), (20, 1), (20, 3), (21, 1), (21, 3), (22, 1), (22, 2), (23, 1),
         (24, 1), (24, 2), (26, 1), (27, 1), (28, 1)]


def transform(plan, src, dst, batch, inverse, pre=None, post=None):
    import torch
    if pre is None and post is None:
        (plan.dev_inverse if inverse else plan.dev_forward)(src.data_ptr(), dst.data_ptr(), batch)
    else:
        plan.dev_weighted(src.data_ptr(), dst.data_ptr(), batch, None if pre is None else pre.data_ptr(),
                          None if post is None else post.data_ptr(), inverse)
    torch.cuda.synchronize()
    plan.check()


@pytest.mark.parametrize("log2n,batch", CASES)
def test_default_plan_equals_plain_passes(ofb, log2n, batch):
    import torch
    n = 1 << log2n
    g = torch.Generator(device="cuda").manual_seed(log2n * 10 + batch)
    x = torch.randn(2 * n * batch, device="cuda", generator=g)
    default = ofb.Plan(n)
    assert default.passes() == SPLITS[log2n][0]
    plain = ofb.Plan(n, split=SPLITS[log2n][0], l2_keep=False)
    a, b = (torch.full((2 * n * batch,), 7.0, device="cuda") for _ in range(2))
    pre, post = (torch.randn(2 * n, device="cuda", generator=g) for _ in range(2)) if log2n <= 24 else (None, None)
    for inverse in (False, True):
        for w in ((None, None), (pre, None), (None, post)) if log2n <= 24 else ((None, None),):
            transform(default, x, a, batch, inverse, *w)
            transform(plain, x, b, batch, inverse, *w)
            assert torch.equal(a, b)


@pytest.mark.parametrize("log2n,batch", [(17, 3), (18, 2), (19, 1), (20, 2), (21, 1), (22, 1), (23, 1), (24, 1), (26, 1)])
def test_unaligned_buffers_take_the_plain_table(ofb, log2n, batch):
    import torch
    n = 1 << log2n
    g = torch.Generator(device="cuda").manual_seed(log2n)
    x = torch.randn(2 * n * batch + 2, device="cuda", generator=g)[2:]
    a, b = (torch.empty(2 * n * batch + 2, device="cuda")[2:] for _ in range(2))
    plain = ofb.Plan(n, split=SPLITS[log2n][1], l2_keep=False)
    for inverse in (False, True):
        transform(ofb.Plan(n), x, a, batch, inverse)
        transform(plain, x, b, batch, inverse)
        assert torch.equal(a, b)


@pytest.mark.parametrize("ln,lcols,lblocks,lbig", [(8, 17, 3, 28), (9, 16, 2, 0), (10, 4, 0, 0), (10, 10, 3, 24), (11, 5, 7, 20),
                                                   (11, 8, 1, 24), (12, 4, 4, 24), (12, 9, 0, 0), (13, 12, 5, 30), (16, 9, 4, 32),
                                                   (19, 6, 3, 30), (20, 4, 0, 0), (20, 5, 4, 40)])
def test_column_passes_same_bits_as_unaligned(ofb, ln, lcols, lblocks, lbig):
    """Aligned buffers (wide tiles where the layout allows them: blocks of at least a 16th of a pass's
    extent) against buffers at an odd complex offset, with every combination of the exchanges."""
    import torch
    values = 1 << (ln + lcols)
    col0 = 2 << lcols if lbig else 0
    c = ofb.Columns(1 << ln, 1 << lcols, 1 << lblocks, 1 << lbig if lbig else 0, col0 if lbig and 3 << (ln + lcols) <= 1 << lbig else 0)
    x = torch.randn(2 * values, device="cuda", generator=torch.Generator(device="cuda").manual_seed(ln * 32 + lcols))
    xs = torch.empty(2 * values + 2, device="cuda")[2:]
    xs.copy_(x)
    a, b = torch.empty_like(x), torch.empty(2 * values + 2, device="cuda")[2:]
    stream = torch.cuda.current_stream().cuda_stream
    for flags in (0, ofb.SWAP_IN, ofb.SWAP_OUT, ofb.SWAP_IN | ofb.SWAP_OUT):
        c.execute(x.data_ptr(), a.data_ptr(), flags, stream)
        c.execute(xs.data_ptr(), b.data_ptr(), flags, stream)
        torch.cuda.synchronize()
        c.check()
        assert torch.equal(a, b)


@pytest.mark.parametrize("log2n", [18, 20, 24])
def test_expired_wait_is_reported(ofb, log2n):
    import torch
    n = 1 << log2n
    x = torch.randn(2 * n, device="cuda")
    out = torch.full_like(x, 7.0)
    plan = ofb.Plan(n)
    ofb.lib().onefft_debug_expire_waits(1)
    try:
        plan.dev_forward(x.data_ptr(), out.data_ptr(), 1)
        torch.cuda.synchronize()
    finally:
        ofb.lib().onefft_debug_expire_waits(0)
    assert plan.status() != 0 and plan.status() == 0
    assert bool((out == 7.0).all())
    transform(plan, x, out, 1, False)
    want = torch.fft.fft(torch.view_as_complex(x.view(-1, 2)).to(torch.complex128))
    assert float((torch.view_as_complex(out.view(-1, 2)) - want).abs().norm() / want.abs().norm()) < 1e-6


@pytest.mark.parametrize("log2n,batch", [(18, 3), (19, 2), (20, 3), (21, 1), (22, 2), (23, 1), (24, 1), (28, 1), (29, 1), (30, 1)])
@pytest.mark.parametrize("shift", [0, 1])  # offset of the weights in complex values: 1 = not 16-byte aligned
def test_weights_equal_plain_passes(ofb, log2n, batch, shift):
    """Both weights at once, aligned and not, where weighted passes split between the wide tiles and
    k_pass_tma: the bits of the plain passes of the same split; nothing is written past the output."""
    import torch
    if shift and log2n > 28:
        pytest.skip("one case of the sizes that hold tens of gigabytes")
    n = 1 << log2n
    splits = {**SPLITS, 29: ((9, 10, 10),), 30: ((10, 10, 10),)}
    g = torch.Generator(device="cuda").manual_seed(log2n)
    x = torch.randn(2 * n * batch, device="cuda", generator=g)
    pre, post = (torch.randn(2 * n + 2 * shift, device="cuda", generator=g)[2 * shift:] for _ in range(2))
    a, b = (torch.full((2 * n * batch + 4,), 7.0, device="cuda") for _ in range(2))
    default, plain = ofb.Plan(n), ofb.Plan(n, split=splits[log2n][0], l2_keep=False)
    for inverse in (False, True):
        transform(default, x, a, batch, inverse, pre, post)
        transform(plain, x, b, batch, inverse, pre, post)
        assert torch.equal(a, b)
        assert bool((a[-4:] == 7.0).all())
