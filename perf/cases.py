"""Workloads of onefft_b200 as its users run them, each through the public entry points.

A case is a dict of plain values; ``kind`` says which call it makes:

  transform  Plan.dev_forward / dev_inverse on a batch of equal transforms ("both": forward, then
             inverse of the spectrum)
  filter     Plan.dev_weighted: forward with the filter's response applied to the spectrum as it is
             written, then dev_inverse (circular convolution of a batch)
  uneven     UnevenBatch.execute: many transforms of different sizes, half of them inverse
  loss       torch_fft.weighted_power_loss_fused and its backward (a differentiable layer's step)
  autograd   torch_fft.fft and its backward with a given upstream gradient
  columns    Columns.execute twice: one rank's two local steps of a distributed four-step transform

Buffers, plans, batch objects and filters are made once (``prepare``), as a program that calls the
library in a loop keeps them; ``run`` is one pass. Every transform is unnormalised.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import onefft_b200 as ofb
from onefft_b200 import torch_fft

MAX_LOG2 = 27         # largest transform and largest batch, in complex values (1 GiB)
COLUMNS_MAX_LOG2 = 27


def listed():
    return [
        # one short transform there and back: what a latency-bound caller pays per call pair
        {"name": "pair_1024", "kind": "transform", "log2n": 10, "batch": 1, "direction": "both"},
        # a ragged batch of very short transforms (OFDM-like symbols), synthesis direction
        {"name": "batch_64", "kind": "transform", "log2n": 6, "batch": 100003, "direction": "inverse"},
        # a batch of frames filtered in the frequency domain; the count fills no tile evenly
        {"name": "filter_512", "kind": "filter", "log2n": 9, "batch": 10007},
        # the batched benchmark workload: 16384 transforms of 4096 points
        {"name": "batch_4096", "kind": "transform", "log2n": 12, "batch": 16384, "direction": "forward"},
        # the longest transforms that run as one kernel, an odd count of them, inverse
        {"name": "batch_2p14", "kind": "transform", "log2n": 14, "batch": 1021, "direction": "inverse"},
        # a batch of medium transforms (two passes)
        {"name": "batch_2p16", "kind": "transform", "log2n": 16, "batch": 256, "direction": "forward"},
        # single large transforms of the benchmark: one that fits the L2 cache, there and back ...
        {"name": "single_2p20", "kind": "transform", "log2n": 20, "batch": 1, "direction": "both"},
        # ... one whose array is about the size of the L2 cache ...
        {"name": "single_2p24", "kind": "transform", "log2n": 24, "batch": 1, "direction": "forward"},
        # ... and one far beyond it, inverse
        {"name": "single_2p27", "kind": "transform", "log2n": 27, "batch": 1, "direction": "inverse"},
        # 20000 transforms of 2^4 .. 2^16 points packed back to back, in one launch
        {"name": "uneven_20000", "kind": "uneven", "count": 20000, "lo": 4, "hi": 16, "mix": 1},
        # one training step of the differentiable layer: 512 signals of 8192 points
        {"name": "loss_512x8192", "kind": "loss", "log2n": 13, "batch": 512},
        # rank 3 of 8 in a distributed transform of 2^30 points: 2^10-point columns, then 2^20-point ones
        {"name": "columns_2p30_rank", "kind": "columns", "log2n1": 10, "log2n2": 20, "log2p": 3, "rank": 3},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _batch(rng, log2n, max_log2, min_values=1):
    """A batch count, log-uniform over what fits, odd more often than not."""
    top = max(1, (1 << max_log2) >> log2n)
    low = min(top, max(1, min_values >> log2n))
    b = min(top, _log_uniform(rng, low, top))
    return b | 1 if rng.random() < 0.6 and (b | 1) <= top else b


def draw(rng):
    p = rng.random()
    if p < 0.58:
        m = rng.randint(0, MAX_LOG2)
        return {"kind": "transform", "log2n": m, "batch": _batch(rng, m, MAX_LOG2, 1 << 12),
                "direction": rng.choice(["forward", "inverse", "both"]) if m < MAX_LOG2 else rng.choice(["forward", "inverse"])}
    if p < 0.70:
        m = rng.randint(3, 22)
        return {"kind": "filter", "log2n": m, "batch": _batch(rng, m, 25, 1 << 14)}
    if p < 0.80:
        lo = rng.randint(0, 10)
        return {"kind": "uneven", "count": _log_uniform(rng, 200, 20000), "lo": lo, "hi": rng.randint(lo + 2, 16),
                "mix": rng.randint(2, 1 << 20)}
    if p < 0.88:
        m = rng.randint(4, 14)
        return {"kind": "loss", "log2n": m, "batch": _batch(rng, m, 25, 1 << 16)}
    if p < 0.92:
        m = rng.randint(4, 20)
        return {"kind": "autograd", "log2n": m, "batch": _batch(rng, m, 24, 1 << 16)}
    # a rank's block of 2^20 .. 2^27 values, either factor of the transform between 2^8 and 2^20
    lp = rng.randint(1, 4)
    total = rng.randint(20, COLUMNS_MAX_LOG2) + lp
    l1 = rng.randint(max(8, lp + 4, total - 20), min(20, total - max(8, lp + 4)))
    return {"kind": "columns", "log2n1": l1, "log2n2": total - l1, "log2p": lp, "rank": rng.randrange(1 << lp)}


# ---- inputs -----------------------------------------------------------------------------------------


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _complex(values, gen, dev, uniform=False):
    """`values` complex64 numbers, standard normal (or uniform in [-1, 1)) parts."""
    r = torch.empty(2 * values, dtype=torch.float32, device=dev)
    if uniform:
        r.uniform_(-1.0, 1.0, generator=gen)
    else:
        r.normal_(generator=gen)
    return torch.view_as_complex(r.view(values, 2))


def _inputs(case, seed):
    """The case's input tensors, from the seed alone."""
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(seed)
    kind = case["kind"]
    if kind == "columns":
        values = 1 << (case["log2n1"] + case["log2n2"] - case["log2p"])
        # the second step's input stands for what the exchange delivers: data of its own
        return {"x": _complex(values, gen, dev), "z": _complex(values, gen, dev)}
    if kind == "uneven":
        return {"x": _complex(int(_descriptors(case)[3]), gen, dev, uniform=True)}
    n, batch = 1 << case["log2n"], case["batch"]
    d = {"x": _complex(n * batch, gen, dev).view(batch, n)}
    if kind == "filter":
        d["h"] = _complex(n, gen, dev)
    elif kind == "loss":
        d["w"] = torch.empty(n, dtype=torch.float32, device=dev).uniform_(0.0, 1.0, generator=gen)
    elif kind == "autograd":
        d["g"] = _complex(n * batch, gen, dev).view(batch, n)
    return d


def _descriptors(case):
    """log2 n, direction and offset of every transform of an uneven batch, and the span."""
    r = np.random.RandomState(case["mix"])
    m = r.randint(case["lo"], case["hi"] + 1, case["count"])
    inv = r.randint(0, 2, case["count"])
    size = np.int64(1) << m.astype(np.int64)
    off = np.concatenate([[0], np.cumsum(size)[:-1]])
    return m.astype(np.int32), inv.astype(np.int32), off.astype(np.int64), int(size.sum())


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case)
    kind = case["kind"]
    if kind == "transform":
        s["plan"] = ofb.Plan(1 << case["log2n"])
        s["y"] = torch.empty_like(s["x"])
        if case["direction"] == "both":
            s["z"] = torch.empty_like(s["x"])
    elif kind == "filter":
        s["plan"] = ofb.Plan(1 << case["log2n"])
        s["y"], s["z"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
    elif kind == "uneven":
        s["batch"] = ofb.UnevenBatch(*_descriptors(case)[:3])
        s["y"] = torch.empty_like(s["x"])
    elif kind in ("loss", "autograd"):
        s["x"].requires_grad_(True)
    elif kind == "columns":
        l1, l2, lp = case["log2n1"], case["log2n2"], case["log2p"]
        c2, r1 = 1 << (l2 - lp), 1 << (l1 - lp)
        s["step1"] = ofb.Columns(1 << l1, c2, 1 << lp, 1 << (l1 + l2), case["rank"] * c2)
        s["step3"] = ofb.Columns(1 << l2, r1)
        s["send"], s["out"] = torch.empty_like(s["x"]), torch.empty_like(s["z"])
    return s


# ---- one pass ---------------------------------------------------------------------------------------


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("loss", "autograd"):
        s["x"].grad = None
        if kind == "loss":
            loss = torch_fft.weighted_power_loss_fused(s["x"], s["w"])
            loss.backward()
            return {"loss": loss.detach(), "grad": s["x"].grad}
        y = torch_fft.fft(s["x"])
        y.backward(s["g"])
        return {"y": y.detach(), "grad": s["x"].grad}
    stream = torch.cuda.current_stream().cuda_stream
    x = s["x"]
    if kind == "columns":
        s["step1"].execute(x.data_ptr(), s["send"].data_ptr(), 0, stream)
        s["step3"].execute(s["z"].data_ptr(), s["out"].data_ptr(), 0, stream)
        return {"send": s["send"], "out": s["out"]}
    y = s["y"]
    if kind == "uneven":
        s["batch"].execute(x.data_ptr(), y.data_ptr(), stream)
        return y
    plan, batch = s["plan"], case["batch"]
    if kind == "filter":
        z = s["z"]
        plan.dev_weighted(x.data_ptr(), y.data_ptr(), batch, None, s["h"].data_ptr(), False, stream)
        plan.dev_inverse(y.data_ptr(), z.data_ptr(), batch, stream)
        return {"spectrum": y, "filtered": z}
    if case["direction"] == "inverse":
        plan.dev_inverse(x.data_ptr(), y.data_ptr(), batch, stream)
        return y
    plan.dev_forward(x.data_ptr(), y.data_ptr(), batch, stream)
    if case["direction"] == "forward":
        return y
    z = s["z"]
    plan.dev_inverse(y.data_ptr(), z.data_ptr(), batch, stream)
    return {"spectrum": y, "back": z}


# ---- what a pass cannot do without --------------------------------------------------------------------


def work(case):
    """Bytes: each input read once, each output written once (8 bytes a complex value); flops:
    5 n log2 n a transform and 6 (8) for a complex product (a loss term with its gradient)."""
    kind = case["kind"]
    if kind == "columns":
        l1, l2 = case["log2n1"], case["log2n2"]
        values = 1 << (l1 + l2 - case["log2p"])
        return {"bytes": 32 * values, "flops": 5 * values * (l1 + l2) + 6 * values}
    if kind == "uneven":
        m, _, _, span = _descriptors(case)
        return {"bytes": 16 * span, "flops": int(np.sum(5.0 * m * 2.0 ** m))}
    n, batch = 1 << case["log2n"], case["batch"]
    values, flops = n * batch, 5 * n * batch * max(1, case["log2n"])
    if kind == "transform":
        k = 2 if case["direction"] == "both" else 1
        # there and back: x read, the spectrum and the result written, the spectrum read back
        return {"bytes": k * 16 * values, "flops": k * flops}
    if kind == "filter":
        return {"bytes": 32 * values + 8 * n, "flops": 2 * flops + 6 * values}
    if kind == "loss":
        return {"bytes": 16 * values + 4 * n, "flops": 2 * flops + 8 * values}
    return {"bytes": 32 * values, "flops": 2 * flops}  # autograd: x, y, g, the gradient


# ---- the same in 64 bits ------------------------------------------------------------------------------


def _fft64(x, inverse, dim=-1):
    """Unnormalised complex128 transform, `inverse` with exp(+2 pi i ...)."""
    return torch.fft.ifft(x, dim=dim, norm="forward") if inverse else torch.fft.fft(x, dim=dim)



def _columns64(x, n, cols, blocks, big_n, col0):
    """Columns.execute's statement: out[((k / r) cols + b) r + k mod r] = Y_b[k] w_big_n^((col0 + b) k)."""
    y = _fft64(x.view(n, cols).to(torch.complex128), False, dim=0)
    if big_n:
        step = max(1, (1 << 24) // cols)
        b = torch.arange(cols, device=x.device, dtype=torch.int64) + col0
        for k0 in range(0, n, step):
            k = torch.arange(k0, min(n, k0 + step), device=x.device, dtype=torch.int64)
            angle = ((k[:, None] * b[None, :]) % big_n).to(torch.float64) * (-2.0 * math.pi / big_n)
            y[k0:k0 + step] *= torch.polar(torch.ones_like(angle), angle)
    r = n // blocks
    return y.view(blocks, r, cols).permute(0, 2, 1).reshape(-1)


def exact(case, seed):
    d = _inputs(case, seed)
    kind, x = case["kind"], d["x"]
    if kind == "columns":
        l1, l2, lp = case["log2n1"], case["log2n2"], case["log2p"]
        c2, r1 = 1 << (l2 - lp), 1 << (l1 - lp)
        send = _columns64(x, 1 << l1, c2, 1 << lp, 1 << (l1 + l2), case["rank"] * c2)
        out = _columns64(d["z"], 1 << l2, r1, 1, 0, 0)
        return {"send": send, "out": out}
    if kind == "uneven":
        m, inv, off, _ = _descriptors(case)
        y = torch.empty(x.numel(), dtype=torch.complex128, device=x.device)
        for log2n in np.unique(m):
            for direction in (0, 1):
                sel = off[(m == log2n) & (inv == direction)]
                lane = torch.arange(1 << int(log2n), device=x.device)
                for part in np.array_split(sel, max(1, len(sel) >> max(0, 24 - int(log2n)))):
                    if len(part):
                        idx = torch.from_numpy(part).to(x.device)[:, None] + lane[None, :]
                        y[idx] = _fft64(x[idx].to(torch.complex128), bool(direction))
        return y
    x = x.to(torch.complex128)
    if kind == "transform":
        if case["direction"] == "inverse":
            return _fft64(x, True)
        y = _fft64(x, False)
        return y if case["direction"] == "forward" else {"spectrum": y, "back": x * (1 << case["log2n"])}
    if kind == "filter":
        y = _fft64(x, False) * d["h"].to(torch.complex128)
        return {"spectrum": y, "filtered": _fft64(y, True)}
    if kind == "loss":
        w = d["w"].to(torch.float64)
        y = _fft64(x, False)
        loss = (torch.view_as_real(y).square().sum(-1) * w.square()).sum()
        return {"loss": loss, "grad": _fft64(2.0 * w.square() * y, True)}
    return {"y": _fft64(x, False), "grad": _fft64(d["g"].to(torch.complex128), True)}
