"""Whole-vocabulary rows of every kind take about the time of rows of normally distributed logits: sums that begin late (grammar masks, late
peaks), that come from a few elements (low temperatures) or that leave elements out (min-p) are no special case of the walk over a
row's segments.  The work of a row is a few passes over it whatever it holds, so twice the time is allowed; where the walk falls back to
adding the row's 501 segments one by one, or makes its guesses anew time after time, it takes four to thirteen times as long."""
import ctypes

import numpy as np
import pytest

from tests import sampler_harness as H

pytestmark = pytest.mark.gpu

ROWS, VOCAB = 96, 128256


@pytest.fixture(scope="module")
def gpu():
    return H.GpuSampler()


def logits_of(kind):
    import torch
    g = torch.Generator(device="cuda").manual_seed(17)
    x = torch.randn(ROWS, VOCAB, generator=g, device="cuda") * 2
    if kind == "last_ids":
        x[:, : VOCAB - 200] = -float("inf")
    elif kind == "few_ids":
        keep = torch.randint(0, VOCAB, (ROWS, 20), generator=g, device="cuda")
        x = torch.full_like(x, -float("inf")).scatter_(1, keep, x.gather(1, keep))
    elif kind == "upper_half":
        x[:, : VOCAB // 2] = -float("inf")
    elif kind == "spikes":
        x.scatter_add_(1, torch.randint(0, VOCAB, (ROWS, 8), generator=g, device="cuda"), torch.full((ROWS, 8), 15.0, device="cuda"))
    elif kind == "late":
        x[:, VOCAB - VOCAB // 8] = 60.0
    return x


def time_of(gpu, x, further=0, **options):
    """Median time of a step with so many further draws per row, in us (nothing of the logits changes: the rows have no penalties)."""
    import torch
    rows = H.make_rows(ROWS, **options)
    staged = gpu.stage(rows, None, x.device)
    args = H.step_args(x, staged["rows"], None, staged["tok"], staged["lp"], ptr=lambda t: t.data_ptr())
    args.num_rows = ROWS
    args.num_logit_rows, args.vocab = x.shape
    args.stream = 1
    if further:
        offs = torch.arange(ROWS + 1, device="cuda") * further
        us = torch.rand(ROWS * further, generator=torch.Generator(device="cuda").manual_seed(5), device="cuda")
        tokens, log_probs = torch.zeros(ROWS * further, dtype=torch.int64, device="cuda"), torch.zeros(ROWS * further, device="cuda")
        args.extra_offsets, args.extra_rand_u = offs.data_ptr(), us.data_ptr()
        args.extra_out_token, args.extra_out_log_prob = tokens.data_ptr(), log_probs.data_ptr()
    times = []
    for i in range(12):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        rc = gpu.lib.sampler_b200_step(gpu.h, ctypes.byref(args))
        b.record()
        torch.cuda.synchronize()
        assert rc == 0
        if i >= 3:
            times.append(a.elapsed_time(b) * 1e3)
    return float(np.median(times))


@pytest.mark.parametrize("top_p", [1.0, 0.95])
@pytest.mark.parametrize("kind,options", [
    ("last_ids", {}), ("few_ids", {}), ("upper_half", {}), ("last_ids", dict(temperature=0.1)), ("spikes", dict(temperature=0.1)),
    ("late", dict(temperature=0.1)), ("normal", dict(temperature=0.01)), ("normal", dict(min_p=0.05)), ("spikes", dict(min_p=0.05)),
])
def test_no_kind_of_row_takes_twice_the_time_of_flat_ones(gpu, kind, options, top_p):
    flat = time_of(gpu, logits_of("normal"), top_p=top_p)
    took = time_of(gpu, logits_of(kind), top_p=top_p, **options)
    print(f"{kind} {options} top_p {top_p}: {took:.0f} us, flat rows {flat:.0f} us")
    assert took < 2 * flat


def test_further_draws_of_peaked_rows_do_not_pass_over_the_row(gpu):
    """Sixteen further draws of rows that keep a handful of elements: each looks into what the first one found.  (A draw takes a few
    microseconds, half of the step's own time all together; with a pass over the row for each the step takes 2.5 times as long.)"""
    x = logits_of("spikes")
    once, often = time_of(gpu, x, top_p=0.9, temperature=0.7), time_of(gpu, x, further=16, top_p=0.9, temperature=0.7)
    print(f"{often:.0f} us with 16 further draws per row, {once:.0f} us without")
    assert often < 1.8 * once
