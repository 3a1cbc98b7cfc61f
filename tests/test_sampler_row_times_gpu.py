"""Whole-vocabulary rows of every kind take about the time of rows of normally distributed logits: sums that begin late (grammar masks, late
peaks), that come from a few elements (low temperatures) or that leave elements out (min-p) are no special case of the walk over a
row's segments.  The work of a row is a few passes over it whatever it holds, so twice the time is allowed; where the walk falls back to
adding the row's 501 segments one by one, or makes its guesses anew time after time, it takes four to thirteen times as long."""
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


def time_of(gpu, x, **options):
    """Median time of a step, in us (nothing of the logits changes: the rows have no penalties)."""
    import torch
    rows = H.make_rows(ROWS, **options)
    staged = gpu.stage(rows, None, x.device)
    times = []
    for i in range(12):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        rc, _, _ = gpu.step_device(x, rows, staged=staged)
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
