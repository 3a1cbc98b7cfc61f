"""The first step of a new sampler handle: for a few rows nothing is allocated, which would take several times as long as the step."""
import numpy as np
import pytest

from tests import sampler_harness as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,v", [(1, 262144), (2, 151936), (3, 128256), (5, 32000), (9, 32000), (16, 32000)])
def test_a_small_first_step_takes_no_device_memory(n, v):
    import torch
    x = torch.randn(n, v, device="cuda")
    rows = H.make_rows(n, top_k=50)
    warm = H.GpuSampler()                     # the kernels are loaded once per process
    staged = warm.stage(rows, None, x.device)
    assert warm.step_device(x, rows, staged=staged)[0] == 0
    new = H.GpuSampler()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    rc, tok, _ = new.step_device(x, rows, staged=staged)
    torch.cuda.synchronize()
    assert rc == 0 and torch.cuda.mem_get_info()[0] == free


def test_steps_of_small_and_large_scratch_take_turns():
    """Whole-vocabulary rows on either side of the limit, on one handle: the tokens of a handle of their own."""
    rng = np.random.default_rng(2)
    handle = H.GpuSampler()
    for n, v in [(2, 32000), (40, 50257), (16, 32000), (17, 32000), (3, 151936), (64, 50257)]:
        x = (rng.standard_normal((n, v)) * 2).astype(np.float32)
        rows = H.make_rows(n, top_p=0.95, seeds=rng.integers(1, 1000, n))
        rc, tok, lp, _ = handle.step_host(x, rows)
        rc_own, tok_own, lp_own, _ = H.GpuSampler().step_host(x, rows)
        assert rc == 0 and rc_own == 0
        assert np.array_equal(tok, tok_own) and np.array_equal(lp, lp_own)
