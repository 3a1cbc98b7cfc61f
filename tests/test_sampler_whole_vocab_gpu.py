"""Whole-vocabulary rows at the edges of the kernel's pieces: blocks of 256 elements, tiles of 32 segments, the vocabulary from
which segments are longer (163 840), chunks of shared memory (46 592 elements), bins too full to be sorted, rows off 16-byte
boundaries (every odd vocabulary).  Token ids must be the oracle's, except inside a run of equal probabilities."""
import numpy as np
import pytest

from tests import sampler_harness as H
from oracle import sampler_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    return H.GpuSampler()


def _logits(kind, rng, n, v):
    x = (rng.standard_normal((n, v)) * 2).astype(np.float32)
    if kind == "flat":            # a few hundred elements per bin
        x *= 0.1
    elif kind == "narrow":        # thousands per bin: finer levels
        x *= 1e-4
    elif kind == "quantised":
        x = np.round(x * 4) / 4
    elif kind == "equal":
        x[:] = 1.5
    elif kind == "peaks":         # most of the mass early, the rest of the sum just below one
        x[:, : max(1, v // 50)] += 12
    elif kind == "masked":
        x[:, ::2] = -np.inf
        x[:, : v // 3] = -np.inf
        x[:, -1] = 0.5
    return np.ascontiguousarray(x.astype(np.float32))


@pytest.mark.parametrize("v", [1, 2, 255, 256, 257, 8191, 8193, 46593, 65537, 163837, 163841, 200001])
@pytest.mark.parametrize("kind", ["normal", "flat", "narrow", "quantised", "equal", "peaks", "masked"])
def test_tokens_at_the_edges(gpu, kind, v):
    rng = np.random.default_rng(v + 7 * len(kind))
    options = [dict(top_p=0.9), dict(top_p=0.99999), dict(top_p=0.05), dict(temperature=0.7), dict(min_p=0.05, top_p=0.95), dict(min_p=0.3, temperature=1.3)]
    x = _logits(kind, rng, len(options), v)
    rows = np.concatenate([H.make_rows(1, logits_rows=np.array([r], np.int64), **kw) for r, kw in enumerate(options) for _ in range(3)])
    rows["rand_u"] = np.tile(np.array([0.0, 0.37, 0.9999999], np.float32), len(options))
    rc_o, tok_o, lp_o, _ = H.run_oracle(x, rows)
    rc_g, tok_g, lp_g, _ = gpu.step_host(x, rows)
    assert rc_o == 0 and rc_g == 0
    for i in np.flatnonzero(tok_o != tok_g):
        p, _, _ = sampler_oracle.transform(0, x[rows["logits_row"][i]], float(rows["temperature"][i]))
        assert p[tok_g[i]] == p[tok_o[i]], (options[i // 3], rows["rand_u"][i], tok_o[i], tok_g[i])
    assert np.allclose(lp_o, lp_g, atol=2e-6, rtol=1e-6, equal_nan=True), (lp_o, lp_g)   # (two logarithms, rounded once each)
