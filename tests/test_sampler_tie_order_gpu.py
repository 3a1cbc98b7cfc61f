"""The token a top-p draw gives when it falls among equal probabilities: the reference's std::sort leaves their order open, the kernel takes
them in index order.  So every row has exactly one right answer: a stable descending sort, float32 sums one by one, the first sum above
total * u.  Also in runs of many thousands, which other tests accept any element of."""
import ctypes

import numpy as np
import pytest

from tests import sampler_harness as H
from oracle import sampler_oracle


def expected_tokens(probs, top_p, min_p, draws):
    """For one row's probabilities (float32): the token of every number in `draws`."""
    order = np.argsort(-probs, kind="stable")
    p = probs[order]
    if min_p > 0:
        p = p[p >= np.float32(min_p) * p[0]]
    sums = np.add.accumulate(p, dtype=np.float32)      # one by one, each rounded to float32
    above = np.flatnonzero(sums > np.float32(top_p))
    kept = above[0] + 1 if len(above) else len(p)
    sums = sums[:kept]
    tokens = []
    for u in draws:
        hit = np.flatnonzero(sums > sums[-1] * np.float32(u))
        tokens.append(order[hit[0] if len(hit) else kept - 1])
    return np.array(tokens, np.int64)


def logits_of(kind, rng, v):
    x = rng.standard_normal(v) * 2
    if kind == "equal":
        x[:] = 1.5
    elif kind == "two_values":
        x = np.where(rng.random(v) < 0.5, 0.25, 0.75)
    elif kind == "quantised":
        x = np.round(x * 4) / 4
    elif kind == "bf16":
        x = (x.astype(np.float32).view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)
    elif kind == "masked":
        x = np.where(np.arange(v) % 3 == 0, 0.5, -np.inf)
    return np.ascontiguousarray(x.astype(np.float32))


KINDS = ["equal", "two_values", "quantised", "bf16", "masked"]
OPTIONS = [dict(top_p=0.9), dict(top_p=0.3), dict(top_p=0.99999), dict(top_p=0.95, min_p=0.02)]
DRAWS = np.array([0.0, 0.11, 0.37, 0.5, 0.76, 0.9999999], np.float32)


def test_the_expectation_follows_the_oracle():
    """CPU: where no probability occurs twice among the drawn, the oracle gives the same tokens."""
    rng = np.random.default_rng(3)
    x = rng.standard_normal((1, 3001)).astype(np.float32)
    rows = np.concatenate([H.make_rows(1, logits_rows=np.array([0], np.int64), **kw) for kw in OPTIONS for _ in DRAWS])
    rows["rand_u"] = np.tile(DRAWS, len(OPTIONS))
    rc, tok, _, _ = H.run_oracle(x, rows)
    p, _, _ = sampler_oracle.transform(0, x[0], 1.0)
    want = np.concatenate([expected_tokens(p, kw["top_p"], kw.get("min_p", 0.0), DRAWS) for kw in OPTIONS])
    assert rc == 0
    for got, token in zip(tok, want):
        assert p[got] == p[token] and (got == token or (p == p[token]).sum() > 1)


@pytest.mark.gpu
@pytest.mark.parametrize("v", [300, 4096, 4097, 50257, 128256, 200001])
@pytest.mark.parametrize("kind", KINDS)
def test_draws_among_equal_probabilities_follow_the_index(kind, v):
    x = logits_of(kind, np.random.default_rng(v), v)[None]
    rows = np.concatenate([H.make_rows(1, logits_rows=np.array([0], np.int64), **kw) for kw in OPTIONS for _ in DRAWS])
    rows["rand_u"] = np.tile(DRAWS, len(OPTIONS))
    rc, tok, _, _ = H.GpuSampler().step_host(x, rows)
    assert rc == 0
    p, _, _ = sampler_oracle.transform(0, x[0], 1.0)
    want = np.concatenate([expected_tokens(p, kw["top_p"], kw.get("min_p", 0.0), DRAWS) for kw in OPTIONS])
    assert np.array_equal(tok, want), [(i // len(DRAWS), float(DRAWS[i % len(DRAWS)]), int(tok[i]), int(want[i])) for i in np.flatnonzero(tok != want)]


@pytest.mark.gpu
@pytest.mark.parametrize("v", [163838, 262144, 327677, 327681, 400001, 655357, 700001])
@pytest.mark.parametrize("kind", ["bf16", "masked", "two_values"])
def test_segments_of_several_blocks(kind, v):
    """Vocabularies around those from which a segment has two, four and more blocks of 256 elements."""
    test_draws_among_equal_probabilities_follow_the_index(kind, v)


@pytest.mark.gpu
@pytest.mark.parametrize("v", [300, 4096, 50257, 128256])
@pytest.mark.parametrize("kind", KINDS + ["peaks", "steps"])
def test_further_draws_of_a_row_follow_the_index_too(kind, v):
    """Several draws of one row, which find their elements in a list where few are kept: as many as fit, one more, runs of equal ones in it."""
    rng = np.random.default_rng(v + 1)
    if kind == "peaks":
        x = (rng.standard_normal(v) * 2).astype(np.float32)
        x[rng.choice(v, size=min(v, 40), replace=False)] += 15
    elif kind == "steps":      # 100 values, each a run of v / 100 elements
        x = (rng.permutation(v) % 100 * 0.125).astype(np.float32)
    else:
        x = logits_of(kind, rng, v)
    x = np.ascontiguousarray(np.tile(x, (len(OPTIONS), 1)))
    rows = np.concatenate([H.make_rows(1, logits_rows=np.array([i], np.int64), **kw) for i, kw in enumerate(OPTIONS)])
    us = rng.random((len(rows), 24)).astype(np.float32)
    rows["rand_u"] = us[:, 0]
    offs = np.arange(len(rows) + 1, dtype=np.int64) * (us.shape[1] - 1)
    extra_u = np.ascontiguousarray(us[:, 1:]).ravel()
    tok, lp = np.full(len(rows), -7, np.int64), np.zeros(len(rows), np.float32)
    xtok, xlp = np.full(len(extra_u), -7, np.int64), np.zeros(len(extra_u), np.float32)
    a = H.step_args(x, rows, None, tok, lp)
    a.extra_offsets, a.extra_rand_u = offs.ctypes.data, extra_u.ctypes.data
    a.extra_out_token, a.extra_out_log_prob = xtok.ctypes.data, xlp.ctypes.data
    gpu = H.GpuSampler()
    assert gpu.lib.sampler_b200_step_host(gpu.h, ctypes.byref(a), 0) == 0
    p, _, _ = sampler_oracle.transform(0, x[0], 1.0)
    for i, kw in enumerate(OPTIONS):
        want = expected_tokens(p, kw["top_p"], kw.get("min_p", 0.0), us[i])
        got = np.concatenate([tok[i:i + 1], xtok[offs[i]:offs[i + 1]]])
        assert np.array_equal(got, want), (kw, np.flatnonzero(got != want), got[got != want], want[got != want])
