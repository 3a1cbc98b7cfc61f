"""Forms of the PagedAttention inputs that decide which branch of a kernel runs, against the CPU oracle: head sizes, block sizes
and head counts of the rotation, query rows that are scaled before they are packed beside rows that are not, and a query and
caches that do not start on a boundary of the wide loads and stores."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests import pa_harness as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cache", ["f16", "bf16", "u8"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("bs", [16, 32])
@pytest.mark.parametrize("hkv", [1, 2, 3])
def test_rotated_blocks_are_bit_exact(cache, d, bs, hkv):
    """A block's (kv head, token) units in whole passes of the CTA, in less than one (16 or 32 units of 32 or 64 per pass)
    and with a partial last pass (48 of 32 + 16): units without work take part in the shuffles and write nothing."""
    from openvino_genai_b200 import workloads
    act = torch.float16 if cache == "f16" else torch.bfloat16
    wl = H.small_workload(hq=2 * hkv, hkv=hkv, d=d, bs=bs, act=act, cache=cache, past=[200, 96], new=[1, 1], seed=53 + hkv)
    first, second = wl.block_indices_begins[:2]
    wl.rotated_block_indices = np.concatenate([wl.block_indices[first:first + 200 // bs], wl.block_indices[second + 1:second + 3]]).astype(np.int32)
    wl.rotation_deltas = (np.arange(len(wl.rotated_block_indices)) * 5 % 9).astype(np.int32)
    wl.rotation_trig_lut = workloads.rotation_trig_lut(9, bs, d, 1e6)
    res = H.run_both(wl)
    assert res["status"] == 0
    assert np.array_equal(res["kc_gpu"], res["kc_ref"]) and np.array_equal(res["vc_gpu"], res["vc_ref"])


@pytest.mark.parametrize("act,cache", [(torch.float16, "u8"), (torch.bfloat16, "u8"), (torch.float32, "u8"), (torch.float16, "f16"), (torch.bfloat16, "f16")])
@pytest.mark.parametrize("d,hq,hkv", [(64, 8, 2), (128, 14, 2)])
def test_rows_scaled_for_the_tensor_cores_beside_rows_that_are_not(act, cache, d, hq, hkv):
    """Query rows of magnitudes 1, 300, 5000 and 15000 in one warp: those above 256 are packed with a power of two of their own,
    which the row's softmax scale takes back out.  Compared row by row, so that a factor given to a neighbour shows.

    Bound: the logits of the largest rows reach about 3 x 4.5; rounding q to f16 moves them by 2^-11 of that, rounding the
    exponent of P to f16 (up to 19.5 in base 2: half an ulp is 2^-7) by 0.0054, P and the output have 2^-10 and 2^-9:
    0.016 in all."""
    wl = H.small_workload(hq=hq, hkv=hkv, d=d, bs=32, act=act, cache=cache, past=[300, 40, 0], new=[70, 1, 33], seed=131, scale=1.0 / (5000.0 * d ** 0.5))
    wl.score_aggregation_window = np.array([5, 1, 3], np.int32)
    q, k, v, fill, pk, pv = H.make_host_data(wl)
    mag = torch.from_numpy(np.random.default_rng(7).choice([1.0, 300.0, 5000.0, 15000.0], size=(q.shape[0], hq, 1)).astype(np.float32))
    q = (q.float().clamp(-4, 4).view(q.shape[0], hq, d) * mag).view(q.shape).to(act)
    data = (q, k, v, fill, pk, pv)
    res = H.run_oracle(wl, data)
    res.update(H.run_gpu(wl, data))
    assert res["status"] == 0 and res["prefill_kernel"] == "tcgen05"
    out, ref = (res[x].reshape(-1, hq, d).astype(np.float64) for x in ("out_gpu", "out_ref"))
    err = np.abs(out - ref).max(-1) / np.abs(ref).max(-1)
    assert err.max() < 2e-2, (err.max(), np.argwhere(err >= 2e-2)[:8], mag.view(-1, hq)[np.unravel_index(err.argmax(), err.shape)])
    assert H.rel_err(res["scores_gpu"], res["scores_ref"]) < 2e-2


@pytest.mark.parametrize("act,cache,d", [(torch.float16, "f16", 128), (torch.bfloat16, "bf16", 64), (torch.float32, "f16", 64), (torch.bfloat16, "u8", 64)])
def test_decode_query_off_a_pair_boundary(act, cache, d):
    """Query rows are read in pairs where the buffer allows it; one element further on, they are read one by one."""
    wl = H.small_workload(hq=6, hkv=2, d=d, bs=32, act=act, cache=cache, past=[100, 31, 777], new=[1, 1, 1], seed=17)
    q, k, v, fill, pk, pv = H.make_host_data(wl)
    op = H.make_op(wl)
    ref = H.run_gpu(wl, (q, k, v, fill, pk, pv), op=op)
    flat = torch.zeros(q.numel() + 8, dtype=q.dtype, device="cuda")
    flat[1:1 + q.numel()] = q.cuda().view(-1)
    moved = flat[1:1 + q.numel()].view(q.shape)
    assert moved.data_ptr() % 8 == q.element_size()
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    out = torch.zeros_like(q, device="cuda")
    kc, vc = t(ref["kc_gpu"]), t(ref["vc_gpu"])   # the step's rows are in it already and are written again
    op.evaluate({"query": moved, "key": k.cuda(), "value": v.cuda(), "key_cache": kc, "value_cache": vc, "past_lens": t(wl.past_lens),
                 "subsequence_begins": t(wl.subsequence_begins), "block_indices": t(wl.block_indices), "block_indices_begins": t(wl.block_indices_begins),
                 "scale": wl.scale, "max_context_len": wl.max_context_len}, {"output": out})
    torch.cuda.synchronize()
    assert op.device_status() == 0
    want = H.run_oracle(wl, (q, k, v, fill, pk, pv))
    assert H.rel_err(ref["out_gpu"], want["out_ref"]) < 1e-2
    # the order in which partials are added may differ: one rounding of the output
    assert H.rel_err(out.float().cpu().numpy(), ref["out_gpu"]) < (2 ** -7 if act == torch.bfloat16 else 2 ** -10)


@pytest.mark.parametrize("cache,act,shift", [("u8", torch.bfloat16, 4), ("f16", torch.float16, 2), ("bf16", torch.float32, 8)])
def test_chunk_writes_into_caches_off_a_16_byte_boundary(cache, act, shift):
    """Enough rows for groups of tokens, whose stores are up to 16 bytes wide: caches that start elsewhere get the same bytes
    row by row (and nothing around them is touched)."""
    wl = H.small_workload(hq=10, hkv=5, d=128, bs=32, act=act, cache=cache, past=[0, 5, 31], new=[701, 33, 1], seed=19)
    assert (wl.num_tokens - 3) * 5 >= 3072 + 3 * 5 // 2
    _, k, v, _, _, _ = H.make_host_data(wl)
    op = H.make_op(wl)
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    kd, vd = k.cuda(), v.cuda()
    n = wl.num_blocks * H.block_bytes(wl)
    def write(off):
        flat = [torch.full((n + 64,), 0xA5, dtype=torch.uint8, device="cuda") for _ in range(2)]
        for x in flat:
            x[off:off + n] = 0
        kc, vc = (x[off:off + n] for x in flat)
        args = op.make_args(kd, kd, vd, kd, kc, vc, t(wl.past_lens), t(wl.subsequence_begins), t(wl.block_indices), t(wl.block_indices_begins),
                            wl.scale, wl.max_context_len)
        op._check(op.lib.pa_b200_write_kv(op._h, C.byref(args)))
        torch.cuda.synchronize()
        assert op.device_status() == 0
        for x in flat:
            assert bool((x[:off] == 0xA5).all()) and bool((x[off + n:] == 0xA5).all())
        return kc.cpu().numpy(), vc.cpu().numpy()
    want, got = write(0), write(shift)
    assert want[0].any() and np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])
