"""Performance cases of the framework: what a continuous-batching engine asks of it in one step.

An engine step is, per layer, one call of the PagedAttention operator (`PagedAttentionExtension.evaluate`: cache write,
optional re-rotation of evicted-neighbour blocks, attention of decode rows and prefill chunks, optional score output)
and, once, one call of the sampler (`SamplerStep.step`).  The cases below are those calls, over the sizes and options an
engine meets: one user's chat up to a full batch, one prompt up to a batch of chunks, every cache type, and the sampling
options requests come with.  Lengths follow from the case alone (`layout` seeds them); values, block tables and random
numbers follow from the seed.

`exact` restates the documented arithmetic (cache layout, by-token u8 quantiser, rotation, attention, scores, penalties,
top-k / top-p draw) in plain torch with 64-bit sums.
"""
import math

import numpy as np
import torch

import __graft_entry__ as entry   # the package folder has a dot in its name: this loads it as `openvino_genai_b200`

pkg = entry.load_package()
from openvino_genai_b200 import _sampler_abi as sampler_abi, sampler as sampler_mod  # noqa: E402

DEV = "cuda:0"
ACT = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
ROTATION_ROWS = 513      # rows of the rotation table: block distances 1 .. 512
ROTATION_THETA = 1e6


# ---- the cases -------------------------------------------------------------------------------------------------------
def _attn(name, **kw):
    case = {"kind": "attn", "hq": 32, "hkv": 8, "d": 128, "bs": 32, "act": "bf16", "cache": "u8", "decode": 0, "past_lo": 0,
            "past_hi": 0, "log_past": False, "chunks": 0, "chunk_lo": 0, "chunk_hi": 0, "chunk_past_hi": 0, "scores": False,
            "rotated": 0.0, "layout": 1}
    case.update(kw)
    if name:
        case["name"] = name
    return case


def _samp(name, **kw):
    case = {"kind": "sampler", "rows": 256, "vocab": 151936, "mode": "top_k", "top_k": 50, "temperature": 0.7, "top_p": 0.9,
            "penalties": False, "history": 0, "spikes": 8, "layout": 1}
    case.update(kw)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # a handful of chats on a small model (TinyLlama shape, f16 everywhere): a layer's call is a few microseconds of work
        _attn("decode_f16_d64_8", hq=32, hkv=4, d=64, act="f16", cache="f16", decode=8, past_lo=64, past_hi=2048, layout=11),
        # one user with a long conversation (Qwen2.5-7B shape): the whole chip works on one sequence
        _attn("decode_u8_single_9k", hq=28, hkv=4, decode=1, past_lo=9001, past_hi=9001, layout=12),
        # the ordinary decode step of a served Llama-3-8B shape, u8 cache
        _attn("decode_u8_64", decode=64, past_lo=512, past_hi=8192, layout=13),
        # the same with an unquantised cache, a ragged number of rows
        _attn("decode_bf16_51", cache="bf16", decode=51, past_lo=512, past_hi=8192, layout=14),
        # one rank's share of a large step of a Llama-3-70B shape, block size 16, log-uniform contexts
        _attn("decode_u8_b16_128", hq=64, bs=16, decode=128, past_lo=1024, past_hi=32768, log_past=True, layout=15),
        # prompts in chunks over contexts already in the cache (Qwen2.5-7B shape)
        _attn("prefill_u8_16x512", hq=28, hkv=4, chunks=16, chunk_lo=512, chunk_hi=512, chunk_past_hi=8192, layout=16),
        # fresh prompts of ragged lengths, unquantised cache
        _attn("prefill_bf16_ragged", cache="bf16", chunks=9, chunk_lo=37, chunk_hi=2048, layout=17),
        # a mixed step with cache eviction on: chunks and decode rows, scores for the eviction policy, a tenth of the
        # blocks re-rotated
        _attn("mixed_u8_scores", hq=28, hkv=4, decode=240, past_lo=256, past_hi=16384, chunks=16, chunk_lo=256, chunk_hi=256,
              chunk_past_hi=4096, scores=True, rotated=0.1, layout=18),
        # a chat server's sampling: top-k, top-p, temperature, the three penalties over the generated history
        _samp("sample_topk_256", penalties=True, history=1024, layout=21),
        # the same options for a handful of requests on a small vocabulary
        _samp("sample_topk_5", rows=5, vocab=32000, penalties=True, history=200, layout=22),
        # nucleus sampling over the whole vocabulary, a rank's share of a large batch, flat logits
        _samp("sample_topp_128", rows=128, vocab=128256, mode="top_p", temperature=1.0, top_p=0.95, spikes=0, layout=23),
        # a batch whose requests differ: greedy, top-k, top-p and plain temperature rows side by side
        _samp("sample_mixed_200", rows=200, vocab=151936, mode="mixed", penalties=True, history=300, layout=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    layout = rng.randrange(1, 1 << 30)
    kind = rng.choice(["decode", "decode", "prefill", "mixed", "sampler", "sampler"])
    if kind == "sampler":
        mode = rng.choice(["top_k", "top_p", "mixed", "greedy"])
        pen = mode != "top_p" and rng.random() < 0.6
        return _samp(None, rows=_log_int(rng, 1, 256), vocab=_log_int(rng, 31999, 151936), mode=mode,
                     top_k=rng.choice([20, 40, 50, 64]), temperature=1.0 if mode == "top_p" else rng.choice([0.7, 0.8, 1.0]),
                     top_p=0.95 if mode == "top_p" else 0.9, penalties=pen, history=_log_int(rng, 30, 1024) if pen else 0,
                     spikes=rng.choice([0, 8]), layout=layout)
    hq, hkv, d, bs = rng.choice([(32, 4, 64, 32), (32, 8, 128, 32), (28, 4, 128, 32), (64, 8, 128, 16)])
    act, cache = rng.choice([("bf16", "u8"), ("bf16", "u8"), ("f16", "u8"), ("f16", "f16"), ("bf16", "bf16")])
    base = dict(hq=hq, hkv=hkv, d=d, bs=bs, act=act, cache=cache, layout=layout)
    if kind == "decode":
        n = _log_int(rng, 1, 192)
        most = 2000000 if cache == "u8" else 1000000              # total context: no more bytes than the largest listed step
        hi = min(32768, _log_int(rng, 300, most) // n + 200)
        lo = max(1, hi // rng.choice([2, 8, 16]))
        return _attn(None, decode=n, past_lo=lo, past_hi=max(lo, hi * 3 // 4), log_past=rng.random() < 0.5, **base)
    if kind == "prefill":
        chunk = _log_int(rng, 17, 1500)
        n = max(1, min(16, _log_int(rng, 17, 4096) // chunk))
        return _attn(None, chunks=n, chunk_lo=max(2, chunk // rng.choice([1, 3])), chunk_hi=chunk,
                     chunk_past_hi=rng.choice([0, _log_int(rng, 50, 6000)]), **base)
    n = _log_int(rng, 4, 120)
    chunk = _log_int(rng, 17, 256)
    return _attn(None, decode=n, past_lo=100, past_hi=_log_int(rng, 300, 12000), chunks=rng.randrange(1, 9), chunk_lo=max(2, chunk // 2),
                 chunk_hi=chunk, chunk_past_hi=_log_int(rng, 50, 4096), scores=True, rotated=rng.choice([0.0, 0.1]), **base)


# ---- attention: lengths, cache, inputs ---------------------------------------------------------------------------------
def _lengths(case):
    rng = np.random.default_rng(case["layout"])
    def spread(lo, hi, n, log):
        if n == 0:
            return np.zeros(0, np.int64)
        if log:
            return np.exp(rng.uniform(math.log(max(lo, 1)), math.log(max(hi, 1) + 1), size=n)).astype(np.int64)
        return rng.integers(lo, hi + 1, size=n)
    chunks = spread(case["chunk_lo"], case["chunk_hi"], case["chunks"], False)
    past = np.concatenate([spread(0, case["chunk_past_hi"], case["chunks"], False),
                           spread(case["past_lo"], case["past_hi"], case["decode"], case["log_past"])]).astype(np.int64)
    new = np.concatenate([np.maximum(chunks, 1), np.ones(case["decode"], np.int64)]).astype(np.int64)
    return past, new


def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFFFFFF)
    return g


def _quantise(x):
    """By-token asymmetric u8 of the last dimension: bytes, scale, zero-point (f32 steps as documented)."""
    mn, mx = x.amin(-1, keepdim=True), x.amax(-1, keepdim=True)
    scale = (mx - mn) / 255.0
    scale = torch.where(mx > mn, scale, torch.ones_like(scale))
    zp = -mn / scale
    inv = 1.0 / scale
    q = torch.round(x.double() * inv.double() + zp.double()).clamp_(0, 255).to(torch.uint8)
    return q, scale.squeeze(-1), zp.squeeze(-1)


def _record_bytes(case):
    return case["bs"] * (case["d"] + 8) if case["cache"] == "u8" else case["bs"] * case["d"] * 2


def _pack(case, x, value):
    """x f32 [blocks, Hkv, bs, D] -> the cache bytes [blocks, Hkv, record]."""
    n, h, bs, d = x.shape
    if case["cache"] != "u8":
        return x.to(ACT[case["cache"]]).contiguous().view(torch.uint8).reshape(n, h, -1)
    q, s, z = _quantise(x)
    if value:
        q = q.transpose(2, 3)
    return torch.cat([q.reshape(n, h, bs * d), s.contiguous().view(torch.uint8).reshape(n, h, 4 * bs),
                      z.contiguous().view(torch.uint8).reshape(n, h, 4 * bs)], dim=2)


def _unpack(case, rec, value):
    """Cache bytes [blocks, Hkv, record] -> f64 [blocks, Hkv, bs, D]."""
    n, h = rec.shape[:2]
    bs, d = case["bs"], case["d"]
    if case["cache"] != "u8":
        return rec.contiguous().view(ACT[case["cache"]]).reshape(n, h, bs, d).double()
    q = rec[:, :, :bs * d]
    q = q.reshape(n, h, d, bs).transpose(2, 3) if value else q.reshape(n, h, bs, d)
    s = rec[:, :, bs * d:bs * d + 4 * bs].contiguous().view(torch.float32).reshape(n, h, bs, 1)
    z = rec[:, :, bs * d + 4 * bs:].contiguous().view(torch.float32).reshape(n, h, bs, 1)
    return (q.double() - z.double()) * s.double()


def _attn_inputs(case, seed):
    past, new = _lengths(case)
    bs, hkv, d, B = case["bs"], case["hkv"], case["d"], len(past)
    nblk = (past + new + bs - 1) // bs
    total = int(nblk.sum())
    pool = total + total // 10 + 1
    rng = np.random.default_rng(int(seed) + 7)
    table = rng.permutation(pool)[:total].astype(np.int32)
    begins = np.concatenate([[0], np.cumsum(nblk)]).astype(np.int32)
    sub = np.concatenate([[0], np.cumsum(new)]).astype(np.int32)
    x = {"past": past, "new": new, "table": table, "begins": begins, "sub": sub, "pool": pool}
    rec = _record_bytes(case)
    g = _gen(seed, 1)
    for which in ("key_cache", "value_cache"):
        cache = torch.empty((pool, hkv, rec), dtype=torch.uint8, device=DEV)
        step = max(1, (1 << 26) // (hkv * bs * d))
        for b in range(0, pool, step):
            n = min(step, pool - b)
            cache[b:b + n] = _pack(case, torch.randn((n, hkv, bs, d), generator=g, device=DEV), which == "value_cache")
        x[which] = cache.reshape(-1)
    tokens, act = int(new.sum()), ACT[case["act"]]
    mk = lambda h: torch.randn((tokens, h * d), generator=g, device=DEV).to(act)
    x["query"], x["key"], x["value"] = mk(case["hq"]), mk(hkv), mk(hkv)
    x["scores_len"] = int((past + new).sum()) if case["scores"] else 0
    if case["scores"]:
        x["window"] = np.where(new > 1, np.minimum(8, new), 1).astype(np.int32)
    if case["rotated"] > 0:
        rot = []
        for s in range(B):
            full = int(past[s]) // bs
            k = int(full * case["rotated"])
            if k:
                rot.append(table[begins[s] + rng.choice(full, size=k, replace=False)])
        if rot:
            x["rot"] = np.concatenate(rot).astype(np.int32)
            x["delta"] = rng.integers(1, ROTATION_ROWS, size=len(x["rot"])).astype(np.int32)
            j = np.arange(d // 2, dtype=np.float64)
            ang = np.arange(ROTATION_ROWS, dtype=np.float64)[:, None] * bs * np.power(ROTATION_THETA, -2.0 * j / d)[None, :]
            x["lut"] = np.concatenate([np.cos(ang), -np.sin(ang)], axis=1).astype(np.float32)
    return x


def _prepare_attn(case, seed):
    x = _attn_inputs(case, seed)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    op = pkg.PagedAttentionExtension(case["hq"], case["hkv"], case["d"], case["bs"], ACT[case["act"]], case["cache"])
    inputs = {"query": x["query"], "key": x["key"], "value": x["value"], "key_cache": x["key_cache"], "value_cache": x["value_cache"],
              "past_lens": dev(x["past"].astype(np.int32)), "subsequence_begins": dev(x["sub"]), "block_indices": dev(x["table"]),
              "block_indices_begins": dev(x["begins"]), "max_context_len": int((x["past"] + x["new"]).max())}
    outputs = {"output": torch.empty_like(x["query"])}
    if case["scores"]:
        inputs["score_aggregation_window"] = dev(x["window"])
        outputs["scores"] = torch.zeros(x["scores_len"], dtype=torch.float32, device=DEV)
    if "rot" in x:
        inputs["rotated_block_indices"], inputs["rotation_deltas"], inputs["rotation_trig_lut"] = dev(x["rot"]), dev(x["delta"]), dev(x["lut"])
    return {"kind": "attn", "op": op, "inputs": inputs, "outputs": outputs}


def _exact_attn(case, seed):
    x = _attn_inputs(case, seed)
    bs, hkv, hq, d = case["bs"], case["hkv"], case["hq"], case["d"]
    G = hq // hkv
    shape = (x["pool"], hkv, _record_bytes(case))
    kc, vc = x["key_cache"].view(shape), x["value_cache"].view(shape)
    if "rot" in x:
        for b in range(0, len(x["rot"]), 1024):
            idx = torch.from_numpy(x["rot"][b:b + 1024].astype(np.int64)).to(DEV)
            row = torch.from_numpy(x["lut"][x["delta"][b:b + 1024]]).to(DEV).view(-1, 1, 1, d)
            c, s = row[..., :d // 2], row[..., d // 2:]
            k = _unpack(case, kc[idx], False)
            k = k.float()
            lo, hi = k[..., :d // 2], k[..., d // 2:]
            n_lo = ((-hi).double() * s.double() + (lo * c).double()).float()
            n_hi = (lo.double() * s.double() + (hi * c).double()).float()
            kc[idx] = _pack(case, torch.cat([n_lo, n_hi], -1), False)
    out = torch.empty((int(x["new"].sum()), hq, d), dtype=torch.float64, device=DEV)
    scores = torch.zeros(x["scores_len"], dtype=torch.float64, device=DEV)
    off = 0
    for s in range(len(x["past"])):
        p, n, t0 = int(x["past"][s]), int(x["new"][s]), int(x["sub"][s])
        idx = torch.from_numpy(x["table"][x["begins"][s]:x["begins"][s + 1]].astype(np.int64)).to(DEV)
        kv = []
        for cache, act, value in ((kc, x["key"], False), (vc, x["value"], True)):
            new = act[t0:t0 + n].float().view(n, hkv, 1, d).transpose(1, 2).reshape(n, 1, hkv, d)
            new = new.permute(0, 2, 1, 3)                      # [n, Hkv, 1, D]
            if case["cache"] == "u8":
                q, sc, zp = _quantise(new)
                new = (q.double() - zp.double().unsqueeze(-1)) * sc.double().unsqueeze(-1)
            else:
                new = new.to(ACT[case["cache"]]).double()
            old = _unpack(case, cache[idx], value).permute(1, 0, 2, 3).reshape(hkv, -1, d)[:, :p]
            kv.append(torch.cat([old, new.reshape(n, hkv, d).transpose(0, 1)], 1))
        q = x["query"][t0:t0 + n].double().view(n, hkv, G, d).permute(1, 2, 0, 3)     # [Hkv, G, n, D]
        w = int(x["window"][s]) if case["scores"] else 0
        acc = torch.zeros(p + n, dtype=torch.float64, device=DEV)
        for h in range(hkv):
            a = torch.matmul(q[h].reshape(G * n, d), kv[0][h].T).view(G, n, p + n) / math.sqrt(d)
            if n > 1:
                a.masked_fill_(torch.arange(p + n, device=DEV)[None, :] > p + torch.arange(n, device=DEV)[:, None], -math.inf)
            a = torch.softmax(a, -1)
            out[t0:t0 + n, h * G:(h + 1) * G] = torch.matmul(a.view(G * n, p + n), kv[1][h]).view(G, n, d).transpose(0, 1)
            if w:
                acc += a[:, n - w:].sum((0, 1))
        if w:
            scores[off:off + p + n] = acc
            off += p + n
    res = {"output": out.view(-1, hq * d), "key_cache": None, "value_cache": None}
    if case["scores"]:
        res["scores"] = scores
    return res


# ---- sampler -------------------------------------------------------------------------------------------------------------
def _row_modes(case):
    """Per row: does it sample, its top_k (0 = off), its top_p."""
    n, mode = case["rows"], case["mode"]
    kinds = [("greedy", "top_k", "top_p", "temperature")[i % 4] for i in range(n)] if mode == "mixed" else [mode] * n
    return [(k != "greedy", case["top_k"] if k == "top_k" else 0, case["top_p"] if k in ("top_k", "top_p") else 1.0) for k in kinds]


def _sampler_inputs(case, seed):
    n, V = case["rows"], case["vocab"]
    g = _gen(seed, 2)
    logits = torch.randn((n, V), generator=g, device=DEV) * 2.0
    rng = np.random.default_rng(int(seed) + 9)
    if case["spikes"]:
        at = torch.from_numpy(np.stack([rng.choice(V, size=case["spikes"], replace=False) for _ in range(n)])).to(DEV)
        logits.scatter_add_(1, at, torch.full(at.shape, 15.0, device=DEV))
    hist = None
    if case["history"]:
        offs, ids, meta = [0], [], []
        for _ in range(n):
            uniq, count = np.unique(rng.integers(0, V, size=case["history"]), return_counts=True)
            ids.append(uniq)
            meta.append((count << 3) | sampler_abi.HIST_GENERATED)
            offs.append(offs[-1] + len(uniq))
        hist = (np.array(offs, np.int64), np.concatenate(ids).astype(np.int32), np.concatenate(meta).astype(np.uint32))
    par = np.zeros(n, dtype=np.dtype(sampler_abi.ROW_DTYPE))
    par["logits_row"] = np.arange(n)
    par["repetition_penalty"] = 1.1 if case["penalties"] else 1.0
    par["presence_penalty"] = 0.2 if case["penalties"] else 0.0
    par["frequency_penalty"] = 0.1 if case["penalties"] else 0.0
    par["rand_u"] = rng.random(n, dtype=np.float32)
    for r, (sample, top_k, top_p) in enumerate(_row_modes(case)):
        par["do_sample"][r] = 1 if sample else 0
        par["temperature"][r] = case["temperature"] if sample else 1.0
        par["top_k"][r] = top_k if top_k else sampler_abi.TOP_K_OFF
        par["top_p"][r] = top_p if sample else 1.0
    return logits, par, hist


def _prepare_sampler(case, seed):
    logits, par, hist = _sampler_inputs(case, seed)
    step = sampler_mod.SamplerStep(0)
    state = {"kind": "sampler", "step": step, "staged": step.stage(par, hist), "logits": logits, "at": None}
    if hist is not None:
        # the step applies the penalties in place, on logits that the model writes anew before every step: the entries
        # it changes are written back before each pass
        flat = np.repeat(np.arange(case["rows"], dtype=np.int64), np.diff(hist[0])) * case["vocab"] + hist[1]
        state["at"] = torch.from_numpy(flat).to(DEV)
        state["fresh"] = logits.view(-1)[state["at"]].clone()
    return state


def _exact_sampler(case, seed):
    logits, par, hist = _sampler_inputs(case, seed)
    n = case["rows"]
    x = logits.double().cpu().numpy()
    if hist is not None:
        for r in range(n):
            a, b = hist[0][r], hist[0][r + 1]
            ids, count = hist[1][a:b], (hist[2][a:b] >> 3).astype(np.float64)
            v = x[r, ids]
            rep, pres, freq = (float(par[k][r]) for k in ("repetition_penalty", "presence_penalty", "frequency_penalty"))
            v = np.where(v >= 0, v / rep, v * rep)
            v = np.where(v >= 0, v - pres, v + pres)
            v = np.where(v >= 0, v - freq * count, v + freq * count)
            x[r, ids] = v
    res = {"tokens": None, "log_probs": None}
    if case["mode"] == "greedy":
        res["tokens"] = x.argmax(1)
    if case["mode"] == "top_k":
        # softmax of the K largest, the shortest descending prefix above top_p, the draw by inverse transform
        lp = np.zeros(n)
        for r in range(n):
            top = np.sort(np.partition(x[r], -case["top_k"])[-case["top_k"]:])[::-1]
            p = np.exp((top - top[0]) * (1.0 / float(par["temperature"][r])))
            p /= p.sum()
            keep = int(np.argmax(np.cumsum(p) > float(par["top_p"][r]))) + 1
            c = np.cumsum(p[:keep])
            pick = min(int(np.searchsorted(c, c[-1] * float(par["rand_u"][r]), side="right")), keep - 1)
            lp[r] = math.log(p[pick] / c[-1])
        res["log_probs"] = lp
    if hist is not None:
        res["logits"] = torch.from_numpy(x).to(DEV)
    return res


# ---- the interface -----------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    return _prepare_attn(case, seed) if case["kind"] == "attn" else _prepare_sampler(case, seed)


def run(state):
    if state["kind"] == "attn":
        state["op"].evaluate(state["inputs"], state["outputs"])
        res = {"output": state["outputs"]["output"], "key_cache": state["inputs"]["key_cache"], "value_cache": state["inputs"]["value_cache"]}
        if "scores" in state["outputs"]:
            res["scores"] = state["outputs"]["scores"]
        return res
    if state["at"] is not None:
        state["logits"].view(-1).index_copy_(0, state["at"], state["fresh"])
    tokens, log_probs = state["step"].step(state["logits"], state["staged"])
    res = {"tokens": tokens, "log_probs": log_probs}
    if state["at"] is not None:
        res["logits"] = state["logits"]
    return res


def work(case):
    if case["kind"] == "sampler":
        # every logit once, the history read and its logits written
        return {"bytes": 4 * case["rows"] * case["vocab"] + 12 * case["rows"] * case["history"] + 60 * case["rows"], "flops": 0}
    past, new = _lengths(case)
    hq, hkv, d, bs = case["hq"], case["hkv"], case["d"], case["bs"]
    act = 4 if case["act"] == "f32" else 2
    per = d + 8 if case["cache"] == "u8" else 2 * d
    tokens = int(new.sum())
    bytes_ = int(past.sum()) * 2 * hkv * per + tokens * 2 * hkv * per + tokens * (2 * hq + 2 * hkv) * d * act
    if case["scores"]:
        bytes_ += 4 * int((past + new).sum())
    if case["rotated"] > 0:
        bytes_ += 2 * hkv * bs * per * int(sum(int((int(p) // bs) * case["rotated"]) for p in past))
    flops = 4 * hq * d * int((new * past + new * (new + 1) // 2).sum())
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    if case["kind"] == "sampler":
        return {"rel": 1e-6}          # ids are whole values: none may differ
    # four times the measured distance to the 64-bit result (1.6e-3 .. 2.3e-3 with bf16 output, 4e-4 with f16 throughout;
    # probabilities in f16 over the u8 cache)
    return {"rel": 8e-3 if case["act"] == "bf16" or case["cache"] == "u8" else 1.6e-3}


def exact(case, seed):
    if case["kind"] == "sampler":
        # nucleus rows over a whole vocabulary follow the float sums' own rounding: no 64-bit value to compare with
        return None if case["mode"] == "top_p" else _exact_sampler(case, seed)
    return _exact_attn(case, seed)
