"""The work a decode loop has this library do, as cases that can be timed one by one.

A case names an entry point (`path`), a block of logits (`rows` x `vocab`), how the rows are
sampled (`settings`) and the options of the call. The five families of settings are the ones the
benchmark configurations use, plus the two defaults of a sampler: greedy, and a temperature alone.

    greedy   temperature 0: what a request that says nothing gets
    chat     temperature 0.7, top-k 40, top-p 0.9, repetition penalty 1.1 over a short window
    nucleus  temperature 1, top-p 0.95, presence and frequency penalties over a long, repetitive window
    mixed    every row its own: temperature 0..1.5 (some greedy), top-k 0..100, top-p 0.5..1, some
             min-p, some typical-p, repetition penalties: the streams of a shared server
    wide     temperature 0.9, top-k 1024, top-p 0.99 over rows with a few dominant tokens
    open     temperature 1 and nothing else

Logits are 3 N(0,1) - 1.2 ln(1 + rank) with a random rank per token: a heavy head over a long noisy
tail, the shape of a language model's logit row.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from molla_b200 import sampler as S

DEVICE = "cuda:0"
MAX_LOGITS = 1 << 28   # no case is larger than 1024 rows of 262144


def listed():
    return [
        # one stream through the host-side sampler object, one token at a time: pure call latency
        dict(name="pick-1x32000-chat", path="pick", rows=1, vocab=32000, settings="chat", window=64),
        # a small server's streams through the batched form of the same loop
        dict(name="pick-24x49152-mixed", path="pick", rows=24, vocab=49152, settings="mixed", window=64),
        # one stream with its state on the device: the shortest decode step there is
        dict(name="step-1x128256-chat", path="step", rows=1, vocab=128256, settings="chat", window=64, softcap=0.0),
        # a few streams of a model that caps its final logits, the largest vocabulary in use
        dict(name="step-16x262144-mixed-softcap", path="step", rows=16, vocab=262144, settings="mixed", window=256,
             softcap=30.0),
        # greedy decoding of a full batch: one maximum per row
        dict(name="batch-128x128256-greedy", path="batch", rows=128, vocab=128256, settings="greedy", window=0, top_n=0),
        # plain sampling, and a vocabulary whose rows do not start on 16-byte boundaries
        dict(name="batch-48x50257-open", path="batch", rows=48, vocab=50257, settings="open", window=0, top_n=0),
        # a wide nucleus with penalties over a long window, logprobs in the response
        dict(name="batch-64x151936-nucleus-top5", path="batch", rows=64, vocab=151936, settings="nucleus", window=512,
             top_n=5),
        # the batch of a shared server, every row with its own settings
        dict(name="batch-256x151936-mixed", path="batch", rows=256, vocab=151936, settings="mixed", window=256, top_n=0),
        # the largest block, with a wide top-k
        dict(name="batch-1024x262144-wide", path="batch", rows=1024, vocab=262144, settings="wide", window=0, top_n=0),
        # constrained decoding: a grammar allows a part of the vocabulary
        dict(name="mask-32x151936-chat", path="mask", rows=32, vocab=151936, settings="chat", window=64, allowed=0.1),
        # a caller that still holds its logits in host memory
        dict(name="host-32x128256-mixed", path="host", rows=32, vocab=128256, settings="mixed", window=64, top_n=0),
        # logprobs of whole rows: scoring a prompt
        dict(name="logprobs-64x128256", path="logprobs", rows=64, vocab=128256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: any entry point, vocabularies of 2000 to 262144 (odd ones
    among them), one row up to what fits the largest block."""
    path = rng.choice(["pick", "step", "batch", "batch", "batch", "batch", "mask", "host", "logprobs"])
    vocab = _log_int(rng, 2000, 262144)
    if rng.random() < 0.5:
        vocab = max(2000, vocab // 64 * 64)   # most models pad their vocabulary, some do not
    top = {"pick": 64, "step": 512, "batch": 1024, "mask": 256, "host": 64, "logprobs": 512}[path]
    rows = min(_log_int(rng, 1, top), MAX_LOGITS // vocab)
    case = dict(path=path, rows=rows, vocab=vocab)
    if path == "logprobs":
        return case
    case["settings"] = rng.choice(["greedy", "chat", "nucleus", "mixed", "mixed", "wide", "open"])
    case["window"] = {"greedy": 0, "open": 0, "wide": 0, "chat": 64, "nucleus": _log_int(rng, 64, 1024),
                      "mixed": _log_int(rng, 16, 512)}[case["settings"]]
    if path == "step":
        case["softcap"] = rng.choice([0.0, 0.0, 30.0])
    elif path in ("batch", "host"):
        case["top_n"] = rng.choice([0, 0, 1, 5, 20])
    elif path == "mask":
        case["allowed"] = round(math.exp(rng.uniform(math.log(0.01), math.log(0.9))), 3)
    return case


# ---- inputs --------------------------------------------------------------------------------------

def _logits(rows, vocab, seed, boost):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    x = torch.rand((rows, vocab), generator=gen, device=DEVICE).mul_(vocab).floor_().log1p_().mul_(-1.2)
    x.add_(torch.randn((rows, vocab), generator=gen, device=DEVICE), alpha=3.0)
    if boost:
        at = torch.randint(0, vocab, (rows, boost), generator=gen, device=DEVICE)
        x.scatter_(1, at, x.gather(1, at) + 12.0)
    return x


def _settings(kind, rows, rng):
    """The fields of SamplerConfig, one array each."""
    p = dict(temperature=np.zeros(rows, np.float32), top_k=np.zeros(rows, np.int32), top_p=np.ones(rows, np.float32),
             min_p=np.zeros(rows, np.float32), typical_p=np.ones(rows, np.float32),
             repeat_penalty=np.ones(rows, np.float32), frequency_penalty=np.zeros(rows, np.float32),
             presence_penalty=np.zeros(rows, np.float32))
    if kind == "chat":
        p["temperature"][:], p["top_k"][:], p["top_p"][:], p["repeat_penalty"][:] = 0.7, 40, 0.9, 1.1
    elif kind == "nucleus":
        p["temperature"][:], p["top_p"][:] = 1.0, 0.95
        p["presence_penalty"][:], p["frequency_penalty"][:] = 0.5, 0.3
    elif kind == "mixed":
        p["temperature"][:] = rng.uniform(0.0, 1.5, rows)
        p["temperature"][::16] = 0.0
        p["top_k"][:] = rng.choice(np.array([0, 1, 20, 50, 100], np.int32), size=rows)
        p["top_p"][:] = np.minimum(rng.uniform(0.5, 1.0, rows).astype(np.float32), np.float32(1.0))
        p["min_p"][3::8] = 0.05
        p["typical_p"][(np.arange(rows) % 8 == 5) & (p["top_k"] > 1)] = 0.9
        p["repeat_penalty"][:] = rng.uniform(1.0, 1.3, rows)
    elif kind == "wide":
        p["temperature"][:], p["top_k"][:], p["top_p"][:] = 0.9, 1024, 0.99
    elif kind == "open":
        p["temperature"][:] = 1.0
    return p


def _windows(kind, rows, vocab, window, rng):
    if kind == "nucleus":   # a repetitive text: token frequencies follow a power law
        rank = np.minimum(rng.zipf(1.1, size=(rows, window)), vocab) - 1
        return (rank * 7919 + rng.integers(0, vocab, size=(rows, 1))) % vocab
    return rng.integers(0, vocab, size=(rows, window))


def _arrays(case, seed):
    """The parallel arrays of the batched entry points."""
    rows, vocab, window = case["rows"], case["vocab"], case["window"]
    rng = np.random.default_rng(seed)
    w = _settings(case["settings"], rows, rng)
    w["seed"] = rng.integers(0, 2**63, size=rows, dtype=np.uint64)
    w["drawn"] = rng.integers(0, 4096, size=rows).astype(np.uint64)
    w["window_on"] = np.full(rows, 1 if window else 0, np.uint8)
    w["hist"] = _windows(case["settings"], rows, vocab, window, rng).reshape(-1).astype(np.int64)
    w["hist_off"] = (np.arange(rows + 1) * window).astype(np.int32)
    return w


def prepare(case, seed):
    path, rows, vocab = case["path"], case["rows"], case["vocab"]
    logits = _logits(rows, vocab, seed, 8 if case.get("settings") == "wide" else 0)
    state = dict(path=path, logits=logits)
    if path == "logprobs":
        return state
    if path in ("batch", "mask"):
        w = _arrays(case, seed)
        state["params"] = S.upload_params(w, DEVICE)
        state["top_n"] = case.get("top_n", 0)
        state["workspace"] = S.Workspace(rows, vocab, state["top_n"], DEVICE)
        if path == "mask":
            gen = torch.Generator(device=DEVICE)
            gen.manual_seed(seed + 1)
            words = (vocab + 31) // 32
            bits = (torch.rand((rows, words, 32), generator=gen, device=DEVICE) < case["allowed"]).to(torch.int32)
            bits[:, 0, :4] = 1   # a grammar allows at least something
            shift = torch.arange(32, device=DEVICE, dtype=torch.int32)
            state["params"]["mask"] = torch.bitwise_left_shift(bits, shift).sum(2, dtype=torch.int32).contiguous()
    elif path == "host":
        w = _arrays(case, seed)
        w["logits"] = logits.cpu().numpy()
        state["block"] = S.HostBlock(w, DEVICE, top_n=case["top_n"], want_logprob=case["top_n"] > 0)
        del state["logits"]
    else:
        w = _arrays(case, seed)
        window = case["window"]
        configs = [S.SamplerConfig(temperature=float(w["temperature"][r]), top_k=int(w["top_k"][r]),
                                   top_p=float(w["top_p"][r]), min_p=float(w["min_p"][r]),
                                   typical_p=float(w["typical_p"][r]), repeat_penalty=float(w["repeat_penalty"][r]),
                                   frequency_penalty=float(w["frequency_penalty"][r]),
                                   presence_penalty=float(w["presence_penalty"][r]), repeat_last_n=window,
                                   seed=int(w["seed"][r])) for r in range(rows)]
        if path == "pick":
            state["samplers"] = [S.Sampler(c, vocab, device=DEVICE) for c in configs]
            for r, s in enumerate(state["samplers"]):
                for t in w["hist"][r * window:(r + 1) * window]:
                    s.observe(int(t))
        else:
            ds = S.DeviceSamplers(rows, vocab, ring_cap=max(window, 1), device=DEVICE)
            for r, c in enumerate(configs):
                ds.assign(r, c, stop_token=2)
            if window:
                ds.ring.copy_(torch.from_numpy(w["hist"].reshape(rows, window)))
                ds.ring_filled.fill_(window)
            rng = np.random.default_rng(seed + 2)
            order = lambda: torch.from_numpy(rng.permutation(rows).astype(np.int32)).to(DEVICE)
            state.update(samplers=ds, rows=order(), slots=order(), softcap=case["softcap"])
    return state


# ---- one pass ------------------------------------------------------------------------------------

def run(state):
    path = state["path"]
    if path == "logprobs":
        return S.logprobs_block(state["logits"])
    if path == "pick":
        return np.array(S.pick_rows(state["logits"], state["samplers"]), np.int64)
    if path == "host":
        hb = state["block"]
        S.sample_batch_host(hb)
        out = dict(tokens=hb.tokens, row_status=hb.status)
        if hb.top_n:
            out.update(chosen_logprob=hb.chosen, top_ids=hb.top_ids, top_logprobs=hb.top_lps)
        return out
    if path == "step":
        ds = state["samplers"]
        out = ds.step(state["logits"], state["rows"], state["slots"], final_softcap=state["softcap"])
        out = {k: v for k, v in out.items() if v is not None}
        out.update(drawn=ds.drawn, ring=ds.ring, ring_head=ds.ring_head, ring_filled=ds.ring_filled)
        return out
    out = S.sample_batch(state["logits"], state["params"], top_n=state["top_n"], want_logprob=state["top_n"] > 0,
                         workspace=state["workspace"])
    return {k: v for k, v in out.items() if v is not None}


def work(case):
    """One read of the logits (and of the mask), of the windows and of about 48 bytes of settings a
    row; the answers written once. Per logit a comparison and, where the row is sampled or its
    logprobs are wanted, an exponential and an addition."""
    rows, vocab, path = case["rows"], case["vocab"], case["path"]
    n = rows * vocab
    if path == "logprobs":
        return dict(bytes=8 * n, flops=4 * n)
    top_n = case.get("top_n", 0)
    out = 8 * rows + (4 * rows * (1 + 2 * top_n) if top_n else 0)
    mask = rows * ((vocab + 31) // 32) * 4 if path == "mask" else 0
    flops = n * (1 if case["settings"] == "greedy" and not top_n else 3)
    return dict(bytes=4 * n + mask + rows * (8 * case["window"] + 48) + out, flops=flops)


def tolerance(case):
    """Tokens, status words, windows and counters are the same whatever computes them. Logprobs are
    fp32 results of a sum over the vocabulary."""
    if case["path"] == "logprobs" or case.get("top_n", 0):
        return dict(rel=2e-6, max=1e-5)
    return "exact"
