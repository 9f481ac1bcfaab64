"""The decode-step form of the sampler (`molla_sample_decode_step`): logit rows picked by
`rows[]`, settings and state per sampler slot kept on the device, the final-logit softcap
fused into the read. Checked against oracle-backed samplers that keep their state on the host
the way the reference's `Sampler` does (src/molla/engine/sample.mojo:157-363) and, for the
softcap, against the oracle's restatement of the reference's device kernel
(src/molla/nn/gpu_ops.mojo:302-317, :607-623) applied to the block beforehand."""
import numpy as np
import pytest
import torch

from helpers import ROUTES, OracleSampler
from molla_b200 import capi, sampler as S

pytestmark = pytest.mark.gpu

CONFIGS = [
    dict(),                                                                    # greedy, window of 64 cut to the capacity
    dict(frequency_penalty=0.4, presence_penalty=0.2, repeat_last_n=8),        # greedy with penalties
    dict(temperature=0.8, top_k=40, top_p=0.9, repeat_penalty=1.2, repeat_last_n=16, seed=5),
    dict(temperature=1.0, top_p=0.95, seed=6, repeat_last_n=0),                # no window at all
    dict(temperature=1.3, seed=7, repeat_last_n=4, frequency_penalty=0.1),     # nothing sorted
    dict(temperature=0.7, top_k=20, min_p=0.05, seed=8, repeat_last_n=16, presence_penalty=0.5),
    dict(temperature=0.9, top_k=12, typical_p=0.8, seed=9, repeat_last_n=8),
    dict(temperature=1.1, top_k=1, seed=10, repeat_last_n=16, repeat_penalty=1.3),
    dict(temperature=0.5, top_p=0.5, seed=11, repeat_last_n=16),
    dict(temperature=2.0, top_k=300, top_p=0.99, seed=12, repeat_last_n=16, repeat_penalty=1.1),
]


def make(dev, oracle, V, ring_cap):
    ds = S.DeviceSamplers(len(CONFIGS), V, ring_cap=ring_cap, device=dev)
    host = []
    for slot, kw in enumerate(CONFIGS):
        kw = dict(kw)
        kw["repeat_last_n"] = min(kw.get("repeat_last_n", 64), ring_cap)
        bias = [(3, 2.5), (3, 0.5), (V - 1, -4.0)] if slot in (2, 5) else []
        ds.assign(slot, S.SamplerConfig(**kw), stop_token=7 if slot % 2 == 0 else -1, bias=bias)
        o = OracleSampler(oracle, V, **kw)
        for t, a in bias:
            o.bias(t, a)
        host.append(o)
    return ds, host


@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("softcap", [0.0, 30.0])
def test_decode_steps_match_host_kept_samplers(dev, lib, oracle, softcap):
    V, ring_cap, n_block = 3000, 16, 14
    ds, host = make(dev, oracle, V, ring_cap)
    rng = np.random.default_rng(77)
    for step in range(9):
        block = (3.0 * rng.standard_normal((n_block, V))).astype(np.float32)
        block[:, 7] += 4.0  # the stop token turns up now and then
        active = rng.permutation(len(CONFIGS))[: 6 + step % 4]
        rows = rng.permutation(n_block)[: len(active)]
        got = ds.step(torch.from_numpy(block).to(dev), torch.tensor(rows, dtype=torch.int32, device=dev),
                      torch.tensor(active, dtype=torch.int32, device=dev), final_softcap=softcap, want_logprob=True)
        torch.cuda.synchronize()
        st = got["row_status"].cpu().numpy()
        assert not np.any(st & np.uint32(capi.ROW_ERROR_BITS)), st
        seen = oracle.softcap(block, softcap) if softcap > 0 else block
        tok = got["tokens"].cpu().numpy()
        stopped = got["stopped"].cpu().numpy()
        lp = oracle.logprobs_batch(seen[rows], tokens=tok, top_n=0)
        assert np.max(np.abs(got["chosen_logprob"].cpu().numpy() - lp["chosen_logprob"])) <= 1e-5
        for i, slot in enumerate(active):
            want = host[slot].pick(seen[rows[i]])
            tie = st[i] & np.uint32(capi.ROW_TIE_BITS)
            if not tie:
                assert tok[i] == want, (step, slot, tok[i], want)
            elif tok[i] != want and host[slot].recent:  # keep the two histories the same past an order-dependent pick
                h = host[slot]
                h.recent[(h.head - 1) % len(h.recent)] = int(tok[i])
            assert stopped[i] == (1 if (slot % 2 == 0 and tok[i] == 7) else 0)
        # the state the kernel left is the state the host samplers are in
        drawn = ds.drawn.cpu().numpy()
        head, filled, ring = ds.ring_head.cpu().numpy(), ds.ring_filled.cpu().numpy(), ds.ring.cpu().numpy()
        for slot, h in enumerate(host):
            assert drawn[slot] == h.drawn
            assert filled[slot] == h.filled and (head[slot] == h.head or not h.recent)
            assert ring[slot, : h.filled].tolist() == h.recent[: h.filled]


@pytest.mark.usefixtures("route")
def test_softcap_alone_gives_the_oracles_tokens_and_logprobs(dev, lib, oracle):
    """Greedy tokens and their logprobs of capped rows (no penalties, no bias). The capped values bit for bit: below."""
    V = 5000
    rng = np.random.default_rng(3)
    block = (40.0 * rng.standard_normal((4, V))).astype(np.float32)
    ds = S.DeviceSamplers(4, V, ring_cap=8, device=dev)
    for slot in range(4):
        ds.assign(slot, S.SamplerConfig(repeat_last_n=8))  # greedy
    got = ds.step(torch.from_numpy(block).to(dev), None, None, final_softcap=50.0, want_logprob=True)
    capped = oracle.softcap(block, 50.0)
    assert got["tokens"].cpu().numpy().tolist() == [int(np.argmax(r)) for r in capped]
    lp = oracle.logprobs_batch(capped, tokens=got["tokens"].cpu().numpy(), top_n=0)
    assert np.max(np.abs(got["chosen_logprob"].cpu().numpy() - lp["chosen_logprob"])) <= 1e-5
    assert np.all(np.abs(capped) <= 50.0)


def test_softcap_quotients_are_the_divisions(dev, lib):
    """(1 - e) / (1 + e) by a reciprocal, for every float e from 0 to 1."""
    with capi.testing_library() as T:
        assert T.molla_sample_debug_softcap_quotients() == 0


@pytest.mark.parametrize("cap", [1e-38, 9.0e-13, 9.2e-13, 1e-3, 1.0, 30.0, 50.0, 1e5, 1.09e12, 1.2e12, 1e38])
def test_softcap_four_at_a_time_is_the_oracles(dev, lib, oracle, cap):
    """Over every exponent, subnormal and infinite logits included, and around the cap. (Zeros are equal whatever their
    sign: a subnormal logit's depends on how x / cap is rounded, and nothing distinguishes them.)"""
    cap = np.float32(cap)
    rng = np.random.default_rng(1)
    bits = np.concatenate([np.arange(0, 2 ** 31, 20011, dtype=np.uint32), np.arange(300, dtype=np.uint32), [0x7f800000, 0x7f7fffff, 0x7fc00000]]).astype(np.uint32)
    x = np.concatenate([bits, bits | np.uint32(1 << 31)]).view(np.float32)
    x = np.concatenate([x, (min(float(cap), 1e37) * rng.uniform(-12, 12, 100001)).astype(np.float32)])
    at, out = torch.from_numpy(x).to(dev), torch.empty(x.size, device=dev)
    with capi.testing_library() as T:
        T.molla_sample_debug_softcap(at.data_ptr(), x.size, float(cap), out.data_ptr())
    got, ref = out.cpu().numpy(), oracle.softcap(x, float(cap))
    assert np.array_equal(got, ref, equal_nan=True)   # (of finite floats only the two zeros are equal without being the same)


def test_bad_arguments_are_refused_before_any_launch(dev, lib):
    ds = S.DeviceSamplers(2, 100, ring_cap=8, device=dev)
    ds.assign(0, S.SamplerConfig(repeat_last_n=8))
    ds.assign(1, S.SamplerConfig(repeat_last_n=0))
    with pytest.raises(ValueError):
        ds.assign(0, S.SamplerConfig(repeat_last_n=9))
    with pytest.raises(ValueError):
        ds.assign(5, S.SamplerConfig(repeat_last_n=8))
    with pytest.raises(ValueError):
        ds.step(torch.zeros((2, 99), device=dev), None, None)
    with pytest.raises(capi.MollaSampleError):
        ds.step(torch.zeros((2, 100), device=dev), None, None, final_softcap=-1.0)


@pytest.mark.usefixtures("route")
def test_stale_row_and_slot_indices_touch_nothing(dev, lib):
    """`pick` refuses a row outside the block (sample.mojo:316-322). The device form reports such a
    row (and a slot outside the samplers) in its status word and reads and writes nothing of it.
    The tensors here are larger than the sizes declared to the call, so that a missing check would
    land in owned memory rather than fault."""
    V, declared_rows, declared_slots = 1000, 4, 3
    ds = S.DeviceSamplers(8, V, ring_cap=8, device=dev)          # 8 slots allocated, 3 declared
    for slot in range(8):
        ds.assign(slot, S.SamplerConfig(temperature=0.8, top_k=10, seed=slot, repeat_last_n=8))
    ds.n_slots = declared_slots
    block = torch.randn((8, V), device=dev)                      # 8 rows allocated, 4 declared
    rows = torch.tensor([0, 5, 2, -1, 3], dtype=torch.int32, device=dev)
    slots = torch.tensor([0, 1, 6, 2, 2], dtype=torch.int32, device=dev)
    before = {k: getattr(ds, k).clone() for k in ("drawn", "ring", "ring_head", "ring_filled")}
    got = ds.step(block[:declared_rows], rows, slots, want_logprob=True, top_n=3)
    torch.cuda.synchronize()
    st = got["row_status"].cpu().numpy().astype(np.uint32)
    tok = got["tokens"].cpu().numpy()
    for i in (1, 2, 3):   # row 5 of 4, slot 6 of 3, row -1
        assert st[i] & capi.ROW_INVALID_CONFIG and tok[i] == -1, (i, st[i], tok[i])
    assert st[0] == 0 and tok[0] >= 0 and (st[4] & capi.ROW_ERROR_BITS) == 0 and tok[4] >= 0
    drawn = ds.drawn.cpu().numpy()
    assert drawn[0] == 1 and drawn[2] == 1 and drawn[1] == 0 and drawn[6] == 0
    for k in ("ring", "ring_head", "ring_filled"):
        assert torch.equal(getattr(ds, k)[[1, 6]], before[k][[1, 6]]), k
    assert np.all(got["top_ids"].cpu().numpy()[[1, 3]] == -1)


@pytest.mark.parametrize("switch", [0, ROUTES["tiles"], ROUTES["clusters"]])
def test_a_wait_that_ran_out_fails_the_row_and_keeps_its_state(dev, lib, switch):
    """The bounded wait on a row's load reports in one warp only. The testing build can pretend
    that it ran out (nothing is withheld, nothing is left waiting): every such row must come back
    with MOLLA_ROW_LOAD_TIMEOUT and token -1, and the sampler in its slot must be as it was."""
    V = 20000
    ds = S.DeviceSamplers(4, V, ring_cap=8, device=dev)
    for slot in range(4):
        ds.assign(slot, S.SamplerConfig(temperature=0.0 if slot == 0 else 0.9, top_k=[0, 1, 20, 0][slot],
                                        top_p=0.9, seed=slot, repeat_last_n=8))
    block = torch.randn((4, V), device=dev)
    before = {k: getattr(ds, k).clone() for k in ("drawn", "ring", "ring_head", "ring_filled")}
    with capi.testing_library() as T:
        T.molla_sample_debug_knobs(16 | switch)
        try:
            got = ds.step(block, None, None)
            torch.cuda.synchronize()
        finally:
            T.molla_sample_debug_knobs(0)
    st = got["row_status"].cpu().numpy().astype(np.uint32)
    assert np.all(st & capi.ROW_LOAD_TIMEOUT), st
    assert np.all(got["tokens"].cpu().numpy() == -1)
    for k, v in before.items():
        assert torch.equal(getattr(ds, k), v), k
    # and the same samplers work on the next call
    got = ds.step(block, None, None)
    torch.cuda.synchronize()
    assert not np.any(got["row_status"].cpu().numpy().astype(np.uint32) & capi.ROW_ERROR_BITS)
    assert np.all(ds.drawn.cpu().numpy() == 1)


def test_status_words_follow_the_window_the_row_was_sampled_with(dev, lib):
    """Rows whose running sum jumps (2^-48 before the largest term) are looked at once more after their token is
    known, for MOLLA_ROW_SLOW_PATH. The window is full and holds one token, which the answer replaces: it is
    ten above everything else unless its penalty is taken off. The same rows with their windows as lists, which no
    call writes to, say what the status words are."""
    B, V = 256, 8192   # (more rows than the chip holds clusters: the tile kernels)
    rng = np.random.default_rng(11)
    x = rng.uniform(-47.0, -40.0, (B, V)).astype(np.float32)
    top = rng.integers(V // 4, V, B)
    old = rng.integers(0, V // 4, B)
    x[np.arange(B), top] = 0.0
    x[np.arange(B), old] = 10.0
    logits = torch.from_numpy(x).to(dev)
    ds = S.DeviceSamplers(B, V, ring_cap=1, device=dev)
    for r in range(B):
        ds.assign(r, S.SamplerConfig(temperature=1.0, top_k=[40, 0, 0][r % 3], top_p=[0.9, 1.0, 0.999][r % 3],
                                     presence_penalty=60.0, repeat_last_n=1, seed=r))
    ds.ring.copy_(torch.from_numpy(old[:, None]))
    ds.ring_filled.fill_(1)
    p = dict(temperature=ds.temperature, top_k=ds.top_k, top_p=ds.top_p, presence_penalty=ds.presence_penalty, seed=ds.seed,
             hist=torch.from_numpy(old).to(dev), hist_off=torch.arange(B + 1, dtype=torch.int32, device=dev))
    ref = S.sample_batch(logits, p)
    got = ds.step(logits, None, None)
    torch.cuda.synchronize()
    st = ref["row_status"].cpu().numpy()
    slow = int(((st & capi.ROW_SLOW_PATH) != 0).sum())
    assert 4 <= slow < B and not np.any(st & capi.ROW_ERROR_BITS), slow
    assert np.array_equal(got["row_status"].cpu().numpy(), st)
    assert torch.equal(got["tokens"], ref["tokens"])
    # and the state has moved on
    assert torch.equal(ds.ring[:, 0], got["tokens"].long()) and bool((ds.drawn == 1).all()) and bool((ds.ring_filled == 1).all())
