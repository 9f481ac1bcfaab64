"""The row kernels at the sizes where they can go wrong, against the CPU oracle: as the library chooses
between them, and all sizes through the tile kernels and through the cluster kernel."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from helpers import ROUTES, OracleSampler, half_a_unit_tails
from molla_b200 import capi, sampler as S, workloads as W
from test_parity_gpu import compare, run_gpu

pytestmark = pytest.mark.gpu


def _kinds(w, B, V):
    """Rows of every way through the kernels: greedy, top-k of one, sorted head, wide top-k, a nucleus past
    the head, nothing sorted (with min-p too), typical-p."""
    w["temperature"][:] = np.float32([0.0, 0.7, 0.7, 1.0, 1.4, 1.0, 1.2, 0.9])[np.arange(B) % 8]
    w["top_k"][:] = np.int32([0, 1, 40, 1024, 0, 0, 0, 50])[np.arange(B) % 8]
    w["top_p"][:] = np.float32([1, 1, 0.9, 0.99, 0.98, 1, 1, 0.95])[np.arange(B) % 8]
    w["min_p"][:] = np.float32([0, 0, 0, 0, 0, 0, 1e-4, 0])[np.arange(B) % 8]
    w["typical_p"][:] = np.float32([1, 1, 1, 1, 1, 1, 1, 0.9])[np.arange(B) % 8]
    return w


@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("V", [33, 1023, 1024, 1025, 4095, 4096, 4097, 8191, 8193, 16385, 50257])
def test_tile_edges(dev, lib, oracle, V):
    B = 16
    w = _kinds(W.config3(seed=V, B=B, V=V, H=16), B, V)
    compare(w, dev, oracle, f"V={V}", top_n=min(5, V), max_exception_frac=0.2)
    compare(w, dev, oracle, f"V={V}, odd stride", stride=V + 3, offset=1, max_exception_frac=0.2)


@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("V", [3000, 9000, 16000, 40000])
def test_sums_that_stay_near_a_power_of_two(dev, lib, oracle, V):
    """Hundreds of chunks whose sum may lie in either of two binades: some, more than have places for their
    values, more than the row kernel takes."""
    B = 16
    rng = np.random.default_rng(V)
    w = _kinds(W.config3(seed=V + 1, B=B, V=V, H=4), B, V)
    w["temperature"][:] = np.where(w["temperature"] > 0, np.float32(1.0), np.float32(0.0))
    x = (-15.5 + rng.standard_normal((B, V)) * 0.2).astype(np.float32)
    x[:, 0] = 0.0
    x[:, 1] = np.log(np.maximum(1.0 - 2.1e-7 * V * rng.random(B), 0.5)).astype(np.float32)
    w["logits"] = x
    compare(w, dev, oracle, f"near two, V={V}", max_exception_frac=0.3)


@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("low,high", [(18, 26), (0, 30), (22, 25)])
@pytest.mark.parametrize("V", [33, 1025, 9000, 40000])
def test_sums_full_of_rounding_ties(dev, lib, oracle, V, low, high):
    """Exponentials that are powers of two, down to a quarter of the sum's last bit: most additions are rounding ties,
    whose direction depends on the sum before them. Equal values at every edge, which the rows are marked for; the
    softmax denominator and the draw in vocabulary order have to be the sequential ones all the same."""
    B = 16
    rng = np.random.default_rng(V + low)
    w = _kinds(W.config3(seed=V + low, B=B, V=V, H=4), B, V)
    w["temperature"][:] = np.where(w["temperature"] > 0, np.float32(1.0), np.float32(0.0))
    w["typical_p"][:] = 1.0
    k = rng.integers(low, high, (B, V))
    k[np.arange(B), rng.integers(0, V, B)] = 0
    k[::2, 0] = 0
    w["logits"] = (-np.log(2.0) * k).astype(np.float32)
    compare(w, dev, oracle, f"ties, V={V}", max_exception_frac=1.0)


@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("V", [9000, 30000, 60000, 131072, 262144])
def test_tails_of_half_a_unit(dev, lib, oracle, V):
    """Values that add nothing in the binade their chunk expects may add something in the one the sum is still in."""
    compare(half_a_unit_tails(_kinds(W.config3(seed=V, B=64, V=V, H=4), 64, V)), dev, oracle, f"half a unit, V={V}", max_exception_frac=0.5)

@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("first", [-30000.0, -9000.0, 25000.0])
def test_sums_of_rows_whose_scaled_logits_round_coarsely(dev, lib, oracle, first):
    """A logit over a temperature of 0.05 is rounded to a sixteenth or so here, its exponential with it. First some values whose
    exponentials are past two in all before that rounding and below two after it, then a tail that adds a unit each below two
    and nothing above."""
    B, V, T, x0 = 16, 6000, np.float32(0.05), np.float32(first)
    rng = np.random.default_rng(int(abs(first)))
    v = (x0 - np.arange(1, 800, dtype=np.float32) * np.spacing(np.float32(abs(first)))).astype(np.float32)
    real = np.exp((v.astype(np.float64) - x0) / float(T))
    got = np.exp((v / T).astype(np.float32).astype(np.float64) - np.float32(x0 / T))
    low = np.argsort(got / real)[:200]
    low = low[real[low] > 0.003]
    w = _kinds(W.config3(seed=1, B=B, V=V, H=4), B, V)
    w["temperature"][:] = T
    w["typical_p"][:], w["repeat_penalty"][:], w["top_p"][:] = 1.0, 1.0, 1.0
    w["frequency_penalty"][:] = w["presence_penalty"][:] = 0.0
    x = np.full((B, V), x0 - 200.0, np.float32)
    x[:, 0] = x0
    for r in range(B):
        while True:
            some = rng.choice(low, rng.integers(3, 9), replace=False)
            if real[some].sum() > 1 + 2 ** -8.5 and got[some].sum() < 1 - 2 ** -11:
                break
        x[r, 1:1 + len(some)] = v[some]
    x[:, 1024:4000] = x0 - np.float32(16.3 * 0.05)
    w["logits"] = x
    compare(w, dev, oracle, f"coarse, first={first}", max_exception_frac=1.0)

@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("V", [1000, 4097])
def test_pick_rows_in_place(dev, lib, oracle, V):
    """Samplers on the host, logit rows in any order and twice, a block with a stride, biases and windows."""
    rng = np.random.default_rng(V)
    wide = torch.from_numpy((3 * rng.standard_normal((6, V + 5))).astype(np.float32)).to(dev)
    block = wide[:, 2:V + 2]
    rows = [4, 0, 4, 5, 1]
    mine, ref = [], []
    for i in range(len(rows)):
        kw = dict(temperature=0.3 * i, top_k=20 * (i % 2), repeat_penalty=1.2, repeat_last_n=8 * i, seed=i)
        mine.append(S.Sampler(S.SamplerConfig(**kw), V, dev))
        ref.append(OracleSampler(oracle, V, **kw))
        for t in range(i):
            mine[i].bias(7 * t + 1, 1.5 - t)
            ref[i].bias(7 * t + 1, 1.5 - t)
    host = block.cpu().numpy()
    for _ in range(12):
        got = S.pick_rows(block, mine, rows)
        assert got == [r.pick(host, row) for r, row in zip(ref, rows)]
        assert [m.recent[: m.filled] for m in mine] == [r.recent[: r.filled] for r in ref]


@pytest.mark.parametrize("B,V,per_logit", [(32, 131072, 0.01), (16, 262144, 0.01), (64, 131072, 8.0), (200, 3000, 100.0)])
def test_pick_rows_asks_for_what_its_kernels_use(dev, lib, B, V, per_logit):
    """Rows in thread-block clusters need no scratch; the tile kernels' is some 6 bytes a logit and, a row, 250 KB of
    lists and tables. It may hold anything: two calls, one of them on a buffer of 0xff."""
    need = lib.molla_sample_pick_workspace_bytes(B, V, 0, 0)
    assert 0 < need <= B * V * per_logit + (1 << 20) and (per_logit < 1 or need > 4 * B * V), need
    block = torch.randn((B, V), device=dev) * 3
    cfg = [S.SamplerConfig(temperature=1.2, top_k=[40, 0, 0][i % 3], top_p=[0.9, 1.0, 0.97][i % 3], seed=i) for i in range(B)]
    got = []
    for fill in (0xff, 0):
        S._scratch.__dict__.clear()
        S._scratch.bufs = {block.device: torch.full((max(need, 1 << 20),), fill, dtype=torch.uint8, device=dev)}
        kept = S._scratch.bufs[block.device].data_ptr()
        got.append(S.pick_rows(block, [S.Sampler(c, V, dev) for c in cfg]))
        assert S._scratch.bufs[block.device].data_ptr() == kept   # large enough
    S._scratch.__dict__.clear()
    assert got[0] == got[1]


@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("steps", [0, 16])
@pytest.mark.parametrize("V", [2049, 3000, 4064, 4097, 20000, 40000, 65536, 65537])
def test_heads_of_short_rows(dev, lib, oracle, V, steps):
    """Nuclei that end in the head's near list, in its far one and behind both; a top-k that asks for more
    elements than the row has lanes; min-p; logits of many values and of few (whole sixteenths: equal values at
    every edge, more candidates than the head has room for)."""
    B = 40
    w = W.config3(seed=V + steps, B=B, V=V, H=16)
    rng = np.random.default_rng(V + steps)
    w["temperature"][:] = rng.uniform(0.2, 1.6, B)
    w["top_k"][:] = np.int32([0, 0, 0, 100, 127, 0, 600, 1025, 1026, 1500])[np.arange(B) % 10]
    w["top_p"][:] = rng.choice(np.float32([0.3, 0.6, 0.9, 0.95, 0.999]), B)
    w["min_p"][::7] = rng.choice(np.float32([0.001, 0.05]), len(w["min_p"][::7]))
    w["typical_p"][:] = np.where((w["top_k"] > 0) & (w["top_k"] < 128) & (np.arange(B) % 4 == 0), np.float32(0.9), np.float32(1.0))
    if steps:
        w["logits"] = (np.round(w["logits"] * steps) / steps).astype(np.float32)
    # (every mismatch has to be explained by a mark: with few values most rows have equal ones at an edge)
    compare(w, dev, oracle, f"V={V} steps={steps}", max_exception_frac=1.0 if steps else 0.1)


@pytest.mark.parametrize("V", [2000, 8193, 38404, 50257, 151936])
def test_both_kinds_report_rows_that_jump_alike(dev, lib, V):
    """Sharp rows, whose sum jumps by 2^40 and more somewhere: one thread-block cluster a row and tiles spread over the
    chip give the same tokens, sums and status words, MOLLA_ROW_SLOW_PATH among them. (Blocks and groups that begin
    inside a tile, groups in the first tile, windows and min-p.)"""
    B = 128
    w = W.config3(seed=V + 7, B=B, V=V, H=48)
    rng = np.random.default_rng(V)
    w["temperature"][:] = rng.uniform(0.02, 0.2, B)
    w["min_p"][::5] = 1e-3
    w["top_k"][1::5] = 0
    w["top_p"][1::5] = 1.0
    w["min_p"][1::10] = 1e-5
    got = []
    for knob in ROUTES.values():
        with capi.testing_library() as T:
            T.molla_sample_debug_knobs(knob)
            try:
                got.append(run_gpu(w, dev))
            finally:
                T.molla_sample_debug_knobs(0)
    a, b = got
    assert np.array_equal(a["tokens"], b["tokens"]) and np.array_equal(a["diag"].view(np.uint32), b["diag"].view(np.uint32))
    slow = np.uint32(capi.ROW_SLOW_PATH)
    assert np.array_equal(a["row_status"] & ~slow, b["row_status"] & ~slow)
    # (one row in some thousands has a sum so near a power of two that the rounding of the estimate decides)
    assert ((a["row_status"] ^ b["row_status"]) != 0).sum() <= 1 and np.any(b["row_status"] & slow)


@pytest.mark.parametrize("B", [14, 15, 16, 17])
def test_rows_around_what_is_resident_at_once(dev, lib, B):
    """Clusters of eight blocks: 15 or 16 of them fit a device, the next row sends the batch to the tile kernels. The
    library's choice and either kind for all rows: the same tokens, sums and status words."""
    V = 262144
    w = _kinds(W.config3(seed=B, B=B, V=V, H=16), B, V)
    got = []
    for knob in (0, *ROUTES.values()):
        with capi.testing_library() as T:
            T.molla_sample_debug_knobs(knob)
            try:
                got.append(run_gpu(w, dev))
            finally:
                T.molla_sample_debug_knobs(0)
    for other in got[1:]:
        for key in ("tokens", "row_status"):
            assert np.array_equal(got[0][key], other[key]), key
        assert np.array_equal(got[0]["diag"][:, :3].view(np.uint32), other["diag"][:, :3].view(np.uint32))


@pytest.mark.parametrize("V,softcap", [(140000, 0.0), (240000, 0.0), (262144, 30.0)])
def test_two_rounds_of_clusters_where_tiles_would_lose(dev, lib, V, softcap):
    """16 rows, of which 15 or 16 are resident: in clusters either way up to 240000 logits, and with a softcap."""
    ds = S.DeviceSamplers(16, V, ring_cap=1, device=dev)
    for slot in range(16):
        ds.assign(slot, S.SamplerConfig(temperature=1.0, top_k=40, repeat_last_n=0))
    counts = (C.c_int64 * 2)()
    with capi.testing_library() as T:
        T.molla_sample_debug_launches(counts)
        ds.step(torch.randn(16, V, device=dev), None, None, final_softcap=softcap)
        T.molla_sample_debug_launches(counts)
    assert list(counts) == [1, 0]


@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("V", [3072, 9000])
def test_a_tile_of_equal_values_below_a_quarter_of_the_sum(dev, lib, oracle, V):
    """1024 exponentials 2^(j-1) (1 - 2^-24) while the sum is expected in [2^j, 2^(j+1)): each rounds to 2^22 units without a
    tie, all of them together are 2^32. Rows that sort nothing add their probabilities in the same way: Z is 2048 in the even
    ones, 1 / 2048 before the tile three times."""
    B = 32
    w = _kinds(W.config3(seed=V, B=B, V=V, H=4), B, V)
    w["temperature"][:] = np.where(w["temperature"] > 0, np.float32(1.0), np.float32(0.0))
    w["typical_p"][:] = 1.0
    w["repeat_penalty"][:] = 1.0
    w["frequency_penalty"][:] = w["presence_penalty"][:] = 0.0
    x = np.full((B, V), -200.0, np.float32)
    x[:, [3, 500, 1000]] = 0.0
    x[:, 1024:2048] = -2.0 ** -24
    x[::2, 2048:2048 + 1021] = 0.0
    half = np.arange(B) % 4 == 3   # the same at half the size, below a maximum that comes last
    x[np.ix_(half, [3, 500, 1000])] = -np.log(2.0)
    x[half, 1024:2048] = np.float32(-0.69314724)
    x[half, 3000] = 0.0
    assert oracle.expf(x[1, 1024:1025])[0] == 1.0 - 2.0 ** -24 and oracle.expf(x[3, 1024:1025])[0] == 0.5 - 2.0 ** -25
    w["logits"] = x
    compare(w, dev, oracle, f"equal values, V={V}", max_exception_frac=1.0)


@pytest.mark.parametrize("tiles,head", [(190, True), (225, True), (240, False)])
def test_rows_of_many_careful_chunks_end_in_row_head(dev, lib, oracle, tiles, head):
    """Three values a tile, each in a chunk of its own, while the sum stays near a power of two: three careful chunks a tile,
    of which row_head takes 704. Rows of more go through the last kernel's general form, to the same result."""
    B, V = 8, 1024 * tiles
    rng = np.random.default_rng(tiles)
    w = W.config3(seed=tiles, B=B, V=V, H=4)
    w["temperature"][:] = 1.0
    w["top_k"][:], w["top_p"][:], w["min_p"][:], w["typical_p"][:] = 40, 0.9, 0.0, 1.0
    w["repeat_penalty"][:] = 1.0
    w["frequency_penalty"][:] = w["presence_penalty"][:] = 0.0
    x = np.full((B, V), -200.0, np.float32)
    at = (1024 * np.arange(tiles)[:, None] + [70, 500, 990]).ravel()
    x[:, at] = rng.uniform(-15.9, -14.5, (B, at.size))   # the sum grows by 2e-4 in all
    x[:, 0] = 0.0
    x[:, 1] = np.log(1.0 - 1e-4 * rng.random(B))
    w["logits"] = x
    stamps = torch.zeros((B, 32), dtype=torch.int64, device=dev)
    with capi.testing_library() as T:
        T.molla_sample_debug_knobs(ROUTES["tiles"])
        T.molla_sample_debug_profile(stamps.data_ptr())
        try:
            compare(w, dev, oracle, f"{tiles} tiles", max_exception_frac=0.3)
        finally:
            T.molla_sample_debug_knobs(0)
            T.molla_sample_debug_profile(None)
    assert stamps[:, 24].tolist() == [0 if head else 2] * B   # why a row was queued: not at all, or for its records


@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("top", [-9e4, -2e3, 3e2, 4e3, 9e4])
def test_denominators_of_rows_far_from_zero(dev, lib, oracle, top):
    """Maxima over temperature of up to 1e5, temperatures from 0.05 to 20: what a tile adds to the sum is told by hardware
    exponentials where their error, which grows with both, leaves no doubt. The denominator is the sequential one, bit for bit."""
    B, V = 24, 60000
    w = W.config3(seed=7, B=B, V=V, H=4)
    w["temperature"][:] = np.geomspace(0.05, 20.0, B).astype(np.float32)
    w["temperature"][::6] = 1.0
    w["top_k"][:], w["top_p"][:], w["min_p"][:], w["typical_p"][:] = 40, 0.95, 0.0, 1.0
    w["repeat_penalty"][:] = 1.0
    w["frequency_penalty"][:] = w["presence_penalty"][:] = 0.0
    T = w["temperature"][:, None]
    x = np.where(np.arange(B)[:, None] % 2 == 0, w["logits"], w["logits"] * T)   # (spread by the temperature, or as it is)
    w["logits"] = (x - x.max(1, keepdims=True) + np.float32(top) * T).astype(np.float32)
    compare(w, dev, oracle, f"top={top}", max_exception_frac=1.0)


@pytest.mark.parametrize("chunks,V", [(1, 131072), (3, 131072), (7, 131072), (7, 30000)])
def test_cluster_sums_of_many_careful_chunks(dev, lib, oracle, chunks, V):
    """Every warp with some chunks, too few to be one stretch, whose sum may lie in either of two binades. Of 131072 logits in
    eight blocks: 128 of them, which the leader strings together; 384, more than it has records for, and 896, more than 64
    of a block, which it goes through one by one. The same for 30000 logits in eight blocks, with chunks of nine."""
    B = 8
    rng = np.random.default_rng(chunks)
    w = _kinds(W.config3(seed=V, B=B, V=V, H=4), B, V)
    w["temperature"][:] = np.where(w["temperature"] > 0, np.float32(1.0), np.float32(0.0))
    w["typical_p"][:] = 1.0
    w["repeat_penalty"][:] = 1.0
    w["frequency_penalty"][:] = w["presence_penalty"][:] = 0.0
    per = {131072: 33, 30000: 9}[V]   # logits a thread: a range of V / 8 over 512 threads, odd
    x = np.full((B, V), -200.0, np.float32)
    for block in range(0, V, V // 8):
        for warp in range(block, min(block + V // 8, V), 32 * per):
            at = warp + 3 + per * np.linspace(1, 30, chunks).astype(int)
            at = at[at < min(block + V // 8, V)]
            x[:, at] = rng.uniform(-15.9, -14.5, (B, at.size))   # the sum grows by 3e-4 at most
    x[:, 0] = 0.0
    x[:, 1] = np.log(1.0 - 1e-4 * rng.random(B))
    w["logits"] = x
    counts = (C.c_int64 * 2)()
    with capi.testing_library() as T:
        T.molla_sample_debug_launches(counts)
        compare(w, dev, oracle, f"{chunks} chunks, V={V}", max_exception_frac=0.5)
        T.molla_sample_debug_launches(counts)
    assert counts[0] > 0 and counts[1] == 0


def test_logprobs_of_a_block_too_large_to_run_beside_it(dev, lib):
    """More than eight times the rows that are in flight together: the logprobs' own pass has no memory to spare beside the last
    kernels and comes behind them. Tokens and logprobs are those of the rows sampled a few at a time."""
    B, V = 1500, 720896
    x = torch.randn(B, V, generator=torch.Generator(dev).manual_seed(5), device=dev) * 3
    w = W.config3(seed=5, B=B, V=64, H=16)
    def sample(rows):
        part = {k: (w[k][rows] if k not in ("hist", "hist_off", "bias_ids", "bias_vals", "bias_off") else w[k]) for k in W.SAMPLER_KEYS}
        n = len(part["temperature"])
        part["hist"], part["hist_off"] = w["hist"][rows.start * 16:(rows.start + n) * 16], np.arange(n + 1, dtype=np.int32) * 16
        part["bias_ids"], part["bias_vals"], part["bias_off"] = np.zeros(0, np.int64), np.zeros(0, np.float32), np.zeros(n + 1, np.int32)
        return S.sample_batch(x[rows], S.upload_params(part, dev), top_n=5, want_logprob=True)
    whole = sample(slice(0, B))
    for a in (0, 160, 1440):
        part = sample(slice(a, a + 60))
        for k in ("tokens", "chosen_logprob", "top_ids", "top_logprobs"):
            assert torch.equal(whole[k][a:a + 60], part[k]), (a, k)


@pytest.mark.usefixtures("route")
@pytest.mark.parametrize("seed", [905217, 905230, 12])
def test_draws_from_sets_that_end_by_count_past_the_head(dev, lib, oracle, seed):
    """Flat rows and a top-k of some thousands: the cut is found by counting, and the draw starts from what that walk has left,
    rounding ties among it. (Two rows of the first two seeds' draws fall behind such a tie.)"""
    rng = np.random.default_rng(seed)
    B, V = 48, int(round(np.exp(rng.uniform(np.log(3000), np.log(60000)))))
    w = W.config3(seed=3, B=B, V=64, H=4)
    w["logits"] = (rng.uniform(0.5, 4) * rng.standard_normal((B, V))).astype(np.float32)
    w["temperature"][:] = rng.choice(np.float32([1.0, 2.0, 4.0, 10.0]), B)
    w["top_k"][:] = rng.choice([0, 1100, 2000, 3000, 5000], B)
    w["top_p"][:] = rng.choice(np.float32([1.0, 0.9, 0.95, 0.5, 0.99]), B)
    w["min_p"][:], w["typical_p"][:], w["repeat_penalty"][:] = 0.0, 1.0, 1.0
    w["seed"][:] = rng.integers(0, 2 ** 63, B).astype(np.uint64)
    compare(w, dev, oracle, f"counted, V={V}", max_exception_frac=0.3)
