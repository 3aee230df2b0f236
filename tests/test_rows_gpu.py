"""The batch kernel (k_rows: a row cut over a cluster of 1, 2, 4 or 8 CTAs, any alignment) against the oracle, at the sizes
where it can go wrong, and what a batch may cost when its histories or masks are not noise."""
import numpy as np
import pytest

from flintnsteel_b200 import workloads as wl
from flintnsteel_b200.sampler import BF16, F32, Sampler, cands_tensor, cands_to_numpy, make_params, params_to_device

from .test_parity_gpu import check_against_oracle, dev, run_rows, upload  # noqa: F401  (dev is a fixture)

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def batch(g, rows, n, bf16=False, hist=64, top_hist=False, fractions=(1.0, 0.5, 0.05, 0.004, 0.0005), masked=True, runs=True):
    x = wl.gaussian_logits(g, rows, n, 2.5, spikes=min(8, n))
    if bf16:
        x = wl.bf16_bits_to_f32(wl.f32_to_bf16_bits(x))
    masks = None
    if masked:
        masks = np.stack([(wl.run_mask if runs else wl.random_mask)(g, n, fractions[r % len(fractions)]) for r in range(rows)])
    h = np.argsort(-x, axis=1)[:, :hist].astype(np.int32) if top_hist else g.integers(-2, n + 2, size=(rows, hist), dtype=np.int32)
    if hist >= 10:
        h[:, 1::5] = h[:, ::5][:, : h[:, 1::5].shape[1]]  # repeats
    p = make_params(rows, temperature=0.8, top_p=0.95, repetition=1.2, presence=0.3, frequency=0.2, seed=3)
    p["top_k"] = g.choice(np.array([0, 1, 20, 64], np.int32), size=rows)
    p["temperature"][::4] = 0.0
    p["repetition"][1::6] = 0.7   # penalties that raise values
    p["frequency"][2::6] = -0.3
    p["repetition"][3::6], p["presence"][3::6], p["frequency"][3::6] = 1.0, 0.0, 0.0
    logits = wl.f32_to_bf16_bits(x) if bf16 else x
    return wl.Workload("rows", logits, p, masks, np.ascontiguousarray(h), np.full(rows, hist, np.int32), bf16=bf16)


def plan_slices(w, max_history):
    s = Sampler(0, max_rows=w.rows, max_vocab=w.vocab, k_cap=w.k_cap, max_history=max_history)
    s.set_cluster_rows(0)
    slices = s.plan(BF16 if w.bf16 else F32, w.vocab, w.rows, max_history)["slices"]
    s.close()
    return slices


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n", [1, 3, 7, 255, 256, 257, 4095, 32_768, 65_537, 131_071])
@pytest.mark.parametrize("rows", [5, 37])
def test_rows_of_any_length_packed_side_by_side(dev, oracle, n, rows, bf16):
    """Rows that start on every element of a 16-byte vector, runs and scattered bits, top history, every penalty sign."""
    g = wl.rng(17 * n + rows + bf16)
    hist = min(64, n)
    for masked in (True, False):
        w = batch(g, rows, n, bf16, hist=hist, top_hist=rows == 5, masked=masked, runs=rows == 5)
        check_against_oracle(oracle, w, *run_rows(w, dev, max_history=hist, cluster_rows=0))


@pytest.mark.parametrize("rows", [16, 64, 150])
def test_slices_of_a_full_vocabulary(dev, oracle, rows):
    """4, 4 and 2 CTAs per row; more history ids among the best than the bound allows for, so that it is lowered; allowed
    ids in one slice only; few allowed ids, so that there is no bound."""
    g = wl.rng(rows)
    n = wl.V_QWEN
    w = batch(g, rows, n, hist=400, top_hist=True, fractions=(1.0, 0.3, 0.01, 0.003, 0.0005))
    w.masks[1::7] = 0
    w.masks[1::7, 100:170] = 0xFFFFFFFF
    assert plan_slices(w, 400) == {16: 4, 64: 4, 150: 2}[rows]
    check_against_oracle(oracle, w, *run_rows(w, dev, max_history=400, cluster_rows=0))
    check_against_oracle(oracle, w, *run_rows(w, dev, k_cap=128, max_history=400, cluster_rows=0), k_cap=128)


def test_more_rows_than_six_per_sm_without_a_mask(dev, oracle):
    w = batch(wl.rng(5), 1000, 4096, hist=100, masked=False)
    check_against_oracle(oracle, w, *run_rows(w, dev, max_history=100))


@pytest.mark.parametrize("cluster_rows", [0, 12])
def test_masks_that_leave_a_few_hundred_ids(dev, oracle, cluster_rows):
    """From fewer ids than k to more than a CTA's buffer holds: with and without a bound, in one slice and in all."""
    g = wl.rng(9)
    n, rows = wl.V_QWEN, 12
    w = batch(g, rows, n, hist=50)
    for r, allowed in enumerate((1, 40, 65, 130, 260, 500, 700, 1000, 1500, 2200, 3000, 6000)):
        w.masks[r] = wl.run_mask(g, n, allowed / n, 20 if r % 2 else 2)
    check_against_oracle(oracle, w, *run_rows(w, dev, max_history=50, cluster_rows=cluster_rows))


def test_crowds_of_equal_values(dev, oracle):
    """Equal values overflow the list and the buffer of every CTA, and history ids are among them."""
    n = 65_536
    x = np.zeros((8, n), np.float32)
    x[1] = -0.0
    x[2, ::3] = np.inf
    x[3] = np.repeat(np.arange(n // 512, dtype=np.float32), 512)
    x[4, 5] = np.nan
    x[5] = -np.finfo(np.float32).max
    masks = np.stack([wl.random_mask(wl.rng(r), n, 0.9) for r in range(8)])
    hist = np.tile(np.arange(600, dtype=np.int32) * 7, (8, 1))
    p = make_params(8, temperature=0.9, top_k=64, top_p=0.99, repetition=1.2, presence=0.4, frequency=0.01, seed=2)
    p["frequency"][7] = -0.5
    w = wl.Workload("crowds", x, p, masks, hist, np.full(8, 600, np.int32))
    check_against_oracle(oracle, w, *run_rows(w, dev, max_history=600, cluster_rows=0))


def hot_history(g, x, masks, hist, hot, spread):
    """hist ids per row of which the first ones are the row's `hot` best allowed ids, the rest drawn from the vocabulary; `spread`
    > 0: drawn again with repeats from that many different ones."""
    rows, n = x.shape
    h = g.integers(0, n, size=(rows, hist), dtype=np.int32)
    for r in range(rows):
        xr = x[r].copy()
        if masks is not None:
            xr[~wl.mask_allows(masks[r], np.arange(n))] = -np.inf
        best = np.argsort(-xr, kind="stable")[:min(hot, hist)]
        h[r, :best.size] = best
        if spread:
            h[r] = g.choice(h[r, :spread], size=hist)
    return h


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("hot, hist, spread", [(100, 300, 0), (400, 2048, 0), (2048, 2048, 0), (200, 2048, 600), (300, 16_384, 0)])
@pytest.mark.parametrize("n, rows", [(151_936, 7), (32_003, 37)])
def test_the_best_ids_are_in_the_history(dev, oracle, n, rows, hot, hist, spread, bf16):
    """Rows whose best ids are penalised, once each and with repeats, few and so many that history ids lie in every cell; cut
    rows, whole rows and rows off a 16-byte boundary; with and without a frequency penalty, strong and raising ones."""
    g = wl.rng(hot + hist + spread + n + bf16)
    x = wl.gaussian_logits(g, rows, n, 2.5)
    if bf16:
        x = wl.bf16_bits_to_f32(wl.f32_to_bf16_bits(x))
    masks = np.stack([wl.run_mask(g, n, f) for f in (1.0, 0.5, 0.05, 0.01, 0.004)[:rows] * -(-rows // 5)])[:rows]
    h = hot_history(g, x, masks, hist, hot, spread)
    p = make_params(rows, temperature=0.8, top_p=0.95, repetition=1.1, presence=0.5, frequency=0.3, seed=3)
    p["top_k"] = g.choice(np.array([0, 1, 20, 64], np.int32), size=rows)
    p["repetition"][1::5], p["presence"][1::5], p["frequency"][1::5] = 2.0, 0.0, 0.0
    p["repetition"][2::5], p["presence"][2::5], p["frequency"][2::5] = 1.0, 0.0, 1.0
    p["repetition"][3::5] = 0.8
    p["frequency"][4::5] = 0.0
    w = wl.Workload("hot", wl.f32_to_bf16_bits(x) if bf16 else x, p, masks, h, np.full(rows, hist, np.int32), bf16=bf16)
    check_against_oracle(oracle, w, *run_rows(w, dev, max_history=hist, cluster_rows=0))


def test_whole_rows_of_more_than_32_cells(dev, oracle):
    """223 rows and more are not cut; the best ids and the history lie behind cell 32 of 38 (element 131,072 on)."""
    g = wl.rng(38)
    rows, n = 224, wl.V_QWEN
    x = wl.gaussian_logits(g, rows, n, 2.5)
    x[:, 131_072:] += 4.0
    masks = np.full((rows, n // 32), 0xFFFFFFFF, np.uint32)
    masks[::3] = wl.random_mask(g, n, 0.7)
    w = wl.Workload("deep", x, make_params(rows, temperature=0.8, top_p=0.95, top_k=50, repetition=1.2, presence=0.3, frequency=0.2, seed=2),
                    masks, None, None)
    w.params["temperature"][::4] = 0.0
    w.history = g.integers(131_000, n, size=(rows, 300), dtype=np.int32)
    w.history[1::2, :40] = np.argsort(-x[1::2], axis=1)[:, :40]
    w.history_len = np.full(rows, 300, np.int32)
    assert plan_slices(w, 300) == 1
    check_against_oracle(oracle, w, *run_rows(w, dev, max_history=300, cluster_rows=0))


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows", [6, 40])
def test_a_shard_with_a_history_of_global_ids(dev, oracle, rows, bf16):
    """select_rows with id_base: masks, a history of ids inside and outside the shard, k_cap 64 and 128."""
    g = wl.rng(rows + bf16)
    base, n = 65_536, 40_001
    x = wl.gaussian_logits(g, rows, n, 2.5)
    if bf16:
        x = wl.bf16_bits_to_f32(wl.f32_to_bf16_bits(x))
    masks = np.stack([wl.run_mask(g, n, (1.0, 0.2, 0.01)[r % 3]) for r in range(rows)])
    h = g.integers(0, 2 * base, size=(rows, 500), dtype=np.int32)
    h[:, :60] = base + np.argsort(-x, axis=1)[:, :60]
    h[:, 60:80] = h[:, :20]
    p = make_params(rows, temperature=0.8, top_k=0, repetition=1.2, presence=0.3, frequency=0.2)
    lg = torch.from_numpy(wl.f32_to_bf16_bits(x).view(np.int16)).to(dev).view(torch.bfloat16) if bf16 else torch.from_numpy(x).to(dev)
    for k in (64, 128):
        s = Sampler(0, max_rows=rows, max_vocab=n, k_cap=k, max_history=500)
        s.set_cluster_rows(0)
        cd = cands_tensor(rows, k, dev)
        s.select_rows(lg, params_to_device(p, dev), cd, id_base=base, masks=torch.from_numpy(masks.view(np.int32)).to(dev),
                      history=torch.from_numpy(h).to(dev), history_len=torch.full((rows,), 500, dtype=torch.int32, device=dev))
        torch.cuda.synchronize()
        got = cands_to_numpy(cd)
        s.close()
        for r in range(rows):
            inside = h[r][(h[r] >= base) & (h[r] < base + n)] - base
            y = oracle.penalize(x[r], inside, None, 1.2, 0.3, 0.2)
            cv, ci, nk = oracle.topk(y, masks[r], k, base)
            assert np.array_equal(got["id"][r][:nk], ci[:nk])
            assert np.array_equal(got["value"][r][:nk].view(np.uint32), (cv[:nk] + np.float32(0.0)).view(np.uint32))


def us_per_call(w, dev):
    """Device time of a call, the best of six runs of eight calls."""
    s = Sampler(0, max_rows=w.rows, max_vocab=w.vocab, k_cap=w.k_cap, max_history=w.history.shape[1])
    lg, masks, h, hl = upload(w, dev)
    pd, out = params_to_device(w.params, dev), torch.empty(w.rows, dtype=torch.int32, device=dev)
    best = float("inf")
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(8):
            s.sample_rows(lg, pd, out, masks=masks, history=h, history_len=hl)
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / 8)
    s.close()
    return best


def timed_batch(rows, bf16, masked, k_cap=64):
    """32 different rows over and over, masks of 0.1 to 100 % of the ids, a history of noise."""
    g = wl.rng(rows)
    n = wl.V_QWEN
    x = np.tile(wl.gaussian_logits(g, 32, n, 2.5), (rows // 32, 1))
    masks = np.stack([wl.run_mask(g, n, 10.0 ** g.uniform(-3, 0)) for _ in range(rows)]) if masked else None
    p = make_params(rows, temperature=0.8, top_k=50 if k_cap == 64 else 0, top_p=0.95, repetition=1.1, presence=0.5, frequency=0.3)
    noise = g.integers(0, n, size=(rows, 2048), dtype=np.int32)
    return g, x, wl.Workload("timed", wl.f32_to_bf16_bits(x) if bf16 else x, p, masks, noise, np.full(rows, 2048, np.int32), bf16=bf16,
                             k_cap=k_cap)


@pytest.mark.parametrize("rows, bf16, masked", [(256, False, True), (1024, True, False)])
def test_a_history_that_repeats_itself_costs_little(dev, rows, bf16, masked):
    """600 different ids in 2,048, as text has them, against noise.  Taking the repeats down one by one, and reading the history
    again one id at a time, took 2.5 and 1.8 times as long; it is 1.1 times."""
    g, x, w = timed_batch(rows, bf16, masked)
    noise = us_per_call(w, dev)
    ids = g.integers(0, w.vocab, size=(rows, 600), dtype=np.int32)
    at = np.minimum((600.0 ** g.random((rows, 2048))).astype(np.int64), 599)
    w.history = np.take_along_axis(ids, at, axis=1)
    assert us_per_call(w, dev) < 1.6 * noise


@pytest.mark.parametrize("rows, bf16, masked", [(256, False, True), (1024, True, False)])
def test_a_history_of_the_best_ids_does_not_cost_a_multiple(dev, rows, bf16, masked):
    """A row whose best 400 ids are in the history against one whose history is noise.  A bound that could be in the history,
    lowered step by step and then given up, took 18 and 11.8 times as long; it is 3.2 and 2.4 times."""
    g, x, w = timed_batch(rows, bf16, masked)
    noise = us_per_call(w, dev)
    w.history = hot_history(g, x, w.masks, 2048, 400, 0) if masked else np.tile(hot_history(g, x[:32], None, 2048, 400, 0), (rows // 32, 1))
    assert us_per_call(w, dev) < 5.0 * noise


def test_rows_that_allow_little_do_not_hold_up_a_batch(dev):
    """k = 128 over rows of which some allow a few hundred to a few thousand ids, too few for a bound from groups of threads:
    without one for such rows the batch took 184 us, 5 times what it takes when every id is allowed."""
    _, _, w = timed_batch(128, True, True, k_cap=128)
    some = us_per_call(w, dev)
    w.masks = np.full_like(w.masks, 0xFFFFFFFF)
    assert some < 2.5 * us_per_call(w, dev)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows, slices", [(16, 8), (37, 8), (38, 4), (55, 4)])
def test_the_longest_rows(dev, oracle, rows, slices, bf16):
    """V = 262,144 under masks in eight CTAs per row and in four; rows on and off 16-byte boundaries."""
    g = wl.rng(rows + bf16)
    for n in (262_144, 262_147):
        w = batch(g, rows, n, bf16, hist=200, top_hist=True, fractions=(1.0, 0.3, 0.01, 0.003, 0.0005))
        assert plan_slices(w, 200) == slices
        check_against_oracle(oracle, w, *run_rows(w, dev, max_history=200, cluster_rows=0))
