"""The passes of the row clusters over a row's logits: overrides around the size at which their table gives way to the
histogram, and logits whose tiles weigh next to nothing, or everything, against the row's maximum."""
import numpy as np
import pytest

from tests import parity

pytestmark = pytest.mark.gpu


def _run(logits, params, hist=None, seed=5, max_top_k=8):
    from opentail.stingray_b200 import BatchSampler, workloads as W

    rows, vocab = logits.shape
    rng = np.random.default_rng(seed)
    ids = off = None
    if hist is not None:
        ids = np.concatenate(hist).astype(np.int32)
        off = np.concatenate([[0], np.cumsum([len(h) for h in hist])]).astype(np.int32)
    w = W.SampleWorkload("s", np.ascontiguousarray(logits), params, W.uniforms24(rng, rows), ids, off, None)
    bs = BatchSampler(max_rows=rows, max_vocab=vocab, max_history=2048, max_top_k=max_top_k)
    try:
        gpu = parity.run_gpu(bs, w, want_topk=int(params["top_k"].max()))
        stats = parity.compare(w, gpu)
        assert stats["mismatch"] == stats["boundary_draws"] <= 1
        return gpu["flags"].view(np.uint32)
    finally:
        bs.close()


def _params(rows):
    from opentail.stingray_b200 import workloads as W

    p = W._params(rows)
    p["temperature"] = np.resize([0.8, 1.0, 1.3], rows)
    p["top_p"] = np.resize([0.9, 1.0, 0.99, 0.5], rows)
    p["min_p"] = np.resize([0.0, 0.0, 0.0, 0.0, 0.02], rows)
    return p


@pytest.mark.parametrize("entries", [1, 511, 512, 513, 2048])
@pytest.mark.parametrize("rows,vocab", [(6, 32_000), (80, 16_640)])
def test_override_table_beside_and_over_the_histogram(rows, vocab, entries):
    """The longest row's history decides nothing for the others: every row's table has its own size."""
    rng = np.random.default_rng(entries)
    p = _params(rows)
    p["repetition_penalty"], p["presence_penalty"], p["repeat_last_n"] = 1.2, 0.3, 0
    hist = [rng.integers(0, vocab, entries if r % 2 == 0 else max(1, entries // 3)) for r in range(rows)]
    _run(rng.normal(0, 2.5, (rows, vocab)).astype(np.float32), p, hist)


@pytest.mark.parametrize("vocab", [32_000, 50_257])
def test_tiles_of_very_different_weight(vocab):
    """Tiles far below the maximum (their exp values zero, subnormal or the only ones for a while), a row that rises to its
    maximum, one whose logits are a thousand times larger, one that is -infinity but for a few."""
    rng = np.random.default_rng(9)
    x = rng.normal(0, 1.5, (12, vocab)).astype(np.float32)
    half = vocab // 2
    x[0, :half] -= 300.0                                   # underflow to zero
    x[1, :half] -= 88.0                                    # subnormal exp values in front of the others
    x[2, half:] -= 1e5
    x[3] += np.linspace(-200.0, 0.0, vocab, dtype=np.float32)
    x[4] += np.linspace(0.0, -90.0, vocab, dtype=np.float32)
    x[5] *= 1000.0
    x[6] = -np.inf
    x[6, rng.integers(0, vocab, 40)] = rng.normal(0, 1, 40)
    x[7, : vocab - 300] = -np.inf
    x[8] = 0.25                                            # all equal
    x[9] = np.round(x[9])                                  # ties at every bin
    x[10, 777] = 80.0
    x[11] += 3e4
    p = _params(12)
    p["temperature"] = 1.0
    _run(x, p)
    p["top_p"] = 1.0
    p["min_p"] = 0.0
    _run(x, p)


@pytest.mark.parametrize("top_k", [63, 64, 127, 128, 255, 256])
@pytest.mark.parametrize("rows", [8, 300])
def test_top_k_with_ties_and_penalties_around_the_cut(top_k, rows):
    """Logits in steps of 1/4, penalised in small steps, 20 to 90 % of the tokens near the cut in the history; top_k up to the
    largest the short finish takes."""
    from opentail.stingray_b200 import workloads as W

    vocab = 32_000
    rng = np.random.default_rng(top_k)
    x = (np.round(rng.normal(0, 2.0, (rows, vocab)) * 4) / 4).astype(np.float32)
    hist = []
    for r in range(rows):
        order = np.argsort(-x[r], kind="stable")[: 2 * top_k]
        hist.append(order[rng.random(order.size) < (0.2, 0.5, 0.9)[r % 3]])
    p = W._params(rows)
    p["temperature"], p["top_p"], p["top_k"], p["repeat_last_n"] = 0.9, 0.98, top_k, 0
    p["repetition_penalty"] = np.resize([1.0, 1.1, 1.25], rows)
    p["presence_penalty"] = np.resize([0.25, 0.0, 0.5, 0.125], rows)
    _run(x, p, hist, max_top_k=512)


def test_top_p_next_to_one():
    """The cut lies where the sorted sum is nearly flat: tens of thousands of tokens within the estimate's error of it."""
    from opentail.stingray_b200 import workloads as W

    rows, vocab = 12, 151_936
    rng = np.random.default_rng(21)
    p = W._params(rows)
    p["temperature"] = np.resize([0.7, 1.1, 0.4], rows)
    p["top_p"] = np.resize([0.9997, 0.9999, 0.99995, 0.99999, 0.999999], rows)
    _run(rng.normal(0, 2.5, (rows, vocab)).astype(np.float32), p)


@pytest.mark.parametrize("top_p", [0.997, 0.999, 0.9995, 0.9997, 0.9998])
def test_top_p_near_one_is_no_reason_to_redo_a_row(top_p):
    from opentail.stingray_b200 import workloads as W

    rows, vocab = 12, 151_936
    p = W._params(rows, top_p=top_p)
    p["temperature"] = np.resize([0.4, 0.7, 0.9, 1.1], rows)
    flags = _run(np.random.default_rng(22).normal(0, 2.5, (rows, vocab)).astype(np.float32), p)
    assert not (flags >> 8 & 1).any()


# ---- temperatures so small that neighbouring logits lie far apart, or fall together, once scaled -------------------------------

SMALL_T = [1e-7, 3e-7, 5e-7, 7e-7, 1e-6]
# a softmax sum that is off by a tenth shows in where these cut; Normalize hides it from the probabilities themselves
CUTS = [0.9, 0.35, 0.7, 1.0, 0.55]


def _near_maximum(rng, temperature, count):
    """(A, B, maximum) triples whose exp values are other than their distance in the unscaled logits says: behind A alone the
    sum is in the binade expected, B looks like less than a quarter of that binade and is half of it or more."""
    inv = np.float32(1.0) / np.float32(temperature)
    m = rng.uniform(15.0, 31.0, 8000).astype(np.float32)
    found = []
    for i, j in ((0, 1), (1, 2), (2, 3)):  # units of A and B below the maximum
        a, b = ((m.view(np.uint32) - np.uint32(k)).view(np.float32) for k in (i, j))
        real = [np.exp((v * inv).astype(np.float64) - (m * inv)) for v in (a, b)]
        seen = [np.exp((v.astype(np.float64) - m) * float(inv)) for v in (a, b)]
        with np.errstate(divide="ignore"):
            g = np.floor(np.log2(seen[0]))
            hit = (np.floor(np.log2(real[0])) == g) & (real[1] >= 2.0 ** (g - 1)) & (seen[1] < 2.0 ** (g - 2)) & (real[0] > 1e-4)
        found += [(a[t], b[t], m[t]) for t in np.flatnonzero(hit)[:count]]
    assert len(found) >= count
    return [found[t] for t in rng.permutation(len(found))[:count]]


def _near_rows(temperature, rows, vocab, seed=31):
    rng = np.random.default_rng(seed)
    x = rng.normal(0, 2.5, (rows, vocab)).astype(np.float32)
    for r, (a, b, m) in enumerate(_near_maximum(rng, temperature, rows)):
        x[r, 100] = a
        x[r, 256 * int(rng.integers(2, vocab // 512)) + int(rng.integers(0, 256))] = b
        x[r, 256 * int(rng.integers(vocab // 512, vocab // 256)) + int(rng.integers(0, 256))] = m
    return x


@pytest.mark.parametrize("temperature", SMALL_T)
@pytest.mark.parametrize("vocab", [32_000, 151_936])
def test_near_the_maximum_at_small_temperatures(temperature, vocab):
    from opentail.stingray_b200 import workloads as W

    rows = 24
    p = W._params(rows)
    p["temperature"] = temperature
    p["top_p"] = np.resize(CUTS, rows)
    _run(_near_rows(temperature, rows, vocab), p)


def test_near_the_maximum_behind_penalties():
    """bf16 logits that a repetition penalty leaves one unit away from unpenalised ones (31.875 / 1.2 beside 26.5625), at
    temperatures that make the two equal."""
    from opentail.stingray_b200 import workloads as W

    rows, vocab = 24, 32_000
    rng = np.random.default_rng(33)
    x = rng.normal(0, 2.5, (rows, vocab)).astype(np.float32)
    p = W._params(rows)
    p["repeat_last_n"] = 0
    p["top_p"] = np.resize(CUTS, rows)
    hist = []
    bf16 = (np.arange(0x4180, 0x4280, dtype=np.uint32) << 16).view(np.float32)  # 16 .. 64
    for r in range(rows):
        rep = np.float32([1.05, 1.2, 1.3][r % 3])
        q = bf16 / rep
        plain = ((q.view(np.uint32) + 0x7FFF) >> 16 << 16).view(np.float32)
        pick = rng.choice(np.flatnonzero((np.abs(q.view(np.int32) - plain.view(np.int32)) == 1) & (q > 14.0)))
        t = rng.uniform(1e-7, 1e-6, 1000).astype(np.float32)
        inv = np.float32(1.0) / t
        t = t[(q[pick] * inv == plain[pick] * inv) & (abs(float(q[pick]) - float(plain[pick])) * inv > 2.0)][0]
        p["repetition_penalty"][r], p["temperature"][r] = rep, t
        # the larger one in tile 0 and near the row's end, the smaller one in between
        low = 256 * int(rng.integers(2, 60)) + int(rng.integers(0, 256))
        high = np.array([100, 256 * int(rng.integers(61, vocab // 256)) + int(rng.integers(0, 256))])
        pen, raw = (np.array([low]), high) if q[pick] < plain[pick] else (high, np.array([low]))
        x[r, pen], x[r, raw] = bf16[pick], plain[pick]
        hist.append(np.concatenate([pen, rng.integers(0, 50, 20)]))
    _run(W.to_bf16_bits(x), p, hist)


@pytest.mark.parametrize("temperature", SMALL_T)
def test_distributions_near_the_maximum(temperature):
    import torch
    from opentail.stingray_b200 import BatchSampler, workloads as W
    from oracle import oracle as orc

    rows, vocab = 12, 32_000
    x = _near_rows(temperature, rows, vocab, seed=35)
    p = W._params(rows)
    p["temperature"] = temperature
    p["top_p"] = np.resize(CUTS, rows)
    bs = BatchSampler(max_rows=rows, max_vocab=vocab, max_history=1, max_top_k=8)
    try:
        u = torch.full((rows,), 0.7, device="cuda")
        beside = bs.sample_with_distribution(torch.from_numpy(x).cuda(), p, uniforms=u)[1].cpu().numpy()
        alone = bs.build_distribution(torch.from_numpy(x).cuda(), p).cpu().numpy()
    finally:
        bs.close()
    for r in range(rows):
        want = orc.build_filtered_distribution(x[r], orc.OrcParams(*[p[r][n].item() for n in p.dtype.names]))[0]
        for got in (beside[r], alone[r]):
            np.testing.assert_allclose(got, want, rtol=2e-5, atol=1e-30)


@pytest.mark.parametrize("temperature", SMALL_T)
def test_verification_near_the_maximum(temperature):
    from opentail.stingray_b200 import workloads as W
    from tests.test_gpu_spec_shard import _check_spec

    n, L, vocab = 4, 2, 32_000
    rng = np.random.default_rng(37)
    rows = _near_rows(temperature, n * (2 * L + 1), vocab, seed=39)
    target, draft = rows[: n * (L + 1)].reshape(n, L + 1, vocab), rows[n * (L + 1):].reshape(n, L, vocab)
    p = W._params(n, temperature=temperature)
    p["top_p"] = CUTS[:n]
    _check_spec(W.SpecWorkload("near", target, draft, draft.argmax(2).astype(np.int32), p, rng.random((n, L + 2))))


@pytest.mark.parametrize("top_p,min_p", [(1.0, 0.0), (0.9, 0.0), (0.9, 0.02)])
def test_not_a_number_wherever_it_stands(top_p, min_p):
    """A NaN logit among -infinities, a whole tile of them, and one among ordinary logits make the same of a row."""
    import torch
    from opentail.stingray_b200 import BatchSampler, workloads as W

    rows, vocab = 16, 32_000
    x = np.random.default_rng(4).normal(0, 2.5, (rows, vocab)).astype(np.float32)
    x[:, 5120:5376] = x[:, 5400] = -np.inf
    p = W._params(rows, temperature=0.8, top_p=top_p, min_p=min_p)
    u = torch.from_numpy(W.uniforms24(np.random.default_rng(5), rows)).cuda()
    bs = BatchSampler(max_rows=rows, max_vocab=vocab, max_history=1, max_top_k=8)
    got = []
    try:
        for where in (slice(5400, 5401), slice(5200, 5201), slice(5120, 5376)):
            y = x.copy()
            y[:, where] = np.nan
            out = bs.sample_rows(torch.from_numpy(y).cuda(), p, uniforms=u, want_probs=True)
            got.append((out["tokens"].cpu().numpy(), out["probs"].cpu().numpy()))
    finally:
        bs.close()
    for tokens, probs in got[1:]:
        np.testing.assert_array_equal(tokens, got[0][0])
        np.testing.assert_array_equal(probs, got[0][1])


@pytest.mark.parametrize("vocab", [32_000, 50_257])
def test_masks_of_a_few_tokens_per_lane(vocab):
    """Rows closed up as they are read, eight tokens to a lane: none or one allowed in each, up to two (taken one after the
    other), up to three and up to all of them (taken by predicate)."""
    from opentail.stingray_b200 import BatchSampler, workloads as W

    rows, words = 12, (vocab + 31) // 32
    rng = np.random.default_rng(vocab)
    allowed = np.zeros((rows, words * 32), bool)
    for r in range(rows):
        most = (1, 2, 3, 8)[r % 4]
        pick = rng.permuted(np.tile(np.arange(8), (words * 4, 1)), axis=1)
        n = rng.integers(0, most + 1, words * 4) * (rng.random(words * 4) < (0.02, 0.5, 1.0)[r % 3])
        if r % 4 == 3:
            n = np.where(rng.random(n.size) < 0.4, n, 0)
        np.put_along_axis(allowed[r].reshape(-1, 8), pick, np.arange(8) < n[:, None], axis=1)
    mask = np.packbits(allowed, axis=1, bitorder="little").view(np.uint32)
    w = W.SampleWorkload("m", rng.normal(0, 2.5, (rows, vocab)).astype(np.float32), _params(rows), W.uniforms24(rng, rows), None, None, mask)
    bs = BatchSampler(max_rows=rows, max_vocab=vocab, max_history=1, max_top_k=8)
    try:
        stats = parity.compare(w, parity.run_gpu(bs, w))
        assert stats["mismatch"] == stats["boundary_draws"] <= 1
    finally:
        bs.close()


# ---- the finish of the top-k rows: 8 rows take its 512-thread form, 300 the 256-thread form, 600 the full-size one ---------------


@pytest.mark.parametrize("rows", [8, 300, 600])
@pytest.mark.parametrize("length", [500, 1500, 1850])
def test_top_k_candidate_lists_behind_long_histories(rows, length):
    """Beside the hash of 1,025 tokens and more the 256-thread form has room for the values of some 3,500 candidates, in
    registers and shared memory; the lists hold 2,000 to 9,000."""
    from opentail.stingray_b200 import workloads as W

    vocab = 16_640
    rng = np.random.default_rng(length)
    x = rng.normal(0, 2.5, (rows, vocab)).astype(np.float32)
    x[1::3] = np.round(x[1::3] * 16) / 16
    p = W._params(rows, temperature=0.9, top_p=0.98, top_k=40, repeat_last_n=0)
    p["repetition_penalty"] = np.resize([1.1, 1.0, 1.3], rows)
    p["frequency_penalty"] = np.resize([0.0, 0.25], rows)
    # every other history holds what would have been drawn
    hist = [rng.integers(0, vocab, length) if r % 2 else rng.permutation(np.argsort(-x[r])[: 2 * length])[:length] for r in range(rows)]
    _run(x, p, hist, max_top_k=64)


def test_a_long_history_costs_no_second_selection():
    """Rows whose hash leaves little room beside it were once selected anew from their lists, which took 5.7 times as long as
    rows of two thirds of their history; here they may take twice as long."""
    import torch
    from opentail.stingray_b200 import BatchSampler, workloads as W

    rows, vocab = 300, 32_000
    rng = np.random.default_rng(41)
    x = torch.from_numpy(rng.normal(0, 2.5, (rows, vocab)).astype(np.float32)).cuda()
    p = W._params(rows, temperature=0.9, top_p=0.98, top_k=40, repetition_penalty=1.1, repeat_last_n=0)
    u = torch.from_numpy(W.uniforms24(rng, rows)).cuda()
    bs = BatchSampler(max_rows=rows, max_vocab=vocab, max_history=2048, max_top_k=64)
    best = {}
    try:
        for length in (1000, 1500):
            kw = dict(history_ids=torch.from_numpy(rng.integers(0, vocab, rows * length).astype(np.int32)).cuda(),
                      history_offsets=np.arange(rows + 1, dtype=np.int32) * length, uniforms=u)
            out, times = None, []
            for _ in range(20):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                out = bs.sample_rows(x, p, out=out, **kw)
                b.record()
                torch.cuda.synchronize()
                times.append(a.elapsed_time(b))
            best[length] = min(times)
    finally:
        bs.close()
    assert best[1500] < 2 * best[1000], best


@pytest.mark.parametrize("rows", [8, 300, 600])
@pytest.mark.parametrize("lowered,plain", [(0, 2000), (600, 600), (300, 600), (20, 491)])
def test_top_k_cut_among_equal_candidates(rows, lowered, plain):
    """Around and beyond the 512 candidates that are put in order: `plain` logits of 6.5 and `lowered` ones of 7.0 that a
    presence penalty makes equal to them, which come first; among equals the lower token does."""
    from opentail.stingray_b200 import workloads as W

    vocab = 16_640
    rng = np.random.default_rng(lowered + plain)
    x = np.minimum(rng.normal(0, 2.0, (rows, vocab)), 6.0).astype(np.float32)
    hist = []
    for r in range(rows):
        t = rng.permutation(vocab)[: 10 + lowered + plain + 1300]
        x[r, t[:10]] = 8.0 + np.arange(10) / 8
        x[r, t[10:10 + plain]] = 6.5
        x[r, t[10 + plain:10 + plain + lowered]] = 7.0
        x[r, t[10 + plain + lowered:]] = -1.0
        hist.append(t[10 + plain:])
    p = W._params(rows, temperature=0.9, top_p=1.0, top_k=40, presence_penalty=0.5, repeat_last_n=0)
    # (of some rows in a hundred the list overflows, whose bound is the smallest of a few group maxima)
    assert (_run(x, p, hist, max_top_k=64) >> 8 & 1).mean() < 0.05, "read a second time"
