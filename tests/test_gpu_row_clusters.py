"""The kernels that give a row to a cluster of CTAs (full-vocabulary rows, speculative draws), the finish
that sorts a top-k row's candidates in registers, and the streaming pass's piece sizes, against the
oracle at the sizes where they can go wrong: edges of 256-element tiles, vocabularies that are not aligned,
one row (the largest cluster) and many (the smallest), nuclei narrow and wide, equal values at the cut,
list lengths around the K2 of a warp's sort."""
import numpy as np
import pytest

from opentail.stingray_b200 import workloads as W
from tests import parity

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bs():
    from opentail.stingray_b200 import BatchSampler

    s = BatchSampler(max_rows=320, max_vocab=262144, max_history=600, max_top_k=320, max_spec_draft=3)
    yield s
    s.close()


def _workload(rows, vocab, bf16, seed, topk=False, sigma=2.5):
    rng = np.random.default_rng(seed)
    x = rng.normal(0, sigma, (rows, vocab)).astype(np.float32)
    x[::3, rng.integers(0, vocab, 8)] += 7.0  # peaked rows beside flat ones: narrow nuclei beside wide ones
    p = W._params(rows, repetition_penalty=1.1, repeat_last_n=48)
    p["temperature"] = rng.choice(np.array([0.4, 1.0, 1.3], np.float32), rows)
    p["top_p"] = rng.choice(np.array([0.5, 0.9, 0.99, 0.9995, 1.0], np.float32), rows)
    p["min_p"] = rng.choice(np.array([0.0, 0.0, 0.02], np.float32), rows)
    p["frequency_penalty"] = rng.choice(np.array([0.0, 0.5], np.float32), rows)
    if topk:
        p["top_k"] = rng.choice(np.array([1, 31, 63, 64, 127, 128, 255, 256]), rows)
    hist = W.zipf_ids(rng, rows, 96, vocab)
    ids, off = W._csr(np.array(hist))
    return W.SampleWorkload("rows", W.to_bf16_bits(x) if bf16 else x, p, W.uniforms24(rng, rows), ids, off)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows,vocab", [(1, 255), (2, 256), (3, 257), (1, 4095), (5, 50257), (1, 151936), (3, 262144), (40, 33001)])
def test_full_vocabulary_rows(bs, rows, vocab, bf16):
    w = _workload(rows, vocab, bf16, 7 * vocab + rows)
    stats = parity.compare(w, parity.run_gpu(bs, w))
    assert stats["boundary_draws"] <= 1


def test_more_rows_than_clusters_fit_at_once(bs):
    w = _workload(310, 16640, False, 5)
    stats = parity.compare(w, parity.run_gpu(bs, w))
    assert stats["boundary_draws"] <= 1


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows,vocab", [(1, 16384), (2, 20481), (1, 151936), (64, 33000), (3, 262144)])
def test_top_k_rows(bs, rows, vocab, bf16):
    w = _workload(rows, vocab, bf16, 11 * vocab + rows, topk=True)
    stats = parity.compare(w, parity.run_gpu(bs, w, want_topk=256))
    assert stats["boundary_draws"] <= 1


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("top_k,run", [(1, 2), (4, 2), (31, 5), (40, 31), (40, 40), (100, 2)])
def test_penalised_logits_that_come_out_equal(bs, top_k, run, bf16):
    """Pairs like 11 / 1.1^2 and 10 / 1.1 among the best, and runs of equal values up to and beyond what is
    ordered in place: the order among them is that of the raw logits."""
    rows, vocab = 3, 33000
    rng = np.random.default_rng(top_k)
    x = rng.normal(0, 1.0, (rows, vocab)).astype(np.float32)
    hist = []
    for r in range(rows):
        tok = rng.permutation(vocab)[: 2 * run + 12]
        x[r, tok[:run]], x[r, tok[run:2 * run]] = 11.0, 10.0
        x[r, tok[2 * run:]] = np.repeat(np.float32([22, 20, 5.5, 5, 8.8125, 8.0]), 2)
        h = np.concatenate([np.repeat(tok[:run], 2), tok[run:2 * run], np.repeat(tok[2 * run::2], 2), tok[2 * run + 1::2]])
        hist.append(rng.permutation(h))
    p = W._params(rows, repetition_penalty=1.1)
    p["temperature"], p["top_p"], p["top_k"], p["repeat_last_n"] = 1.0, 0.999, top_k, 256
    ids, off = W._csr(np.array(hist))
    w = W.SampleWorkload("ties", W.to_bf16_bits(x) if bf16 else x, p, W.uniforms24(rng, rows), ids, off)
    parity.compare(w, parity.run_gpu(bs, w, want_topk=100))


def _row_of_many_equal_top_logits(rng, vocab):
    """Over a thousand tokens of one exp value just above 1/4 whose lower mantissa bits are high - together more than 20 bits
    hold - bring the sum of the probabilities to just above 1/2; behind them a few single tokens, then half of the mass in
    bins of two or three hundred.  Those differ a little: of hundreds of equal addends half a unit of the sum off its grid, a
    last bit of exp decides the rounding of all."""
    v = 0.25 + 2000.0 * 2.0 ** -25
    while True:
        n, over = int(rng.integers(1055, 1110)), rng.uniform(7e-5, 9e-5)
        total = 2.0 * (1.0 + n * v) / (1.0 + over)
        if abs((v / total * 2.0 ** 25 + 0.5) % 1.0 - 0.5) < 0.03:  # the sequential sum stays close to the real one
            break
    bins = 0.0078125 * 2.0 ** (-(np.arange(260) // 128)) * (1.0 - (np.arange(260) % 128 + 0.5) / 256.0)
    single, rest = bins[:8], bins[8:]
    counts = np.full(rest.size, int((total - 1.0 - n * v) / rest.sum()))
    left = total - 1.0 - n * v - single.sum() - (counts * rest).sum()
    for i in range(rest.size):  # what is missing, a token at a time
        more = int(left / rest[i]) if i + 40 > rest.size else min(int(left / rest[i]), 1)
        counts[i] += more
        left -= more * rest[i]
    rest = np.repeat(rest, counts)
    e = np.concatenate([[1.0], np.full(n, v), single, rest * (1.0 + rng.uniform(-1e-3, 1e-3, rest.size))])
    x = np.full(vocab, -80.0, np.float32)
    x[:e.size] = np.log(e)
    return rng.permutation(x)


@pytest.mark.parametrize("rows", [1, 20, 80])
def test_a_thousand_equal_top_logits(bs, rows):
    """The histogram's masses of such a row have to be good to 6e-5 for the binades of the nucleus sum to be known, else the
    row is done twice."""
    vocab = 131072
    rng = np.random.default_rng(rows)
    p = W._params(rows, top_p=0.9)
    w = W.SampleWorkload("equal", np.stack([_row_of_many_equal_top_logits(rng, vocab) for _ in range(rows)]), p, W.uniforms24(rng, rows))
    gpu = parity.run_gpu(bs, w)
    stats = parity.compare(w, gpu)
    assert stats["boundary_draws"] <= 1
    assert not (gpu["flags"].view(np.uint32) >> 8 & 1).any()


@pytest.mark.parametrize("below", [1e-4, 9e-4])
@pytest.mark.parametrize("rows,vocab", [(1, 300), (7, 40000)])
def test_min_p_leaves_less_than_top_p(bs, rows, vocab, below):
    """A token a little below min-p's threshold, whose mass is what the survivors lack to top_p: the sum never gets there and
    every survivor stays.  Nothing has to be done twice for that."""
    rng = np.random.default_rng(vocab)
    p = W._params(rows)
    x = np.full((rows, vocab), -40.0, np.float32)
    for r in range(rows):
        min_p = np.float32(rng.uniform(0.01, 0.1))
        e = np.concatenate([[1.0], rng.uniform(1.5 * min_p, 0.9, 12), [min_p * (1.0 - below)], rng.uniform(0, 0.3 * min_p, 100)])
        x[r, rng.permutation(vocab)[: e.size]] = np.log(e)
        p["min_p"][r], p["top_p"][r] = min_p, (e[:13].sum() + 0.5 * e[13]) / e.sum()
    w = W.SampleWorkload("min_p", x, p, W.uniforms24(rng, rows))
    gpu = parity.run_gpu(bs, w)
    parity.compare(w, gpu)
    assert not (gpu["flags"].view(np.uint32) >> 8 & 1).any()
