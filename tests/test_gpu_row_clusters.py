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
