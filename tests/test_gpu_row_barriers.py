"""The cluster barriers of the full-vocabulary kernels (stg_row.cu), on rows that put the least work between them, and the
rounds in which the nucleus sum asks for a histogram bin whose order it was not expected to need."""
import numpy as np
import pytest

from opentail.stingray_b200 import workloads as W
from tests import parity

pytestmark = pytest.mark.gpu

BINS = 100       # histogram bins (1/128 of a binade wide) a row's values lie in
HIDDEN = -80.0   # a logit that weighs nothing


def _row_that_asks_for_a_bin(rng, vocab):
    """(logits, top_p): neighbouring bins of a few hundred equal values each.  Equal addends round the same way every
    time - here by 0.3 of a unit of sums above 1/2, all up or all down - so the sequential fp32 sum runs away from the
    real one; top_p lies between the two at the end of a bin, so that the sum meets it in the neighbour of the bin it
    should.  None when this draw holds no such place."""
    counts = rng.integers(300, 700, BINS)
    counts[0] = 1  # the maximum: exp value 1, a bin of its own
    mid = 1.0 - (np.arange(BINS - 1) + 0.5) / 256.0  # the middles of the bins below 1
    part = rng.choice([0.3, 0.7])
    e = mid.copy()
    for _ in range(8):  # the values decide the sum, which decides what a unit is
        unit = 2.0 ** -24 * float(1.0 + (counts[1:] * e).sum())
        e = (np.round(mid / unit - part) + part) * unit
    logit = np.concatenate([[0.0], np.log(e)]).astype(np.float32)
    seq = np.repeat(np.exp(logit).astype(np.float32), counts)
    p = seq * (np.float32(1.0) / np.cumsum(seq, dtype=np.float32)[-1])
    run, real = np.cumsum(p, dtype=np.float32), np.cumsum(p.astype(np.float64))
    ends = np.cumsum(counts) - 1
    off = run[ends].astype(np.float64) - real[ends]
    usable = np.flatnonzero((np.abs(off) > 2e-4) & (real[ends] > 0.55) & (real[ends] < 0.95))  # the kernel allows for 6e-5
    if usable.size == 0 or seq.size > vocab:
        return None
    k = rng.choice(usable)
    x = np.full(vocab, HIDDEN, np.float32)
    x[:seq.size] = np.repeat(logit, counts)
    return rng.permutation(x), np.float32(real[ends[k]] + 0.7 * off[k])


def rows_that_ask_for_bins(rows, vocab, seed):
    rng = np.random.default_rng(seed)
    x, top_p = np.empty((rows, vocab), np.float32), np.empty(rows, np.float32)
    for r in range(rows):
        made = None
        while made is None:
            made = _row_that_asks_for_a_bin(rng, vocab)
        x[r], top_p[r] = made
    p = W._params(rows)
    p["top_p"] = top_p
    return W.SampleWorkload("bins", x, p, W.uniforms24(rng, rows))


@pytest.fixture(scope="module")
def bs():
    from opentail.stingray_b200 import BatchSampler

    s = BatchSampler(max_rows=320, max_vocab=262144, max_history=64, max_top_k=64, max_spec_draft=3)
    yield s
    s.close()


@pytest.mark.parametrize("rows,vocab", [(1, 151936), (2, 262144), (12, 131077), (30, 131072), (60, 131072), (150, 131072)])
def test_a_sum_that_asks_for_more_bins(bs, rows, vocab):
    """Clusters of 16, 8, 4, 2 and 1 CTAs; no bin is asked for by a rounding tie, so the first round hands nothing over
    and the CTAs meet only where the cut has been looked for."""
    w = rows_that_ask_for_bins(rows, vocab, 3 * vocab + rows)
    for _ in range(3):
        stats = parity.compare(w, parity.run_gpu(bs, w))
        assert stats["boundary_draws"] <= 1


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows,vocab", [(1, 4096), (1, 262144), (12, 33001), (40, 151936), (150, 32000), (310, 4095)])
def test_rows_of_a_few_allowed_tokens(bs, rows, vocab, bf16):
    """Nothing to read and nothing to sum: every CTA reaches its first push to the others at once."""
    rng = np.random.default_rng(vocab + rows)
    x = rng.normal(0, 2.5, (rows, vocab)).astype(np.float32)
    mask = np.zeros((rows, (vocab + 31) // 32), np.uint32)
    for r in range(rows):
        for t in rng.integers(0, vocab, 1 + r % 3):
            mask[r, t >> 5] |= np.uint32(1) << np.uint32(t & 31)
    p = W._params(rows, temperature=0.8)
    p["top_p"] = rng.choice(np.array([0.7, 0.95, 1.0], np.float32), rows)
    w = W.SampleWorkload("few", W.to_bf16_bits(x) if bf16 else x, p, W.uniforms24(rng, rows), None, None, mask)
    stats = parity.compare(w, parity.run_gpu(bs, w))
    assert stats["boundary_draws"] <= 1
