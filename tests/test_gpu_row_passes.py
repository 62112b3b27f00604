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
        stats = parity.compare(w, parity.run_gpu(bs, w, want_topk=int(params["top_k"].max())))
        assert stats["mismatch"] == stats["boundary_draws"] <= 1
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
def test_top_k_at_the_sizes_of_the_register_sort(top_k, rows):
    """Where the sort takes twice as many keys and the history's hash, filled ahead of the candidates, lies elsewhere: logits in
    steps of 1/4, penalised in small steps, half of the tokens near the cut in the history."""
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
