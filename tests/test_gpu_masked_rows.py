"""Full-vocabulary rows without a finite logit - a grammar that has come to a dead end, a row of -infinity - in every form of
the call: every token has probability 1/V, the filters and the draw work on equal values, and the row is done once."""
import itertools

import numpy as np
import pytest

from opentail.stingray_b200 import workloads as W
from oracle import oracle as orc
from tests import parity
from tests.test_gpu_spec_shard import _check_spec

pytestmark = pytest.mark.gpu


def _masked(vocab, seed, by_mask):
    """Every combination of the filters, each with the uniforms where a sum of equal values can go wrong; one live row."""
    rng = np.random.default_rng(seed)
    knobs = list(itertools.product([1.0, 0.5, 0.9, 0.99999, 1e-6], [0.0, 0.05, 1.0, 1.5], [0.0, 0.37, 0.9999999]))
    p = W._params(len(knobs) + 1, repetition_penalty=1.1)
    p["temperature"] = 0.7
    for i, (top_p, min_p, _) in enumerate(knobs):
        p["top_p"][i], p["min_p"][i] = top_p, min_p
    u = np.array([k[2] for k in knobs] + [0.5], np.float32)
    x = rng.normal(0, 2.5, (p.size, vocab)).astype(np.float32)
    mask = None
    if by_mask:
        mask = np.zeros((p.size, (vocab + 31) // 32), np.uint32)
        mask[-1] = 0xFFFFFFFF
        # tokens that are allowed but have no finite logit: the row is closed up to them first
        few = rng.integers(0, vocab, 3)
        x[::2, few] = -np.inf
        for t in few:
            mask[:-1:2, t >> 5] |= np.uint32(1) << np.uint32(t & 31)
        x[-1] = rng.normal(0, 2.5, vocab)
    else:
        x[:-1] = -np.inf
    ids, off = W._csr(W.zipf_ids(rng, p.size, 20, vocab))
    return W.SampleWorkload("masked", x, p, u, ids, off, mask)


@pytest.mark.parametrize("by_mask", [False, True])
@pytest.mark.parametrize("vocab", [1, 2, 3, 255, 4096, 33001, 151936, 262144])
def test_sampled(vocab, by_mask):
    from opentail.stingray_b200 import BatchSampler

    w = _masked(vocab, vocab, by_mask)
    bs = BatchSampler(max_rows=w.rows, max_vocab=vocab, max_history=20, max_top_k=8)
    try:
        gpu = parity.run_gpu(bs, w)
        parity.compare(w, gpu)
        flags = gpu["flags"].view(np.uint32)
        assert (flags[:-1] >> 6 & 1).all() and not flags[-1] >> 6 & 1
        assert not (flags[:-1] >> 8 & 1).any(), "done twice"
        assert bs.stats()["fully_masked_rows"] == w.rows - 1
    finally:
        bs.close()


@pytest.mark.parametrize("by_mask", [False, True])
@pytest.mark.parametrize("vocab", [1, 257, 151936])
def test_distributions(vocab, by_mask):
    import torch
    from opentail.stingray_b200 import BatchSampler

    w = _masked(vocab, vocab + 1, by_mask)
    want = np.stack([orc.build_filtered_distribution(parity.row_logits_f32(w, r), orc.OrcParams(*[w.params[r][n].item() for n in w.params.dtype.names]),
                                                     history=parity.row_history(w, r))[0] for r in range(w.rows - 1)])
    dev = parity.to_device(w)
    kw = dict(history_ids=dev["history_ids"], history_offsets=w.history_offsets)
    if by_mask:
        kw["mask"] = dev["mask"]
    bs = BatchSampler(max_rows=w.rows, max_vocab=vocab, max_history=20, max_top_k=8)
    try:
        drawn, beside = bs.sample_with_distribution(dev["logits"], w.params, uniforms=dev["uniforms"], **kw)
        alone = bs.build_distribution(dev["logits"], w.params, **kw)
        tokens = bs.sample_rows(dev["logits"], w.params, uniforms=dev["uniforms"], **kw)["tokens"]
        torch.cuda.synchronize()
        for got in (beside, alone):
            np.testing.assert_allclose(got.cpu().numpy()[:-1], want, rtol=1e-6, atol=0)
        assert torch.equal(drawn, tokens)
        assert bs.stats()["reread_rows"] == 0
    finally:
        bs.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_speculative_verification(mode):
    """Target and draft rows without a finite logit among ordinary ones."""
    rng = np.random.default_rng(8)
    n, L, vocab = 6, 3, 40000
    draft = rng.normal(0, 2.5, (n, L, vocab)).astype(np.float32)
    target = np.concatenate([draft + rng.normal(0, 0.5, draft.shape), rng.normal(0, 2.5, (n, 1, vocab))], 1).astype(np.float32)
    target[0, 0] = target[1, :] = target[2, 3] = -np.inf
    draft[1, 0] = draft[3, 1] = -np.inf
    p = W._params(n, top_p=0.9)
    p["min_p"][::2] = 0.01
    w = W.SpecWorkload("masked", target, draft, rng.integers(0, 40, (n, L)).astype(np.int32), p, rng.random((n, L + 2)))
    _check_spec(w, mode=mode, p_min=1e-5)
