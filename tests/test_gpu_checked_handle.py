"""A handle created with STG_CHECKED=1 keeps 256 guard bytes behind each of its device buffers; after
a tour of the entry points over awkward shapes (ragged vocabularies, full capacities, bf16 with masks,
wide nuclei, speculative verification, device-resident histories, the mask cache) every guard must
still hold its pattern.  This stands in for a memory checker, which cannot be run where these tests run."""
import ctypes as C
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _checked(**kw):
    from opentail.stingray_b200 import BatchSampler

    os.environ["STG_CHECKED"] = "1"
    try:
        return BatchSampler(**kw)
    finally:
        del os.environ["STG_CHECKED"]


def _guards(bs):
    n, bad = C.c_int32(0), C.c_int32(0)
    rc = bs._lib.stg_debug_check_guards(bs._h, C.byref(n), C.byref(bad))
    assert rc == 0
    return n.value, bad.value


def test_guards_survive_a_tour_of_the_entry_points():
    import torch
    from opentail.stingray_b200 import workloads as W
    from tests import parity

    rows, vocab = 40, 151936
    bs = _checked(max_rows=rows, max_vocab=262144, max_history=512, max_top_k=128, max_bias=8, max_spec_draft=3,
                  max_cached_masks=3, host_logits=True)
    try:
        n0, bad0 = _guards(bs)
        assert n0 > 20 and bad0 == -1
        # mixed rows at full row capacity, histories at full length
        w = W.config2(rows=rows, seed=3)
        parity.compare(w, parity.run_gpu(bs, w, want_topk=int(w.params["top_k"].max())))
        # bf16 + masks, the widest vocabulary
        w3 = W.config3(rows=rows, seed=4)
        parity.compare(w3, parity.run_gpu(bs, w3))
        # a ragged vocabulary and host-resident inputs
        rng = np.random.default_rng(5)
        v = 151936 - 13
        x = rng.normal(0, 2.5, (rows, v)).astype(np.float32)
        p = W._params(rows, temperature=1.1, top_p=0.97)
        p["top_k"][::3] = 64
        bs.sample_rows(x, p, uniforms=rng.random(rows).astype(np.float32), want_probs=True, want_flags=True)
        bs.build_distribution(torch.from_numpy(x[:4]).cuda(), p[:4])
        # speculative verification at the draft capacity
        w4 = W.config4(n_seq=8, n_draft=3, vocab=32000, seed=6)
        bs.spec_verify(torch.from_numpy(w4.target).cuda(), torch.from_numpy(w4.draft).cuda(), torch.from_numpy(w4.draft_tokens).cuda(),
                       w4.params, torch.from_numpy(w4.uniforms).cuda())
        # device-resident histories run to their capacity and beyond
        bs.history_reset()
        pr = W._params(rows, top_k=40, repetition_penalty=1.2)
        pr["repeat_last_n"] = 64
        lg = torch.from_numpy(x).cuda()
        for r in range(rows):
            bs.history_load(r, rng.integers(0, v, 510).astype(np.int32))
        for _ in range(4):
            out = bs.sample_rows(lg, pr, uniforms=torch.from_numpy(rng.random(rows).astype(np.float32)).cuda(), history_ring=True)
            bs.history_append(out["tokens"])
        # the mask cache filled past its capacity
        words = (v + 31) // 32
        for key in (1, 2, 3, 4):
            bs.mask_cache_put(key, rng.integers(0, 1 << 32, words, dtype=np.uint64).astype(np.uint32), v)
        bs.mask_compose(np.array([[2, 3, 4]] * rows, np.uint64), v, "and")
        bs.argmax_rows(lg)
        torch.cuda.synchronize()
        n1, bad1 = _guards(bs)
        assert n1 >= n0 and bad1 == -1, f"guard of buffer {bad1} was overwritten"
    finally:
        bs.close()


def test_unchecked_handles_carry_no_guards():
    from opentail.stingray_b200 import BatchSampler

    bs = BatchSampler(max_rows=4, max_vocab=4096)
    try:
        assert _guards(bs) == (0, -1)
    finally:
        bs.close()


@pytest.mark.parametrize("drilled_pass", ["1", "2"])
def test_a_row_that_is_given_up_costs_a_second_pass_not_the_result(drilled_pass):
    """k_row works with bounds that the exact sums behind them check; a row whose check fails is left to the row kernel.
    The drill makes k_row give every row up, before its sum (1) or at its draw (2).  Tokens and probabilities
    must still be the oracle's, every full-vocabulary row must report the second pass, and the handle must keep
    working."""
    from opentail.stingray_b200 import BatchSampler
    from opentail.stingray_b200 import workloads as W
    from tests import parity

    w = W.config2(rows=24, seed=11)
    os.environ["STG_ROW_DRILL"] = drilled_pass
    try:
        bs = BatchSampler(max_rows=w.rows, max_vocab=w.vocab, max_history=512, max_top_k=128)
    finally:
        del os.environ["STG_ROW_DRILL"]
    try:
        for _ in range(2):
            gpu = parity.run_gpu(bs, w, want_topk=int(w.params["top_k"].max()))
            parity.compare(w, gpu)
            flags = gpu["flags"].view(np.uint32)
            full = (flags & 7) == 3
            assert full.any() and ((flags[full] >> 8) & 1).all(), "every full-vocabulary row should have been redone"
        assert bs.stats()["reread_rows"] >= int(full.sum())
    finally:
        bs.close()


def test_target_and_draft_rows_redone_side_by_side():
    """Both descriptor passes of a speculative step have every row redone at once, in the same scratch rows: more target
    rows than their share of it, more draft rows than theirs."""
    from opentail.stingray_b200 import workloads as W
    from tests.test_gpu_spec_shard import _check_spec

    rng = np.random.default_rng(12)
    n, L, vocab = 44, 3, 20011
    draft = rng.normal(0, 2.5, (n, L, vocab)).astype(np.float32)
    target = np.concatenate([draft + rng.normal(0, 0.5, draft.shape), rng.normal(0, 2.5, (n, 1, vocab))], 1).astype(np.float32)
    p = W._params(n, temperature=0.9)
    p["top_p"][::2] = 0.95
    w = W.SpecWorkload("redo", target, draft, draft.argmax(-1).astype(np.int32), p, rng.random((n, L + 2)))
    os.environ["STG_ROW_DRILL"] = "1"
    try:
        for _ in range(2):
            _check_spec(w)
    finally:
        del os.environ["STG_ROW_DRILL"]


def test_a_handle_for_drafts_costs_little_more():
    """What a handle with room for draft tokens takes more than one without: descriptors and small arrays, no rows of V."""
    import torch
    from opentail.stingray_b200 import BatchSampler

    def taken(**kw):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        bs = BatchSampler(max_rows=8, max_vocab=262144, max_history=8, max_top_k=8, **kw)
        try:
            return before - torch.cuda.mem_get_info()[0]
        finally:
            bs.close()

    taken()  # the library's own context and modules
    assert taken(max_spec_draft=7) - taken() <= 16 << 20


def test_phase_stamps_of_rows_that_were_not_redone():
    """The stamps of a row's phases are k_row's: the redo pass behind it leaves those of the rows it skips alone."""
    from opentail.stingray_b200 import BatchSampler
    from opentail.stingray_b200 import workloads as W
    from tests import parity

    w = W.config2(rows=8, seed=2)
    w.params["top_k"], w.params["top_p"], w.params["temperature"] = 0, 1.0, 1.0  # the phases of a full row, one after the other
    os.environ["STG_PHASE_TICKS"] = "1"
    try:
        bs = BatchSampler(max_rows=w.rows, max_vocab=w.vocab, max_history=512, max_top_k=8)
    finally:
        del os.environ["STG_PHASE_TICKS"]
    try:
        gpu = parity.run_gpu(bs, w)
        assert not (gpu["flags"].view(np.uint32) >> 8 & 1).any()
        stamps, n = np.zeros((w.rows, 32), np.uint64), C.c_int32(0)
        assert bs._lib.stg_debug_phase_ticks(bs._h, stamps.ctypes.data, w.rows, C.byref(n)) == 0 and n.value == w.rows
        order = stamps[:, [0, 1, 2, 3, 4, 5, 10, 11, 12]].astype(np.int64)
        assert (np.diff(order, axis=1) >= 0).all() and (order[:, -1] - order[:, 0] < 10_000_000).all()
    finally:
        bs.close()
