"""Repeatability: the same batch on the same handle must give the same tokens, flags and probabilities
every time, whatever the handle ran before.  The sweep's batches are repeated in random order on one
handle, on the legacy default stream (direct launches) and on a stream of the test's own (where the
library replays repeated steps as CUDA graphs); the first run of each batch is checked against the
oracle, every later run against the first.  Results that depend on what a CTA processed before, or
on how the streams happened to interleave, show up here and nowhere else."""
import numpy as np
import pytest

from tests import parity
from tests.test_gpu_random_sweep import _workload

pytestmark = pytest.mark.gpu

CASES = [0, 1, 2, 3, 4, 9, 11, 69, 78, 141, 149, 171, 195]


def _run(bs, w, dev, outs, it):
    import torch

    kw = dict(uniforms=dev["uniforms"], want_probs=True, want_flags=True, want_topk=512)
    if w.history_ids is not None:
        kw.update(history_ids=dev["history_ids"], history_offsets=w.history_offsets)
    if w.mask is not None:
        kw["mask"] = dev["mask"]
    outs[it] = bs.sample_rows(dev["logits"], w.params, out=outs.get(it), **kw)
    torch.cuda.synchronize()
    return {k: v.cpu().numpy() for k, v in outs[it].items()}


@pytest.mark.parametrize("own_stream", [False, True])
def test_repeated_batches_in_random_order(own_stream):
    import torch
    from opentail.stingray_b200 import BatchSampler

    bs = BatchSampler(max_rows=64, max_vocab=262144, max_history=1024, max_top_k=512)
    st = torch.cuda.Stream() if own_stream else torch.cuda.current_stream()
    try:
        with torch.cuda.stream(st):
            ws = {it: _workload(it) for it in CASES}
            devs = {it: parity.to_device(ws[it]) for it in CASES}
            first, outs = {}, {}
            rng = np.random.default_rng(7)
            for rep in range(25):
                for it in (rng.permutation(CASES) if rep else CASES):
                    it = int(it)
                    # a step is replayed when it follows itself: a batch of another kind has another plan
                    for _ in range(3 if own_stream else 1):
                        gpu = _run(bs, ws[it], devs[it], outs, it)
                        if it not in first:
                            parity.compare(ws[it], gpu)
                            first[it] = gpu
                            continue
                        for key in ("tokens", "flags", "probs"):
                            np.testing.assert_array_equal(gpu[key].view(np.uint32), first[it][key].view(np.uint32),
                                                          err_msg=f"case {it}, repeat {rep}: {key} differ from the first run")
        # (a replay also needs the same output buffers, which a batch keeps here)
        assert (bs.stats()["graph_replays"] > 100) == own_stream
    finally:
        bs.close()


def test_penalised_top_k_rows_keep_every_candidate():
    """Rows whose candidates are looked up in a long history: three rows of the sweep's batch 1, repeated.  With a lookup that
    lanes left one by one, and a register sort behind it, a warp's candidates were lost once in a few hundred to a few
    thousand steps."""
    import torch
    from opentail.stingray_b200 import BatchSampler, workloads as W

    w, rows = _workload(1), [10, 22, 32]
    h = int(w.history_offsets[1])
    w = W.SampleWorkload("s", np.ascontiguousarray(w.logits[rows]), w.params[rows].copy(), w.uniforms[rows].copy(),
                         np.concatenate([w.history_ids[r * h:(r + 1) * h] for r in rows]), np.arange(4, dtype=np.int32) * h, None)
    bs = BatchSampler(max_rows=4, max_vocab=262144, max_history=1024, max_top_k=64)
    try:
        dev = parity.to_device(w)
        kw = dict(uniforms=dev["uniforms"], history_ids=dev["history_ids"], history_offsets=w.history_offsets,
                  want_probs=True, want_flags=True, want_topk=40)
        out = bs.sample_rows(dev["logits"], w.params, **kw)
        torch.cuda.synchronize()
        parity.compare(w, {k: v.cpu().numpy() for k, v in out.items()})
        first = {k: v.clone() for k, v in out.items()}
        differ = torch.zeros(1, dtype=torch.int64, device="cuda")
        for _ in range(10_000):
            out = bs.sample_rows(dev["logits"], w.params, out=out, **kw)
            differ += (out["topk_ids"] != first["topk_ids"]).any() | (out["probs"] != first["probs"]).any()
        assert int(differ) == 0
    finally:
        bs.close()


def test_full_rows_with_long_histories_repeat():
    """Loops that lanes leave one by one ahead of warp-wide operations: the overrides of a lane's own tokens, and the rounding
    ties of a wide nucleus.  Five thousand steps of rows full of both."""
    import torch
    from opentail.stingray_b200 import BatchSampler, workloads as W

    rows, vocab, h = 6, 50_257, 1200
    rng = np.random.default_rng(51)
    x = rng.normal(0, 2.5, (rows, vocab)).astype(np.float32)
    x[::2] = np.round(x[::2] * 8) / 8
    p = W._params(rows, top_p=0.95, repetition_penalty=1.1, presence_penalty=0.25, repeat_last_n=0)
    p["temperature"] = np.resize([1.0, 0.9, 1.2], rows)
    # tokens side by side, so that a lane has several overrides
    hist = np.concatenate([(rng.integers(0, vocab // 64, h) * 64 + rng.integers(0, 12, h)) % vocab for _ in range(rows)]).astype(np.int32)
    w = W.SampleWorkload("s", x, p, W.uniforms24(rng, rows), hist, np.arange(rows + 1, dtype=np.int32) * h, None)
    bs = BatchSampler(max_rows=rows, max_vocab=vocab, max_history=2048, max_top_k=8)
    try:
        dev = parity.to_device(w)
        kw = dict(uniforms=dev["uniforms"], history_ids=dev["history_ids"], history_offsets=w.history_offsets,
                  want_probs=True, want_flags=True)
        out = bs.sample_rows(dev["logits"], w.params, **kw)
        torch.cuda.synchronize()
        parity.compare(w, {k: v.cpu().numpy() for k, v in out.items()})
        first = {k: v.clone() for k, v in out.items()}
        differ = torch.zeros(1, dtype=torch.int64, device="cuda")
        for _ in range(5_000):
            out = bs.sample_rows(dev["logits"], w.params, out=out, **kw)
            differ += (out["tokens"] != first["tokens"]).any() | (out["probs"] != first["probs"]).any() | (out["flags"] != first["flags"]).any()
        assert int(differ) == 0
    finally:
        bs.close()
