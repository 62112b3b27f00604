"""What a user of the sampling library has it do, as cases that can be timed and compared.

A serving engine keeps one library handle, a stream of its own and fixed output buffers; every decode
step it hands the step's logits over and takes tokens (and the probability of each) back.  The cases
are such steps from a single chat to a 512-row shard, the drop-in call on host logits, speculative
verification, and the draw that returns the distribution beside the token.  Sizes and value
distributions are those of the configurations in ``opentail/stingray_b200/workloads.py`` and of the
tests, or lie between them; all inputs are generated, on the GPU, from the seed.

Kinds (``case["kind"]``):

  step     ``BatchSampler.sample_rows``, everything resident on the GPU, one batch composition
  turn     ``BatchSampler.sample_rows`` with host-resident histories that grow by a token per step, so
           that every step brings a new batch description (continuous batching without device histories)
  loop     ``sample_rows(history_ring=True)`` followed by ``history_append`` (device-resident histories),
           with the alternatives of every token asked for
  greedy   ``BatchSampler.argmax_rows``
  single   ``Sampler.Sample`` on host logits: the managed API's own signature
  spec     ``BatchSampler.spec_verify``
  dist     ``BatchSampler.sample_with_distribution``: the draft side of speculative decoding
"""
import numpy as np
import torch

from opentail.stingray_b200 import BatchSampler, Sampler, SamplingParams
from opentail.stingray_b200.sampler import PARAMS_DTYPE, Random

SHORT, LONG = 32_000, 262_144  # vocabularies of the tests and configurations lie between these
MAX_HISTORY = 512


# ---- the cases -----------------------------------------------------------------------------------------

def _case(name, kind, rows, vocab, dtype="f32", mix="topk", history=0, mask=False, logits="peaked", draft=0):
    c = {"kind": kind, "rows": rows, "vocab": vocab, "dtype": dtype, "mix": mix, "history": history, "mask": mask,
         "logits": logits, "draft": draft}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one chat: repetition penalty over 64 tokens, top-k 40, top-p 0.95, min-p 0.05 (the single-row configuration)
        _case("chat_top_k", "step", 1, 151_936, history=64),
        # one chat on a small vocabulary with bf16 logits and no top-k: the whole vocabulary takes part in the draw
        _case("chat_nucleus", "step", 1, 32_000, dtype="bf16", mix="nucleus", history=64),
        # the managed API as it is called today: one row of host logits in, one token out
        _case("chat_host_logits", "single", 1, 151_936, history=64),
        # a server's decode step, mixed requests (the batched server-decode configuration, the benchmark's headline)
        _case("server_mixed", "step", 256, 151_936, mix="mixed", history=512, logits="flat"),
        # a small server whose sessions differ in history length and whose vocabulary is odd, so rows are not aligned;
        # the histories live on the host and grow with every step
        _case("server_ragged", "turn", 24, 50_257, mix="mixed", history=300),
        # a decode loop with device-resident histories and bf16 logits, alternatives of every token returned
        _case("server_loop", "loop", 96, 151_936, dtype="bf16", history=256),
        # an evaluation run: every row plain arg-max
        _case("greedy_batch", "greedy", 256, 151_936, mix="greedy", logits="flat"),
        # structured output: an allowed-token bitmask per row (the grammar configuration)
        _case("grammar", "step", 64, 262_144, dtype="bf16", mix="nucleus", mask=True, logits="flat"),
        # one GPU's rows of the large multi-GPU configuration
        _case("large_top_k", "step", 512, 256_000, history=256, logits="flat"),
        # speculative decoding for one chat
        _case("spec_chat", "spec", 1, 151_936, mix="nucleus", draft=4),
        # speculative decoding for a batch (the verification configuration)
        _case("spec_batch", "spec", 32, 151_936, mix="full", draft=8, logits="flat"),
        # the draft model's side of it: tokens together with the distributions they were drawn from
        _case("draft_draw", "dist", 16, 151_936, mix="nucleus", history=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(2.0 ** rng.uniform(np.log2(lo), np.log2(hi))))


def draw(rng):
    """Another case of the same ranges.  Vocabularies from 32,000 to 262,144, mostly padded to a multiple
    of 64 as model heads are, some only even or odd; row counts over the range of each kind, limited so
    that no case costs more than the listed ones do."""
    kind = rng.choice(["step", "step", "step", "step", "turn", "loop", "greedy", "single", "spec", "spec", "dist"])
    vocab = _log_int(rng, SHORT, LONG)
    pad = rng.choice([64, 64, 64, 64, 2, 1])
    vocab = min(LONG, (vocab + pad - 1) // pad * pad)
    dtype = rng.choice(["f32", "f32", "bf16"])
    logits = rng.choice(["flat", "peaked"])
    history = rng.choice([0, 64, _log_int(rng, 1, MAX_HISTORY), MAX_HISTORY])

    def rows(limit_elements, most):
        return max(1, min(_log_int(rng, 1, most), limit_elements // vocab))

    if kind == "step":
        mix = rng.choice(["topk", "topk", "mixed", "mixed", "nucleus"])
        limit = {"topk": 120_000_000, "mixed": 40_000_000, "nucleus": 12_000_000}[mix]
        return _case(None, kind, rows(limit, 512), vocab, dtype, mix, history, rng.random() < 0.25, logits)
    if kind == "turn":
        return _case(None, kind, rows(12_000_000, 128), vocab, dtype, rng.choice(["topk", "mixed"]), max(8, history), False, logits)
    if kind == "loop":
        return _case(None, kind, rows(60_000_000, 256), vocab, dtype, "topk", max(64, history), False, logits)
    if kind == "greedy":
        return _case(None, kind, rows(100_000_000, 512), vocab, dtype, "greedy", 0, False, logits)
    if kind == "single":
        return _case(None, kind, 1, vocab, "f32", rng.choice(["topk", "nucleus"]), history, False, logits)
    if kind == "spec":
        draft = rng.randint(1, 8)
        n = max(1, min(_log_int(rng, 1, 32), 40_000_000 // (vocab * (2 * draft + 1))))
        return _case(None, kind, n, vocab, dtype, rng.choice(["full", "nucleus"]), 0, False, logits, draft)
    return _case(None, kind, rows(3_000_000, 32), vocab, dtype, "nucleus", history, False, logits)


# ---- inputs --------------------------------------------------------------------------------------------

def _logits(g, rows, vocab, how, dtype, dev):
    """flat: N(0, 2.5^2), as in the configurations.  peaked: N(0, 3^2) with 16 ids boosted by 2 to 10, the
    shape a model's head gives when it has an idea what comes next."""
    x = torch.randn((rows, vocab), generator=g, device=dev)
    x *= 2.5 if how == "flat" else 3.0
    if how == "peaked":
        ids = torch.randint(0, vocab, (rows, 16), generator=g, device=dev)
        x.scatter_add_(1, ids, 2.0 + 8.0 * torch.rand((rows, 16), generator=g, device=dev))
    return x.to(torch.bfloat16) if dtype == "bf16" else x


def _uniforms(g, shape, dev, dtype=torch.float32):
    """(j + 0.5) / 2^24: never 0 or 1, exactly representable."""
    return ((torch.randint(0, 1 << 24, shape, generator=g, device=dev).double() + 0.5) / float(1 << 24)).to(dtype)


def _histories(g, rows, length, vocab, dev):
    """Token ids by Zipf(1.1) over the ranks, as text repeats itself."""
    w = torch.arange(1, vocab + 1, device=dev, dtype=torch.float64).pow(-1.1)
    cdf = torch.cumsum(w, 0)
    u = torch.rand((rows, length), generator=g, device=dev, dtype=torch.float64) * cdf[-1]
    return torch.searchsorted(cdf, u).clamp_(max=vocab - 1).to(torch.int32)


def _mask(g, rows, vocab, dev):
    """Allowed-token bits, density log-uniform in [0.1 %, 30 %], at least one bit set per row."""
    words = (vocab + 31) // 32
    dens = torch.exp(torch.empty(rows, 1, device=dev).uniform_(float(np.log(0.001)), float(np.log(0.30)), generator=g))
    bits = torch.zeros((rows, words * 32), dtype=torch.bool, device=dev)
    bits[:, :vocab] = torch.rand((rows, vocab), generator=g, device=dev) < dens
    bits[torch.arange(rows, device=dev), torch.randint(0, vocab, (rows,), generator=g, device=dev)] = True
    weights = torch.ones(32, dtype=torch.int64, device=dev) << torch.arange(32, device=dev)
    out = torch.empty((rows, words), dtype=torch.int32, device=dev)
    for r in range(0, rows, 32):  # a block of rows at a time: the sum below is 64-bit
        v = (bits[r:r + 32].view(-1, words, 32).to(torch.int64) * weights).sum(-1)
        out[r:r + 32] = torch.where(v >= 1 << 31, v - (1 << 32), v).to(torch.int32)
    return out


def _params(rng, rows, mix, history):
    """Per-row request parameters.  The kind of every row follows from its index, so that two seeds cost
    the same; temperatures and thresholds are the seed's."""
    p = np.zeros(rows, PARAMS_DTYPE)
    p["temperature"], p["top_p"], p["repetition_penalty"], p["repeat_last_n"] = 1.0, 1.0, 1.0, 64
    if mix == "greedy":
        p["temperature"] = 0.0
        return p
    if mix == "full":
        return p  # temperature 1, nothing filtered
    p["temperature"] = rng.uniform(0.5, 1.1, rows).astype(np.float32)
    if mix == "topk":
        p["top_k"] = np.array([40, 50, 20, 64])[np.arange(rows) % 4]
        p["top_p"] = rng.uniform(0.85, 0.98, rows).astype(np.float32)
        p["min_p"] = np.where(np.arange(rows) % 2 == 0, 0.05, 0.0)
        if history:
            p["repetition_penalty"] = 1.1
    elif mix == "nucleus":
        p["top_p"] = rng.uniform(0.85, 0.98, rows).astype(np.float32)
        p["min_p"] = np.where(np.arange(rows) % 4 == 1, 0.02, 0.0)
        if history:
            p["repetition_penalty"] = 1.1
    else:  # mixed: the server-decode configuration
        p["temperature"] = rng.uniform(0.3, 1.2, rows).astype(np.float32)
        p["top_k"] = np.array([0, 20, 50, 100])[np.arange(rows) % 4]
        p["top_p"] = rng.uniform(0.8, 1.0, rows).astype(np.float32)
        if history:
            p["frequency_penalty"], p["presence_penalty"] = 0.5, 0.3
    return p


_engine_stream = None


def _stream(dev):
    """The engine's stream.  The whole program runs on it, as bench.py does."""
    global _engine_stream
    if _engine_stream is None:
        _engine_stream = torch.cuda.Stream(dev)
    torch.cuda.set_stream(_engine_stream)
    return _engine_stream


class _State:
    pass


def prepare(case, seed):
    dev = torch.device("cuda", 0)
    s = _State()
    s.kind, s.stream, s.out, s.calls = case["kind"], _stream(dev), None, 0
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    rows, vocab, hist = case["rows"], case["vocab"], case["history"]
    if s.kind == "spec":
        _prepare_spec(s, case, g, rng, dev)
        return s
    s.logits = _logits(g, rows, vocab, case["logits"], case["dtype"], dev)
    s.params = _params(rng, rows, case["mix"], hist)
    if s.kind == "greedy":
        s.sampler = BatchSampler(max_rows=rows, max_vocab=vocab, max_history=1, max_top_k=1)
        return s
    ids = _histories(g, rows, hist, vocab, dev) if hist else None
    if s.kind == "single":
        s.logits = s.logits[0].cpu().numpy()
        p = s.params[0]
        s.params = SamplingParams(Temperature=float(p["temperature"]), TopK=int(p["top_k"]), TopP=float(p["top_p"]),
                                  MinP=float(p["min_p"]), RepetitionPenalty=float(p["repetition_penalty"]),
                                  PreviousTokens=ids[0].tolist() if hist else None)
        s.rng = Random(int(seed))
        return s
    s.sampler = BatchSampler(max_rows=rows, max_vocab=vocab, max_history=max(hist, 1), max_top_k=128)
    s.uniforms = _uniforms(g, (rows,), dev)
    s.inputs = {"uniforms": s.uniforms}
    if case["mask"]:
        s.inputs["mask"] = _mask(g, rows, vocab, dev)
    if s.kind == "loop":
        s.sampler.history_reset()
        host = ids.cpu().numpy()
        for r in range(rows):
            s.sampler.history_load(r, host[r])
        s.inputs["history_ring"] = True
        s.want_topk = int(s.params["top_k"].max())
        torch.cuda.synchronize()  # the loads read `host`
    elif s.kind == "turn":
        # sessions of different lengths; step k of four has k more tokens in each
        full = ids.cpu().numpy()
        base = rng.integers(max(1, hist // 8), hist - 3, rows)
        s.turns = []
        for k in range(4):
            n = base + k
            s.turns.append((np.concatenate([full[r, :n[r]] for r in range(rows)]),
                            np.concatenate([[0], np.cumsum(n)]).astype(np.int32)))
    elif hist:
        s.inputs.update(history_ids=ids.reshape(-1), history_offsets=(np.arange(rows + 1) * hist).astype(np.int32))
    return s


def _prepare_spec(s, case, g, rng, dev):
    n, vocab, L = case["rows"], case["vocab"], case["draft"]
    draft = _logits(g, n * L, vocab, case["logits"], "f32", dev).view(n, L, vocab)
    s.target = torch.empty((n, L + 1, vocab), device=dev)
    s.target[:, :L] = draft + 0.5 * torch.randn((n, L, vocab), generator=g, device=dev)
    s.target[:, L] = _logits(g, n, vocab, case["logits"], "f32", dev)
    s.params = _params(rng, n, case["mix"], 0)
    t = torch.from_numpy(s.params["temperature"].copy()).to(dev)
    probs = torch.softmax(draft / t[:, None, None], -1).view(n * L, vocab)
    s.tokens = torch.multinomial(probs, 1, generator=g).view(n, L).to(torch.int32)
    s.draft = draft
    if case["dtype"] == "bf16":
        s.target, s.draft = s.target.to(torch.bfloat16), draft.to(torch.bfloat16)
    s.uniforms = _uniforms(g, (n, L + 2), dev, torch.float64)
    s.sampler = BatchSampler(max_rows=n * (L + 1), max_vocab=vocab, max_history=1, max_top_k=8, max_spec_draft=L)


# ---- one pass ------------------------------------------------------------------------------------------

def run(s):
    if s.kind == "step":
        s.out = s.sampler.sample_rows(s.logits, s.params, want_probs=True, stream=s.stream, out=s.out, **s.inputs)
        return s.out
    if s.kind == "turn":
        ids, offsets = s.turns[s.calls & 3]
        s.calls += 1
        s.out = s.sampler.sample_rows(s.logits, s.params, history_ids=ids, history_offsets=offsets, want_probs=True,
                                      stream=s.stream, out=s.out, **s.inputs)
        return s.out
    if s.kind == "loop":
        s.out = s.sampler.sample_rows(s.logits, s.params, want_probs=True, want_topk=s.want_topk, stream=s.stream,
                                      out=s.out, **s.inputs)
        s.sampler.history_append(s.out["tokens"], stream=s.stream)
        # a row's alternatives end at its own top_k; what lies behind them in the buffers is not written
        return {"tokens": s.out["tokens"], "probs": s.out["probs"], "topk_ids": s.out["topk_ids"][:, :20],
                "topk_logits": s.out["topk_logits"][:, :20], "topk_probs": s.out["topk_probs"][:, :20]}
    if s.kind == "greedy":
        return s.sampler.argmax_rows(s.logits, stream=s.stream)
    if s.kind == "single":
        return Sampler.Sample(s.logits, s.params, s.rng)
    if s.kind == "spec":
        return s.sampler.spec_verify(s.target, s.draft, s.tokens, s.params, s.uniforms, want_probs=True, stream=s.stream)
    return s.sampler.sample_with_distribution(s.logits, s.params, stream=s.stream, **s.inputs)




# ---- what a pass cannot do without, and how far a correct result may be off ------------------------------

def work(case):
    rows, vocab = case["rows"], case["vocab"]
    esz = 2 if case["dtype"] == "bf16" else 4
    if case["kind"] == "spec":
        elements = rows * (2 * case["draft"] + 1) * vocab
        return {"bytes": elements * esz + rows * (case["draft"] * 8 + (case["draft"] + 2) * 8 + 48), "flops": 6 * elements}
    elements = rows * vocab
    b = elements * esz + rows * (32 + 4 + 8 + 4 * case["history"])
    if case["mask"]:
        b += rows * ((vocab + 31) // 32) * 4
    if case["kind"] == "dist":
        b += elements * 4
    if case["kind"] == "loop":
        b += rows * 64 * 12
    return {"bytes": b, "flops": elements if case["mix"] in ("greedy", "topk") else 6 * elements}


def tolerance(case):
    if case["kind"] in ("greedy", "single"):
        return "exact"
    return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
