"""The paged, batched engine against the naive oracle on the tiny CPU config."""
import pytest
import torch

from stkernel_b200.config import CacheConfig, EngineConfig, SchedulerConfig, tiny_config
from stkernel_b200.models.dsv4 import DictSource, build_model_weights
from stkernel_b200.models.dsv4_oracle import OracleModel, index_cache_computes
from stkernel_b200.models.weights import init_random_weights
from stkernel_b200.ops import functional as Fn
from stkernel_b200.runtime.engine import Engine, SamplingParams


@pytest.fixture(autouse=True)
def fp32_acts():
    Fn.set_cpu_act_dtype(torch.float32)
    yield
    Fn.set_cpu_act_dtype(torch.bfloat16)


def close(got, ref, tol=5e-3, frac=0.9):
    """The layer input is rounded to bf16 by design, so a 1e-6 difference upstream can move an
    element by one bf16 ulp and, rarely, flip a router or top-k choice for one token.  Require
    most positions to agree tightly and the whole tensor to agree in norm."""
    err = (got.float() - ref).abs().amax(-1)
    assert (err < tol).float().mean().item() >= frac, err
    assert ((got.float() - ref).norm() / ref.norm()).item() < 5e-2


def make_engine(cfg, w, chunk=4096, seqs=4):
    ec = EngineConfig(model=cfg, sched=SchedulerConfig(max_model_len=512, max_num_seqs=seqs, max_num_batched_tokens=chunk,
                                                       graph_cap=0)).validate()
    weights = build_model_weights(cfg, DictSource(w), "cpu")
    return Engine(ec, weights, "cpu", max_context=512)


def test_index_cache_rule():
    cfg = tiny_config(num_hidden_layers=8, compress_ratios=(4, 0, 4, 4, 0, 4, 4, 4), index_topk_freq=3)
    flags = [index_cache_computes(cfg, i) for i in range(8)]
    assert flags == [True, False, False, False, False, True, False, False]
    cfg1 = tiny_config(num_hidden_layers=3, compress_ratios=(0, 4, 4), index_topk_freq=7)
    assert [index_cache_computes(cfg1, i) for i in range(3)] == [False, True, False]   # first C4A always computes


@pytest.mark.parametrize("chunk", [4096, 24])
def test_prefill_and_greedy_decode_match_oracle(chunk):
    torch.manual_seed(0)
    cfg = tiny_config()
    w = init_random_weights(cfg, seed=0)
    oracle = OracleModel(cfg, w)
    eng = make_engine(cfg, w, chunk=chunk)
    prompts = [torch.randint(0, cfg.vocab_size, (64,)).tolist() for _ in range(2)]
    steps = 32 if chunk == 4096 else 8
    outs = eng.generate(prompts, SamplingParams(temperature=0.0, max_tokens=steps))
    for p, o in zip(prompts, outs):
        ref_ids, ref_logits = oracle.greedy_decode(torch.tensor(p), steps)
        assert o == ref_ids.tolist()


def test_logits_match_oracle_mixed_batch():
    torch.manual_seed(1)
    cfg = tiny_config(num_hidden_layers=3, compress_ratios=(4, 0, 4), index_topk_freq=2)
    w = init_random_weights(cfg, seed=3)
    oracle = OracleModel(cfg, w)
    eng = make_engine(cfg, w)
    a = torch.randint(0, cfg.vocab_size, (50,))
    b = torch.randint(0, cfg.vocab_size, (37,))
    # drive the model directly through two ragged steps to compare full logits
    from stkernel_b200.runtime.engine import Request, ScheduledSeq
    ra, rb = Request(0, a.tolist(), SamplingParams()), Request(1, b.tolist(), SamplingParams())
    ra.row, rb.row = eng.kv.alloc_row(), eng.kv.alloc_row()
    seqs = [ScheduledSeq(ra, 0, 30, False), ScheduledSeq(rb, 0, 37, True)]
    t, n, ns = eng._stage(seqs)
    eng._upload(t, n, ns)
    meta = eng._build_meta(t, n, 16)
    lg1 = eng.model.forward(meta)
    seqs = [ScheduledSeq(ra, 30, 20, True)]
    t, n, ns = eng._stage(seqs)
    eng._upload(t, n, ns)
    meta = eng._build_meta(t, n, 16)
    lg2 = eng.model.forward(meta)
    ref_a, ref_b = oracle.logits(a), oracle.logits(b)
    close(lg1[:30], ref_a[:30])
    close(lg1[30:], ref_b)
    close(lg2, ref_a[30:])


def test_quantised_storage_matches_quant_aware_oracle():
    torch.manual_seed(2)
    cfg = tiny_config(dense_dtype="bf16", kv_cache_dtype="fp8_ds_mla", expert_dtype="nvfp4")
    w = init_random_weights(cfg, seed=5)
    oracle = OracleModel(cfg, w)
    eng = make_engine(cfg, w)
    p = torch.randint(0, cfg.vocab_size, (48,))
    from stkernel_b200.runtime.engine import Request, ScheduledSeq
    r = Request(0, p.tolist(), SamplingParams())
    r.row = eng.kv.alloc_row()
    t, n, ns = eng._stage([ScheduledSeq(r, 0, 48, True)])
    eng._upload(t, n, ns)
    lg = eng.model.forward(eng._build_meta(t, n, 16))
    ref = oracle.logits(p)
    close(lg, ref, tol=1e-2)


def test_padded_decode_bucket_ignores_stale_sample_rows():
    """A decode bucket wider than the step (3 requests in a 4-row bucket) must not read the staged row list: the
    entries past the uploaded ones still hold the row numbers of an earlier, larger step (here a 4-prompt prefill
    whose last sampling row is far beyond the bucket)."""
    torch.manual_seed(3)
    cfg = tiny_config()
    w = init_random_weights(cfg, seed=0)
    eng = make_engine(cfg, w)
    lens = (40, 33, 21, 50)
    ids = [eng.add_request(torch.randint(0, cfg.vocab_size, (n,)).tolist(),
                           SamplingParams(max_tokens=1 if i == 3 else 4)) for i, n in enumerate(lens)]
    eng.step()                                    # one mixed step: all four prompts prefill and sample
    assert eng.requests[ids[3]].finished
    stale = eng.buf.d_logit_rows[:4].tolist()
    assert max(stale) >= 4                        # what a 4-row decode graph would have indexed with
    seqs = eng.sched.schedule()
    assert len(seqs) == 3 and all(s.n == 1 for s in seqs)
    t, n_req, ns = eng._stage(seqs)
    eng._upload(t, n_req, ns)
    eng.buf.d_qstart[n_req + 1:5].fill_(n_req)    # the padding rule of `_decode_graph`
    ref = eng._run_model(t, n_req, ns, 16)
    eng.buf.d_logit_rows.fill_(10 ** 6)           # poison: any read of it would raise on this path
    got = eng._run_model(4, 4, 4, 16, identity_rows=True)
    assert got[:3].tolist() == ref.tolist()


def test_nonzero_device_status_fails_step_and_disables_symmetric_path():
    """Host-side injection: the status word the engine reads after a step says a peer-flag wait ran out.  The step
    must raise, be counted, and switch the symmetric collectives off so that later all-reduces take the library path."""
    from stkernel_b200.runtime.engine import DeviceStatusError

    class FakeSymm:
        enabled = True
        reason = None

        def eligible(self, x):
            return self.enabled

        def all_reduce(self, x):
            return x if self.enabled else None

        def disable(self, reason):
            self.enabled, self.reason = False, reason

    class FakeComm:
        def __init__(self):
            self.symm, self.world_size, self.library_calls = FakeSymm(), 2, 0

        def all_reduce(self, x):
            if self.symm.eligible(x) and self.symm.all_reduce(x) is not None:
                return x
            self.library_calls += 1
            return x

    torch.manual_seed(4)
    cfg = tiny_config()
    eng = make_engine(cfg, init_random_weights(cfg, seed=0))
    eng.model.comm = FakeComm()
    eng.add_request(torch.randint(0, cfg.vocab_size, (12,)).tolist(), SamplingParams(max_tokens=4))
    eng.step()
    assert eng.metrics.device_status_errors == 0
    eng._read_status = lambda: (2, 5)
    with pytest.raises(DeviceStatusError) as ei:
        eng.step()
    assert ei.value.code == 2 and ei.value.detail == 5
    assert eng.metrics.device_status_errors == 1
    assert eng.model.comm.symm.enabled is False and "device status 2" in eng.model.comm.symm.reason
    eng.model.comm.all_reduce(torch.zeros(4))
    assert eng.model.comm.library_calls == 1
    assert "stk:device_status_errors_total" in eng.metrics.render()


def test_indexer_scoring_in_query_subchunks_under_a_logits_budget():
    """With a logits budget of a few hundred bytes the indexer scores a prefill chunk a handful of query rows at a
    time; the selected rows, hence the text, must not change."""
    torch.manual_seed(5)
    cfg = tiny_config()
    w = init_random_weights(cfg, seed=0)
    prompts = [torch.randint(0, cfg.vocab_size, (n,)).tolist() for n in (90, 41)]
    sp = SamplingParams(temperature=0.0, max_tokens=6)
    ref = make_engine(cfg, w).generate(prompts, sp)
    eng = make_engine(cfg, w)
    eng.model.indexer_logits_bytes = 256
    calls = []
    from stkernel_b200.ops import attention as A
    orig = A.indexer_scores
    try:
        A.indexer_scores = lambda q, *a, **k: (calls.append(q.shape[0]), orig(q, *a, **k))[1]
        out = eng.generate(prompts, sp)
    finally:
        A.indexer_scores = orig
    assert out == ref
    assert len(calls) > 20 and max(calls) * 4 * 22 <= 256 + 4 * 22          # rows x compressed rows x 4 bytes within budget


def test_log_probabilities_match_the_oracle_and_do_not_change_the_text():
    torch.manual_seed(0)
    cfg = tiny_config()
    w = init_random_weights(cfg, seed=0)
    eng = make_engine(cfg, w, chunk=48)
    p = torch.randint(0, cfg.vocab_size, (30,)).tolist()
    a = eng.add_request(p, SamplingParams(temperature=0.0, max_tokens=5, logprobs=3))
    b = eng.add_request(p, SamplingParams(temperature=0.0, max_tokens=5))            # same batch, not asking
    while eng.has_work():
        eng.step()
    ra, rb = eng.requests[a], eng.requests[b]
    assert ra.output == rb.output and len(ra.logprobs) == 5 and rb.logprobs == []
    _, logits = OracleModel(cfg, w).greedy_decode(torch.tensor(p), 5)
    ref = torch.log_softmax(logits.float(), -1)
    for i, (lp, top) in enumerate(ra.logprobs):
        assert abs(lp - float(ref[i, ra.output[i]])) < 2e-3
        assert len(top) == 3 and top[0][0] == ra.output[i]
        assert [t for t, _ in top] == ref[i].topk(3).indices.tolist()
    # sampled (temperature 1): the reported value is the model's log-probability of the token that was drawn
    c = eng.add_request(p, SamplingParams(temperature=1.0, seed=5, max_tokens=4, logprobs=0))
    while eng.has_work():
        eng.step()
    rc = eng.requests[c]
    assert len(rc.logprobs) == 4 and all(top == [] and lp <= 0 for lp, top in rc.logprobs)


@pytest.mark.parametrize("seqs", [1, 3, 5, 8, 33])
def test_step_buffers_hold_the_padded_batch(seqs):
    """A captured step of n requests reads the query ranges, rows and sampling inputs of the next power of two."""
    from stkernel_b200.runtime.engine import step_bucket
    cfg = tiny_config()
    eng = make_engine(cfg, init_random_weights(cfg, seed=1), seqs=seqs)
    bucket = step_bucket(seqs)
    assert bucket >= seqs and bucket & (bucket - 1) == 0 and bucket < 2 * seqs
    b = eng.buf
    assert b.d_qstart.numel() >= bucket + 1
    assert min(x.numel() for x in (b.d_tokens, b.d_rows, b.d_start, b.d_temp, b.d_seed, b.d_pos, b.d_topk, b.d_topp)) >= bucket


class PlainStep:
    """Stands for a captured step without a GPU: `replay` runs the step's body over the padded batch."""

    def __init__(self, eng, bucket, rows_bucket, logits=False):
        self.body = lambda: eng._run_logits(bucket, rows_bucket)

    def replay(self):
        return self.body()


@pytest.mark.parametrize("wanted", [([0, 0], []), ([], [0, 0]), ([0], [0]), ([0, 0], [0]), ([], [0])])
def test_captured_feed_steps_give_the_wanted_rows(wanted, monkeypatch):
    """Places that are repeated or absent: the logits are those of an engine that never captures, in the order asked for."""
    from stkernel_b200.runtime import engine as E
    monkeypatch.setattr(E, "DecodeGraph", PlainStep)
    monkeypatch.setattr(Engine, "FEED_EAGER_STEPS", 0)
    torch.manual_seed(4)
    cfg = tiny_config()
    w = init_random_weights(cfg, seed=2)
    tokens = torch.randint(0, cfg.vocab_size, (2, 24)).tolist()
    outs = []
    for captured in (False, True):
        ec = EngineConfig(model=cfg, sched=SchedulerConfig(max_model_len=64, max_num_seqs=2, max_num_batched_tokens=64, graph_cap=8)).validate()
        eng = Engine(ec, build_model_weights(cfg, DictSource(w), "cpu"), "cpu", max_context=64)
        eng.use_graphs = captured
        a, b = eng.open_sequence(), eng.open_sequence()
        eng.feed([(a, tokens[0][:20], []), (b, tokens[1][:17], [])])
        outs.append(eng.feed([(a, [tokens[0][20]], wanted[0]), (b, [tokens[1][17]], wanted[1])]))
    assert outs[0].shape[0] == len(wanted[0]) + len(wanted[1])
    assert outs[0].shape == outs[1].shape and float((outs[0] - outs[1]).norm()) <= 1e-5 * float(outs[0].norm())


def test_feed_steps_of_several_ranks_or_with_recorded_loads_are_not_captured(monkeypatch):
    """Full rows gathered over the ranks stay outside captured steps; recorded expert loads count the fed tokens alone."""
    import dataclasses
    from stkernel_b200.parallel.eplb import LoadRecorder
    from stkernel_b200.runtime import engine as E
    monkeypatch.setattr(E, "DecodeGraph", PlainStep)
    monkeypatch.setattr(Engine, "FEED_EAGER_STEPS", 0)
    cfg = tiny_config()
    ec = EngineConfig(model=cfg, sched=SchedulerConfig(max_model_len=64, max_num_seqs=4, max_num_batched_tokens=64, graph_cap=8)).validate()
    eng = Engine(ec, build_model_weights(cfg, DictSource(init_random_weights(cfg, seed=2)), "cpu"), "cpu", max_context=64)
    eng.use_graphs = True
    assert eng._feed_graph(3, 1) is not None
    eng.cfg = dataclasses.replace(ec, parallel=dataclasses.replace(ec.parallel, tp_size=2))
    assert eng._feed_graph(3, 1) is None
    eng.cfg = ec
    eng.model.load_recorder = rec = LoadRecorder(cfg.num_hidden_layers, cfg.n_routed_experts, torch.device("cpu"))
    assert eng._feed_graph(3, 1) is None
    seqs = [eng.open_sequence() for _ in range(3)]
    for i in range(4):
        eng.feed([(s, [7 + i], [0]) for s in seqs])
    assert rec.counts.sum().item() == 4 * 3 * cfg.num_experts_per_tok * cfg.num_hidden_layers


def test_feed_graphs_are_counted_padded_and_bounded_by_the_graph_that_serves_them(monkeypatch):
    """Each graph is captured after its own eager steps, also when a sequence grows into the next one; padding is small and within
    the step's buffers; the graphs held are bounded and the least recently used one goes."""
    from stkernel_b200.runtime import engine as E
    built = []

    class Step(PlainStep):
        def __init__(self, eng, bucket, rows_bucket, logits=False):
            super().__init__(eng, bucket, rows_bucket, logits)
            built.append((bucket, rows_bucket))

    monkeypatch.setattr(E, "DecodeGraph", Step)
    cfg = tiny_config()
    ec = EngineConfig(model=cfg, sched=SchedulerConfig(max_model_len=64, max_num_seqs=256, max_num_batched_tokens=256, graph_cap=256)).validate()
    eng = Engine(ec, build_model_weights(cfg, DictSource(init_random_weights(cfg, seed=2)), "cpu"), "cpu", max_context=64)
    eng.use_graphs = True
    eng.model.decode_bucket = lambda rows: 64 * (rows // 64 + 1)
    for n in range(1, 257):
        b = E.feed_bucket(n)
        assert n <= b <= n + 7 and b <= E.step_bucket(n) and (n > 8 or b == n)
    steps = Engine.FEED_EAGER_STEPS
    # 9 to 16 sequences share a graph and its count
    assert all(eng._feed_graph(9 + i % 8, 1) is None for i in range(steps))
    assert eng._feed_graph(12, 1) is not None and built == [(16, 64)]
    assert eng.buf.d_qstart[13:17].tolist() == [12] * 4
    # more rows: another graph, with eager steps of its own
    assert all(eng._feed_graph(12, 64) is None for _ in range(steps))
    assert eng._feed_graph(12, 64) is not None and built == [(16, 64), (16, 128)]
    assert eng._feed_graph(16, 1) is not None and len(built) == 2
    for n in range(1, 256, 8):
        for _ in range(steps + 1):
            eng._feed_graph(n, 1)
        eng._feed_graph(12, 64)                       # kept in use
        assert sum(k[0] == "feed" for k in eng._graphs) <= Engine.FEED_MAX_GRAPHS
    assert ("feed", 16, 128) in eng._graphs and ("feed", 24, 64) not in eng._graphs
    assert len(built) == len(set(built))
