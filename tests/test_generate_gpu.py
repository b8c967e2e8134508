"""Generation on the GPU: sampling kernels against their host twin, greedy generation through
the Python entry point against the plain model, sessions, long decoding, the first tokens of
a sequence, and the scheduler under a pool too small for everyone."""

import pytest
import torch

import plain_model
from tiny_configs import CONFIGS, random_tokens

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def folders(tmp_path_factory):
    from ninfer_amd_mi50_b200.weights import write_random_model
    out = {}
    for name, (cfg, seed) in CONFIGS.items():
        d = str(tmp_path_factory.mktemp("gen") / name)
        write_random_model(cfg, seed, d)
        out[name] = (d, cfg) + plain_model.read_model_folder(d)
    return out


def test_argmax_takes_the_first_maximum():
    from ninfer_amd_mi50_b200 import kernels
    l = torch.randn(5, 2003, device="cuda")
    l[1, 77] = l[1, 1500] = 50.0
    l[3, 2002] = 60.0
    got = kernels.argmax_rows(l).tolist()
    assert got == torch.argmax(l, dim=-1).tolist() and got[1] == 77 and got[3] == 2002
    # a long row is cut into pieces: ties across pieces and inside one, the last element, a
    # length that is no multiple of the piece
    for V in (16384, 151936, 40001):
        l = torch.randn(6, V, device="cuda")
        l[1, 77] = l[1, V - 5] = 50.0
        l[2, 5000] = l[2, 5001] = 50.0
        l[3, V - 1] = 60.0
        l[4] = 1.0                                   # all equal: the first index
        got = kernels.argmax_rows(l).tolist()
        assert got == torch.argmax(l, dim=-1).tolist()
        assert got[1] == 77 and got[2] == 5000 and got[3] == V - 1 and got[4] == 0


@pytest.mark.parametrize("V", [515, 2003, 151936])
@pytest.mark.parametrize("temperature,top_k,top_p", [(0.8, 50, 0.95), (1.3, 1, 1.0), (0.5, 1024, 0.5),
                                                     (1.0, 10**9, 1.0), (0.7, 7, 1.0)])
def test_sampler_matches_its_host_twin(V, temperature, top_k, top_p):
    from ninfer_amd_mi50_b200.sampling import Sampler, SamplingParams, sample_reference, uniform_draw
    g = torch.Generator().manual_seed(V + top_k % 1000)
    R = 6
    logits = (torch.randn(R, V, generator=g) * 2).cuda()
    params = [SamplingParams(temperature, top_k, top_p, seed=11 + r) for r in range(R)]
    counters = list(range(R))
    got = Sampler(V, "cuda").sample(logits, params, counters=counters).tolist()
    agree = 0
    for r in range(R):
        u = uniform_draw(params[r].seed, counters[r])
        want = sample_reference(logits[r].cpu(), params[r], draw=u)
        if got[r] == want:
            agree += 1
        else:
            # a draw within rounding of a boundary of the running sum may fall either way:
            # then the two picks are neighbours in the order of the draw
            lo = sample_reference(logits[r].cpu(), params[r], draw=max(0.0, u - 1e-4))
            hi = sample_reference(logits[r].cpu(), params[r], draw=min(1.0, u + 1e-4))
            assert got[r] in (lo, hi), (r, got[r], want, lo, hi)
    assert agree >= R - 1


def test_sampler_distribution_and_penalty():
    from ninfer_amd_mi50_b200.sampling import Sampler, SamplingParams
    V = 64
    logits = torch.full((1, V), -30.0, device="cuda")
    logits[0, 3], logits[0, 9] = 1.0, 0.0        # p = e/(e+1) = 0.731, 0.269
    s = Sampler(V, "cuda")
    n = 4000
    params = [SamplingParams(1.0, 50, 1.0, seed=5)] * n
    picks = s.sample(logits.expand(n, V).contiguous(), params, counters=list(range(n))).tolist()
    assert set(picks) <= {3, 9} and abs(picks.count(3) / n - 0.731) < 0.03
    # repetition penalty divides a positive logit and multiplies a negative one, once per occurrence
    l = torch.zeros((1, V), device="cuda")
    l[0, 5], l[0, 6], l[0, 7] = 4.0, 3.9, -1.0
    greedy = [SamplingParams(0.0, repetition_penalty=1.5)]
    assert s.sample(l, greedy, recent=[[5]]).tolist() == [6]          # 4.0 / 1.5 < 3.9
    assert s.sample(l, greedy, recent=[[5, 6, 6]]).tolist() == [5]    # 3.9 / 1.5^2 < 4.0 / 1.5
    assert s.sample(l, [SamplingParams(0.0)], recent=[[5]]).tolist() == [5]


def test_sampler_refuses_what_it_cannot_do():
    from ninfer_amd_mi50_b200.sampling import SamplingParams, check_params
    with pytest.raises(ValueError, match="top_k"):
        check_params(SamplingParams(0.7, 5000, 0.9), 151936)
    check_params(SamplingParams(0.7, 5000, 1.0), 4000)       # above the vocabulary means no limit
    check_params(SamplingParams(0.0, 5000, 0.9), 151936)     # greedy ignores both


@pytest.mark.parametrize("name", ["A", "B", "C", "D"])
def test_greedy_generation_through_the_entry_point(folders, name):
    from ninfer_amd_mi50_b200.api import Ninfer
    d, cfg, pcfg, weights = folders[name]
    prompts = [random_tokens(n, cfg["vocab_size"], 70 + n) for n in (7, 16, 33)]
    want = [plain_model.plain_greedy(pcfg, weights, p, 8) for p in prompts]
    eng = Ninfer(d, max_context=128, prefill_chunk=16, num_sequences=3, dtype="float32")
    assert eng.generate(prompts, max_new_tokens=8, temperature=0.0) == want
    st = eng.stats()
    assert st["finished"] == 3 and st["live_requests"] == 0 and st["decode_tokens"] == 21
    eng.close()
    eng = Ninfer(d, max_context=128, prefill_chunk=16, num_sequences=3, dtype="bfloat16")
    got = eng.generate(prompts, max_new_tokens=8, temperature=0.0)
    # bfloat16 may part from the plain tokens where two logits are within rounding, and the
    # sequences differ from there on.  So every token is judged on the engine's own prefix: the
    # plain model, given prompt and the tokens generated so far, must rate the engine's next
    # token within twice the rounding bound (1.5 % of the largest logit) of its own best.
    for p, g in zip(prompts, got):
        assert len(g) == 8
        logits = plain_model.plain_forward(pcfg, weights, p + g)[len(p) - 1:-1]
        scale = logits.abs().max().item()
        for i, tok in enumerate(g):
            assert logits[i, tok].item() >= logits[i].max().item() - 3e-2 * scale, \
                f"token {i} ({tok}) is not among the plain model's best"
    eng.close()


def test_temperature_generation_is_seeded_and_independent_of_batching(folders):
    """Same seed, same tokens: whatever the batch, the portions, or a pool so small that a
    request is preempted and recomputed."""
    from ninfer_amd_mi50_b200.api import Ninfer
    d, cfg, _, _ = folders["B"]
    prompts = [random_tokens(n, cfg["vocab_size"], 80 + n) for n in (14, 15, 30, 31)]
    runs = []
    for nseq, chunk, page, pool in ((4, 16, 64, None), (2, 64, 64, None), (4, 16, 16, 96)):
        eng = Ninfer(d, max_context=64, prefill_chunk=chunk, num_sequences=nseq, dtype="float32",
                     page_size=page, cache_tokens=pool)
        runs.append(eng.generate(prompts, max_new_tokens=12, temperature=0.8, seed=99))
        if pool:
            assert eng.stats()["preemptions"] >= 1 and eng.stats()["out_of_cache"] == 0
        eng.close()
    assert runs[0] == runs[1] == runs[2]
    assert all(len(r) == 12 for r in runs[0])
    eng = Ninfer(d, max_context=64, num_sequences=4, dtype="float32")
    assert eng.generate(prompts, max_new_tokens=12, temperature=0.8, seed=100) != runs[0]
    eng.close()


def test_sessions_prefill_decode_and_decode_batch(folders):
    from ninfer_amd_mi50_b200.api import Ninfer, NinferError
    d, cfg, pcfg, weights = folders["A"]
    eng = Ninfer(d, max_context=128, prefill_chunk=8, num_sequences=2, dtype="float32")
    a, b = random_tokens(21, 1024, 1), random_tokens(9, 1024, 2)
    wa, wb = plain_model.plain_forward(pcfg, weights, a), plain_model.plain_forward(pcfg, weights, b)
    with eng.session() as s, eng.session() as t:
        assert {s.slot, t.slot} == {0, 1}
        la = s.prefill(a[:19])                     # three portions of 8, 8, 3
        torch.testing.assert_close(torch.from_numpy(la), wa[18], rtol=1e-4, atol=1e-5)
        lb = t.prefill(b[:8])
        torch.testing.assert_close(torch.from_numpy(lb), wb[7], rtol=1e-4, atol=1e-5)
        both = eng.decode_batch([s, t], [a[19], b[8]])
        torch.testing.assert_close(torch.from_numpy(both[0]), wa[19], rtol=1e-4, atol=1e-5)
        torch.testing.assert_close(torch.from_numpy(both[1]), wb[8], rtol=1e-4, atol=1e-5)
        assert (s.length, t.length) == (20, 9)
        torch.testing.assert_close(torch.from_numpy(s.decode(a[20])), wa[20], rtol=1e-4, atol=1e-5)
        t.reset()
        assert t.length == 0
        torch.testing.assert_close(torch.from_numpy(t.prefill(a[:3])), wa[2], rtol=1e-4, atol=1e-5)
        with pytest.raises(NinferError, match="capacity"):
            s.prefill([1] * 200)
        with pytest.raises(NinferError):
            eng.session()                          # both slots are taken
    assert eng.pages_free == [eng._runner.cache.groups[0].pool.num_pages]
    assert eng.kv_bytes_per_token == 2 * 2 * 2 * 64 * 4
    tok = eng.sample(la, temperature=0.0)
    assert tok == int(torch.argmax(wa[18]))
    eng.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_long_decoding_and_first_tokens(folders, dtype):
    """A prompt of one token, then 330 tokens one by one across several pages; the first
    positions (1, 2, 3 tokens of context) are checked like the rest."""
    import schedules
    from test_replay_gpu import check, make_runner, want_for
    d, cfg, pcfg, weights = folders["C"]
    toks = random_tokens(331, cfg["vocab_size"], 3)
    want = plain_model.plain_forward(pcfg, weights, toks)
    runner = make_runner(d, dtype, 384)
    routing = {}
    got = schedules.run_schedule(runner, schedules.tail_decoded({"r": toks}, tail=330), routing)["r"]
    want = want_for((pcfg, weights), {"r": toks}, {"r": want}, dtype, routing, "long decode")["r"]
    check(got, want, dtype, "long decode")
    check(got[:3], want[:3], dtype, "first tokens")


@pytest.mark.parametrize("dtype,count", [("float32", 11), ("bfloat16", 11), ("bfloat16", 40)])
def test_graph_replay_equals_host_driven_steps(folders, dtype, count):
    """Decode-only steps are replayed from CUDA graphs, with padding rows when the number of
    live requests is not one a graph was built for; the logits must be those of the same
    step driven from the host."""
    from ninfer_amd_mi50_b200.api import Ninfer
    d, cfg, _, _ = folders["A"]
    outs = []
    for use_graph in (False, True):
        eng = Ninfer(d, max_context=256, prefill_chunk=32, num_sequences=count + 1, dtype=dtype, use_graph=use_graph)
        assert (eng._runner.graphs is not None) == use_graph
        sessions = [eng.session() for _ in range(count)]
        for i, s in enumerate(sessions):
            s.prefill(random_tokens(3 + 7 * (i % 11), 1024, 90 + i))
        logs = []
        for step in range(5):
            # 11, 9, 7, 5, 3 rows: padded and exact graphs; 40 .. 32 rows: the shared expert's
            # branch starts after the router
            live = sessions[:count - 2 * step]
            logs.append(torch.from_numpy(eng.decode_batch(live, [(5 * step + j) % 1024 for j in range(len(live))])))
        outs.append(logs)
        if use_graph:
            assert sorted(k[0] for k in eng._runner.graphs.graphs) == ([3, 5, 7, 16] if count == 11 else [32, 64])
        for s in sessions:
            s.close()
        eng.close()
    for a, b in zip(*outs):
        if count <= 16:
            torch.testing.assert_close(a, b, rtol=0, atol=0)
        else:
            # the graph is built for 64 rows and the host drives 40 and fewer: the library's
            # dense products may round differently for the two row counts, so the bound is the
            # one of bfloat16 rounding (a wrong row, page or branch order moves a row by the scale)
            scale = b.abs().max().item()
            row_err = (a - b).abs().max(dim=1).values
            assert (row_err > 1.5e-2 * scale).sum().item() <= max(1, len(row_err) // 10)
            assert row_err.max().item() <= 0.1 * scale


def test_capture_survives_an_older_engine_waiting_for_the_collector(folders, monkeypatch):
    """An engine that died inside a reference cycle keeps its CUDA graphs until the cyclic
    collector runs.  If that happened during a later engine's capture, the graphs would be
    destroyed inside the capture and invalidate it; the capture therefore holds the collector
    off.  Here the older engine becomes garbage in the middle of the capture, followed by
    enough cyclic garbage to set an enabled collector off."""
    import gc
    from ninfer_amd_mi50_b200.api import Ninfer
    from ninfer_amd_mi50_b200.engine.step import ModelRunner
    d, cfg, _, _ = folders["A"]
    first = Ninfer(d, max_context=128, prefill_chunk=32, num_sequences=2, dtype="bfloat16", use_graph=True)
    s = first.session()
    s.prefill(random_tokens(5, 1024, 7))
    ref = first.decode_batch([s], [3]).copy()
    assert first._runner.graphs.graphs                      # a graph was captured
    s.close()
    del s
    held = [first]
    del first
    seen = []
    plain_run = ModelRunner.run

    def run(self, ctx):
        if torch.cuda.is_current_stream_capturing() and held:
            ring = [held.pop()]
            ring.append(ring)
            del ring
            for _ in range(5000):                            # far beyond the collector's thresholds
                c = []
                c.append(c)
            seen.append(gc.isenabled())
        return plain_run(self, ctx)

    monkeypatch.setattr(ModelRunner, "run", run)
    second = Ninfer(d, max_context=128, prefill_chunk=32, num_sequences=2, dtype="bfloat16", use_graph=True)
    s = second.session()
    s.prefill(random_tokens(5, 1024, 7))
    out = second.decode_batch([s], [3])
    assert seen == [False] and gc.isenabled()
    assert (out == ref).all()
    s.close()
    second.close()


@pytest.mark.parametrize("temperature", [0.0, 0.9])
def test_running_ahead_changes_no_token(folders, temperature):
    """Decode steps are launched before the host has read the tokens of the step before (they
    travel inside the device).  Same tokens as without, also when requests stop on a stop token
    (their row in the step ahead was computed for nothing) or finish by length at different
    times; and every page comes back."""
    from ninfer_amd_mi50_b200.api import Ninfer
    d, cfg, _, _ = folders["A"]
    prompts = [random_tokens(n, cfg["vocab_size"], 300 + n) for n in (5, 9, 17, 3, 12)]
    runs, stats = [], []
    for ahead in (False, True):
        eng = Ninfer(d, max_context=128, prefill_chunk=32, num_sequences=5, dtype="bfloat16", run_ahead=ahead)
        free = eng.stats()["pages_free"]
        base = eng.generate(prompts, max_new_tokens=40, temperature=temperature, seed=5)
        # stop ids taken from what the requests generate: some stop early, at different steps
        stops = {base[0][7], base[1][20], base[3][2]}
        outs = [base, eng.generate(prompts, max_new_tokens=40, temperature=temperature, seed=5, stop_ids=stops)]
        # lengths that differ per request (finishing by length is known in advance)
        from ninfer_amd_mi50_b200.sampling import SamplingParams
        ps = [SamplingParams(temperature, 50, 0.95, 1.0, 5, n) for n in (3, 40, 11, 1, 25)]
        outs.append(eng._engine.generate(prompts, ps))
        runs.append(outs)
        stats.append(eng.stats())
        assert eng.stats()["pages_free"] == free and eng.stats()["live_requests"] == 0
        eng.close()
    assert runs[0] == runs[1]
    assert stats[0]["ahead_steps"] == 0 and stats[1]["ahead_steps"] > 50
    assert any(len(o) < 40 for o in runs[1][1])          # some request did stop early


@pytest.mark.parametrize("name,rows,chained", [("A", 3, -1), ("C", 3, -1), ("A", 40, -1), ("C", 40, -1), ("C", 3, 1)])
def test_a_replayed_step_gives_the_same_bits_every_time(folders, name, rows, chained):
    """A captured decode step, replayed on unchanged inputs, must give the same logits bit for
    bit.  With the kernels of the step launched chained (each may begin while its predecessor
    drains), the first kernel after a wait on another stream - the shared expert's branch, and
    the combine that joins it - must be an ordinary launch: chained, it began before the other
    stream's kernel had finished, and every replay of the step differed.  With 40 rows the
    shared expert's branch starts after the router instead of beside it.

    `chained` = 1 chains the streaming products only.  That timing showed a second fault: the
    shared expert's second product, already resident while the first still ran beside the
    high-priority router, read its input rows through the non-coherent path and got rows of an
    earlier layer; a quarter of the replays differed.  A chained kernel reads what its
    predecessor wrote with coherent loads issued after the wait."""
    from ninfer_amd_mi50_b200 import kernels
    from ninfer_amd_mi50_b200.config import EngineOptions
    from ninfer_amd_mi50_b200.engine import StepEntry, load_runner
    d, cfg, _, _ = folders[name]
    kernels.load().nf_set_chained_launch(chained)
    try:
        _replay_and_compare(d, cfg, rows)
    finally:
        kernels.load().nf_set_chained_launch(-1)


def _replay_and_compare(d, cfg, rows):
    from ninfer_amd_mi50_b200.config import EngineOptions
    from ninfer_amd_mi50_b200.engine import StepEntry, load_runner
    runner = load_runner(d, options=EngineOptions(dtype="bfloat16", page_size=64, num_sequences=rows + 1,
                                                   max_context=256, cache_tokens=256 * (rows + 1)))
    for r in range(rows):
        runner.open(r)
        runner.step([StepEntry(r, random_tokens(70 + 9 * (r % 7), cfg["vocab_size"], 500 + r), [])])
    for s in range(2):
        runner.step([StepEntry(r, [5 + s + r], [0]) for r in range(rows)])
    torch.cuda.synchronize()
    (graph,) = runner.graphs.graphs.values()
    graph.graph.replay()
    torch.cuda.synchronize()
    ref = graph.logits.clone()
    for _ in range(300 if rows < 8 else 100):
        graph.graph.replay()
        assert torch.equal(graph.logits, ref)


def _staging_runner(folders, rows, **more):
    from ninfer_amd_mi50_b200.config import EngineOptions
    from ninfer_amd_mi50_b200.engine import StepEntry, load_runner
    d, cfg, _, _ = folders["A"]
    runner = load_runner(d, options=EngineOptions(dtype="bfloat16", page_size=16, num_sequences=rows, **more))
    return runner, StepEntry, cfg["vocab_size"]


def test_steps_prepared_far_ahead_of_the_device(folders):
    """More decode steps than there are staging buffers, of two graphs in turn, queued behind a busy device: the logits of
    steps taken one at a time."""
    outs = []
    for waits in (True, False):
        runner, StepEntry, vocab = _staging_runner(folders, 4, max_context=256, cache_tokens=1024)
        for r in range(3):
            runner.open(r)
            runner.step([StepEntry(r, random_tokens(20 + 7 * r, vocab, 40 + r), [])])
        for n in (3, 1):                                      # both graphs exist before the device is kept busy
            runner.step([StepEntry(r, [1], [0]) for r in range(n)])
        a = torch.randn((8192, 8192), device="cuda")
        torch.cuda.synchronize()
        if not waits:
            for _ in range(30):
                a @ a
        got = []
        for s in range(50):
            n = 1 if s % 3 == 2 else 3
            got.append(runner.step([StepEntry(r, [(37 * s + 11 * r) % vocab], [0]) for r in range(n)]).clone())
            if waits:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        outs.append(got)
    assert all(torch.equal(x, y) for x, y in zip(*outs))


def test_staging_memory_does_not_grow_with_the_graphs(folders):
    """A service whose context passes one bound after another, with many rows and with few."""
    pinned = lambda: torch.cuda.memory.host_memory_stats()["allocated_bytes.current"]
    runner, StepEntry, vocab = _staging_runner(folders, 16, max_context=4096, cache_tokens=16 * 2048)
    for r in range(16):
        runner.open(r)
    before = pinned()
    sizes = []
    for bound in range(3):
        runner.step([StepEntry(0, random_tokens(500, vocab, bound), [])])
        for n in (16, 5):
            runner.step([StepEntry(r, [3], [0]) for r in range(n)])
            sizes.append(pinned() - before)
    assert len(runner.graphs.graphs) == 6
    assert sizes[-1] == sizes[0] > 0
