"""Sampling rows served from per-chunk results (4096 logits a chunk): truncated and untruncated draws, edits, top lists,
against the CPU restatement on the same logits, at vocabulary sizes around the chunk's edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _transformed(logits, sp):
    """The logits the draw works on: bias, then top_k (ties: lowest ids), then min_p."""
    l = logits.copy()
    for token, bias in sp.logit_bias:
        l[token] = np.float32(l[token] + np.float32(bias))
    if 0 < sp.top_k < l.size:
        order = np.argsort(-l, kind="stable")
        l[order[sp.top_k :]] = -np.inf
    if sp.min_p > 0:
        l[l < l.max() + np.log(np.float32(sp.min_p))] = -np.inf
    return l


@pytest.mark.parametrize("vocab", [260, 4096, 4097, 12293])
def test_chunked_rows_match_the_restatement(rb, oracle, models, vocab):
    path = models(f"sampling_{vocab}", arch="llama", layers=1, d=256, heads=4, kv_heads=4, ff=256, vocab=vocab, dtype="q8_0", seed=9)
    far = vocab - 1
    options = [dict(temperature=1.0), dict(temperature=0.7), dict(temperature=1.3, logit_bias=[(5, 2.0), (far, 3.5)]), dict(top_k=2),
               dict(top_k=20), dict(temperature=0.8, top_k=40, top_p=0.95, min_p=0.05), dict(temperature=1.2, top_k=128, top_p=0.5),
               dict(top_k=7, logit_bias=[(far, 4.0), (17, -50.0)]), dict(top_k=129), dict(top_k=20, top_p=1e-4), dict(top_k=1, logit_bias=[(far, 9.0)])]
    with rb.Engine(str(path), rb.EngineConfig(n_ctx=1024, n_seq_max=len(options), n_batch=256, n_ubatch=256)) as engine:
        out = rb.StepOutput()
        prompt = np.arange(3, 12).tolist()
        for draw in range(6):
            params = [rb.SamplingParamsV2(seed=50 + i, **o) for i, o in enumerate(options)]
            rows = [rb.StepRow(i, i, prompt if draw == 0 else [out.row(i).token], 0 if draw == 0 else len(prompt) + draw - 1, True, sp, 5, True)
                    for i, sp in enumerate(params)]
            engine.step(rows, out)
            for i, sp in enumerate(params):
                logits, o = engine.last_logits(i), out.row(i)
                l = _transformed(logits, sp)
                want, margin = oracle.sample_philox(l, sp.temperature, sp.top_p, sp.seed, draw)
                # the two sums differ in the order of their additions: a draw within 1e-9 of a border may fall on either side
                assert o.token == want or margin < 1e-9, (sp, o.token, want, margin)
                assert o.logprob == pytest.approx(float(oracle.token_logprob(logits, o.token)), abs=2e-6)
                p = np.exp((l.astype(np.float64) - l.max()) / sp.temperature)
                if sp.top_p < 1 or sp.top_k == 1:
                    order = np.argsort(-p, kind="stable")
                    keep = 1 if sp.top_k == 1 else int(np.searchsorted(np.cumsum(p[order]), sp.top_p * p.sum()) + 1)
                    mask = np.zeros(p.size)
                    mask[order[:keep]] = 1
                    p = p * mask
                p /= p.sum()
                assert o.sampled_logprob == pytest.approx(np.log(p[o.token]), abs=1e-5)
                ids, lps = out.top(i)
                order = np.lexsort((np.arange(p.size), -np.where(p > 0, l, -np.inf)))
                assert list(ids) == order[:5].tolist()
                with np.errstate(divide="ignore"):
                    np.testing.assert_allclose(lps, np.log(p[order[:5]]), atol=1e-5)


def test_rows_of_ties_take_the_lowest_ids(rb, models):
    """A model of zero weights: every logit is equal, so the candidate lists overflow and the general passes serve the row."""
    path = models("sampling_ties", arch="llama", layers=1, d=256, heads=4, kv_heads=4, ff=256, vocab=9000, dtype="f32", std=0, seed=1)
    with rb.Engine(str(path), rb.EngineConfig(n_ctx=256, n_seq_max=2, n_batch=64, n_ubatch=64)) as engine:
        out = rb.StepOutput()
        seen = set()
        for trial in range(12):
            for slot in (0, 1):
                engine.seq_rm(slot)
            rows = [rb.StepRow(10 + trial, 0, [5, 6], 0, True, rb.SamplingParamsV2(top_k=5, seed=trial), 3, True),
                    rb.StepRow(100 + trial, 1, [5], 0, True, rb.SamplingParamsV2(top_k=0, seed=trial))]
            engine.step(rows, out)
            seen.add(out.row(0).token)
            assert 0 <= out.row(0).token < 5 and list(out.top(0)[0]) == [0, 1, 2]
            assert out.row(0).sampled_logprob == pytest.approx(np.log(0.2), abs=1e-6)
            assert out.row(0).logprob == pytest.approx(-np.log(9000), abs=1e-6)
        assert len(seen) > 1


@pytest.mark.parametrize("vocab", [260, 9000])
def test_rows_with_a_nan_or_an_infinity_keep_the_general_rules(rb, oracle, models, tmp_path, vocab):
    """Output rows of NaN and of infinities: a NaN counts against top_k (its order key is above every number) and is never drawn
    or listed; an infinite logit leaves no probability. The order of the selection and that of the list differ for these."""
    gguf = pytest.importorskip("gguf")
    path = models(f"sampling_f32_{vocab}", arch="llama", layers=1, d=256, heads=4, kv_heads=4, ff=256, vocab=vocab, dtype="f32", seed=11)
    for values in ({7: np.nan}, {7: np.nan, vocab - 2: np.nan, 130: np.nan}, {9: np.inf}, {9: -np.inf}):
        file = tmp_path / "odd.gguf"
        file.write_bytes(path.read_bytes())
        reader = gguf.GGUFReader(str(file), "r+")
        weight = next(t for t in reader.tensors if t.name == "output.weight").data
        assert weight.shape == (vocab, 256)
        for token, value in values.items():
            weight[token, :] = 0
            weight[token, 3] = value
        weight.flush()
        del reader, weight
        options = [dict(top_k=5), dict(top_k=40, temperature=0.8), dict(), dict(top_k=1), dict(temperature=1.2)]
        with rb.Engine(str(file), rb.EngineConfig(n_ctx=512, n_seq_max=8, n_batch=64, n_ubatch=64)) as engine:
            out = rb.StepOutput()
            for draw in range(4):
                params = [rb.SamplingParamsV2(seed=30 + i, **o) for i, o in enumerate(options)]
                engine.step([rb.StepRow(i, i, [5 + draw], draw, True, sp, 4, True) for i, sp in enumerate(params)], out)
                for i, sp in enumerate(params):
                    l, o = engine.last_logits(i), out.row(i)
                    nan = np.isnan(l)
                    assert nan.sum() == sum(np.isnan(v) for v in values.values()) and 0 <= o.token < vocab
                    if nan.any():
                        assert not nan[o.token] and np.isnan(o.logprob)
                    if sp.top_k == 1 or np.nanmax(l) == np.inf:
                        continue
                    kept = l.copy()
                    if sp.top_k:
                        order = np.lexsort((np.arange(vocab), -np.where(nan, np.inf, l)))      # NaNs first
                        kept[order[sp.top_k :]] = -np.inf
                    want, margin = oracle.sample_philox(np.where(np.isnan(kept), np.float32(-np.inf), kept), sp.temperature, 1.0, sp.seed, draw)
                    assert o.token == want or margin < 1e-9
                    p = np.exp((kept.astype(np.float64) - np.nanmax(kept)) / sp.temperature)
                    p /= np.nansum(p)
                    assert o.sampled_logprob == pytest.approx(np.log(p[o.token]), abs=1e-5)
                    n = int((p > 0).sum())
                    best = np.lexsort((np.arange(vocab), -np.where(p > 0, kept, -np.inf)))[: min(n, 4)]
                    assert list(out.top(i)[0][: len(best)]) == best.tolist()


def test_edits_that_overflow_to_a_nan_keep_the_general_rules(rb, oracle, models):
    """Each edit's parts are finite, the edited logit of a repeated token is not: (l + 3e38) / 1e-3 - 2 * 3e38 = inf - inf."""
    path = models("sampling_edits", arch="llama", layers=1, d=256, heads=4, kv_heads=4, ff=256, vocab=6000, dtype="q8_0", seed=12)
    with rb.Engine(str(path), rb.EngineConfig(n_ctx=512, n_seq_max=4, n_batch=64, n_ubatch=64)) as engine:
        out = rb.StepOutput()
        force = rb.SamplingParamsV2(top_k=1, logit_bias=[(4321, 100.0)])
        for pos in range(2):
            engine.step([rb.StepRow(0, 0, [5], pos, True, force)], out)
            assert out.row(0).token == 4321
        # the history is 4321 twice: its edit is a NaN, which takes one of the six places
        sp = rb.SamplingParamsV2(top_k=6, seed=0, logit_bias=[(4321, 3e38), (17, 2.0)], repeat_penalty=1e-3, frequency_penalty=3e38)
        engine.step([rb.StepRow(0, 0, [5], 2, True, sp, 8, True)], out)
        l, o = engine.last_logits(0).copy(), out.row(0)
        l[17] += np.float32(2.0)
        l[4321] = -np.inf
        order = np.argsort(-l, kind="stable")
        l[order[5:]] = -np.inf
        want, margin = oracle.sample_philox(l, 1.0, 1.0, 0, 2)
        assert o.token == want or margin < 1e-9
        p = np.exp(l.astype(np.float64) - l.max())
        assert o.sampled_logprob == pytest.approx(np.log(p[o.token] / p.sum()), abs=1e-5) and np.isfinite(o.logprob)
        # (the listing has probability zero after the five, in id order; the NaN is not in it)
        assert list(out.top(0)[0]) == order[:5].tolist() + [i for i in range(9) if i not in order[:5]][:3]


def test_negative_zeros_come_after_positive_ones_in_top_k(rb, models):
    """Ten equal logits of zero, two of them turned negative by an edit that underflows: top_k counts the others first."""
    path = models("sampling_zeros", arch="llama", layers=1, d=256, heads=4, kv_heads=4, ff=256, vocab=260, dtype="f32", std=0, seed=1)
    zeros = [3, 4, 50, 51, 90, 91, 92, 200, 201, 259]
    bias = [(i, -1.0) for i in range(260) if i not in zeros]
    with rb.Engine(str(path), rb.EngineConfig(n_ctx=64, n_seq_max=2, n_batch=16, n_ubatch=16)) as engine:
        out = rb.StepOutput()
        for pos, token in enumerate((3, 50)):
            engine.step([rb.StepRow(0, 0, [5], pos, True, rb.SamplingParamsV2(top_k=1, logit_bias=[(token, 5.0)]))], out)
            assert out.row(0).token == token
        sp = rb.SamplingParamsV2(top_k=9, logit_bias=bias + [(3, -1e-44), (50, -1e-44)], repeat_penalty=1e-3)
        engine.step([rb.StepRow(0, 0, [5], 2, True, sp, 9, True)], out)
        assert sorted(out.top(0)[0]) == sorted(i for i in zeros if i != 50)
        assert out.row(0).sampled_logprob == pytest.approx(-np.log(9), abs=1e-6)


def test_top_k_at_the_limits_of_the_candidate_lists(rb, oracle, models):
    """128 256 logits in 32 chunks: 96 candidates a chunk fit the row's list, 97 are left to the general passes, which take one
    launch less. Both draw what the restatement draws."""
    vocab = 128256
    path = models("sampling_128256", arch="llama", layers=1, d=256, heads=4, kv_heads=4, ff=256, vocab=vocab, dtype="q8_0", seed=3)
    launches = {}
    with rb.Engine(str(path), rb.EngineConfig(n_ctx=1024, n_seq_max=4, n_batch=64, n_ubatch=64)) as engine:
        out = rb.StepOutput()
        for request, top_k in enumerate((64, 96, 97, 100, 128)):
            for draw in range(3):
                sp = rb.SamplingParamsV2(top_k=top_k, seed=request, temperature=1.5)
                rows = [rb.StepRow(10 * request + slot, slot, [5 + draw + slot], 3 * request + draw, True, sp, 3, True) for slot in range(3)]
                engine.step(rows, out)
                launches[top_k] = engine.last_step_stats()[1]
                for slot in range(3):
                    l = _transformed(engine.last_logits(slot), sp)
                    want, margin = oracle.sample_philox(l, sp.temperature, 1.0, sp.seed, draw)
                    assert out.row(slot).token == want or margin < 1e-9
                    assert list(out.top(slot)[0]) == np.argsort(-l, kind="stable")[:3].tolist()
    assert launches[64] == launches[96] == launches[97] + 1 and launches[97] == launches[100] == launches[128]


@pytest.mark.parametrize("vocab", [260, 8191, 8192, 8193, 16385])
def test_rows_of_the_general_passes_match_the_restatement(rb, oracle, models, vocab):
    """min_p and a nucleus over the whole vocabulary: the row is copied eight times 1024 logits at a time, then transformed."""
    path = models(f"sampling_{vocab}", arch="llama", layers=1, d=256, heads=4, kv_heads=4, ff=256, vocab=vocab, dtype="q8_0", seed=9)
    options = [dict(min_p=0.1), dict(min_p=0.3, temperature=1.5, logit_bias=[(vocab - 1, 4.0)]), dict(top_p=0.8), dict(top_k=129, top_p=0.5)]
    with rb.Engine(str(path), rb.EngineConfig(n_ctx=256, n_seq_max=4, n_batch=64, n_ubatch=64)) as engine:
        out = rb.StepOutput()
        for draw in range(4):
            params = [rb.SamplingParamsV2(seed=20 + i, **o) for i, o in enumerate(options)]
            engine.step([rb.StepRow(i, i, [5 + draw], draw, True, sp, 0, True) for i, sp in enumerate(params)], out)
            for i, sp in enumerate(params):
                logits, o = engine.last_logits(i), out.row(i)
                want, margin = oracle.sample_philox(_transformed(logits, sp), sp.temperature, sp.top_p, sp.seed, draw)
                assert o.token == want or margin < 1e-9
                assert o.logprob == pytest.approx(float(oracle.token_logprob(logits, o.token)), abs=2e-6)


def _penalised(logits, sp, history):
    """Biases summed per id, then the penalties of the window, each step rounded to f32 as the kernel does."""
    l = logits.copy()
    edits = {}
    for token, bias in sp.logit_bias:
        edits.setdefault(token, [np.float32(0), 0])[0] += np.float32(bias)
    window = history[-sp.penalty_window :] if sp.penalty_window else history
    for token in window:
        edits.setdefault(token, [np.float32(0), 0])[1] += 1
    for token, (bias, count) in edits.items():
        t = np.float32(l[token] + bias)
        if count:
            rp = np.float32(sp.repeat_penalty)
            t = np.float32(t * rp) if t <= 0 else np.float32(t / rp)
            t -= np.float32(np.float32(count) * np.float32(sp.frequency_penalty)) + np.float32(sp.presence_penalty)
        l[token] = t
    return l


def test_penalties_over_a_history_and_a_full_bias_list(rb, oracle, models):
    """Rows whose edits grow with their history, and one with 4096 biases (the largest list that is accepted), served from the
    chunks: token, sampled log-probability and top list against the restatement."""
    path = models("sampling_20000", arch="llama", layers=1, d=256, heads=4, kv_heads=4, ff=256, vocab=20000, dtype="q8_0", seed=6)
    bias = [(int(i), float(b)) for i, b in zip(np.random.default_rng(0).permutation(20000)[:4096], np.random.default_rng(1).normal(0, 2, 4096))]
    options = [dict(top_k=3, repeat_penalty=1.3), dict(top_k=30, frequency_penalty=0.7, presence_penalty=0.4), dict(repeat_penalty=0.7, penalty_window=4),
               dict(top_k=2, logit_bias=bias, repeat_penalty=1.1), dict(temperature=0.9, logit_bias=bias)]
    histories = [[] for _ in options]
    with rb.Engine(str(path), rb.EngineConfig(n_ctx=1024, n_seq_max=8, n_batch=64, n_ubatch=64)) as engine:
        out = rb.StepOutput()
        for draw in range(24):
            params = [rb.SamplingParamsV2(seed=70 + i, **o) for i, o in enumerate(options)]
            engine.step([rb.StepRow(i, i, [5 + draw % 3], draw, True, sp, 3, True) for i, sp in enumerate(params)], out)
            for i, sp in enumerate(params):
                logits, o = engine.last_logits(i), out.row(i)
                l = _penalised(logits, sp, histories[i])
                if sp.top_k:
                    l[np.argsort(-l, kind="stable")[sp.top_k :]] = -np.inf
                want, margin = oracle.sample_philox(l, sp.temperature, 1.0, sp.seed, draw)
                assert o.token == want or margin < 1e-9
                p = np.exp((l.astype(np.float64) - l.max()) / np.float32(sp.temperature))
                assert o.sampled_logprob == pytest.approx(np.log(p[o.token] / p.sum()), abs=1e-5)
                assert o.logprob == pytest.approx(float(oracle.token_logprob(logits, o.token)), abs=2e-6)
                assert list(out.top(i)[0]) == np.lexsort((np.arange(l.size), -l))[:3].tolist()
                histories[i].append(o.token)
    assert len(set(histories[0])) > 3


def test_sampled_row_counts_that_rise_and_fall(rb, models):
    """The output projection's activations keep the layout of the most rows so far: 24 rows after 40 give the logits of 24 rows in
    an engine of their own, bit for bit, on the tensor-core path of either weight type."""
    for dtype in ("q4_k", "q8_0"):
        path = models(f"sampling_rows_{dtype}", arch="llama", layers=1, d=512, heads=4, kv_heads=4, ff=512, vocab=1000, dtype=dtype, seed=8)

        def logits(counts):
            with rb.Engine(str(path), rb.EngineConfig(n_ctx=4096, n_seq_max=64, n_batch=256, n_ubatch=256)) as engine:
                out = rb.StepOutput()
                for n in counts:
                    for i in range(n):
                        engine.seq_rm(i)
                    engine.step([rb.StepRow(100 * n + i, i, [5 + i, 7], 0, True, rb.SamplingParamsV2.greedy()) for i in range(n)], out)
                return np.stack([engine.last_logits(i) for i in range(counts[-1])])

        want = logits([24])
        assert np.isfinite(want).all()
        assert np.array_equal(logits([3, 40, 1, 24]), want) and np.array_equal(logits([24, 17, 24]), want)


def test_greedy_chunked_and_v1_rows_across_graph_replays(rb, oracle, models):
    """Rows of every kind side by side, their numbers changing between steps of one shape while the steps are captured and
    replayed: plain greedy rows beside rows of candidate lists (the chunk kernel's other form), untruncated draws, general rows."""
    vocab = 20000
    path = models(f"sampling_{vocab}", arch="llama", layers=1, d=256, heads=4, kv_heads=4, ff=256, vocab=vocab, dtype="q8_0", seed=6)
    greedy, listed, plain, general = dict(top_k=1), dict(top_k=30, temperature=1.3), dict(), dict(min_p=0.1)
    mixes = [[greedy] * 6, [greedy] * 4 + [listed] * 2, [listed] * 3 + [greedy] * 2 + [plain], [greedy, general, listed, greedy, plain, general]]
    with rb.Engine(str(path), rb.EngineConfig(n_ctx=2048, n_seq_max=8, n_batch=64, n_ubatch=64)) as engine:
        out = rb.StepOutput()
        pos, draws = 0, [0] * 24
        for mix in [0, 0, 0, 0, 1, 1, 1, 1, 0, 2, 2, 2, 1, 3, 3, 3, 2, 0, 3, 1]:
            params = [rb.SamplingParamsV2(seed=90 + 6 * mix + i, **o) for i, o in enumerate(mixes[mix])]
            engine.step([rb.StepRow(6 * mix + i, i, [5 + pos % 7 + i], pos, True, sp, 2, True) for i, sp in enumerate(params)], out)
            for i, sp in enumerate(params):
                logits = engine.last_logits(i)
                l = _transformed(logits, sp)
                want, margin = oracle.sample_philox(l, sp.temperature, 1.0, sp.seed, draws[6 * mix + i])
                draws[6 * mix + i] += 1
                assert out.row(i).token == want or margin < 1e-9, (pos, mix, i)
                assert out.row(i).logprob == pytest.approx(float(oracle.token_logprob(logits, want)), abs=2e-6)
                assert list(out.top(i)[0]) == np.lexsort((np.arange(vocab), -l))[:2].tolist()
            pos += 1
        assert engine.graph_stats()[0] >= 6


@pytest.mark.parametrize("vocab", [260, 20000, 128256])
def test_v1_rows_report_the_policy_before_the_draw(rb, oracle, models, vocab):
    """v1 rows from the chunks: the draw at their temperature, token and top log-probabilities of the raw row."""
    path = models(f"sampling_v1_{vocab}", arch="llama", layers=1, d=256, heads=4, kv_heads=4, ff=256, vocab=vocab, dtype="q8_0", seed=5)
    with rb.Engine(str(path), rb.EngineConfig(n_ctx=256, n_seq_max=4, n_batch=64, n_ubatch=64)) as engine:
        for draw in range(5):
            params = [rb.SamplingParams(temperature=t, seed=10 + i) for i, t in enumerate((1.0, 0.6, 1.7))]
            rows, ids, lps = engine.step_v1([rb.StepRow(i, i, [5 + draw], draw, True, sp, 6) for i, sp in enumerate(params)], 6)
            for i, sp in enumerate(params):
                logits = engine.last_logits(i)
                want, margin = oracle.sample_philox(logits, sp.temperature, 1.0, sp.seed, draw)
                assert rows[i].token == want or margin < 1e-9
                assert rows[i].logprob == pytest.approx(float(oracle.token_logprob(logits, rows[i].token)), abs=2e-6)
                want_ids, want_lps = oracle.top_token_logprobs(logits, 6)
                assert ids[i].tolist() == want_ids.tolist()
                np.testing.assert_allclose(lps[i], want_lps, atol=2e-6)
