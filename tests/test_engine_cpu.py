"""The engine loop, the entry points and the sampler's host side, on a CPU with the stand-in kernels."""

from __future__ import annotations

import asyncio

import pytest
import torch

import plain_llama
import tiny_configs


def _prompts(vocab, lengths):
    return [tiny_configs.prompt(vocab, n, i) for i, n in enumerate(lengths)]


def test_greedy_generation_through_llm_matches_plain(cpu_kernels, model_dirs):
    from liteinfer_b200 import LLM, SamplingParams

    config, _, page = tiny_configs.ALL["tiny_b"]
    prompts = _prompts(config["vocab_size"], (3, 30, 11, 1))
    raw, weights = plain_llama.read_model(model_dirs["tiny_b"])
    expected = [plain_llama.greedy(raw, weights, p, 5) for p in prompts]
    # a budget of 16 tokens cuts the 30-token prompt into portions that run beside the others' decodes
    with LLM(str(model_dirs["tiny_b"]), dtype="float32", device="cpu", block_size=page, max_num_seqs=3,
             max_model_len=64, max_num_batched_tokens=16) as llm:
        outs = llm.generate(prompts, SamplingParams(temperature=0.0, max_tokens=5, ignore_eos=True))
        assert [o.token_ids for o in outs] == expected
        assert [o.finish_reason for o in outs] == ["length"] * 4
        assert [o.request_id for o in outs] == ["req-0", "req-1", "req-2", "req-3"]
        assert outs[0].text == " ".join(map(str, expected[0]))        # no tokenizer.json: text is ids
        phases = {s.phase for s in llm.stats.steps}
        assert "mixed" in phases and "decode" in phases
        assert max(s.input_tokens for s in llm.stats.steps) <= 16
        assert llm.engine.runner.cache.live_requests == [] or True
        # strings work too: the tokenizer of a folder without tokenizer.json reads ids
        again = llm.generate(" ".join(map(str, prompts[0])), SamplingParams(temperature=0.0, max_tokens=5))
        assert again[0].token_ids == expected[0]


def test_stop_rules_through_the_engine(cpu_kernels, model_dirs):
    from liteinfer_b200 import LLM, SamplingParams

    config, _, page = tiny_configs.ALL["tiny_a"]
    prompt = tiny_configs.prompt(config["vocab_size"], 7, 0)
    with LLM(str(model_dirs["tiny_a"]), dtype="float32", device="cpu", block_size=page, max_model_len=32) as llm:
        free = llm.generate([prompt], SamplingParams(temperature=0.0, max_tokens=8))[0].token_ids
        stop_at = free[2]
        cut = llm.generate([prompt], SamplingParams(temperature=0.0, max_tokens=8, stop_token_ids=[stop_at]))[0]
        assert cut.finish_reason == "stop" and cut.token_ids == free[:free.index(stop_at) + 1]
        gated = llm.generate([prompt], SamplingParams(temperature=0.0, max_tokens=8, min_tokens=6,
                                                      stop_token_ids=[stop_at]))[0]
        assert len(gated.token_ids) >= 6
        # A stop string is looked for in the text, which is then decoded at every step (otherwise at the end only).
        text_stop = " " + str(free[3])
        by_text = llm.generate([prompt], SamplingParams(temperature=0.0, max_tokens=8, stop=[text_stop]))[0]
        first = next(n for n in range(1, 9) if text_stop in " ".join(map(str, free[:n])))
        assert by_text.finish_reason == "stop" and by_text.token_ids == free[:first]
        assert by_text.text == " ".join(map(str, free[:first]))
        long = llm.generate([prompt], SamplingParams(temperature=0.0, max_tokens=100))[0]
        assert long.finish_reason == "length" and len(prompt) + len(long.token_ids) == 32   # max_model_len
        with pytest.raises(ValueError, match="max_model_len"):
            llm.generate([list(range(40))], SamplingParams(max_tokens=1))
        with pytest.raises(ValueError, match="no tokens"):
            llm.generate([""], SamplingParams(max_tokens=1))


def test_newcomers_wait_for_pages_and_nothing_is_lost(cpu_kernels, model_dirs):
    """Six requests through a cache that holds two of them: all finish, none is aborted, every page comes back."""
    from liteinfer_b200 import LLM, SamplingParams

    config, _, page = tiny_configs.ALL["tiny_a"]
    prompts = _prompts(config["vocab_size"], (20, 25, 18, 30, 9, 22))
    raw, weights = plain_llama.read_model(model_dirs["tiny_a"])
    with LLM(str(model_dirs["tiny_a"]), dtype="float32", device="cpu", block_size=page, max_num_seqs=4,
             max_model_len=64, num_gpu_blocks=5) as llm:
        outs = llm.generate(prompts, SamplingParams(temperature=0.0, max_tokens=4, ignore_eos=True))
        assert [o.token_ids for o in outs] == [plain_llama.greedy(raw, weights, p, 4) for p in prompts]
        assert llm.stats.num_requests_aborted == 0
        cache = llm.engine.runner.cache
        llm.engine.step()                                   # evicts what finished last
        assert all(g.allocator.num_held == 0 for g in cache.groups) and cache.slots.num_held == 0


def test_running_out_of_pages_while_decoding_sheds_the_least_invested(cpu_kernels, model_dirs):
    """Two requests fill the cache while decoding; the step that does not fit aborts one tier and the other goes on."""
    from liteinfer_b200.cache.pages import CacheExhaustedError
    from liteinfer_b200.config.engine_config import EngineConfig
    from liteinfer_b200.engine.core import EngineCore
    from liteinfer_b200.sampling.params import SamplingParams

    config, _, page = tiny_configs.ALL["tiny_a"]          # pages of 16 tokens
    engine = EngineCore(EngineConfig(model=str(model_dirs["tiny_a"]), dtype="float32", device="cpu",
                                     block_size=page, max_num_seqs=4, max_model_len=128, num_gpu_blocks=3))
    engine.load()
    engine.scheduler.ledger = None                          # admit regardless, as the reference does
    params = SamplingParams(temperature=0.0, max_tokens=40, ignore_eos=True)
    a = engine.add_request("a", tiny_configs.prompt(config["vocab_size"], 30, 0), params)
    b = engine.add_request("b", tiny_configs.prompt(config["vocab_size"], 14, 1), params)
    aborted = []
    for _ in range(60):
        if not engine.has_unfinished():
            break
        result = engine.step()
        aborted += result.aborted
    # a needs its third page at 33 tokens, b its second at 17: the pool of three cannot hold both.
    assert len(aborted) == 2 or len(aborted) == 1
    assert all(isinstance(error, CacheExhaustedError) for _, error in aborted)
    assert engine.stats.num_requests_aborted == len(aborted)
    finished = [s for s in (a, b) if s.status.value == "finished_length"]
    assert len(finished) + len(aborted) == 2
    engine.step()
    assert all(g.allocator.num_held == 0 for g in engine.runner.cache.groups)


def test_a_failing_step_aborts_only_its_requests(cpu_kernels, model_dirs, monkeypatch):
    from liteinfer_b200 import LLM, SamplingParams

    config, _, page = tiny_configs.ALL["tiny_a"]
    with LLM(str(model_dirs["tiny_a"]), dtype="float32", device="cpu", block_size=page, max_model_len=64) as llm:
        runner = llm.engine.runner
        real = runner.model.forward
        calls = {"n": 0}

        def flaky(ctx, caches):
            calls["n"] += 1
            if calls["n"] == 2:
                raise RuntimeError("boom")
            return real(ctx, caches)

        monkeypatch.setattr(runner.model, "forward", flaky)
        with pytest.raises(RuntimeError, match="boom"):
            llm.generate([tiny_configs.prompt(config["vocab_size"], 5, 0)], SamplingParams(temperature=0.0, max_tokens=4))
        monkeypatch.setattr(runner.model, "forward", real)
        out = llm.generate([tiny_configs.prompt(config["vocab_size"], 5, 0)], SamplingParams(temperature=0.0, max_tokens=4))
        assert len(out[0].token_ids) == 4                   # the engine is still usable, the cache was rolled back
        runner.cache.check_invariants()


def test_async_llm_generates_and_streams(cpu_kernels, model_dirs):
    from liteinfer_b200 import AsyncLLM, SamplingParams

    config, _, page = tiny_configs.ALL["tiny_b"]
    prompts = _prompts(config["vocab_size"], (4, 12, 7))
    raw, weights = plain_llama.read_model(model_dirs["tiny_b"])
    expected = [plain_llama.greedy(raw, weights, p, 4) for p in prompts]

    async def run():
        async with AsyncLLM(str(model_dirs["tiny_b"]), dtype="float32", device="cpu", block_size=page,
                            max_num_seqs=2, max_model_len=64) as llm:
            outs = await llm.generate(prompts, SamplingParams(temperature=0.0, max_tokens=4, ignore_eos=True))
            events = [e async for e in llm.stream(prompts[1], SamplingParams(temperature=0.0, max_tokens=4,
                                                                              ignore_eos=True))]
            with pytest.raises(ValueError):
                await llm.generate([[]], SamplingParams(max_tokens=1))
            return outs, events

    outs, events = asyncio.run(run())
    assert [o.token_ids for o in outs] == expected
    assert [len(e.output_token_ids) for e in events] == [1, 2, 3, 4]
    assert events[-1].is_finished and events[-1].finish_reason == "length" and not events[0].is_finished
    assert events[-1].output_token_ids == expected[1]


def test_sampling_params_checks():
    from liteinfer_b200 import SamplingParams

    for bad in ({"temperature": -1}, {"top_p": 0.0}, {"top_p": 1.5}, {"top_k": 0}, {"max_tokens": 0},
                {"min_tokens": -1}, {"min_tokens": 9, "max_tokens": 3}):
        with pytest.raises(ValueError):
            SamplingParams(**bad)
    assert SamplingParams(temperature=0).greedy and SamplingParams(top_k=1).greedy and not SamplingParams().greedy
    assert SamplingParams().id != SamplingParams().id


def test_steps_name_their_single_tokens_longest_first():
    """Of a step's entries and of padding, by falling context, equal ones in their order; a list of its own beside the batch's."""
    from liteinfer_b200.engine.runner import _Batch, _longest_first, _write_padding
    import numpy as np

    lengths = np.array([5, 9, 9, 1, 30, 9], dtype=np.int32)
    assert _longest_first(np.array([0, 1, 2, 3, 4, 5], dtype=np.int32), lengths).tolist() == [4, 1, 2, 5, 0, 3]
    assert _longest_first(np.array([5, 3, 0], dtype=np.int32), lengths).tolist() == [5, 0, 3]
    assert _longest_first(np.array([], dtype=np.int32), lengths).tolist() == []
    batch = _Batch(3, 3, 3, [2], 3, 0)
    views = batch.views(np.zeros(batch.total, dtype=np.int32))
    _write_padding(views)
    assert views.dlong.tolist() == views.dseq.tolist() == [-1] * 3


def test_steps_sort_their_single_tokens_where_a_launch_reads_the_order():
    """Sorting is host work in every step: only for as many sequences as have more blocks than the device has places."""
    from types import SimpleNamespace
    from liteinfer_b200.engine.runner import _Batch, _context, _order_pays
    from liteinfer_b200.ops import kernels
    from liteinfer_b200.parts.context import KVNeed

    held = lambda *needs: SimpleNamespace(groups=[SimpleNamespace(need=need) for need in needs])
    for need in (KVNeed(8, 64), KVNeed(8, 128), KVNeed(2, 128, v_head_dim=256)):
        each = need.kv_heads * need.value_dim // need.head_dim
        most = kernels.decode_capacity(need.head_dim, True) // each
        for cache in (held(need), held(KVNeed(1, 64), need)):
            assert [_order_pays(cache, n, None) for n in (0, 1, most, most + 1)] == [False, False, False, True]
            assert _order_pays(cache, most // 4 + 1, 4) and not _order_pays(cache, most // 4, 4)
    assert not _order_pays(held(KVNeed(8, 96)), 1000, None) and not _order_pays(held(), 1000, None)      # (no streaming kernel)
    for ordered in (False, True):
        batch = _Batch(3, 3, 3, [2], 3, 0, ordered)
        plan = _context(batch, torch.zeros(batch.total, dtype=torch.int32), "cpu", [1] * 3, [5] * 3, None, 5).plan
        assert (plan.decode_longest_first is not None) == ordered and plan.decode_tokens.numel() == 3


def test_sampler_streams_do_not_depend_on_the_batch(cpu_kernels):
    """A seeded request draws the same tokens alone and beside others; greedy rows are the arg-max."""
    from liteinfer_b200 import SamplingParams
    from liteinfer_b200.sampling.sampler import Sampler

    g = torch.Generator().manual_seed(0)
    logits = torch.randn(3, 50, generator=g)
    seeded = SamplingParams(temperature=1.0, top_k=20, top_p=0.9, seed=7)
    alone = [int(Sampler(1)(logits[1:2], [seeded], ["r"])[0]) for _ in range(1)]
    sampler = Sampler(99)
    mixed = sampler(logits, [SamplingParams(temperature=0.0), seeded, SamplingParams(temperature=0.8)], ["a", "r", "c"])
    assert int(mixed[1]) == alone[0] and int(mixed[0]) == int(torch.argmax(logits[0]))
    draws_a = [int(Sampler(5)(logits[2:3], [SamplingParams(temperature=1.5, seed=3)], ["x"])[0]) for _ in range(2)]
    assert draws_a[0] == draws_a[1]                                    # same seed, same first draw
    s = Sampler(5)
    p = SamplingParams(temperature=1.5, seed=3)
    many = {int(s(logits[2:3], [p], ["x"])[0]) for _ in range(40)}
    assert len(many) > 3                                               # the stream advances between steps
    with pytest.raises(ValueError):
        s(logits, [p])


@pytest.mark.parametrize("keys", [["a"], ["a", "b"]])
def test_sampler_refuses_fewer_keys_than_rows(cpu_kernels, keys):
    """One key for three rows is not the first row's parameters for all of them."""
    from liteinfer_b200 import SamplingParams
    from liteinfer_b200.sampling.sampler import Sampler

    with pytest.raises(ValueError):
        Sampler(5)(torch.zeros(3, 50), [SamplingParams(temperature=t) for t in (0.0, 1.0, 2.0)], keys)


def test_sample_rule_properties():
    """The row-by-row rule the kernel is tested against: top-k keeps exactly k, the entry crossing p is kept."""
    from torch_kernels import sample_row

    logits = torch.tensor([1.0, 3.0, 3.0, 2.0, -1.0])
    draws = {sample_row(logits, 1.0, 2, 1.0, u / 100) for u in range(100)}
    assert draws == {1, 2}                                             # ties at the top: exactly two survive
    draws = {sample_row(logits, 1.0, 3, 1.0, u / 100) for u in range(100)}
    assert draws == {1, 2, 3}
    probs = torch.softmax(logits, -1)
    p_just_below_top_two = float(probs[1] + probs[2]) - 1e-3
    draws = {sample_row(logits, 1.0, 0, p_just_below_top_two, u / 200) for u in range(200)}
    assert draws == {1, 2}                                             # the second entry crosses p and is kept
    draws = {sample_row(logits, 1.0, 0, float(probs[1]) - 1e-3, u / 50) for u in range(50)}
    assert draws == {1}
    assert sample_row(logits, 0.0, 0, 1.0, 0.5) == 1                   # temperature 0: the first arg-max


def test_bench_run_reports_the_references_summaries(cpu_kernels, model_dirs, capsys):
    """`bench run` on a CPU with the stand-in kernels: forced output lengths, the two modes' fields."""
    import json

    from liteinfer_b200.benchmark import make_prompts, percentile
    from liteinfer_b200.cli import main

    assert percentile([1.0, 2.0, 3.0, 4.0], 50) == 2.5 and percentile([5.0], 99) == 5.0
    mixed = make_prompts(100, None, 200, 64, 0)
    assert all(1 <= len(p) <= 64 for p in mixed) and len({len(p) for p in mixed}) > 10
    assert make_prompts(100, 7, 3, 64, 0) == make_prompts(100, 7, 3, 64, 0)
    code = main(["bench", "run", "--model", str(model_dirs["tiny_a"]), "--isl", "9", "--osl", "4", "-n", "5",
                 "--dtype", "float32", "--device", "cpu", "--max-num-seqs", "2", "--max-model-len", "32"])
    assert code == 0
    result = json.loads(capsys.readouterr().out.strip().splitlines()[-1])
    assert result["dataset"]["num_samples"] == 5 and result["dataset"]["input_tokens"] == 45
    assert set(result["summary"]["throughput"]) == {"output_tokens_per_s", "requests_per_s", "wall_time_s", "step_phases"}
    assert set(result["summary"]["latency"]) == {"ttft_p50_ms", "ttft_p95_ms", "ttft_p99_ms", "itl_p50_ms",
                                                 "itl_p95_ms", "itl_p99_ms", "e2e_p50_ms"}
    assert result["summary"]["throughput"]["output_tokens_per_s"] > 0


def test_padded_shapes_of_the_step_graphs():
    """The ladder that steps are rounded up to before they are replayed from a graph: never below the step, less
    than 16 tokens or an eighth of the next power of two above it, few distinct shapes, and stable (a padded size
    pads to itself)."""
    from liteinfer_b200.engine.runner import _pow2, _token_bucket

    shapes = set()
    for n in range(1, 8193):
        padded = _token_bucket(n)
        shapes.add(padded)
        assert padded >= n and _token_bucket(padded) == padded
        assert padded - n < max(16, _pow2(n) // 8)
    assert len(shapes) <= 48
    assert [_pow2(n) for n in (0, 1, 2, 3, 4, 5, 33, 64)] == [1, 1, 2, 4, 4, 8, 64, 64]


def test_steps_launched_ahead_give_the_same_outputs(cpu_kernels, model_dirs):
    """The engine launches a step before it has read the tokens of the step before.  With every kind of ending
    (a stop id early or late, min_tokens, max_tokens, the context limit), prompts cut by the budget and a cache
    that makes newcomers wait, the outputs are those of the engine that reads every step before the next."""
    from liteinfer_b200 import LLM, SamplingParams

    config, _, page = tiny_configs.ALL["tiny_a"]
    vocab = config["vocab_size"]
    prompts = _prompts(vocab, (5, 21, 9, 30, 2, 14, 17, 40))
    common = dict(dtype="float32", device="cpu", block_size=page, max_num_seqs=3, max_model_len=48,
                  max_num_batched_tokens=12, num_gpu_blocks=7)
    with LLM(str(model_dirs["tiny_a"]), async_scheduling=False, **common) as llm:
        free = [o.token_ids for o in llm.generate(prompts, SamplingParams(temperature=0.0, max_tokens=12))]
    params = [
        SamplingParams(temperature=0.0, max_tokens=12, stop_token_ids=[free[0][0]]),            # the very first token ends it
        SamplingParams(temperature=0.0, max_tokens=12, stop_token_ids=[free[1][4]]),
        SamplingParams(temperature=0.0, max_tokens=12, stop_token_ids=[free[2][1]], min_tokens=5),
        SamplingParams(temperature=0.0, max_tokens=100),                                          # the context limit
        SamplingParams(temperature=0.0, max_tokens=1),
        SamplingParams(temperature=0.0, max_tokens=12, stop=[" " + str(free[5][3])]),            # a stop string
        SamplingParams(temperature=0.7, top_k=5, seed=3, max_tokens=9),                           # a seeded stream
        SamplingParams(temperature=0.0, max_tokens=7, stop_token_ids=[free[7][6]]),              # stop id and length at once
    ]
    runs = []
    for ahead in (False, True):
        with LLM(str(model_dirs["tiny_a"]), async_scheduling=ahead, **common) as llm:
            outs = llm.generate(prompts, params)
            runs.append([(o.token_ids, o.finish_reason, o.text) for o in outs])
            assert llm.stats.num_requests_aborted == 0
            llm.engine.step()
            cache = llm.engine.runner.cache
            cache.check_invariants()
            assert all(g.allocator.num_held == 0 for g in cache.groups) and cache.slots.num_held == 0
            assert not llm.engine.has_unfinished()
    assert runs[0] == runs[1]
    assert runs[1][0][0] == free[0][:1] and runs[1][0][1] == "stop"
    assert runs[1][3][1] == "length" and len(prompts[3]) + len(runs[1][3][0]) == 48
    assert all(-1 not in tokens for tokens, _, _ in runs[1])


@pytest.mark.parametrize("family,name", [("tiny", "tiny_a"), ("gifudra", "gif_a"), ("karupel", "kar_a"), ("kegizen", "keg_a"),
                                         ("kutolix", "kut_a"), ("lulisun", "lul_a"), ("sogazen", "sog_a")])
def test_every_weight_of_a_product_is_at_rest(cpu_kernels, monkeypatch, tmp_path, family, name):
    """What a bound model multiplies by may be read before the kernel ahead is done; a computed operand, or a view, may not."""
    import importlib

    from liteinfer_b200 import LLM, SamplingParams, ops
    from liteinfer_b200.weights.random_init import write_random_model

    config, seed, page = importlib.import_module(f"{family}_configs").ALL[name]
    seen = []

    def watched(product):
        def run(x, weight, *args, **kwargs):
            seen.append(weight)
            return product(x, weight, *args, **kwargs)
        return run

    monkeypatch.setattr(ops, "linear", watched(ops.linear))
    monkeypatch.setattr(ops, "batched_linear", watched(ops.batched_linear))
    with LLM(str(write_random_model(config, tmp_path / name, seed)), dtype="float32", device="cpu", block_size=page,
             max_num_seqs=2, max_model_len=64) as llm:
        llm.generate(_prompts(config["vocab_size"] if family == "tiny" else 40, (9, 2)),
                     SamplingParams(temperature=0.0, max_tokens=2, ignore_eos=True))
    assert seen and all(ops.kernels._at_rest(w) for w in seen)
    assert not ops.kernels._at_rest(torch.zeros(2, 2)) and not ops.kernels._at_rest(seen[0][:1])


def test_a_step_says_how_long_its_prompts_contexts_are(cpu_kernels, model_dirs):
    """The plan of a step that runs kernel by kernel has the longest context of the rows that bring several tokens; a graph's
    has the bound of its class."""
    from liteinfer_b200 import LLM
    from liteinfer_b200.engine.runner import StepEntry
    from liteinfer_b200.ops import kernels

    _, _, page = tiny_configs.ALL["tiny_a"]
    with LLM(str(model_dirs["tiny_a"]), dtype="float32", device="cpu", block_size=page, max_num_seqs=4, max_model_len=64) as llm:
        runner = llm.engine.runner
        runner.step([StepEntry("a", list(range(1, 12)), (10,)), StepEntry("b", [1, 2, 3], (2,))])
        entries = [StepEntry("a", [5], (0,)), StepEntry("b", [4, 5], (1,))]
        runner.cache.reserve(["a", "b"], [12, 5])
        plan = runner.build_context(entries).plan
        assert (plan.max_prefill_context_len, plan.max_decode_context_len) == (5, 12)
        runner.cache.rollback(["a", "b"])
        assert runner.build_context([StepEntry("a", [5], (0,))]).plan.max_prefill_context_len == 0
    classes = [kernels.context_class(n, 4096, (64, 448)) for n in (1, 64, 65, 448, 449, 4096)]
    assert classes == [64, 64, 448, 448, 4096, 4096]
    assert [kernels.context_class(n, 64, (64, 448)) for n in (5, 64)] == [64, 64] and kernels.context_class(100, 300, (64, 448)) == 300
    assert kernels.context_class(5, 300, ()) == 300


def test_a_model_names_the_contexts_that_its_kernels_turn_at():
    import kutolix_configs

    from liteinfer_b200.config.registry import resolve
    from liteinfer_b200.ops import kernels
    from liteinfer_b200.parts.model import Model

    def bounds(config, dtype, prompts=1, longest=16):
        arch, typed = resolve(config)
        return Model(arch.build_spec(typed), dtype, torch.device("cpu")).context_bounds(prompts, longest)

    plain = dict(tiny_configs.ALL["tiny_a"][0], head_dim=64, num_attention_heads=8, num_key_value_heads=2)
    few, more = kernels.ATTENTION_CONTEXTS
    assert bounds(plain, torch.bfloat16) == (few,) and bounds(plain, torch.bfloat16, 4, 512) == (more,)
    assert bounds(plain, torch.bfloat16, 8, 512) == () and bounds(plain, torch.bfloat16, 0, 512) == ()
    assert kernels.LATENT_CONTEXTS[0] in bounds(kutolix_configs.ALL["kut_a"][0], torch.bfloat16)
    assert bounds(kutolix_configs.ALL["kut_a"][0], torch.float32) == ()


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(32, 8, 64), (24, 8, 128), (8, 1, 64), (128, 1, 128), (4, 4, 96), (6, 2, 64)])
def test_a_graph_launches_prompt_attention_as_its_steps_would(heads, kv_heads, head_dim):
    """Whether blocks go out in pairs is the same for a step's contexts and for the bound of their class, and a launch whose form
    no context decides has one class."""
    from liteinfer_b200.ops import kernels

    def in_pairs(prompts, longest, context):            # the launch's own rule
        rows = 128 // (heads // kv_heads)
        rows *= 2 if head_dim == 128 and longest > rows else 1
        blocks = kv_heads * prompts * -(-longest // rows)
        return (head_dim in (64, 128) and 2 * blocks <= (296 if head_dim == 64 else 148)
                and context > 64 * (9 if 2 * blocks > 148 else 7))

    for prompts in (1, 2, 4, 16):
        for longest in (16, 112, 448, 512, 576, 640, 1024, 2048):
            bounds = kernels.attention_contexts(heads, kv_heads, head_dim, prompts, longest)
            assert len(bounds) <= 1
            for context in (2, 447, 448, 449, 576, 577, 4000, 4096):
                stated = kernels.context_class(context, 4096, bounds)
                assert in_pairs(prompts, longest, context) == in_pairs(prompts, longest, stated)
            forms = {in_pairs(prompts, longest, context) for context in (2, 4096)}
            assert len(forms) == 1 + len(bounds)
