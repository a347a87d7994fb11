"""The routes a decode step can take through the runner, compared at the level of
logits: launched kernel by kernel, replayed as the captured step (with fewer
requests than the step was captured for, so that some of it is padding), and
packed ahead of time and then replayed (what the engine does while the step before
runs).  The model is drawn so that attention decides the next token."""

import numpy as np
import pytest
import torch

import plain_qwen3 as P
from tiny_configs import CONFIGS, write_model

pytestmark = pytest.mark.gpu


def err(got, want):
    return float(np.abs(got - want).max() / max(1.0, np.abs(want).max()))


@pytest.mark.parametrize("name,dtype", [("D", "bfloat16"), ("D", "float32"), ("B", "bfloat16"), ("W", "bfloat16")])
def test_launched_captured_and_prepacked_steps_give_the_same_logits(tmp_path, name, dtype):
    from paged_llm_rs_b200.engine.runner import ModelRunner
    from paged_llm_rs_b200.engine.step import StepEntry

    cfg, seed = CONFIGS[name]
    model = write_model(tmp_path, name, decisive=True)
    V = cfg["vocab_size"]
    runner = ModelRunner(model, dtype=dtype, page_size=16, num_pages=64, max_requests=8, prefix_cache=False)
    cache = runner.cache
    rng = np.random.default_rng(seed + 40)
    lens = dict(a=70, b=5, c=131)          # three requests: the captured step for four runs with one row of padding
    steps = 12
    toks = {k: rng.integers(0, V, n + steps).tolist() for k, n in lens.items()}
    for k, n in lens.items():
        cache.open(k)
        assert cache.reserve(k, n)
        runner.step([StepEntry(k, toks[k][:n], [])])
        cache.commit(k, n)
    c64, w64 = P.load_model(model, torch.float64)
    want = {k: P.forward(c64, w64, toks[k]).numpy() for k in lens}
    # the plain model's next token depends on what attention adds (else this test could not see the cache)
    silent = {n: (v * 0 if "o_proj" in n else v) for n, v in w64.items()}
    moved = sum(int(P.forward(c64, silent, toks[k])[-1].argmax() != want[k][-1].argmax()) for k in lens)
    assert moved >= 2
    zeros = np.zeros(3, dtype=np.float32)
    tol = 2e-5 if dtype == "float32" else 3e-2
    worst_between = 0.0
    for i in range(steps):
        entries = [StepEntry(k, [toks[k][lens[k] + i]], [0]) for k in lens]
        for k in lens:
            assert cache.reserve(k, 2)      # this step's token and the next one's (the prepacked step stands one further)
        runner.use_graphs = False
        launched, _ = runner.step_and_sample(entries, zeros, zeros)
        launched = launched.cpu().numpy()
        runner.use_graphs = True
        captured, tokens = runner.step_and_sample(entries, zeros, zeros)
        captured, tokens = captured.cpu().numpy(), tokens.cpu().numpy()
        graph = runner._decode_graph(entries)
        assert graph.B == 4 and graph.native is not None
        runner.check_status()
        assert (tokens[1:] == captured.argmax(1)).all()
        worst_between = max(worst_between, err(captured, launched))
        for r, k in enumerate(lens):
            pos = lens[k] + i
            assert err(captured[r][None], want[k][pos][None]) <= tol, (k, i)
            assert err(launched[r][None], want[k][pos][None]) <= tol, (k, i)
            if dtype == "float32":
                assert captured[r].argmax() == want[k][pos].argmax()
        # the same step packed ahead of time: pack while the cache still counts one token less
        if i + 1 < steps:
            nxt = [StepEntry(k, [0], [0]) for k in lens]
            g2 = runner.prepack_decode(nxt, zeros)
            assert g2 is graph
            for k in lens:
                cache.commit(k, 1)
            feed = [toks[k][lens[k] + i + 1] for k in lens]
            ahead, _ = g2.launch_prepacked(feed, None)
            ahead = ahead.cpu().numpy().copy()
            again, _ = runner.step_and_sample([StepEntry(k, [t], [0]) for k, t in zip(lens, feed)], zeros, zeros)
            assert np.array_equal(ahead, again.cpu().numpy()), i      # the same captured kernels: bit for bit
        else:
            for k in lens:
                cache.commit(k, 1)
    assert worst_between <= (2e-5 if dtype == "float32" else 2e-2)
    runner.check_status()
    for k in lens:
        cache.close(k)
    cache.check_invariants()


@pytest.mark.parametrize("budget,total,sizes", [(128, 3, [128, 64, 64]), (128, 64, [128, 64, 64]), (128, 65, [128]), (96, 10, [96, 96]),
                                                (600, 40, [None, 64, 64]), (600, 257, [None, 320, 320]), (600, 590, [600])])
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_a_small_portion_step_gives_the_same_logits_launched_and_at_every_captured_size(tmp_path, dtype, budget, total, sizes):
    from paged_llm_rs_b200.engine.runner import ModelRunner
    from paged_llm_rs_b200.engine.step import StepEntry

    cfg, seed = CONFIGS["D"]
    model = write_model(tmp_path, "D", decisive=True)
    runner = ModelRunner(model, dtype=dtype, page_size=16, num_pages=96, max_requests=8, prefix_cache=False)
    runner.graph_step_tokens = budget
    cache, rng = runner.cache, np.random.default_rng(total)
    toks = rng.integers(0, cfg["vocab_size"], 70 + total).tolist()
    for r, n in (("a", 70), ("b", 23)):        # a request that decodes beside a portion of another, which has 23 tokens behind it
        cache.open(r)
        assert cache.reserve(r, n + total)
        runner.step([StepEntry(r, toks[:n], [])])
        cache.commit(r, n)
    entries = [StepEntry("a", toks[70:71], [0]), StepEntry("b", toks[23:23 + total - 1], [total - 2])]
    zeros = np.zeros(2, dtype=np.float32)
    runner.use_graphs = False
    want = runner.step_and_sample(entries, zeros, zeros)[0].cpu().numpy()
    runner.use_graphs = True
    for size in sizes:
        was = set(runner._graphs)
        got, tokens = runner.step_and_sample(entries, zeros, zeros)
        got, tokens = got.cpu().numpy(), tokens.cpu().numpy()
        runner.check_status()
        assert {k[0] for k in set(runner._graphs) - was} <= {size} and (size is None) == (runner.tokens_host is None)
        assert err(got, want) <= (2e-5 if dtype == "float32" else 3e-2) and (tokens[1:] == got.argmax(1)).all()
    assert {k[0] for k in runner._graphs} == {n for n in sizes if n is not None}


def test_the_captured_step_without_reductions_is_taken_where_nothing_is_split_and_only_there(tmp_path):
    from paged_llm_rs_b200.engine.runner import ModelRunner
    from paged_llm_rs_b200.engine.step import StepEntry

    cfg, seed = CONFIGS["B"]
    model = write_model(tmp_path, "B", decisive=True)
    runner = ModelRunner(model, dtype="float32", page_size=16, num_pages=96, max_requests=8, prefix_cache=False)
    cache, rng = runner.cache, np.random.default_rng(5)
    toks = rng.integers(0, cfg["vocab_size"], 601).tolist()
    for r, n in (("short", 40), ("long", 600)):
        cache.open(r)
        assert cache.reserve(r, n + 1)
        runner.step([StepEntry(r, toks[:n], [])])
        cache.commit(r, n)
    zero = np.zeros(1, dtype=np.float32)
    launches = {}
    for r, n in (("short", 40), ("long", 600), ("short", 40)):
        entries = [StepEntry(r, [toks[n]], [0])]
        runner.use_graphs = False
        want = runner.step_and_sample(entries, zero, zero)[0].cpu().numpy()
        runner.use_graphs = True
        got = runner.step_and_sample(entries, zero, zero)[0].cpu().numpy()
        runner.check_status()
        assert err(got, want) <= 2e-5
        launches.setdefault(r, runner.last_launches)
        assert launches[r] == runner.last_launches
    assert launches["long"] - launches["short"] == cfg["num_hidden_layers"]      # (one reduction a layer)
    assert len(runner._graphs) == 1


def portion_runner(tmp_path, budget, requests=8, num_pages=200, dtype="bfloat16"):
    from paged_llm_rs_b200.engine.runner import ModelRunner
    runner = ModelRunner(write_model(tmp_path, "D", decisive=True), dtype=dtype, page_size=16, num_pages=num_pages, max_requests=requests, prefix_cache=False)
    runner.graph_step_tokens = budget
    return runner, np.random.default_rng(7)


def portion_step(runner, rng, total, requests, vocab):
    """Open ``requests`` requests and give each a portion; ``total`` tokens in all."""
    from paged_llm_rs_b200.engine.step import StepEntry
    entries = []
    for i in range(requests):
        n = total // requests + (i < total % requests)
        r = f"r{total}.{requests}.{i}"
        if not runner.cache.has(r):
            runner.cache.open(r)
            assert runner.cache.reserve(r, n)
        entries.append(StepEntry(r, rng.integers(0, vocab, n).tolist(), [n - 1]))
    return entries, np.zeros(requests, dtype=np.float32)


def close(runner, entries):
    for e in entries:
        runner.cache.close(e.request_id)


def test_a_captured_step_has_one_buffer_of_logits_and_those_of_smaller_portions_share_theirs(tmp_path):
    runner, rng = portion_runner(tmp_path, 1024)
    V = CONFIGS["D"][0]["vocab_size"]
    for requests in (1, 2, 5):
        for total in (40, 100, 300, 600, 1000):
            entries, zeros = portion_step(runner, rng, total, requests, V)
            for _ in range(2):
                runner.step_and_sample(entries, zeros, zeros)
            close(runner, entries)
    held = {k: g for k, g in runner._graphs.items() if len(k) == 3}
    assert {k[0] for k in held} == {64, 128, 320, 640, 1024} and {k[2] for k in held if k[0] < 1024} == {1, 8}
    below = {g.logits.data_ptr() for k, g in held.items() if k[0] < 1024}
    assert len(below) == 2 and len({g.logits.data_ptr() for k, g in held.items() if k[0] == 1024} | below) == 2 + 3
    assert all(len(g.variants) == 2 for g in held.values())


def test_small_portions_results_outlast_the_steps_after_them(tmp_path):
    # (a step that fills its budget's captured step leaves its results in that step's buffers; a smaller one's are the caller's)
    runner, rng = portion_runner(tmp_path, 128)
    V = CONFIGS["D"][0]["vocab_size"]
    a, zeros = portion_step(runner, rng, 50, 1, V)
    b, _ = portion_step(runner, rng, 60, 1, V)
    runner.use_graphs = False
    want = [runner.step_and_sample(e, zeros, zeros)[0].clone() for e in (a, b)]
    runner.use_graphs = True
    assert not torch.equal(*want)
    for _ in range(3):
        got = [runner.step_and_sample(e, zeros, zeros) for e in (a, b)]
        torch.cuda.synchronize()
        for (logits, tokens), w in zip(got, want):
            assert err(logits.cpu().numpy(), w.cpu().numpy()) <= 3e-2 and int(tokens[1]) == int(logits[0].argmax())


def test_captured_portions_are_bounded_and_the_one_used_longest_ago_gives_way(tmp_path, monkeypatch):
    from paged_llm_rs_b200.engine import runner as R
    monkeypatch.setattr(R, "PORTION_CAPTURES", 2)
    runner, rng = portion_runner(tmp_path, 600)
    V = CONFIGS["D"][0]["vocab_size"]
    for total, held in ((40, {64}), (100, {64, 128}), (40, {64, 128}), (200, {64, 256}), (100, {256, 128}), (200, {256, 128})):
        entries, zeros = portion_step(runner, rng, total, 1, V)
        runner.use_graphs = False
        want = runner.step_and_sample(entries, zeros, zeros)[0].cpu().numpy()
        runner.use_graphs = True
        for _ in range(3):
            got = runner.step_and_sample(entries, zeros, zeros)[0]
            assert err(got.cpu().numpy(), want) <= 3e-2
        runner.check_status()
        close(runner, entries)
        assert {k[0] for k in runner._graphs} == held == {k[0] for k in runner._portions}


def test_a_smaller_portion_replays_what_is_captured_before_it_is_captured_itself(tmp_path):
    runner, rng = portion_runner(tmp_path, 600)
    V = CONFIGS["D"][0]["vocab_size"]
    fill, zeros = portion_step(runner, rng, 590, 1, V)
    runner.step_and_sample(fill, zeros, zeros)
    assert {k[0] for k in runner._graphs} == {600}
    close(runner, fill)
    entries, zeros = portion_step(runner, rng, 310, 1, V)      # (more than half of 600, and 320 is not captured)
    for held in ({600}, {600, 320}):
        runner.step_and_sample(entries, zeros, zeros)
        assert runner.tokens_host is not None and {k[0] for k in runner._graphs} == held
    small, zeros = portion_step(runner, rng, 130, 1, V)        # (less than half of 320 and of 600: launched)
    runner.step_and_sample(small, zeros, zeros)
    assert runner.tokens_host is None and {k[0] for k in runner._graphs} == {600, 320}


def test_nothing_is_captured_while_requests_run_after_warming_up(tmp_path):
    from paged_llm_rs_b200 import Engine
    cfg, seed = CONFIGS["D"]
    model = write_model(tmp_path, "D", decisive=True)
    eng = Engine(model, dtype="bfloat16", block_size=16, blocks=400, chunk=300, max_batch=16, max_prefill_seqs=2)
    made = eng.warm_up()
    # 1, 2, 4, 8, 16 requests: decode steps, the budget's; 64 and 128 tokens for 1, 8 and 64 requests
    assert made == 5 + 5 + 2 * 3 and eng.warm_up() == 0
    held = set(eng.runner._graphs)
    rng = np.random.default_rng(3)
    eng.generate([rng.integers(0, cfg["vocab_size"], n).tolist() for n in (5, 70, 299, 310, 420, 17, 64, 129, 200, 33, 600, 3)], max_tokens=20)
    assert set(eng.runner._graphs) == held


@pytest.mark.parametrize("family,name", [("pamarax", "small"), ("pamarax", "wide"), ("bumisun", "small"), ("tebozen", "small"), ("tebozen", "wide"),
                                         ("reperax", "small"), ("tubevik", "small"), ("surelorn", "small")])
def test_small_portions_of_models_with_recurrent_layers_and_experts(tmp_path, family, name):
    # a captured size's padding tokens belong to no request: they must reach no state, and take no expert from another token
    import importlib
    from paged_llm_rs_b200.engine.runner import ModelRunner
    M = importlib.import_module(f"{family}_models")
    runner = ModelRunner(M.write_model(tmp_path, name)[0], dtype="float32", page_size=16, num_pages=100, max_requests=8, prefix_cache=False)
    runner.graph_step_tokens = 600
    rng = np.random.default_rng(11)
    for total, requests in ((3, 1), (70, 2), (257, 3)):
        # (requests that begin here: what a step leaves in their states and pages is what it leaves there again)
        entries, zeros = portion_step(runner, rng, total, requests, runner.vocab_size)
        runner.use_graphs = False
        want = runner.step_and_sample(entries, zeros, zeros)[0].cpu().numpy()
        runner.use_graphs = runner.model.capturable()
        for _ in range(3):
            got, tokens = runner.step_and_sample(entries, zeros, zeros)
            got, tokens = got.cpu().numpy(), tokens.cpu().numpy()
            runner.check_status()
            # (other tiles and splits of the float32 products at the captured size: another order of the sums)
            assert err(got, want) <= 1e-4 and (tokens[1:] == got.argmax(1)).all()
        close(runner, entries)
    assert not runner.use_graphs or {k[0] for k in runner._graphs} == {64, 128, 320}
