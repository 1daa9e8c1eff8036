"""Recorded decode steps whose attention's slices are planned: each replay plans anew from the lengths that the step's copy brought, all layers
use the plan, padding rows are planned with the rest. Against the same steps run eagerly and without plans."""

import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(tmp_path_factory):
    from paged_attention_engine_b200 import Engine

    raw, _, seed = helpers.TINY["tiny_d"]
    return Engine.from_pretrained(helpers.write_model(tmp_path_factory.mktemp("model"), raw, seed, torch.bfloat16, sharpen=4.0), "bfloat16")


def _run(engine, contexts, steps, use_graphs):
    """Logits of decode `steps`, each a list of the requests that bring one token, in that order; `contexts`: tokens in the cache before."""
    from paged_attention_engine_b200 import StepEntry

    vocab, page = 1000, 16
    tokens = {key: helpers.random_tokens(vocab, 512, 900 + key) for key in contexts}
    cache = engine.new_paged_cache(sum(512 // page for _ in contexts), page, len(contexts))
    runner = engine.new_runner(cache, use_graphs=use_graphs)
    at = dict(contexts)
    for key, n in contexts.items():
        assert runner.begin_request(key) and runner.manager.reserve(key, 512).ok
        runner.step([StepEntry(key, tuple(tokens[key][:n]), ())])
    out = []
    for step in steps:
        entries = [StepEntry(key, (tokens[key][at[key]],), (0,)) for key in step]
        out.append(runner.step(entries).logits.float().cpu())
        for key in step:
            at[key] += 1
    return out, runner


def _compare(engine, monkeypatch, contexts, steps):
    from paged_attention_engine_b200.kernels import ops

    monkeypatch.setattr(ops, "use_decode_plans", False)
    want, _ = _run(engine, contexts, steps, use_graphs=False)
    monkeypatch.setattr(ops, "use_decode_plans", True)
    monkeypatch.setattr(ops, "PLANNED_MIN_TILES", 1)
    lib = ops._lib("attention_mma")
    planned = []
    real = lib.pae_paged_attention_decode_planned
    monkeypatch.setattr(lib, "pae_paged_attention_decode_planned", lambda *args: (planned.append(1), real(*args))[1])
    got, runner = _run(engine, contexts, steps, use_graphs=True)
    for i, (g, w) in enumerate(zip(got, want)):
        assert torch.isfinite(g).all()
        gap = (g - w).abs().max().item()
        assert gap <= helpers.tolerance(torch.bfloat16, w), f"step {i}: {gap}"
    ops.check_device_errors()
    return runner, len(planned)


def test_a_replay_plans_for_the_lengths_of_its_own_step(engine, monkeypatch):
    """One recording (ten rows, up to 512 keys): other requests in other places, so that a slice of the step before would be another request's."""
    contexts = dict(enumerate([300, 20, 150, 7, 260, 33, 90, 16, 1, 400, 64]))
    steps = [[0, 1, 2, 3, 4, 5, 6, 7, 8], [8, 7, 6, 5, 4, 3, 2, 1, 0], [9, 3, 1, 8, 7, 5, 10, 6, 2, 4], [1, 3, 5, 7, 8, 10, 6, 2, 9], [4, 9, 0, 2, 6, 10, 5, 1, 3, 7],
             [10, 1, 9, 3, 0, 5, 8, 7, 4]]
    runner, planned = _compare(engine, monkeypatch, contexts, steps)
    if helpers.records_steps():
        assert [key for key in runner.graphs] == [(10, 32, 512, False, True)] and runner.graph_replays == len(steps) - 1
        assert planned == 2, "once a layer, in the recording"


def test_contexts_that_grow_past_the_line_between_planned_and_not(engine, monkeypatch):
    """Four requests of 380 and more of 512 keys: three quarters are filled at 384."""
    runner, planned = _compare(engine, monkeypatch, dict(enumerate([380, 381, 380, 379])), [[0, 1, 2, 3], [3, 1, 0, 2]] * 4)
    if helpers.records_steps():
        assert sorted(key[4] for key in runner.graphs) == [False, True] and runner.graph_replays == 6 and planned == 2
