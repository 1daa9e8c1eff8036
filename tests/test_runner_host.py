"""The step function's recordings, without a device: the model runs on the plain torch stand-in, and what would record
a step runs it instead."""

import pytest
import torch

import helpers
import torch_ops
from paged_attention_engine_b200 import Engine, StepEntry


@pytest.fixture(scope="module")
def folder(tmp_path_factory):
    raw, _, seed = helpers.TINY["tiny_a"]
    return helpers.write_model(tmp_path_factory.mktemp("model"), raw, seed, torch.float32, sharpen=4.0)


def _runner(folder, requests):
    """A runner with `requests` = {key: context} open, the contexts in the cache already."""
    engine = Engine.from_pretrained(folder, "float32", device="cpu", ops=torch_ops)
    page = 16
    cache = engine.new_paged_cache(sum(-(-(c + 16) // page) for c in requests.values()), page, len(requests))
    runner = engine.new_runner(cache)
    for key, context in requests.items():
        assert runner.begin_request(key) and runner.manager.reserve(key, context + 16).ok
        if context:
            runner.step([StepEntry(key, tuple(range(1, context + 1)), ())])
    return runner


def test_a_recording_without_room_leaves_nothing_to_the_eager_step(folder):
    """What the parts keep with the step while it is recorded (the positions' table, a plan of the slices) has not been made when the
    recording ends: the eager step that stands in for a recording without room must not find it."""
    requests = {"a": 5, "b": 20}
    entries = [StepEntry("a", (3, 4), (1,)), StepEntry("b", (7,), ())]
    plain = _runner(folder, requests)
    want = plain.step(entries).logits.clone()
    runner = _runner(folder, requests)
    runner.use_graphs = True
    runner.shapes_seen[runner._shape_key(entries, None)] = 1           # the second time: a recording
    recorded = []

    def out_of_memory(slot, ctx):
        runner._run(ctx)
        assert ctx.memo, "the parts keep something with the step"
        for held in ctx.memo.values():                                   # recorded, not made: whatever the memory held
            if torch.is_tensor(held):
                held.fill_(float("nan"))
        ctx.kv_len.decode_plans = {"unmade": None}
        recorded.append(ctx)
        raise torch.OutOfMemoryError("no room")

    runner._capture = out_of_memory
    ran = []
    run = runner._run
    runner._run = lambda ctx: (ran.append(ctx), run(ctx))[1]
    got = runner.step(entries).logits
    assert len(recorded) == 1 and ran[-1] is not recorded[0]
    assert not hasattr(ran[-1].kv_len, "decode_plans")
    assert torch.equal(got, want)


def _keys(runner, contexts_of_steps):
    """The recordings that decode steps of requests with these contexts ask for."""
    keys = set()
    for contexts in contexts_of_steps:
        runner.manager.num_computed = lambda key, contexts=contexts: contexts[key]
        keys.add(runner._graph_key([StepEntry(i, (1,), (0,)) for i in range(len(contexts))], None))
    return keys


@pytest.mark.parametrize("plans", [False, True])
def test_contexts_of_unequal_lengths_get_recordings_of_their_own_only_where_slices_are_planned(folder, plans):
    runner = _runner(folder, {"a": 0})
    runner.use_graphs = True
    asked = []
    runner.model.plans_decode = lambda seqs, max_kv_len, page_size: (asked.append((seqs, max_kv_len, page_size)), plans and seqs >= 8)[1]
    # Four requests that grow from 16 to 4,095 keys: a recording per longest context rounded up (256, 512, then every 512).
    assert len(_keys(runner, [[n] * 4 for n in range(16, 4096)])) == 9
    assert len(_keys(runner, [[n, 16, 16, 16] for n in range(16, 4096)])) == 9
    # Sixteen: where they are planned, unequal ones another each.
    equal = _keys(runner, [[n] * 16 for n in range(400, 4096, 512)])
    unequal = _keys(runner, [[n] + [16] * 15 for n in range(400, 4096, 512)])
    assert len(equal) == len(unequal) == 8 and (equal.isdisjoint(unequal) if plans else equal == unequal)
    assert len(asked) == len(set(asked)), "asked once per size"


def test_every_decode_step_of_the_largest_batches_finds_room_for_its_recording(folder):
    runner = _runner(folder, {"a": 0})
    runner.use_graphs = True
    runner.model.plans_decode = lambda *sizes: True
    steps = [[n] * b for n in range(15, 4096, 64) for b in range(1, 257)]
    steps += [[n] + [0] * (b - 1) for n in range(15, 4096, 64) for b in range(1, 257)]
    assert len(_keys(runner, steps)) <= runner.MAX_GRAPHS
