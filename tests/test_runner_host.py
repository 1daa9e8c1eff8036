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
