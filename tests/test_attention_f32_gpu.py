"""Float32 attention for head sizes 32, 64 and 128: contexts on both sides of a 16-key tile and of a round of
eight tiles, windows whose earlier pages are released, portions and single tokens; and a query's bits however
the step is cut."""

import pytest
import torch

import torch_ops as ref

pytestmark = pytest.mark.gpu


def _case(q_lens, pos0, heads, kv_heads, d, page, window, seed):
    gen = torch.Generator().manual_seed(seed)
    kv_lens = [p + n for p, n in zip(pos0, q_lens)]
    width = max(-(-n // page) for n in kv_lens)
    pages = sum(-(-n // page) for n in kv_lens) + 2
    order = torch.randperm(pages, generator=gen).tolist()
    keys = torch.randn(pages, kv_heads, page, d, generator=gen)
    values = torch.randn(pages, kv_heads, page, d, generator=gen)
    table = torch.full((len(q_lens), width), -1, dtype=torch.int32)
    for b, n in enumerate(kv_lens):
        released = max(0, pos0[b] - window + 1) // page if window else 0
        for i in range(-(-n // page)):
            at = order.pop()
            if i < released:
                keys[at] = values[at] = float("nan")
            else:
                table[b, i] = at
    qkv = torch.randn(sum(q_lens), (heads + 2 * kv_heads) * d, generator=gen)
    q_start = torch.tensor([0] + torch.tensor(q_lens).cumsum(0).tolist(), dtype=torch.int32)
    return [qkv, keys, values, table, q_start, torch.tensor(pos0, dtype=torch.int32), torch.tensor(kv_lens, dtype=torch.int32)], dict(
        num_heads=heads, num_kv_heads=kv_heads, head_dim=d, page_size=page, max_q_len=max(q_lens), max_kv_len=max(kv_lens),
        scale=d**-0.5 * 2.0, window=window)


@pytest.mark.parametrize("q_lens,pos0", [([1, 1, 1, 1, 1, 1], [0, 15, 16, 127, 128, 1000]), ([1, 3, 4, 5, 70], [300, 126, 0, 14, 40])])
@pytest.mark.parametrize("heads,kv_heads,d,page,window", [(3, 1, 32, 16, 0), (4, 4, 64, 4, 33), (12, 2, 128, 16, 0), (6, 1, 128, 64, 17), (2, 2, 32, 1, 1)])
def test_float32_attention(q_lens, pos0, heads, kv_heads, d, page, window):
    from paged_attention_engine_b200.kernels import ops

    tensors, args = _case(q_lens, pos0, heads, kv_heads, d, page, window, 1)
    want = ref.paged_attention(*tensors, **args)
    got = ops.paged_attention(*[t.cuda() for t in tensors], **args)
    # Sums of d products and of 1,001 weights in float32, exponentials within two units: far inside 2e-5 of the largest value.
    assert float((got.cpu() - want).abs().max()) <= 2e-5 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("d", [32, 64, 128])
def test_a_query_has_the_same_bits_however_the_step_is_cut(d):
    from paged_attention_engine_b200.kernels import ops

    tensors, args = _case([150], [37], 4, 2, d, 16, 0, 2)
    qkv, keys, values, table, _, _, _ = [t.cuda() for t in tensors]
    whole = ops.paged_attention(*[t.cuda() for t in tensors], **args)
    i32 = lambda *a: torch.tensor(a, dtype=torch.int32, device="cuda")  # noqa: E731
    for at, n in ((0, 1), (90, 1), (3, 2), (10, 140)):
        part = ops.paged_attention(qkv[at : at + n].contiguous(), keys, values, table, i32(0, n), i32(37 + at), i32(37 + at + n),
                                   **dict(args, max_q_len=n, max_kv_len=37 + at + n))
        assert torch.equal(part, whole[at : at + n])


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("where", ["query", "key", "all keys"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("q_lens,pos0", [([1, 1], [40, 200]), ([6, 30], [40, 0])])
def test_a_score_that_is_no_number_reaches_the_output(d, where, bad, q_lens, pos0):
    """As a softmax has it: NaN for every query that sees such a score (infinity less infinity among them), the others untouched."""
    from paged_attention_engine_b200.kernels import ops

    page = 16
    tensors, args = _case(q_lens, pos0, 2, 1, d, page, 0, 3)
    qkv, keys, _, table, _, _, _ = tensors
    if where == "query":
        qkv[sum(q_lens) - 1, :d] = bad       # the first head of the last token
    elif where == "key":
        keys[table[0, 0], 0, 3] = bad        # key 3 of the first request
    else:
        keys[table[0, : -(-(pos0[0] + q_lens[0]) // page)].long()] = bad
    want = ref.paged_attention(*tensors, **args)
    got = ops.paged_attention(*[t.cuda() for t in tensors], **args).cpu()
    assert bool(want.isnan().any()) and bool(want.isfinite().any())
    assert torch.equal(got.isnan(), want.isnan())
    there = want.isfinite()
    assert float((got[there] - want[there]).abs().max()) <= 2e-5 * max(1.0, float(want[there].abs().max()))


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("longest", [3, 16, 17, 32, 33, 64, 65, 130])
def test_a_prompt_has_the_same_bits_alone_and_in_a_launch_that_fills_the_gpu(d, longest):
    """Many blocks of short contexts run with fewer warps and fewer registers; windows and lengths off the tiles."""
    from paged_attention_engine_b200.kernels import ops

    heads, window = 8, 0 if longest % 2 else 20
    q_lens = [longest] * 40 + [max(1, longest - 5), max(1, longest // 2), 1, longest]
    pos0 = [0] * 43 + [min(longest, 7)]
    tensors, args = _case(q_lens, pos0, heads, 2, d, 16, window, 4)
    want = ref.paged_attention(*tensors, **args)
    qkv, keys, values, table, q_start, _, kv_len = [t.cuda() for t in tensors]
    got = ops.paged_attention(*[t.cuda() for t in tensors], **args)
    assert float((got.cpu() - want).abs().max()) <= 2e-5 * max(1.0, float(want.abs().max()))
    i32 = lambda *a: torch.tensor(a, dtype=torch.int32, device="cuda")  # noqa: E731
    for b in (0, 40, 41, 42, 43):
        at, n = int(q_start[b]), q_lens[b]
        alone = ops.paged_attention(qkv[at : at + n].contiguous(), keys, values, table[b : b + 1].contiguous(), i32(0, n), i32(pos0[b]), kv_len[b : b + 1],
                                    **dict(args, max_q_len=n, max_kv_len=pos0[b] + n))
        assert torch.equal(alone, got[at : at + n])
