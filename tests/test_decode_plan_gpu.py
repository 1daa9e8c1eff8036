"""Decode attention over planned slices (csrc/attention_mma.cuh: plan_decode_kernel, decode_planned_kernel, merge_planned_kernel): the
plan's slices cover every request's keys once, in order, within its room; and the attention is that of the plain reference, for requests of
one tile and of many, with and without a window, beside requests that bring more than one token, and with one slice a pair."""

import numpy as np
import pytest
import torch

import torch_ops as ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from paged_attention_engine_b200.kernels import ops as kernel_ops

    yield kernel_ops
    kernel_ops.PLANNED_MIN_TILES = 4000


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("lengths,window", [([1], 0), ([16, 17, 1, 4095, 500], 0), ([3000] * 70, 0), (list(range(1, 1100, 3)), 0), ([700, 20, 333], 100),
                                            ([5] * 2048, 0), ([40, 0, 900, 0, 0, 77], 0)])
@pytest.mark.parametrize("kv_heads,items,least", [(2, 1184, 2), (4, 0, 3), (1, 64, 6)])
def test_the_slices_cover_every_request(ops, lengths, window, kv_heads, items, least):
    lib = ops._lib("attention_mma")
    q_lens = [1 if n else 3 for n in lengths]                  # 0 stands for a request of three tokens: no slices
    seqs = len(lengths)
    items = max(items, seqs * kv_heads)
    q_start, kv_len = _i32(np.concatenate(([0], np.cumsum(q_lens)))), _i32([n or 50 for n in lengths])
    plan = torch.full((lib.pae_decode_plan_ints(seqs, kv_heads, items),), -7, dtype=torch.int32, device="cuda")
    assert lib.pae_plan_decode(plan.data_ptr(), q_start.data_ptr(), kv_len.data_ptr(), seqs, kv_heads, window, items, least, 0) == 0
    plan = plan.cpu().numpy()
    slices, pairs = plan[: 4 * items].reshape(items, 4), plan[4 * items :].reshape(seqs, kv_heads, 2)
    # The rule: the shortest slices, in steps of a 32nd and from `least` tiles and an even share on, that are no more than `items`; one a pair at the most.
    tiles = [(n + 15) // 16 - (max(0, n - window) // 16 if window else 0) for n in lengths]
    length = max(least, -(-sum(tiles) * kv_heads // items))
    while sum(-(-t // length) for t in tiles) * kv_heads > items and max(tiles) > length:
        length += max(1, length // 32)
    used = 0
    for b, n in enumerate(lengths):
        base = max(0, n - window) // 16 * 16 if window else 0
        for g in range(kv_heads):
            first, count = pairs[b, g]
            assert first == used and count == -(-tiles[b] // length)
            at = base
            for request, head, begin, end in slices[first : first + count]:
                assert (request, head, begin, end) == (b, g, at, min(n, at + 16 * length)) and begin < end
                at = end
            assert n == 0 or at == n
            used += count
    assert used <= items and (slices[used:, 2] >= slices[used:, 3]).all()


def test_a_request_without_a_key_leaves_zeros(ops):
    """As without a plan: no slice is made for it, and its row is written all the same."""
    heads, kv_heads, d, page, lengths = 4, 2, 64, 16, [70, 0, 33, 1]
    gen = torch.Generator().manual_seed(5)
    qkv = torch.randn((4, (heads + 2 * kv_heads) * d), generator=gen).to(torch.bfloat16).cuda()
    keys, values = (torch.randn((20, kv_heads, page, d), generator=gen).to(torch.bfloat16).cuda() for _ in range(2))
    table, kv_len = torch.arange(20, dtype=torch.int32).view(4, 5).cuda(), _i32(lengths)
    q_start, pos0 = _i32([0, 1, 2, 3, 4]), _i32([n - 1 for n in lengths])
    args = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=d, page_size=page, max_q_len=1, max_kv_len=70, scale=d ** -0.5, window=0)
    alone = ops.paged_attention(qkv, keys, values, table, q_start, pos0, kv_len, **args)
    ops.PLANNED_MIN_TILES = 1
    ops.plan_decode(q_start, kv_len, 70, heads, kv_heads, d, page, 0, torch.bfloat16)
    ops.PLANNED_MIN_TILES = 4000
    torch.full((4, heads * d), float("nan"), dtype=torch.bfloat16, device="cuda")      # what the allocator hands out next
    got = ops.paged_attention(qkv, keys, values, table, q_start, pos0, kv_len, **args)
    assert (alone[1] == 0).all() and (got[1] == 0).all() and torch.isfinite(got).all()
    ops.check_device_errors()


@pytest.mark.parametrize("heads,kv_heads,d,page,window", [(12, 2, 128, 16, 0), (28, 4, 128, 16, 0), (8, 8, 64, 32, 0), (4, 1, 32, 16, 90), (12, 2, 128, 48, 300)])
@pytest.mark.parametrize("lengths", [[1, 900, 17, 16, 33, 2000, 400], [700] * 3 + [5] * 30, [64]])
def test_attention_over_planned_slices(ops, heads, kv_heads, d, page, window, lengths):
    gen = torch.Generator().manual_seed(heads + len(lengths))
    seqs = len(lengths)
    width = max(-(-n // page) for n in lengths)
    counts = [-(-n // page) for n in lengths]
    order = torch.randperm(sum(counts), generator=gen).to(torch.int32)
    table, at = torch.zeros((seqs, width), dtype=torch.int32), 0
    for b, c in enumerate(counts):
        table[b, :c] = order[at : at + c]
        at += c

    def normal(*shape):
        return torch.randn(shape, generator=gen).to(torch.bfloat16)

    qkv = normal(seqs, (heads + 2 * kv_heads) * d)
    keys, values = normal(sum(counts), kv_heads, page, d), normal(sum(counts), kv_heads, page, d)
    q_start, kv_len = torch.arange(seqs + 1, dtype=torch.int32), torch.tensor(lengths, dtype=torch.int32)
    args = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=d, page_size=page, max_q_len=1, max_kv_len=max(lengths), scale=d ** -0.5, window=window)
    tensors = [qkv, keys, values, table, q_start, kv_len - 1, kv_len]
    want = ref.paged_attention(*tensors, **args).float()
    dev = [t.cuda() for t in tensors]
    alone = ops.paged_attention(*dev, **args).cpu().float()
    ops.PLANNED_MIN_TILES = 1
    ops.plan_decode(dev[4], dev[6], max(lengths), heads, kv_heads, d, page, window, torch.bfloat16)
    assert (kv_heads, d, window) in dev[6].decode_plans
    got = ops.paged_attention(*dev, **args).cpu().float()
    # Scores' sums in another order and one rounding of the output: as the sliced kernel's tolerance.
    assert (got - want).abs().max() <= 2.0 ** -6 * max(1.0, float(want.abs().max()))
    assert (got - want).norm() <= 1.05 * (alone - want).norm() + 1e-3
    ops.check_device_errors()
