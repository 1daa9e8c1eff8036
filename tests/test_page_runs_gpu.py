"""Prefill attention brings the pages of a tile that follow one another in the pool in one box, others a box each
(csrc/attention_tcgen05.cu: load_pages): the same keys and values in pages that follow one another, in pages that do so but for some,
in descending order and scattered give the same bits, in both kernels and with their clusters, and those are the plain reference's."""

import pytest
import torch

import torch_ops as ref

pytestmark = pytest.mark.gpu


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("form", [1, 2, 4])
@pytest.mark.parametrize("d,page", [(128, 16), (128, 32), (128, 64), (128, 128), (64, 16), (64, 64)])
@pytest.mark.parametrize("requests,window", [([(0, 70)], 0), ([(0, 129), (70, 200)], 0), ([(500, 300)], 0), ([(700, 150)], 333)])
def test_where_the_pages_lie_changes_no_bit(form, d, page, requests, window):
    from paged_attention_engine_b200.kernels import ops

    heads, kv_heads = 4, 2
    gen = torch.Generator().manual_seed(d + page)
    counts = [-(-(c + n) // page) for c, n in requests]
    total, tokens = sum(counts), sum(n for _, n in requests)

    def normal(*shape):
        return torch.randn(shape, generator=gen).to(torch.bfloat16)

    qkv = normal(tokens, (heads + 2 * kv_heads) * d)
    keys, values = normal(total, kv_heads, page, d), normal(total, kv_heads, page, d)
    q_start = [0]
    for _, n in requests:
        q_start.append(q_start[-1] + n)
    kv_len = [c + n for c, n in requests]
    args = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=d, page_size=page, max_q_len=max(n for _, n in requests), max_kv_len=max(kv_len),
                scale=d ** -0.5, window=window)

    def run(place):
        """Page i of the keys lies at place[i] of a pool with room to spare, which is not a number."""
        pool_k = torch.full((total + 9, kv_heads, page, d), float("nan"), dtype=torch.bfloat16)
        pool_v = pool_k.clone()
        pool_k[place], pool_v[place] = keys, values
        table, at = torch.zeros((len(requests), max(counts)), dtype=torch.int32), 0
        for b, c in enumerate(counts):
            table[b, :c] = place[at : at + c].to(torch.int32)
            at += c
        pos0 = [c for c, _ in requests]
        return ops.paged_attention(qkv.cuda(), pool_k.cuda(), pool_v.cuda(), table.cuda(), _i32(q_start), _i32(pos0), _i32(kv_len), **args, form=form), table

    line = torch.arange(total) + 5
    got, _ = run(line)
    swapped = line.clone()
    swapped[::7], swapped[-1] = line[::7], total + 7
    shuffled = torch.randperm(total + 9, generator=gen)[:total]
    for place in (swapped, line.flip(0), shuffled):
        other, _ = run(place)
        assert torch.equal(got, other)
    table, at = torch.zeros((len(requests), max(counts)), dtype=torch.int32), 0
    for b, c in enumerate(counts):
        table[b, :c] = torch.arange(at, at + c)
        at += c
    want = ref.paged_attention(qkv, keys, values, table, torch.tensor(q_start), torch.tensor([c for c, _ in requests]), torch.tensor(kv_len), **args).float()
    assert (got.cpu().float() - want).abs().max() <= 2.0 ** -6 * max(1.0, float(want.abs().max()))
    ops.check_device_errors()


@pytest.mark.parametrize("form", [1, 2, 4])
def test_a_request_without_a_visible_key_disturbs_nothing(form):
    """A request of 70 tokens whose length says 0: no copy is made for it, and its neighbours' outputs keep their bits."""
    from paged_attention_engine_b200.kernels import ops

    heads, kv_heads, d, page = 4, 2, 128, 16
    gen = torch.Generator().manual_seed(3)
    qkv = torch.randn((70 + 90, (heads + 2 * kv_heads) * d), generator=gen).to(torch.bfloat16).cuda()
    keys, values = (torch.randn((12, kv_heads, page, d), generator=gen).to(torch.bfloat16).cuda() for _ in range(2))
    args = dict(num_heads=heads, num_kv_heads=kv_heads, head_dim=d, page_size=page, max_q_len=90, max_kv_len=90, scale=d ** -0.5, window=0, form=form)
    table = torch.arange(12, dtype=torch.int32).view(2, 6).cuda()
    got = ops.paged_attention(qkv, keys, values, table, _i32([0, 70, 160]), _i32([0, 0]), _i32([0, 90]), **args)
    alone = ops.paged_attention(qkv[70:].contiguous(), keys, values, table[1:].contiguous(), _i32([0, 90]), _i32([0]), _i32([90]), **args)
    assert torch.equal(got[70:], alone)
    ops.check_device_errors()
