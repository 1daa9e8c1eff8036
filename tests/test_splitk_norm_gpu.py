"""A split product's sum with the norm after it, for rows that one block and a cluster of two take: widths around
where the form changes and off the blocks' shares, against the sum in float64; and a row's bits in every batch."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2048, 2052, 3584, 4096, 4100, 5120, 8196])
@pytest.mark.parametrize("splits", [1, 5, 13, 24])
@pytest.mark.parametrize("extras", [False, True])
def test_sum_and_norm(width, splits, extras):
    from paged_attention_engine_b200.kernels import ops

    gen = torch.Generator(device="cuda").manual_seed(0)
    rows = 7
    partial = torch.randn(splits, rows, width, device="cuda", generator=gen)
    bias = torch.randn(width, device="cuda", generator=gen) if extras else None
    residual = torch.randn(rows, width, device="cuda", generator=gen).to(torch.bfloat16) if extras else None
    weight = torch.rand(width, device="cuda", generator=gen) + 0.5
    pending = ops.PendingSum(partial, bias, residual, torch.bfloat16)
    normed = ops.rms_norm(pending, weight, 1e-6)
    total = partial.double().sum(0)
    if extras:
        total = total + bias.double() + residual.double()
    # The value is the sum rounded once (and 26 float32 additions); the norm is of the rounded value, rounded once.
    value = pending.value.double()
    assert bool(((value - total).abs() <= total.abs() * 2.0**-8 + 26 * 2.0**-24 * (partial.abs().double().sum(0) + 2)).all())
    want = value * torch.rsqrt((value * value).mean(-1, keepdim=True) + 1e-6) * weight.double()
    assert bool(((normed.double() - want).abs() <= want.abs() * (2.0**-8 + 2.0**-18)).all())
    few = ops.PendingSum(partial[:, 2:4].contiguous(), bias, residual[2:4].contiguous() if extras else None, torch.bfloat16)
    assert torch.equal(ops.rms_norm(few, weight, 1e-6), normed[2:4])


@pytest.mark.parametrize("width", [2052, 3584, 4100, 5120, 8196])
@pytest.mark.parametrize("splits", [2, 13])
def test_a_row_has_the_same_bits_in_launches_of_every_size(width, splits):
    """Few rows are shared by clusters of two blocks, many are not."""
    from paged_attention_engine_b200.kernels import ops

    gen = torch.Generator(device="cuda").manual_seed(1)
    partial = torch.randn(splits, 400, width, device="cuda", generator=gen)
    bias = torch.randn(width, device="cuda", generator=gen)
    residual = torch.randn(400, width, device="cuda", generator=gen).to(torch.bfloat16)
    weight = torch.rand(width, device="cuda", generator=gen) + 0.5
    whole = ops.PendingSum(partial, bias, residual, torch.bfloat16)
    normed = ops.rms_norm(whole, weight, 1e-6)
    for rows in (1, 64, 148, 149, 300):
        some = ops.PendingSum(partial[:, -rows:].clone(), bias, residual[-rows:].clone(), torch.bfloat16)      # on 16-byte boundaries
        assert torch.equal(ops.rms_norm(some, weight, 1e-6), normed[-rows:]) and torch.equal(some.value, whole.value[-rows:])
