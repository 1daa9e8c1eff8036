"""The float32 products: tokens on both sides of every kernel's range, K and N off every tile, against
the same sums in float64; and a token's bits whatever else is in its batch."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(m, n, k, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(m, k, device="cuda", generator=gen)
    w = torch.randn(n, k, device="cuda", generator=gen) * 0.02
    bias = torch.randn(n, device="cuda", generator=gen)
    residual = torch.randn(m, n, device="cuda", generator=gen)
    return x, w, bias, residual


@pytest.mark.parametrize("m", [1, 2, 3, 8, 9, 16, 17, 32, 33, 64, 65, 130])
@pytest.mark.parametrize("n,k", [(1, 4), (31, 96), (33, 252), (96, 256), (70, 260), (65, 2308), (1537, 1536), (4801, 512), (48, 97)])
@pytest.mark.parametrize("extras", [False, True])
def test_float32_product_is_the_rounded_float64_product(m, n, k, extras):
    from paged_attention_engine_b200.kernels import ops

    x, w, bias, residual = _operands(m, n, k)
    got = ops.linear(x, w, bias if extras else None, residual if extras else None)
    want = x.double() @ w.double().T
    if extras:
        want = want + bias.double() + residual.double()
    # One rounding to float32 of a sum in double: half a unit in the last place of the result, and the
    # sums' own error (2^-53 a step relative to the terms' absolute sum) far below it.
    terms = x.double().abs() @ w.double().abs().T + (bias.abs().double() + residual.abs().double() if extras else 0.0)
    assert bool(((got.double() - want).abs() <= want.abs() * 2**-24 + terms * (k + 2) * 2**-52).all())


@pytest.mark.parametrize("n,k", [(96, 96), (256, 1536), (1536, 2052), (9600, 512)])
def test_a_token_has_the_same_bits_in_every_batch(n, k):
    from paged_attention_engine_b200.kernels import ops

    x, w, bias, residual = _operands(200, n, k, seed=1)
    whole = ops.linear(x, w, bias, residual)
    for m in (1, 2, 7, 9, 16, 17, 32, 33, 64, 100):
        assert torch.equal(ops.linear(x[:m], w, bias, residual[:m]), whole[:m])


@pytest.mark.parametrize("k", [128, 132, 1536, 2308])
def test_the_sums_of_a_token_are_taken_in_the_same_order_by_every_kernel(k):
    """Products that cancel: what is left of a sum is the rounding of its steps in double, which
    another order would change."""
    from paged_attention_engine_b200.kernels import ops

    gen = torch.Generator(device="cuda").manual_seed(3)
    half = torch.randn(200, k // 2, device="cuda", generator=gen)
    w_half = torch.randn(96, k // 2, device="cuda", generator=gen)
    order = torch.randperm(k, device="cuda", generator=gen)
    x = torch.cat((half, -half), 1)[:, order].contiguous()
    w = torch.cat((w_half, w_half), 1)[:, order].contiguous()
    whole = ops.linear(x, w)
    assert float(whole.abs().max()) < 1e-10 and float((whole != 0).float().mean()) > 0.5
    for m in (1, 2, 3, 8, 9, 17, 33, 64):
        assert torch.equal(ops.linear(x[:m], w), whole[:m]), m


def test_misaligned_operands_are_taken():
    from paged_attention_engine_b200.kernels import ops

    x, w, _, _ = _operands(3, 40, 64)
    shifted = torch.empty(3 * 64 + 1, device="cuda")[1:].view(3, 64).copy_(x)
    want = x.double() @ w.double().T
    assert torch.allclose(ops.linear(shifted, w).double(), want, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("m,n,k", [(64, 3584, 18944), (300, 100, 65536), (33, 70, 393216)])
def test_outputs_cut_into_slices_that_share_the_scratch(m, n, k):
    """Sizes whose planes of double do not fit the scratch at once: slices of weight rows, and of tokens too."""
    from paged_attention_engine_b200.kernels import ops

    x, w, bias, residual = _operands(m, n, k, seed=2)
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got = ops.linear(x, w, bias, residual)
    assert torch.cuda.max_memory_allocated() - before <= (96 << 20) + 4 * m * n + 4096
    want = x.double() @ w.double().T + bias.double() + residual.double()
    terms = x.double().abs() @ w.double().abs().T + bias.abs().double() + residual.abs().double()
    assert bool(((got.double() - want).abs() <= want.abs() * 2**-24 + terms * (k + 2) * 2**-52).all())
    for few in (2, 32):
        assert torch.equal(ops.linear(x[:few], w, bias, residual[:few]), got[:few])
