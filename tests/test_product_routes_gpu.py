"""What a product of few or of some tens of tokens hands back: `linear` a finished sum wherever the kernels of few tokens or of clusters run
it, whatever becomes of its operands later."""

import pytest
import torch

pytestmark = pytest.mark.gpu

REL = 3 * 2.0 ** -9        # bfloat16 rounds to 2^-9 relative: two roundings and a sum in another order


@pytest.fixture(scope="module")
def ops():
    from paged_attention_engine_b200.kernels import ops as kernel_ops

    return kernel_ops


def _rand(shape, seed, std=1.0):
    gen = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=gen) * std).to(torch.bfloat16).cuda()


def _near(got, want, rel=REL):
    error = float((got.double() - want).norm() / want.norm())
    assert error <= rel, f"{error} > {rel}"


@pytest.mark.parametrize("tokens,n,k", [(1, 2048, 2048), (8, 3584, 3584), (9, 1024, 1024), (16, 1536, 1536), (24, 896, 896), (40, 1536, 8960),
                                        (64, 2048, 2048), (65, 2048, 11008), (128, 768, 2048)])
def test_a_product_with_a_residual_is_finished_when_it_comes_back(ops, tokens, n, k):
    x, w, r = _rand((tokens, k), 1), _rand((n, k), 2, k ** -0.5), _rand((tokens, n), 3)
    want = x.double() @ w.double().T + r.double()
    got = ops.linear(x, w, residual=r)
    assert type(got) is torch.Tensor and got.shape == (tokens, n)
    torch.cuda.synchronize()
    x.zero_(), r.zero_()
    _near(got + 0, want)
    ops.check_device_errors()
