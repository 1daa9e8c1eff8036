"""Products whose tiles are computed by pairs of SMs: token counts on both sides of a pair's 256 rows and of its
first block's 128, widths off the tiles, every epilogue."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf(gen, *shape, std=1.0):
    return (torch.randn(*shape, device="cuda", generator=gen) * std).to(torch.bfloat16)


def _by_pairs(m, n, k, head_dim=0, swiglu=0):
    from paged_attention_engine_b200.kernels import ops

    return ops._lib("gemm_tcgen05").pae_linear_pair_width(m, n, k, head_dim, swiglu) > 0


def _close(got, want, k, rounded=1):
    """bfloat16 products of k terms summed in float32, rounded `rounded` times on the way: half a unit of the last place each,
    and a float32 sum's error far below it."""
    gap = (got.double() - want).abs()
    limit = want.abs() * 2.0**-8 * rounded + want.abs().amax() * 2.0**-8 * (rounded - 1) + want.abs().amax() * k * 2.0**-23
    assert bool((gap <= limit).all()), float((gap - limit).max())


@pytest.mark.parametrize("m,n,k", [(8192 + 129, 17920, 136), (2049, 17904, 1032), (4096 + 127, 5008, 1032), (8192 - 127, 3592, 2056)])
def test_plain_product(m, n, k):
    from paged_attention_engine_b200.kernels import ops

    assert _by_pairs(m, n, k)
    gen = torch.Generator(device="cuda").manual_seed(0)
    x, w, residual = _bf(gen, m, k), _bf(gen, n, k, std=0.05), _bf(gen, m, n)
    bias = torch.randn(n, device="cuda", generator=gen)
    want = x.double() @ w.double().T + bias.double() + residual.double()
    _close(ops.linear(x, w, bias, residual), want, k)
    _close(ops.linear(x, w, bias, residual.float(), out_dtype=torch.float32), want, k)
    ops.check_device_errors()


@pytest.mark.parametrize("m", [513, 2048, 8191])
def test_gated_product(m):
    from paged_attention_engine_b200.kernels import ops

    gen = torch.Generator(device="cuda").manual_seed(1)
    inter, k = 8960, 1536
    assert _by_pairs(m, 2 * inter, k, swiglu=1)
    x, gate, up = _bf(gen, m, k), _bf(gen, inter, k, std=0.02), _bf(gen, inter, k, std=0.02)
    got = ops.linear_swiglu(x, ops.interleave_gate_up(gate, up))
    g, u = x.double() @ gate.double().T, x.double() @ up.double().T
    _close(got, g * torch.sigmoid(g) * u, k, rounded=3)
    ops.check_device_errors()


@pytest.mark.parametrize("m", [4096, 8192 - 65])
@pytest.mark.parametrize("heads,kv_heads,d", [(12, 2, 128), (28, 4, 64)])
def test_heads_product_with_rotation_and_page_write(m, heads, kv_heads, d):
    """The same numbers as the product followed by the stand-alone rotation and page write."""
    from paged_attention_engine_b200.kernels import ops

    gen = torch.Generator(device="cuda").manual_seed(2)
    k, n, page = 3584, (heads + 2 * kv_heads) * d, 16
    assert _by_pairs(m, n, k, head_dim=d)
    x, w = _bf(gen, m, k), _bf(gen, n, k, std=0.02)
    bias, table = torch.randn(n, device="cuda", generator=gen), torch.randn(m, d, device="cuda", generator=gen)
    slots = torch.randperm(m, device="cuda", generator=gen).to(torch.int32)
    slots[::7] = -1
    shape = (m // page + 1, kv_heads, page, d)
    results = []
    for fused in (True, False):
        keys, values = torch.zeros(shape, dtype=torch.bfloat16, device="cuda"), torch.zeros(shape, dtype=torch.bfloat16, device="cuda")
        if fused:
            out = ops.qkv_projection(x, w, bias, table, slots, keys, values, heads, kv_heads, d, page)
        else:
            out = ops.rotary_qk_cache_write(ops.linear(x, w, bias), table, slots, keys, values, heads, kv_heads, d, page)
        results.append((out, keys, values))
    for a, b in zip(*results):
        assert torch.equal(a, b)
    ops.check_device_errors()


@pytest.mark.parametrize("m,n,k,pairs", [(8192, 3584, 1536, True), (300, 2048, 1024, False)])
def test_a_weight_that_the_call_before_wrote(m, n, k, pairs):
    """The product waits for the kernel before, which starts it early; nothing of the weight is read until then."""
    from paged_attention_engine_b200.kernels import ops

    assert _by_pairs(m, n, k) == pairs
    gen = torch.Generator(device="cuda").manual_seed(4)
    x, a, b = _bf(gen, m, k), _bf(gen, n, 512), _bf(gen, k, 512, std=0.002)
    weight = ops.linear(a, b)
    torch.cuda.synchronize()
    want = ops.linear(x, weight)
    for _ in range(20):
        assert torch.equal(ops.linear(x, ops.linear(a, b)), want)
    ops.check_device_errors()
