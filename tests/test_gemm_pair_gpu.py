"""Products whose tiles are computed by pairs of SMs: every tile width of every epilogue (each is a kernel of its own), token counts on
both sides of a pair's 256 rows and of its first block's 128, sizes off the tiles."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf(gen, *shape, std=1.0):
    return (torch.randn(*shape, device="cuda", generator=gen) * std).to(torch.bfloat16)


def _pair_width(m, n, k, head_dim=0, swiglu=0):
    """The width of the tiles that pairs compute; 0: single blocks do."""
    from paged_attention_engine_b200.kernels import ops

    return ops._lib("gemm_tcgen05").pae_linear_pair_width(m, n, k, head_dim, swiglu)


def _close(got, want, k, rounded=1):
    """bfloat16 products of k terms summed in float32, rounded `rounded` times on the way: half a unit of the last place each,
    and a float32 sum's error far below it."""
    gap = (got.double() - want).abs()
    limit = want.abs() * 2.0**-8 * rounded + want.abs().amax() * 2.0**-8 * (rounded - 1) + want.abs().amax() * k * 2.0**-23
    assert bool((gap <= limit).all()), float((gap - limit).max())


@pytest.mark.parametrize("m,n,k,width", [
    (8192 + 129, 17920, 136, 256), (2049, 17904, 1032, 256), (4096 + 127, 5008, 1032, 256), (8192 - 127, 3592, 2056, 256),
    (1281, 5008, 520, 224), (2500, 4104, 1032, 192), (2049, 1032, 520, 160), (385, 3592, 2056, 128),
])
def test_plain_product(m, n, k, width):
    from paged_attention_engine_b200.kernels import ops

    assert _pair_width(m, n, k) == width
    gen = torch.Generator(device="cuda").manual_seed(0)
    x, w, residual = _bf(gen, m, k), _bf(gen, n, k, std=0.05), _bf(gen, m, n)
    bias = torch.randn(n, device="cuda", generator=gen)
    want = x.double() @ w.double().T + bias.double() + residual.double()
    _close(ops.linear(x, w, bias, residual), want, k)
    _close(ops.linear(x, w, bias, residual.float(), out_dtype=torch.float32), want, k)
    ops.check_device_errors()


@pytest.mark.parametrize("m,inter,k,width", [
    (513, 8960, 1536, 256), (2048, 8960, 1536, 256), (8191, 8960, 1536, 256),
    (1281, 2512, 520, 224), (1025, 4112, 520, 192), (2049, 528, 520, 160), (4095, 528, 2056, 128),
])
def test_gated_product(m, inter, k, width):
    from paged_attention_engine_b200.kernels import ops

    gen = torch.Generator(device="cuda").manual_seed(1)
    assert _pair_width(m, 2 * inter, k, swiglu=1) == width
    x, gate, up = _bf(gen, m, k), _bf(gen, inter, k, std=0.02), _bf(gen, inter, k, std=0.02)
    got = ops.linear_swiglu(x, ops.interleave_gate_up(gate, up))
    g, u = x.double() @ gate.double().T, x.double() @ up.double().T
    _close(got, g * torch.sigmoid(g) * u, k, rounded=3)
    ops.check_device_errors()


@pytest.mark.parametrize("m,heads,kv_heads,d,k,width", [
    (4096, 12, 2, 128, 3584, 256), (8192 - 65, 12, 2, 128, 3584, 256), (4096, 28, 4, 64, 3584, 256), (8192 - 65, 28, 4, 64, 3584, 256),
    (641, 47, 1, 64, 520, 192), (1700, 39, 1, 64, 2056, 128),
    (4223, 51, 3, 32, 1544, 256), (4223, 40, 5, 32, 520, 224), (4223, 60, 4, 32, 520, 192), (2049, 27, 3, 32, 520, 160), (5000, 15, 5, 32, 2056, 128),
])
def test_heads_product_with_rotation_and_page_write(m, heads, kv_heads, d, k, width):
    """The same numbers as the product followed by the stand-alone rotation and page write."""
    from paged_attention_engine_b200.kernels import ops

    gen = torch.Generator(device="cuda").manual_seed(2)
    n, page = (heads + 2 * kv_heads) * d, 16
    assert _pair_width(m, n, k, head_dim=d) == width
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

    assert (_pair_width(m, n, k) > 0) == pairs
    gen = torch.Generator(device="cuda").manual_seed(4)
    x, a, b = _bf(gen, m, k), _bf(gen, n, 512), _bf(gen, k, 512, std=0.002)
    weight = ops.linear(a, b)
    torch.cuda.synchronize()
    want = ops.linear(x, weight)
    for _ in range(20):
        assert torch.equal(ops.linear(x, ops.linear(a, b)), want)
    ops.check_device_errors()
