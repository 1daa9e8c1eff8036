"""Which kernel a product of few or of some tens of tokens goes to, and what the call hands back: `linear` a finished sum wherever the kernels
of few tokens or of clusters run it, whatever becomes of its operands later; a cluster's kernel only where it is the faster one."""

import pytest
import torch

pytestmark = pytest.mark.gpu

REL = 3 * 2.0 ** -9        # bfloat16 rounds to 2^-9 relative: two roundings and a sum in another order


@pytest.fixture(scope="module")
def ops():
    from paged_attention_engine_b200.kernels import ops as kernel_ops

    return kernel_ops


@pytest.fixture()
def ran(ops, monkeypatch):
    """The product kernels that ran, in their order."""
    calls = []
    for library, entries in (("gemm_cluster", ("pae_linear_cluster", "pae_linear_swiglu_cluster", "pae_qkv_cluster")),
                             ("gemv_mma", ("pae_linear_few_tokens", "pae_linear_swiglu_few_tokens", "pae_qkv_few_tokens")),
                             ("gemm_tcgen05", ("pae_linear_tcgen05", "pae_linear_tcgen05_swapped", "pae_linear_swiglu_tcgen05", "pae_linear_rotary_tcgen05"))):
        lib = ops._lib(library)
        for name in entries:
            real = getattr(lib, name)
            monkeypatch.setattr(lib, name, lambda *args, real=real, name=name: (calls.append(name), real(*args))[1])
    return calls


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


@pytest.mark.parametrize("tokens,n,k,kernel", [
    (8, 2048, 2048, "pae_linear_few_tokens"), (8, 3584, 3584, "pae_linear_few_tokens"), (16, 1024, 1024, "pae_linear_few_tokens"),
    (24, 1536, 1536, "pae_linear_few_tokens"), (25, 1536, 1536, "pae_linear_cluster"), (128, 2048, 2048, "pae_linear_cluster")])
def test_a_product_alone(ops, ran, tokens, n, k, kernel):
    x, w, r = _rand((tokens, k), 4), _rand((n, k), 5, k ** -0.5), _rand((tokens, n), 6)
    want = x.double() @ w.double().T + r.double()
    _near(ops.linear(x, w, residual=r), want)
    _near(ops.materialized(ops.linear_before_norm(x, w, residual=r)), want)
    assert ran == [kernel, kernel]
    ops.check_device_errors()


@pytest.mark.parametrize("tokens,width,inter,kernels", [
    # few tokens: as few-token kernels while the layer's gate|up runs at once as one
    (8, 1536, 8960, "few few few few"), (8, 2048, 5504, "few few few few"), (8, 2304, 2304, "cluster cluster cluster cluster"),
    (1, 3584, 9472, "cluster cluster cluster cluster"), (8, 2048, 11008, "few cluster cluster cluster"),
    # some tens, up to the last; gate|up of some more tiles than SMs, or than two an SM, is the many-token kernel's
    (9, 1536, 2048, "cluster cluster cluster cluster"), (16, 896, 1024, "few few few few"), (17, 896, 1024, "cluster cluster cluster cluster"),
    (64, 2048, 11008, "cluster cluster cluster cluster"), (65, 2048, 11008, "cluster other cluster cluster"), (128, 1536, 2048, "cluster cluster cluster cluster"),
    (64, 2048, 20480, "cluster cluster cluster cluster"), (65, 2048, 20480, "cluster other cluster cluster"), (65, 2048, 28672, "cluster cluster cluster cluster"),
])
def test_a_layers_products(ops, ran, tokens, width, inter, kernels):
    """o, norm, gate|up, down, norm, q|k|v: which kernels run them, and that they compute the layer."""
    heads, kv_heads, d = width // 128, 2, 128
    n = (heads + 2 * kv_heads) * d
    a, r = _rand((tokens, width), 7), _rand((tokens, width), 8)
    wo, wgu = _rand((width, width), 9, width ** -0.5), _rand((2 * inter, width), 10, width ** -0.5)
    wd, wqkv = _rand((width, inter), 11, inter ** -0.5), _rand((n, width), 12, width ** -0.5)
    gamma = (1 + 0.1 * torch.randn(width, generator=torch.Generator().manual_seed(13))).cuda()
    y = ops.linear_before_norm(a, wo, None, r)
    hidden = ops.linear_swiglu(ops.rms_norm(y, gamma, 1e-6), wgu)
    z = ops.linear_before_norm(hidden, wd, None, ops.materialized(y))
    q = ops.qkv_projection(ops.rms_norm(z, gamma, 1e-6), wqkv, None, None, None, None, None, heads, kv_heads, d, 16)
    short = ["few" if c.endswith("few_tokens") else "cluster" if c.endswith("cluster") else "other" for c in ran]
    if ops._lib("gemm_tcgen05").pae_sm_count() == 148:
        assert " ".join(short) == kernels

    def norm(v):
        return v * torch.rsqrt((v * v).mean(1, keepdim=True) + 1e-6) * gamma.double()

    stream = (a.double() @ wo.double().T + r.double()).to(torch.bfloat16).double()
    gate_up = (norm(stream) @ wgu.double().T).view(tokens, -1, 2, 16)
    gate = gate_up[:, :, 0]
    stream = stream + (gate * torch.sigmoid(gate) * gate_up[:, :, 1]).reshape(tokens, -1) @ wd.double().T
    _near(ops.materialized(z), stream, 4 * REL)
    _near(q, norm(stream) @ wqkv.double().T, 4 * REL)
    ops.check_device_errors()
