"""The products of some tens of tokens by clusters of blocks (csrc/gemm_cluster.cu) against the plain reference in 64 bits:
tokens on both sides of a multiple of 16, of the columns that tensor memory is asked for and of a block's share; rows that do not fill a
tile; K that is not a multiple of 64; every number of blocks a tile; and a layer's chain of products and norms."""

import pytest
import torch

pytestmark = pytest.mark.gpu

TOKENS = [1, 16, 17, 33, 64, 65, 100, 127, 128]
# bfloat16 rounds to 2^-9 relative: an output of two roundings (a gate's, of rounded gate and up, of three) in norm over norm.
REL = 3 * 2.0 ** -9


@pytest.fixture(scope="module")
def ops():
    from paged_attention_engine_b200.kernels import ops as kernel_ops

    yield kernel_ops
    kernel_ops.use_cluster_products = True


def _rand(shape, seed, std=1.0):
    gen = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=gen) * std).to(torch.bfloat16).cuda()


def _near(got, want, rel=REL):
    assert torch.isfinite(got).all()
    error = float((got.double() - want).norm() / want.norm())
    assert error <= rel, f"{error} > {rel}"


def _p(t):
    return 0 if t is None else t.data_ptr()


def _residual(ops, x, w, r, gamma, shape=(0, 0, 0), early=1, squares=None, eps=0.0):
    lib = ops._lib("gemm_cluster")
    (m, k), n = x.shape, w.shape[0]
    out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    scaled = torch.full_like(out, float("nan"))
    parts = -(-n // shape[0]) if shape[0] else lib.pae_linear_cluster_parts(m, n, k)
    sums = torch.full((parts, m), float("nan"), device="cuda")
    code = lib.pae_linear_cluster(_p(out), _p(x), _p(w), _p(r), _p(gamma), _p(scaled), _p(sums), _p(squares),
                                  0 if squares is None else squares.shape[0], k, eps, m, n, k, early, *shape, ops.error_flag("cuda:0").data_ptr(), 0)
    assert code == 0, lib.pae_last_error().decode()
    return out, scaled, sums


@pytest.mark.parametrize("tokens", TOKENS)
@pytest.mark.parametrize("n,k,shape", [(1536, 1536, (0, 0, 0)), (200, 264, (0, 0, 0)), (8, 8, (0, 0, 0)), (392, 648, (64, 3, 4)), (264, 1032, (128, 7, 2)),
                                       (128, 8960, (128, 8, 3)), (640, 512, (128, 1, 3)), (3584, 3584, (0, 0, 0))])
def test_product_with_residual_and_what_the_next_norm_needs(ops, tokens, n, k, shape):
    if shape[0] and tokens > 64 and shape[1] == 1:
        shape = (shape[0], 1, 4)
    x, w, r = _rand((tokens, k), 1), _rand((n, k), 2, k ** -0.5), _rand((tokens, n), 3)
    gamma = (1 + 0.2 * torch.randn(n, generator=torch.Generator().manual_seed(4))).cuda()
    out, scaled, sums = _residual(ops, x, w, r, gamma, shape, early=tokens % 2)
    _near(out, x.double() @ w.double().T + r.double())
    assert torch.equal(scaled, (out.float() * gamma).to(torch.bfloat16))
    torch.testing.assert_close(sums.double().sum(0), (out.double() ** 2).sum(1), rtol=1e-5, atol=0)
    squares = (x.double() ** 2).view(tokens, 1, -1).sum(2).T.float().contiguous()
    alone, _, _ = _residual(ops, x, w, None, None, shape, squares=squares, eps=1e-5)
    _near(alone, (x.double() @ w.double().T) * torch.rsqrt((x.double() ** 2).mean(1, keepdim=True) + 1e-5))
    ops.check_device_errors()


def _squares(x, parts):
    """The sums of the squares of x's rows over `parts` shares of their columns, as a product before leaves them: [parts, tokens]."""
    return torch.stack([(share.float() ** 2).sum(1) for share in x.chunk(parts, dim=1)]).contiguous()


@pytest.mark.parametrize("gate", ["silu", "relu", "gelu_tanh"])
@pytest.mark.parametrize("normed", [False, True])
@pytest.mark.parametrize("tokens,n,k", [(1, 4096, 2048), (8, 7168, 3584), (17, 32, 64), (33, 352, 192), (64, 17920, 128), (65, 37888, 64), (128, 2080, 1536), (100, 544, 8192)])
def test_gated_product(ops, tokens, n, k, gate, normed):
    lib = ops._lib("gemm_cluster")
    x, w = _rand((tokens, k), 5), _rand((n, k), 6, k ** -0.5)
    out = torch.full((tokens, n // 2), float("nan"), dtype=torch.bfloat16, device="cuda")
    squares = _squares(x, k // 64) if normed else None
    code = lib.pae_linear_swiglu_cluster(_p(out), _p(x), _p(w), _p(squares), 0 if squares is None else squares.shape[0], k, 1e-5, tokens, n, k, ops.GATE_KINDS[gate], 1,
                                         0, 0, 0, ops.error_flag("cuda:0").data_ptr(), 0)
    assert code == 0, lib.pae_last_error().decode()
    z = x.double() @ w.double().T
    if normed:
        z = z * torch.rsqrt((x.double() ** 2).mean(1, keepdim=True) + 1e-5)
    z = z.to(torch.bfloat16).double().view(tokens, -1, 2, 16)
    act = {"silu": torch.nn.functional.silu, "relu": torch.relu, "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[gate]
    _near(out, (act(z[:, :, 0]) * z[:, :, 1]).reshape(tokens, -1))
    ops.check_device_errors()


@pytest.mark.parametrize("tokens,heads,kv_heads,d,k", [(t, *sizes) for t in (17, 40, 64, 65, 100, 127, 128)
                                                       for sizes in ((12, 2, 128, 1536), (14, 2, 64, 896), (3, 1, 32, 192), (5, 5, 16, 64))]
                         + [(1, 16, 4, 128, 2048), (3, 28, 4, 128, 3584), (8, 16, 4, 128, 2048)])
@pytest.mark.parametrize("normed", [False, True])
def test_qkv_with_rotation_and_page_write(ops, tokens, heads, kv_heads, d, k, normed):
    lib = ops._lib("gemm_cluster")
    n, page, pages = (heads + 2 * kv_heads) * d, 16, 10
    x, w = _rand((tokens, k), 7), _rand((n, k), 8, k ** -0.5)
    gen = torch.Generator().manual_seed(9)
    bias, table = torch.randn(n, generator=gen).cuda(), torch.randn((tokens, d), generator=gen).cuda()
    slots = torch.randperm(pages * page, generator=gen)[:tokens].to(torch.int32)
    slots[tokens // 2] = -1
    slots = slots.cuda()
    keys = torch.zeros((pages, kv_heads, page, d), dtype=torch.bfloat16, device="cuda")
    values = torch.zeros_like(keys)
    got = torch.full((tokens, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    squares = _squares(x, k // 64) if normed else None
    ops._set_bounds("gemm_cluster", keys)
    code = lib.pae_qkv_cluster(_p(got), _p(x), _p(w), _p(bias), _p(squares), 0 if squares is None else squares.shape[0], k, 1e-5, _p(table), _p(slots), _p(keys),
                               _p(values), tokens, heads, kv_heads, d, page, k, 1, 0, 0, 0, ops.error_flag("cuda:0").data_ptr(), 0)
    assert code == 0, lib.pae_last_error().decode()
    got = got.view(tokens, -1, d)
    y = x.double() @ w.double().T
    if normed:
        y = y * torch.rsqrt((x.double() ** 2).mean(1, keepdim=True) + 1e-5)
    y = (y + bias.double()).to(torch.bfloat16).double().view(tokens, -1, d)
    c, s = table.double()[:, None, : d // 2], table.double()[:, None, d // 2 :]
    lo, hi = y[..., : d // 2], y[..., d // 2 :]
    rotated = torch.cat((lo * c - hi * s, hi * c + lo * s), -1)
    _near(got, torch.cat((rotated[:, : heads + kv_heads], y[:, heads + kv_heads :]), 1))
    for pool, first in ((keys, heads), (values, heads + kv_heads)):
        want = torch.zeros_like(pool)
        for t, slot in enumerate(slots.tolist()):
            if slot >= 0:
                want[slot // page, :, slot % page] = got[t, first : first + kv_heads]
        assert torch.equal(pool, want)
    ops.check_device_errors()


@pytest.mark.parametrize("tokens", [17, 64, 128])
def test_a_chain_of_products_and_norms(ops, tokens):
    """o, norm, gate|up, down, norm, q|k|v: the norms take no launch, and the values are those of the separate kernels."""
    h, inter, heads, kv_heads, d, page = 384, 512, 3, 1, 128, 16
    a, r = _rand((tokens, h), 10), _rand((tokens, h), 11)
    wo, wgu, wd = _rand((h, h), 12, h ** -0.5), _rand((2 * inter, h), 13, h ** -0.5), _rand((h, inter), 14, inter ** -0.5)
    wqkv = _rand(((heads + 2 * kv_heads) * d, h), 15, h ** -0.5)
    g1, g2 = ((1 + 0.1 * torch.randn(h, generator=torch.Generator().manual_seed(s))).cuda() for s in (16, 17))

    def run():
        before = ops.launches
        y = ops.linear_before_norm(a, wo, None, r)
        normed = ops.rms_norm(y, g1, 1e-6)
        z = ops.linear_before_norm(ops.linear_swiglu(normed, wgu), wd, None, ops.materialized(y))
        normed = ops.rms_norm(z, g2, 1e-6)
        q = ops.qkv_projection(normed, wqkv, None, None, None, None, None, heads, kv_heads, d, page)
        stream = ops.materialized(z)
        count = ops.launches - before
        return q, stream, ops.materialized(normed), count

    q, stream, normed, count = run()
    assert count == 4
    ops.use_cluster_products = False
    try:
        want = run()
    finally:
        ops.use_cluster_products = True
    for got, other in zip((q, stream, normed), want):
        _near(got, other.double(), 4 * REL)
    ops.check_device_errors()


def test_all_clusters_of_a_launch_run_at_once(ops):
    """One cluster more than the chip takes at a time makes the launch last twice as long."""
    lib = ops._lib("gemm_cluster")
    for tokens in TOKENS + [40, 80, 96, 97, 112]:
        for n in [8, 512, 768, 1024, 1536, 2048, 2304, 2560, 3072, 3584, 4096, 4608, 5120, 6144, 8192, 11008, 16384, 18944, 22016, 37888]:
            for k in [64, 192, 512, 768, 1024, 1536, 2048, 3584, 8960, 18944]:
                for gate in (0, 1):
                    assert lib.pae_linear_cluster_rounds(tokens, n, k, gate) <= 1, (tokens, n, k, gate)


@pytest.mark.parametrize("cluster,stages,skip", [(4, 4, (0, 1)), (4, 4, (2, 3)), (2, 8, (1, 5)), (8, 2, (7, 0))])
def test_a_wait_that_runs_out_in_one_block_of_a_cluster(ops, cluster, stages, skip):
    """One block of every cluster never loads one of its k-blocks: its wait gives up after a few thousand polls, the cluster's other blocks
    do their work, all of them end, and the error word says who gave up. The next product is right."""
    tokens, n, k = 40, 384, 1024
    x, w = _rand((tokens, k), 20), _rand((n, k), 21, k ** -0.5)
    out = torch.zeros((tokens, n), dtype=torch.bfloat16, device="cuda")
    ops.check_device_errors()
    lib = ops._lib("gemm_cluster")
    code = lib.pae_linear_cluster_selftest_giveup(_p(out), _p(x), _p(w), tokens, n, k, cluster, stages, *skip, ops.error_flag("cuda:0").data_ptr(), 0)
    assert code == 0, lib.pae_last_error().decode()
    torch.cuda.synchronize()                     # the kernel came back by itself
    assert int(ops.error_flag("cuda:0").item()) == 2, "the MMA issuer's wait is the one that runs out"
    with pytest.raises(ops.KernelError, match="role code 2"):
        ops.check_device_errors()
    got, _, _ = _residual(ops, x, w, None, None, (128, cluster, stages))
    _near(got, x.double() @ w.double().T)
    ops.check_device_errors()


def test_what_the_library_refuses(ops):
    lib = ops._lib("gemm_cluster")
    x, w, out = _rand((4, 64), 1), _rand((64, 64), 2), _rand((4, 64), 3)
    flag = ops.error_flag("cuda:0").data_ptr()

    def call(tokens=4, n=64, k=64, shift=0, shape=(0, 0, 0)):
        return lib.pae_linear_cluster(_p(out), _p(x) + shift, _p(w), 0, 0, 0, 0, 0, 0, 0, 0.0, tokens, n, k, 1, *shape, flag, 0)

    assert call() == 0
    for bad in (dict(tokens=0), dict(tokens=129), dict(n=60), dict(k=60), dict(shift=2), dict(shape=(128, 9, 2)), dict(shape=(96, 1, 2)),
                dict(shape=(128, 2, 2)), dict(shape=(128, 1, 1)), dict(shape=(128, 1, 13))):
        assert call(**bad) != 0, bad
    assert not lib.pae_qkv_cluster_supports(256) and not lib.pae_qkv_cluster_supports(48) and lib.pae_qkv_cluster_supports(64)
    torch.cuda.synchronize()
