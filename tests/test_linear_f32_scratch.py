"""The scratch of a float32 product whose K is shared out over blocks: bounded whatever the sizes. Host arithmetic; no GPU."""

import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    from paged_attention_engine_b200.kernels import build

    lib = ctypes.CDLL(str(build.ensure_built(["gemm_simt"])["gemm_simt"]))
    lib.pae_linear_f32_scratch.restype = ctypes.c_longlong
    return lib


@pytest.mark.parametrize("k", [128, 132, 1536, 8960, 18944, 393216, 393220, 1 << 22])
def test_the_scratch_is_bounded(lib, k):
    shared = 0
    for m in (1, 32, 33, 64, 65, 200, 1000, 4700, 100_000):
        for n in (1, 64, 100, 1536, 3584, 4736, 151_936):
            doubles = lib.pae_linear_f32_scratch(m, n, k)
            assert 0 <= doubles * 8 <= 96 << 20
            launches = lib.pae_linear_f32_launches(m, n, k)
            assert launches >= 2 if doubles else launches == 1
            shared += doubles > 0
    assert (shared > 0) == (128 < k <= 393216)


def test_a_product_that_fits_is_one_slice(lib):
    assert lib.pae_linear_f32_launches(60, 1536, 8960) == 2
    assert lib.pae_linear_f32_scratch(60, 1536, 8960) == 70 * 60 * 1536
    assert lib.pae_linear_f32_launches(64, 3584, 18944) > 2
