"""Host side of the GEMM dispatch: which kernel a problem goes to."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    from cppmega_b200.ops.cuda import build
    if not build.LIB.exists():
        pytest.skip("the kernel library has not been built")
    return ctypes.CDLL(str(build.LIB))


@pytest.mark.parametrize("M,N,K,b_mn,accumulate,want", [
    (8192, 8192, 8192, 0, 0, 1256),             # many waves: pairs
    (300, 24960, 4096, 0, 0, 256),              # two waves of 128 x 256 against three of pairs
    (300, 24960, 4096, 1, 0, 256),
    (64, 512, 4096, 0, 0, 64),                  # one wave of anything: the cheapest
    (4096, 4096, 512, 1, 1, 256),               # a short accumulating reduction: one CTA
    (4096, 4096, 1024, 1, 1, 256),
    (4096, 4096, 2048, 1, 1, 1256),
    (4096, 4096, 512, 1, 0, 1256),
])
def test_dense_plan(lib, M, N, K, b_mn, accumulate, want):
    assert lib.cm_gemm_bf16_plan(148, M, N, K, b_mn, accumulate) == want
