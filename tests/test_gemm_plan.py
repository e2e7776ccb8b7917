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


@pytest.mark.parametrize("used,E,N,K,b_mn,want", [
    (32768, 16, 4096, 896, 0, 1),               # many rows, a short reduction: pairs
    (32768, 16, 4096, 1792, 1, 1),
    (16384, 16, 4096, 896, 0, 1),
    (16384, 16, 4096, 1792, 1, 0),              # shared boundary tiles cost more than the pair saves
    (8192, 16, 4096, 896, 0, 0),
    (32768, 16, 1792, 4096, 0, 0),              # a long reduction
    (16384, 16, 1024, 1024, 0, 0),              # few waves
    (32768, 16, 1024, 1024, 0, 1),
    (64, 16, 4096, 896, 0, 0),
])
def test_expert_products_go_to_pairs_by_the_rows_in_use(lib, used, E, N, K, b_mn, want):
    assert lib.cm_grouped_rows_plan(148, used, E, N, K, b_mn) == want


@pytest.mark.parametrize("used,E,M,accumulate,want", [(64, 16, 1792, 0, 1), (64, 16, 1792, 1, 0), (20479, 16, 1792, 1, 0),
                                                      (20480, 16, 1792, 1, 1), (65536, 16, 128, 0, 0)])
def test_expert_weight_gradients_go_to_pairs(lib, used, E, M, accumulate, want):
    assert lib.cm_grouped_k_plan(used, E, M, accumulate) == want


@pytest.mark.parametrize("M,N,K,fp32,accumulate,want", [
    (8192, 4096, 8192, 0, 0, 1), (4096, 8192, 8192, 0, 0, 1),       # the products of a large projection
    (2048, 2048, 2048, 0, 0, 0), (160, 4096, 8192, 0, 0, 0),        # a single wave
    (2048, 2048, 16384, 0, 0, 1),
    (4096, 4096, 1024, 0, 0, 0), (4096, 4096, 2048, 0, 0, 1),       # by the reduction and the bytes of the result
    (4096, 4096, 2048, 1, 0, 0), (4096, 4096, 3072, 1, 0, 1), (4096, 4096, 3072, 1, 1, 0), (4096, 4096, 4096, 1, 1, 1),
    (1056, 8192, 16384, 0, 0, 0),                                   # three waves of pairs against two
    (128, 8192, 16384, 0, 0, 0),                                    # no second row tile
])
def test_mxfp8_plan(lib, M, N, K, fp32, accumulate, want):
    assert lib.cm_mxfp8_gemm_plan(148, M, N, K, fp32, accumulate) == want


def test_routed_experts_pass_the_rows_in_use_not_the_allocated_ones(monkeypatch):
    """The buffers of an expert-parallel rank hold several times the rows that arrive on average."""
    import types

    import torch
    from cppmega_b200.ops import cuda as cu
    from cppmega_b200.parallel import fused_moe as fm
    calls = []
    entry = lambda *a: calls.append(a) or 0  # noqa: E731
    monkeypatch.setattr(cu, "lib", lambda: types.SimpleNamespace(cm_grouped_gemm_rows_bf16=entry, cm_grouped_gemm_k_bf16=entry))
    monkeypatch.setattr(cu, "err_word", lambda device=None: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(cu, "stream_ptr", lambda: 0)
    plan = types.SimpleNamespace(T=40, k=4, tile_expert=torch.zeros(8, dtype=torch.int32), seg_offsets=torch.zeros(3, dtype=torch.int32))
    x, w = torch.zeros(1024, 16, dtype=torch.bfloat16), torch.zeros(2, 24, 16, dtype=torch.bfloat16)
    y = fm._grouped(x, w, plan, 1024, False)
    fm._grouped_wgrad(y, x, plan, 2)
    assert calls[0][9] == 160 and calls[1][8] == 160
