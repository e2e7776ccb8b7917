"""Kernels launched after another one gave up: they leave as whole blocks and touch nothing."""
import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "cppmega_b200" / "ops" / "csrc"


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_no_thread_leaves_a_tensor_memory_kernel_on_the_error_word_by_itself(path):
    """The word can change while a block starts.  A kernel that sets up barriers and tensor memory must read it once for the
    block (``setup_barrier``, or a shared flag that every role tests), not return on a read of each thread's own."""
    kernels = re.split(r"(?=__global__ )", path.read_text())[1:]
    bad = [re.search(r"(\w+_kernel)\(", k).group(1) for k in kernels
           if "tmem_alloc" in k and re.search(r"if \([^\n]*err[^\n]*!= 0\) return;", k)]
    assert not bad, bad


def _ops():
    from cppmega_b200.ops import cuda as cu, functional as F_
    from cppmega_b200.ops.cuda import extra, kernels4, mxfp8
    bf = lambda *s, std=0.5: (torch.randn(*s, device="cuda") * std).bfloat16().requires_grad_()  # noqa: E731
    f32 = lambda *s: torch.rand(*s, device="cuda").requires_grad_()  # noqa: E731
    counts = torch.tensor([200, 40], device="cuda")
    idx = torch.randint(0, 64, (1, 64, 256), device="cuda").int()

    def mx(x, w):
        return mxfp8.linear(x, w)

    def scan(*t):
        return F_.mimo_scan(*t, 4, 16)

    scan_in = [bf(1, 64, 4, 1, 128), bf(1, 64, 4, 1, 128), bf(1, 64, 2, 64), (-0.1 * torch.rand(1, 2, 64, device="cuda")).requires_grad_(),
               f32(1, 2, 64), f32(1, 2, 64), f32(2, 4, 128), f32(2, 4, 128), f32(2, 4, 64), f32(2, 4, 64), f32(2, 4, 64), f32(1, 64, 2, 32),
               f32(2), bf(1, 64, 2, 64)]
    return {
        "linear_pair": (cu.linear, [bf(4096, 512), bf(4096, 512)]),
        "linear_one_cta": (cu.linear, [bf(64, 512), bf(128, 512)]),
        "mxfp8_linear_small": (mx, [bf(96, 128), bf(96, 128)]),
        "mxfp8_linear_large": (mx, [bf(4096, 4096), bf(4096, 4096)]),
        "experts": (lambda x, w1, w2: extra.moe_experts(x, w1, w2, counts), [bf(240, 128), bf(2, 128, 128), bf(2, 128, 64)]),
        "attention": (lambda q, k, v: F_.causal_attention(q, k, v, 0.1), [bf(1, 384, 2, 128), bf(1, 384, 2, 128), bf(1, 384, 2, 64)]),
        "sparse_attention": (lambda q, kv: F_.sparse_mla(q, kv, idx, 0.1, 64), [bf(1, 64, 32, 128), bf(1, 64, 128)]),
        "head_linear": (F_.head_linear, [bf(200, 4, 64), bf(4, 64, 64)]),
        "scan": (scan, scan_in),
        "indexer": (lambda q, k, w: kernels4.indexer_topk(q.detach(), k.detach(), w.detach(), 64), [bf(1, 256, 32, 64), bf(1, 256, 64), f32(1, 256, 32)]),
    }


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["linear_pair", "linear_one_cta", "mxfp8_linear_small", "mxfp8_linear_large", "experts", "attention",
                                  "sparse_attention", "head_linear", "scan", "indexer"])
def test_kernels_drain_while_the_error_word_is_set(name):
    from cppmega_b200.ops import cuda as cu
    torch.manual_seed(0)
    fn, ins = _ops()[name]

    def once():
        y = fn(*ins)
        if not y.requires_grad:
            return [y.sort(-1).values]
        return [y.detach(), *torch.autograd.grad(y, ins, torch.ones_like(y))]

    cu.check_errors()
    want = once()
    cu.check_errors()
    word = cu.err_word()
    word.fill_(3)
    once()
    torch.cuda.synchronize()
    assert word.item() == 3
    word.zero_()
    for a, b in zip(once(), want):
        assert (a.float() - b.float()).norm() <= 1e-2 * b.float().norm()
    cu.check_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("M", [64, 4096])
def test_a_drained_product_leaves_its_result_alone(M):
    from cppmega_b200.ops import cuda as cu
    a, b = torch.ones(M, 64, device="cuda").bfloat16(), torch.ones(4096, 64, device="cuda").bfloat16()
    out = torch.full((M, 4096), 7.0, device="cuda")
    cu.err_word().fill_(3)
    cu.gemm(a, b, out=out)
    torch.cuda.synchronize()
    cu.err_word().zero_()
    assert (out == 7.0).all()
