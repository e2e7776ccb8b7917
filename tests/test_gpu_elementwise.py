"""Bandwidth-bound kernels and the fused cross-entropy against fp32 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


@pytest.mark.parametrize("rows,H", [(37, 64), (1000, 128), (513, 256), (300, 1024), (257, 4096), (64, 8192)])
def test_rmsnorm(rows, H):
    from cppmega_b200.ops import cuda as cu, reference as ref
    torch.manual_seed(rows)
    x = torch.randn(rows, H, device="cuda").bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16().requires_grad_()
    y = cu.rmsnorm(x, w, 1e-5)
    g = torch.randn_like(y)
    y.backward(g)
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yr = ref.rmsnorm(xr, wr, 1e-5)
    yr.backward(g.float())
    assert _rel(y, yr) < 6e-3
    assert _rel(x.grad, xr.grad) < 8e-3
    assert _rel(w.grad, wr.grad) < 8e-3


@pytest.mark.parametrize("H", [264, 816, 1024, 1032, 3584, 4096, 4104, 16384])
@pytest.mark.parametrize("rows", [1, 297, 887, 889, 1187, 3553, 5003])
def test_rmsnorm_backward_row_groups(rows, H):
    """Row counts on both sides of the thresholds at which a CTA takes two rows at a time (888 and 3552 on 148 SMs), with
    remainders and with fewer and more groups than ring slots, at widths that fill the thread block and that do not.  One bf16 rounding of each result: 2^-9 relative at
    most, 1.7e-3 in the mean; dw is summed in fp32 first."""
    from cppmega_b200.ops import cuda as cu, reference as ref
    torch.manual_seed(rows + H)
    x = torch.randn(rows, H, device="cuda").bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16().requires_grad_()
    y = cu.rmsnorm(x, w, 1e-5)
    g = torch.randn_like(y)
    y.backward(g)
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    ref.rmsnorm(xr, wr, 1e-5).backward(g.float())
    assert _rel(x.grad, xr.grad) < 4e-3
    assert _rel(w.grad, wr.grad) < 4e-3


@pytest.mark.parametrize("n", [8, 8 * 1023, 8 * 512 * 148 * 8 + 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_scale_to_bf16(n, dtype):
    """The same bits as the product and cast of the tensor library."""
    from cppmega_b200.ops import cuda as cu
    torch.manual_seed(n)
    x = torch.randn(n, device="cuda").to(dtype)
    g = torch.tensor([0.37], device="cuda")
    out = torch.empty(n, dtype=torch.bfloat16, device="cuda")
    assert cu.lib().cm_scale_to_bf16(x.data_ptr(), int(dtype == torch.float32), out.data_ptr(), g.data_ptr(), n, cu.stream_ptr()) == 0
    assert torch.equal(out, (x * g.to(dtype)).to(torch.bfloat16))


def test_swiglu():
    from cppmega_b200.ops import cuda as cu, reference as ref
    torch.manual_seed(0)
    x = torch.randn(777, 2 * 896, device="cuda").bfloat16().requires_grad_()
    y = cu.swiglu(x)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    yr = ref.swiglu(xr)
    yr.backward(g.float())
    assert _rel(y, yr) < 6e-3
    assert _rel(x.grad, xr.grad) < 8e-3


@pytest.mark.parametrize("gdt", [torch.float32, torch.bfloat16])
def test_adamw(gdt):
    from cppmega_b200.ops import cuda as cu
    from cppmega_b200.optim.adamw import adamw_reference
    torch.manual_seed(0)
    n = 100_003
    master = torch.randn(n, device="cuda")
    m = torch.randn(n, device="cuda") * 0.1
    v = torch.rand(n, device="cuda") * 0.01
    g = torch.randn(n, device="cuda").to(gdt)
    wd = torch.rand(n, device="cuda") > 0.5
    clip = torch.tensor(0.7, device="cuda")
    ref_state = [t.clone() for t in (master, m, v)]
    out_ref = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    adamw_reference(*ref_state, g, out_ref, wd, clip, 1e-3, 0.9, 0.95, 1e-8, 0.1, 0.1, 0.05)
    out = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    cu.adamw_shard(master, m, v, g, out, wd, clip, 1e-3, 0.9, 0.95, 1e-8, 0.1, 0.1, 0.05)
    for a, b in zip((master, m, v), ref_state):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-6)
    assert torch.allclose(out.float(), out_ref.float(), rtol=1e-2, atol=1e-3)


@pytest.mark.parametrize("T,H,V", [(300, 256, 4096), (5000, 128, 1024)])
def test_linear_ce_weighted(T, H, V):
    from cppmega_b200.ops import cuda as cu, reference as ref
    from cppmega_b200.ops.cuda import extra
    torch.manual_seed(0)
    h = torch.randn(T, H, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(V, H, device="cuda") * 0.1).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[::7] = -100
    rw = torch.rand(T, device="cuda") / T
    total, per = extra.linear_cross_entropy_weighted(h, w, labels, rw, -100)
    (total * 0.5).backward()
    cu.check_errors()
    hr, wr = h.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    pr = ref.linear_cross_entropy(hr, wr, labels, -100, "none")
    tr = (pr * rw).sum()
    (tr * 0.5).backward()
    assert torch.allclose(per, pr, rtol=2e-2, atol=2e-2)
    assert abs(total.item() - tr.item()) < 2e-2 * abs(tr.item()) + 1e-3
    assert _rel(h.grad, hr.grad) < 3e-2
    assert _rel(w.grad, wr.grad) < 3e-2


@pytest.mark.parametrize("T,H,V", [(33, 64, 8), (130, 64, 16392), (70, 64, 65544), (4097, 64, 512)])
def test_linear_ce_chunk_and_vocabulary_edges(T, H, V):
    """A vocabulary of one vector, ones that end inside a group of vectors of either kernel, and a last chunk of one row (the
    first chunk writes dw, the second adds to it)."""
    test_linear_ce_weighted(T, H, V)


def test_linear_ce_batched_upstream_gradients():
    """``is_grads_batched`` gives, slice by slice, the bits of one backward per upstream gradient."""
    from cppmega_b200.ops.cuda import extra
    torch.manual_seed(0)
    h = torch.randn(70, 64, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(512, 64, device="cuda") * 0.1).bfloat16().requires_grad_()
    total, _ = extra.linear_cross_entropy_weighted(h, w, torch.randint(0, 512, (70,), device="cuda"), torch.rand(70, device="cuda"), -100)
    gs = torch.tensor([1.0, 0.37], device="cuda")
    batched = torch.autograd.grad(total, [h, w], gs, is_grads_batched=True, retain_graph=True)
    for i, g in enumerate(gs):
        one = torch.autograd.grad(total, [h, w], g, retain_graph=True)
        assert torch.equal(batched[0][i], one[0]) and torch.equal(batched[1][i], one[1])


@pytest.mark.parametrize("unpack", [lambda t: t.t().contiguous().t(),
                                    lambda t: torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(t.shape),
                                    lambda t: t.double()])
def test_linear_ce_gradients_given_back_in_another_form(unpack):
    """A saved-tensor hook may return a transposed, an unaligned or a wider tensor of the same values: the gradients are those of the same
    values saved plainly, to the one rounding in which a wider product differs."""
    from cppmega_b200.ops.cuda import extra
    torch.manual_seed(0)
    h = torch.randn(72, 64, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(512, 64, device="cuda") * 0.1).bfloat16().requires_grad_()
    lab, rw, g = torch.randint(0, 512, (72,), device="cuda"), torch.rand(72, device="cuda"), torch.tensor(0.37, device="cuda")
    plain = torch.autograd.grad(extra.linear_cross_entropy_weighted(h, w, lab, rw, -100)[0], [h, w], g)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: unpack(t) if t.is_floating_point() else t):
        total = extra.linear_cross_entropy_weighted(h, w, lab, rw, -100)[0]
        other = torch.autograd.grad(total, [h, w], g)
    for a, b in zip(other, plain):
        assert _rel(a, b) < 2.0 ** -8
