"""Backward of the fused vocabulary head and loss in the forms that its kernel does not take."""
import types

import torch


def test_head_gradients_scale_for_batched_upstream_gradients():
    """``is_grads_batched`` runs the backward with an upstream gradient that has no storage to hand to a kernel."""
    from cppmega_b200.ops.cuda.extra import LinearCEWeightedFn
    torch.manual_seed(0)
    dh, dw = torch.randn(5, 8).bfloat16(), torch.randn(16, 8)
    h, w = torch.zeros(5, 8, dtype=torch.bfloat16, requires_grad=True), torch.zeros(16, 8, dtype=torch.bfloat16, requires_grad=True)
    ctx = types.SimpleNamespace(saved_tensors=(dh, dw), w_dtype=torch.bfloat16)

    class Head(torch.autograd.Function):
        @staticmethod
        def forward(_, h, w):
            return h.new_zeros((), dtype=torch.float32)

        @staticmethod
        def backward(_, g):
            return LinearCEWeightedFn.backward(ctx, g, None)[:2]

    gs = torch.tensor([1.0, 0.37, -2.0])
    got_h, got_w = torch.autograd.grad(Head.apply(h, w), [h, w], gs, is_grads_batched=True)
    assert torch.equal(got_h, torch.stack([dh * g.bfloat16() for g in gs]))
    assert torch.equal(got_w, torch.stack([(dw * g).bfloat16() for g in gs]))
