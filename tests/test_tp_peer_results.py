"""Host side of the staged GEMM -> reduce-scatter, with the kernels replaced by tensor arithmetic."""
import types

import pytest
import torch


@pytest.mark.parametrize("me", [0, 1])
def test_partial_products_for_other_ranks_are_marked_as_peer_results(monkeypatch, me):
    """Results that lie in another GPU's memory go to the one-CTA kernel, whose ordinary stores that path was run with on
    several GPUs; this rank's own shard may take any kernel."""
    from cppmega_b200.ops import cuda as cu
    from cppmega_b200.parallel import fused_tp
    tp, B, S, K, N = 2, 1, 8, 16, 24
    tpo = fused_tp.FusedTP.__new__(fused_tp.FusedTP)
    tpo.tp, tpo.rs_epoch, tpo.stage = tp, 0, torch.zeros(tp * B * S * N, dtype=torch.bfloat16)
    owners = [tpo.stage if p == me else torch.zeros_like(tpo.stage) for p in range(tp)]

    def peer_tensor(t, p):
        off = (t.data_ptr() - tpo.stage.data_ptr()) // 2
        return owners[p][off:off + t.numel()].view(t.shape)

    noop = lambda *a: None  # noqa: E731
    tpo.heap = types.SimpleNamespace(me=me, wait=noop, barrier=noop, signal=noop, peer_tensor=peer_tensor)
    seen = {}

    def gemm(a, b, *, b_mn=False, out=None, peer_out=False):
        owner = next(p for p in range(tp) if owners[p].data_ptr() <= out.data_ptr() < owners[p].data_ptr() + owners[p].numel() * 2)
        seen[owner] = peer_out
        out.copy_(a.float() @ (b.float() if b_mn else b.float().t()))

    monkeypatch.setattr(cu, "gemm", gemm)
    monkeypatch.setattr(cu, "stream_ptr", lambda: 0)
    monkeypatch.setattr(fused_tp, "_lib", lambda: types.SimpleNamespace(cm_sum_slots=lambda *a: 0))
    x, w = torch.randn(B, S, K).bfloat16(), torch.randn(N, K).bfloat16()
    tpo._gemm_rs_staged(x, w, False)
    assert seen == {p: p != me for p in range(tp)}
    for p in range(tp):
        slot = owners[p].view(-1)[me * B * (S // tp) * N:][:B * (S // tp) * N].view(S // tp, N)
        assert torch.equal(slot, (x[0, p * 4:(p + 1) * 4].float() @ w.float().t()).bfloat16())


def test_peer_results_take_the_one_cta_kernel(monkeypatch):
    from cppmega_b200.ops import cuda as cu
    calls = []
    entry = lambda name: lambda *a: calls.append((name, a)) or 0  # noqa: E731
    monkeypatch.setattr(cu, "lib", lambda: types.SimpleNamespace(cm_gemm_bf16=entry("planned"), cm_gemm_bf16_tiled=entry("tiled")))
    monkeypatch.setattr(cu, "err_word", lambda device=None: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(cu, "stream_ptr", lambda: 0)
    a, b = torch.zeros(4096, 64, dtype=torch.bfloat16), torch.zeros(4096, 64, dtype=torch.bfloat16)
    cu.gemm(a, b)
    cu.gemm(a, b, peer_out=True)
    assert [n for n, _ in calls] == ["planned", "tiled"]
    assert calls[1][1][13:15] == (0, 256)           # not a CTA pair, 256 columns
