"""Sequence-mixer kernels against the fp32 PyTorch definitions."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


@pytest.mark.parametrize("B,S,H,KD,shared", [(2, 77, 3, 64, True), (1, 130, 5, 16, True), (2, 64, 4, 32, False)])
def test_m2rnn_scan(B, S, H, KD, shared):
    from cppmega_b200.ops import reference as ref
    from cppmega_b200.ops.cuda import kernels2
    torch.manual_seed(0)
    Hq = 1 if shared else H
    dev = "cuda"
    q = (torch.randn(B, S, Hq, KD, device=dev) * 0.5).bfloat16().requires_grad_()
    k = (torch.randn(B, S, Hq, KD, device=dev) * 0.5).bfloat16().requires_grad_()
    v = (torch.randn(B, S, H, 16, device=dev) * 0.5).bfloat16().requires_grad_()
    W = (torch.eye(16, device=dev).repeat(H, 1, 1) + 0.1 * torch.randn(H, 16, 16, device=dev)).bfloat16().requires_grad_()
    f = torch.rand(B, S, H, device=dev).requires_grad_()
    y = kernels2.m2rnn_scan(q, k, v, W, f)
    g = torch.randn_like(y)
    y.backward(g)
    refs = [t.detach().float().requires_grad_() for t in (q, k, v, W, f)]
    yr, _ = ref.m2rnn_scan(*refs)
    yr.backward(g.float())
    assert _rel(y, yr) < 2e-2
    for name, a, b in zip("q k v W f".split(), (q, k, v, W, f), refs):
        assert _rel(a.grad, b.grad) < 4e-2, name


def test_mimo_scan_lean_matches_sequential():
    from cppmega_b200.ops import mimo_scan_ref as R
    from cppmega_b200.ops.mimo_scan_lean import mimo_scan_lean
    torch.manual_seed(0)
    dev = "cuda"
    B, S, Rk, G, N, H, P = 2, 96, 4, 2, 32, 4, 16
    Q = torch.randn(B, S, Rk, G, N, device=dev)
    K = torch.randn(B, S, Rk, G, N, device=dev)
    V = torch.randn(B, S, H, P, device=dev)
    Z = torch.randn(B, S, H, P, device=dev)
    DT = torch.rand(B, H, S, device=dev) * 0.1
    ADT = -DT * torch.rand(B, H, S, device=dev) * 3
    Trap = torch.randn(B, H, S, device=dev)
    Qb, Kb = torch.randn(H, Rk, N, device=dev), torch.randn(H, Rk, N, device=dev)
    Psi, Zeta, Phi = (torch.randn(H, Rk, P, device=dev) for _ in range(3))
    ang = torch.randn(B, S, H, N // 4, device=dev).cumsum(1) * 0.1
    D = torch.randn(H, device=dev)
    args = [Q, K, V, ADT, DT, Trap, Qb, Kb, Psi, Zeta, Phi, ang, D, Z]
    a1 = [t.clone().requires_grad_() for t in args]
    a2 = [t.clone().requires_grad_() for t in args]
    y1 = R.mimo_scan_sequential(*a1, 4)
    y2 = mimo_scan_lean(*a2, 4, 32)
    g = torch.randn_like(y1)
    y1.backward(g)
    y2.backward(g)
    assert _rel(y2, y1) < 2e-2
    for i, (x, r) in enumerate(zip(a2, a1)):
        assert _rel(x.grad, r.grad) < 5e-2, i


def _attn_ref(q, k, v, scale):
    """fp32 causal attention, [B,S,H,D] layout."""
    B, S, H, _ = q.shape
    s = torch.einsum("bihd,bjhd->bhij", q.float(), k.float()) * scale
    s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=q.device).tril(), float("-inf"))
    return torch.einsum("bhij,bjhd->bihd", torch.softmax(s, dim=-1), v.float())


@pytest.mark.parametrize("B,S,H", [(1, 128, 2), (2, 512, 4), (1, 1024, 3)])
def test_dense_causal_attention_kernels(B, S, H):
    """Forward and the three gradients of the tcgen05 attention kernels against the fp32 definition: one key tile, several
    key tiles (online softmax, the state gradients kept in TMEM over the query loop), batch and head strides."""
    from cppmega_b200.ops import cuda as cu
    from cppmega_b200.ops import functional as F_
    torch.manual_seed(S)
    q = (torch.randn(B, S, H, 128, device="cuda") * 0.7).bfloat16().requires_grad_()
    k = (torch.randn(B, S, H, 128, device="cuda") * 0.7).bfloat16().requires_grad_()
    v = torch.randn(B, S, H, 64, device="cuda").bfloat16().requires_grad_()
    scale = 128 ** -0.5
    F_.reset_counters()
    o = F_.causal_attention(q, k, v, scale)
    assert F_.launch_counts().get("causal_attention", 0) == 1 and not F_.fallback_counts()
    g = torch.randn_like(o)
    o.backward(g)
    torch.cuda.synchronize()
    cu.check_errors()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    orf = _attn_ref(qr, kr, vr, scale)
    orf.backward(g.float())
    assert _rel(o, orf) < 1.5e-2
    for name, a, b in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        assert torch.isfinite(a.float()).all(), name
        assert _rel(a, b) < 2.5e-2, (name, _rel(a, b))


@pytest.mark.parametrize("T,H,sliced", [(256, 32, True), (200, 5, False), (1024, 32, False)])
def test_head_linear_kernels(T, H, sliced):
    """Per-head 64 x 64 maps (the absorbed MLA up-projections): output, input gradient and weight gradient against fp32,
    on an operand that is a column slice of a wider tensor (read in place), on a token count that is not a multiple of
    the tile, and on an odd head count (the last head pair of the weight-gradient kernel is half empty)."""
    from cppmega_b200.ops import cuda as cu
    from cppmega_b200.ops import functional as F_
    torch.manual_seed(T + H)
    base = torch.randn(2, T // 2, H, 128 if sliced else 64, device="cuda").bfloat16()
    x = (base[..., :64] if sliced else base).detach().requires_grad_()
    w = (torch.randn(H, 64, 64, device="cuda") * 0.2).bfloat16().requires_grad_()
    F_.reset_counters()
    y = F_.head_linear(x, w)
    assert F_.launch_counts().get("head_linear", 0) == 1 and not F_.fallback_counts()
    g = torch.randn_like(y)
    y.backward(g)
    torch.cuda.synchronize()
    cu.check_errors()
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yr = torch.einsum("bshi,hoi->bsho", xr, wr)
    yr.backward(g.float())
    assert _rel(y, yr) < 1e-2
    assert _rel(x.grad, xr.grad) < 1e-2
    assert _rel(w.grad, wr.grad) < 1e-2
    # the transposed-weight view used by the model (q . W_uk with W_uk stored [H, in, out])
    wt = (torch.randn(H, 64, 64, device="cuda") * 0.2).bfloat16()
    y2 = F_.head_linear(x.detach(), wt.transpose(1, 2))
    assert _rel(y2, torch.einsum("bshi,hio->bsho", x.detach().float(), wt.float())) < 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,C,k,sliced", [(2, 200, 136, 4, True), (1, 64, 64, 2, False), (3, 130, 72, 3, True)])
def test_causal_conv1d_silu_kernels(B, S, C, k, sliced):
    """Depthwise causal conv + SiLU, channels-last, read in place from a wider projection: output, input gradient, weight
    and bias gradients against the fp32 definition (segments of 64 tokens: S = 200 / 130 cross segment boundaries)."""
    from cppmega_b200.ops import cuda as cu
    from cppmega_b200.ops import functional as F_
    from cppmega_b200.ops import reference as ref
    torch.manual_seed(S + C)
    base = torch.randn(B, S, C + 40 if sliced else C, device="cuda").bfloat16()
    x = (base[..., :C] if sliced else base).detach().requires_grad_()
    w = (torch.randn(C, 1, k, device="cuda") * 0.5).bfloat16().requires_grad_()
    b = (torch.randn(C, device="cuda") * 0.1).bfloat16().requires_grad_()
    F_.reset_counters()
    y = F_.causal_conv1d_silu(x, w, b)
    assert F_.launch_counts().get("causal_conv1d_silu", 0) == 1 and not F_.fallback_counts()
    g = torch.randn_like(y)
    y.backward(g)
    torch.cuda.synchronize()
    cu.check_errors()
    xr, wr, br = (t.detach().float().requires_grad_() for t in (x, w, b))
    yr = ref.causal_conv1d_silu(xr, wr.squeeze(1), br)
    yr.backward(g.float())
    assert _rel(y, yr) < 1e-2
    assert _rel(x.grad, xr.grad) < 1.5e-2
    assert _rel(w.grad, wr.grad) < 1.5e-2
    assert _rel(b.grad, br.grad) < 1.5e-2


@pytest.mark.gpu
@pytest.mark.parametrize("variant", ["ssd", "noconv_ssd"])
def test_ssd_variant_mixers_on_gpu_match_the_cpu_fp32_module(variant):
    """The alternative SSM mixers (Mamba2-style SSD with the fused causal conv + SiLU kernel, and the no-conv variant with
    QK-norm / biases / data-dependent A / trapezoid / rotary state) in bf16 on the GPU against the same module in fp32 on
    the CPU: output and input gradient."""
    import copy
    from cppmega_b200.config.model import nam56r_tiny
    from cppmega_b200.models.mamba_variants import build_variant_mixer
    from cppmega_b200.ops import cuda as cu
    from cppmega_b200.ops import functional as F_
    from cppmega_b200.parallel.state import single_process_context
    cfg = nam56r_tiny(seq_length=128, mamba_variant=variant)
    pc = single_process_context()
    ref_mod = build_variant_mixer(cfg, pc, 1, dtype=torch.float32, seed=3, out_std=0.02)
    gpu_mod = copy.deepcopy(ref_mod).to("cuda").to(torch.bfloat16)
    for n, p in gpu_mod.named_parameters():                       # per-head fp32 parameters stay fp32, as in the model
        if p.dim() <= 1 and "norm" not in n and "conv" not in n:
            p.data = p.data.float()
    torch.manual_seed(5)
    x = torch.randn(2, 128, cfg.hidden_size) * 0.5
    g = torch.randn(2, 128, cfg.hidden_size) * 0.1
    xr = x.clone().requires_grad_()
    yr = ref_mod(xr)
    yr.backward(g)
    xg = x.cuda().bfloat16().requires_grad_()
    F_.reset_counters()
    yg = gpu_mod(xg)
    yg.backward(g.cuda().bfloat16())
    torch.cuda.synchronize()
    cu.check_errors()
    if variant == "ssd":
        assert F_.launch_counts().get("causal_conv1d_silu", 0) == 1
    assert _rel(yg.cpu(), yr) < 4e-2
    assert _rel(xg.grad.cpu(), xr.grad) < 6e-2


@pytest.mark.parametrize("B,S,H,KD,shared,offset", [(1, 1, 2, 64, True, 0), (2, 16, 3, 64, False, 0), (1, 33, 5, 32, True, 0),
                                                    (2, 50, 2, 64, True, 1), (1, 19, 3, 16, False, 3)])
def test_m2rnn_blocks_and_unaligned_inputs(B, S, H, KD, shared, offset):
    """Sequence lengths at, below and past the 16-step staging block, and inputs whose storage starts off a 16-byte boundary.
    The state factor is fp32 (three bf16 parts per factor): the fp32 gradient of f agrees to the accuracy of tanh.approx
    (2^-11 of tanh, less in the mean)."""
    from cppmega_b200.ops import reference as ref
    from cppmega_b200.ops.cuda import kernels2
    torch.manual_seed(S)
    Hq = 1 if shared else H

    def make(*shape, std):
        buf = (torch.randn(offset + torch.Size(shape).numel(), device="cuda") * std).bfloat16()
        return buf[offset:].view(shape).detach().requires_grad_()

    q, k, v = make(B, S, Hq, KD, std=0.5), make(B, S, Hq, KD, std=0.5), make(B, S, H, 16, std=0.5)
    W = make(H, 16, 16, std=0.3)
    f = torch.rand(B, S, H, device="cuda").requires_grad_()
    y = kernels2.m2rnn_scan(q, k, v, W, f)
    g = torch.randn_like(y)
    y.backward(g)
    refs = [t.detach().float().requires_grad_() for t in (q, k, v, W, f)]
    yr, _ = ref.m2rnn_scan(*refs)
    yr.backward(g.float())
    assert _rel(y, yr) < 5e-3
    for name, a, b in zip("q k v W f".split(), (q, k, v, W, f), refs):
        if b.grad.norm() > 0:
            assert _rel(a.grad, b.grad) < (1e-3 if name == "f" else 5e-3), name
        else:
            assert a.grad.norm() == 0, name


@pytest.mark.parametrize("B,S,KD", [(1, 1, 64), (1, 16, 16), (1, 16, 32), (2, 16, 64), (1, 19, 64)])
def test_m2rnn_gradients_of_v_and_w_keep_fp32_factors(B, S, KD):
    """dv and dW in fp32, before their rounding, against 64-bit sums of the kernel's own states and da.  With v the j-th unit
    vector in head j, dk is the j-th column of da, exactly.  A few fp32 roundings of 2^-24 give up to 2e-7 here; factors cut
    to two bf16 parts 1e-6 to 4e-6."""
    from cppmega_b200.ops import cuda as cu
    torch.manual_seed(S + KD)
    H = 16
    bf = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    q, k, dy = bf(B, S, H, KD), bf(B, S, H, KD), bf(B, S, H, 16)
    v = torch.eye(16, device="cuda").bfloat16().expand(B, S, 16, 16).contiguous()
    W = (torch.eye(16, device="cuda") + 0.1 * torch.randn(H, 16, 16, device="cuda")).bfloat16().contiguous()
    f32 = lambda *s: torch.empty(*s, device="cuda")  # noqa: E731
    f, y, hist = torch.rand(B, S, H, device="cuda"), torch.empty_like(dy), f32(B, H, S, KD, 16)
    dq, dk, dv, df, dW = f32(B, S, H, KD), f32(B, S, H, KD), f32(B, S, H, 16), f32(B, S, H), torch.zeros(H, 16, 16, device="cuda")
    ptr = lambda *ts: [t.data_ptr() for t in ts]  # noqa: E731
    dims = (B, S, H, H, H, KD, 16, cu.stream_ptr())
    assert cu.lib().cm_m2rnn_fwd(*ptr(q, k, v, W, f, y, hist), None, *dims) == 0
    assert cu.lib().cm_m2rnn_bwd(*ptr(q, k, v, W, f, hist, dy, dq, dk, dv, df, dW), *dims) == 0
    before = torch.zeros_like(hist)
    before[:, :, 1:] = hist[:, :, :-1]
    da, j = dk.double(), torch.arange(16)
    err = lambda a, b: ((a - b).norm() / b.norm().clamp_min(1e-30)).item()  # noqa: E731
    assert err(dv.double()[:, :, j, j], (k.double() * da).sum(-1)) < 2.0 ** -21
    assert err(dW.double()[j, :, j], torch.einsum("bhsku,bshk->hu", before.double(), da)) < 2.0 ** -21
    assert err(dq.double(), torch.einsum("bhskv,bshv->bshk", hist.double(), dy.double())) < 2.0 ** -21


@pytest.mark.parametrize("B,S,H,std,scale", [(1, 128, 1, 0.7, 0.09), (1, 384, 2, 4.0, 0.09), (2, 640, 1, 0.7, -0.05), (1, 384, 2, 4.0, -0.09), (1, 256, 3, 0.7, 0.0)])
def test_dense_causal_attention_tile_pairs(B, S, H, std, scale):
    """Odd and even counts of query tiles (the last pair has one or two), scores large enough that the running maximum grows
    past the rescale threshold between key tiles, and scales of either sign and zero: with std 4 and -0.09 a row spans several hundred
    powers of two, so that only its true maximum serves as the reference."""
    from cppmega_b200.ops import cuda as cu
    from cppmega_b200.ops import functional as F_
    torch.manual_seed(S)
    grow = torch.linspace(0.2, 1.0, S, device="cuda").view(1, S, 1, 1)          # later keys score higher
    q = (torch.randn(B, S, H, 128, device="cuda") * std).bfloat16().requires_grad_()
    k = (torch.randn(B, S, H, 128, device="cuda") * std * grow).bfloat16().requires_grad_()
    v = torch.randn(B, S, H, 64, device="cuda").bfloat16().requires_grad_()
    o = F_.causal_attention(q, k, v, scale)
    g = torch.randn_like(o)
    o.backward(g)
    cu.check_errors()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    orf = _attn_ref(qr, kr, vr, scale)
    orf.backward(g.float())
    assert _rel(o, orf) < 1e-2
    for name, a, b in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        if b.norm() > 0:
            assert _rel(a, b) < 1.5e-2, name
        else:
            assert a.norm() == 0, name


@pytest.mark.parametrize("B,S", [(1, 40), (2, 300)])
def test_sparse_mla_repeated_and_masked_keys(B, S):
    """Rows selected twice by one query, queries with few or no keys, and keys after the query: the gradient rows of a key are
    summed over all of its uses."""
    from cppmega_b200.ops import cuda as cu
    from cppmega_b200.ops import reference as ref
    from cppmega_b200.ops.cuda import kernels4
    torch.manual_seed(S)
    q = (torch.randn(B, S, 32, 128, device="cuda") * 0.5).bfloat16().requires_grad_()
    kv = (torch.randn(B, S, 128, device="cuda") * 0.5).bfloat16().requires_grad_()
    idx = torch.randint(-60, S, (B, S, 256), device="cuda").clamp_min(-1).to(torch.int32)
    idx[:, 3] = -1
    idx[:, 5, 1:] = -1
    o = kernels4.sparse_mla(q, kv, idx, 0.1, 64)
    g = torch.randn_like(o)
    o.backward(g)
    cu.check_errors()
    # the definition has no gradient for a query without keys: give it one key there and no upstream gradient
    some, gr = idx.clone(), g.float().clone()
    some[:, 3, 0] = 0
    gr[:, 3] = 0
    qr, kr = (t.detach().float().requires_grad_() for t in (q, kv))
    orf, _ = ref.sparse_mla(qr, kr, some, 0.1, 64)
    orf.backward(gr)
    assert o[:, 3].norm() == 0
    live = torch.arange(S, device="cuda") != 3
    assert _rel(o[:, live], orf[:, live]) < 1e-2
    assert _rel(q.grad, qr.grad) < 1.5e-2
    assert _rel(kv.grad, kr.grad) < 1.5e-2
