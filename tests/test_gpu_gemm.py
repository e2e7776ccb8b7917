"""tcgen05 GEMM family against fp32 PyTorch matmul."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


@pytest.fixture(scope="module")
def cu():
    from cppmega_b200.ops import cuda
    return cuda


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (1000, 776, 520), (4096, 4096, 1024),
                                   (8, 16, 8), (304, 24960, 256)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_layouts(cu, M, N, K, a_mn, b_mn):
    torch.manual_seed(M + N + K)
    A = torch.randn(M, K, device="cuda").bfloat16()
    B = torch.randn(N, K, device="cuda").bfloat16()
    ref = A.float() @ B.float().t()
    a = A.t().contiguous() if a_mn else A
    b = B.t().contiguous() if b_mn else B
    out = cu.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    cu.check_errors()
    assert out.shape == (M, N)
    assert _rel(out, ref) < 6e-3


def test_gemm_fp32_accumulate(cu):
    torch.manual_seed(1)
    A = torch.randn(512, 320, device="cuda").bfloat16()
    B = torch.randn(384, 320, device="cuda").bfloat16()
    C0 = torch.randn(512, 384, device="cuda")
    out = C0.clone()
    cu.gemm(A, B, out=out, accumulate=True)
    cu.check_errors()
    ref = C0 + A.float() @ B.float().t()
    assert _rel(out, ref) < 1e-4
    out2 = torch.empty(512, 384, device="cuda")
    cu.gemm(A, B, out=out2)
    assert _rel(out2, A.float() @ B.float().t()) < 1e-4


def test_linear_autograd(cu):
    torch.manual_seed(2)
    x = torch.randn(4, 96, 256, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(512, 256, device="cuda") * 0.05).bfloat16().requires_grad_()
    y = cu.linear(x, w)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    yr = xr @ wr.t()
    yr.backward(g.float())
    cu.check_errors()
    assert _rel(y, yr) < 6e-3
    assert _rel(x.grad, xr.grad) < 6e-3
    assert _rel(w.grad, wr.grad) < 6e-3


@pytest.mark.parametrize("counts", [[128, 0, 300, 5], [1, 1, 1, 1], [0, 0, 0, 700], [257, 129, 64, 63]])
def test_grouped_experts(cu, counts):
    from cppmega_b200.ops.cuda import extra
    from cppmega_b200.ops import reference as ref
    torch.manual_seed(3)
    E, H, Fh = len(counts), 256, 192
    T = sum(counts)
    x = torch.randn(T, H, device="cuda").bfloat16().requires_grad_()
    w1 = (torch.randn(E, 2 * Fh, H, device="cuda") * 0.05).bfloat16().requires_grad_()
    w2 = (torch.randn(E, H, Fh, device="cuda") * 0.05).bfloat16().requires_grad_()
    cnt = torch.tensor(counts, device="cuda")
    y = extra.moe_experts(x, w1, w2, cnt)
    g = torch.randn_like(y)
    y.backward(g)
    cu.check_errors()
    xr, w1r, w2r = (t.detach().float().requires_grad_() for t in (x, w1, w2))
    h = ref.grouped_gemm(xr, w1r.transpose(1, 2), counts)
    h = ref.swiglu(h)
    yr = ref.grouped_gemm(h, w2r.transpose(1, 2), counts)
    yr.backward(g.float())
    assert _rel(y, yr) < 1.5e-2
    assert _rel(x.grad, xr.grad) < 1.5e-2
    assert _rel(w1.grad, w1r.grad) < 1.5e-2
    assert _rel(w2.grad, w2r.grad) < 1.5e-2


def test_linear_fp32out_router_shape():
    from cppmega_b200.ops import cuda as cu
    torch.manual_seed(0)
    x = (torch.randn(3000, 512, device="cuda") * 0.5).bfloat16().requires_grad_()
    w = (torch.randn(16, 512, device="cuda") * 0.05).requires_grad_()
    y = cu.linear_fp32out(x, w)
    assert y.dtype == torch.float32
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().clone().requires_grad_()
    yr = torch.nn.functional.linear(xr, wr)
    yr.backward(g)
    rel = lambda a, b: ((a.float() - b.float()).norm() / b.float().norm()).item()
    assert rel(y, yr) < 1e-2
    assert rel(x.grad, xr.grad) < 2e-2
    assert rel(w.grad, wr.grad) < 2e-2
    assert w.grad.dtype == torch.float32


@pytest.mark.parametrize("pair,bn", [(1, 256), (1, 192), (1, 128), (0, 256), (0, 128), (0, 64)])
@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (129, 200, 72), (257, 264, 64), (520, 776, 456), (2056, 1032, 1000)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("out,accumulate", [(torch.bfloat16, False), (torch.float32, False), (torch.bfloat16, True), (torch.float32, True)])
def test_gemm_tile_shapes(cu, pair, bn, M, N, K, a_mn, b_mn, out, accumulate):
    """Every tile shape of the dense dispatch at sizes below, at and past the edges of its tiles, with a padded C pitch that
    must stay untouched.  fp32 results: sums of K <= 1000 products in fp32, relative error well below 1e-5; bf16 results add
    one rounding of 2^-9."""
    if bn == 192 and b_mn:
        pytest.skip("an MN-major B operand comes in runs of 64 columns per CTA")
    torch.manual_seed(M + K)
    M8 = (M + 7) // 8 * 8 if a_mn else M
    A, B = torch.randn(M8, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    buf = torch.randn(M8, N + 8, device="cuda").to(out)
    before = buf.clone()
    a, b = (A.t().contiguous() if a_mn else A), (B.t().contiguous() if b_mn else B)
    rc = cu.lib().cm_gemm_bf16_tiled(a.data_ptr(), b.data_ptr(), buf.data_ptr(), M8, N, K, a.stride(0), b.stride(0), buf.stride(0), int(a_mn),
                                     int(b_mn), int(out == torch.float32), int(accumulate), pair, bn, cu.err_word(a.device).data_ptr(),
                                     cu.stream_ptr())
    assert rc == 0
    cu.check_errors()
    ref = A.double() @ B.double().t() + (before[:, :N].double() if accumulate else 0)
    err = ((buf[:, :N].double() - ref).norm() / ref.norm()).item()
    assert err < (1e-5 if out == torch.float32 else 4e-3)
    assert torch.equal(buf[:, N:], before[:, N:])


@pytest.mark.parametrize("counts", [[700, 0, 1300, 129], [5, 640, 2000, 0], [1025, 1023, 128, 896]])
def test_grouped_experts_pair_tiles(cu, counts):
    """Segments of odd and even tile counts, empty experts, and widths that end inside a tile, through the public entry: the
    products of one CTA and the weight gradients of CTA pairs."""
    from cppmega_b200.ops.cuda import extra
    from cppmega_b200.ops import reference as ref
    torch.manual_seed(4)
    E, H, Fh = len(counts), 328, 232
    x = torch.randn(sum(counts), H, device="cuda").bfloat16().requires_grad_()
    w1 = (torch.randn(E, 2 * Fh, H, device="cuda") * 0.05).bfloat16().requires_grad_()
    w2 = (torch.randn(E, H, Fh, device="cuda") * 0.05).bfloat16().requires_grad_()
    y = extra.moe_experts(x, w1, w2, torch.tensor(counts, device="cuda"))
    g = torch.randn_like(y)
    y.backward(g)
    cu.check_errors()
    xr, w1r, w2r = (t.detach().float().requires_grad_() for t in (x, w1, w2))
    yr = ref.grouped_gemm(ref.swiglu(ref.grouped_gemm(xr, w1r.transpose(1, 2), counts)), w2r.transpose(1, 2), counts)
    yr.backward(g.float())
    for got, want in ((y, yr), (x.grad, xr.grad), (w1.grad, w1r.grad), (w2.grad, w2r.grad)):
        assert _rel(got, want) < 1.5e-2


@pytest.mark.parametrize("pair,bn", [(1, 256), (1, 128), (0, 128), (0, 64)])
@pytest.mark.parametrize("offset,pitch", [(1, 264), (4, 264), (8, 264), (0, 257), (2, 260)])
@pytest.mark.parametrize("out,accumulate", [(torch.bfloat16, False), (torch.float32, False), (torch.bfloat16, True), (torch.float32, True)])
def test_gemm_result_in_an_unaligned_view(cu, pair, bn, offset, pitch, out, accumulate):
    """C starts off a 16-byte boundary, or its rows do: every element is still written, and nothing beside it.  Tolerances as
    for aligned results (test_gemm_tile_shapes)."""
    M, N, K = 200, 256, 136
    torch.manual_seed(offset + pitch)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    buf = torch.randn(offset + M * pitch, device="cuda").to(out)
    before = buf.clone()
    C, C0 = (t[offset:].view(M, pitch)[:, :N] for t in (buf, before))
    rc = cu.lib().cm_gemm_bf16_tiled(a.data_ptr(), b.data_ptr(), C.data_ptr(), M, N, K, K, K, pitch, 0, 0, int(out == torch.float32),
                                     int(accumulate), pair, bn, cu.err_word(a.device).data_ptr(), cu.stream_ptr())
    assert rc == 0
    cu.check_errors()
    ref = a.double() @ b.double().t() + (C0.double() if accumulate else 0)
    assert ((C.double() - ref).norm() / ref.norm()).item() < (1e-5 if out == torch.float32 else 4e-3)
    C.copy_(C0)
    assert torch.equal(buf, before)


@pytest.mark.parametrize("pair,bn", [(1, 256), (1, 192), (1, 128), (0, 256), (0, 128), (0, 64)])
@pytest.mark.parametrize("M,N,K,pitch", [(129, 201, 73, 208), (300, 515, 64, 520), (64, 1, 64, 8), (257, 66, 200, 72), (40, 260, 64, 264)])
@pytest.mark.parametrize("out,accumulate", [(torch.bfloat16, False), (torch.float32, False), (torch.float32, True)])
def test_gemm_result_of_an_odd_width_in_wider_rows(cu, pair, bn, M, N, K, pitch, out, accumulate):
    """Rows that end off a 16-byte boundary inside aligned wider ones (out=buf[:, :N]): the columns beside them stay."""
    torch.manual_seed(N)
    ld = (K + 7) // 8 * 8
    a, b = torch.randn(M, ld, device="cuda").bfloat16(), torch.randn(N, ld, device="cuda").bfloat16()
    buf = torch.randn(M, pitch, device="cuda").to(out)
    before = buf.clone()
    assert cu.lib().cm_gemm_bf16_tiled(a.data_ptr(), b.data_ptr(), buf.data_ptr(), M, N, K, ld, ld, pitch, 0, 0, int(out == torch.float32),
                                       int(accumulate), pair, bn, cu.err_word(a.device).data_ptr(), cu.stream_ptr()) == 0
    cu.check_errors()
    ref = a[:, :K].double() @ b[:, :K].double().t() + (before[:, :N].double() if accumulate else 0)
    assert ((buf[:, :N].double() - ref).norm() / ref.norm()).item() < (1e-5 if out == torch.float32 else 4e-3)
    assert torch.equal(buf[:, N:], before[:, N:])


@pytest.mark.parametrize("ldc", [0, 8, 64])
def test_gemm_single_row_of_any_pitch(cu, ldc):
    """The pitch of a single row is any number (an expanded or reshaped [1, N] view)."""
    torch.manual_seed(ldc)
    a, b = torch.randn(1, 64, device="cuda").bfloat16(), torch.randn(512, 64, device="cuda").bfloat16()
    out = torch.empty(512, device="cuda").bfloat16()
    for pair, bn in ((1, 256), (1, 128), (0, 256), (0, 64)):
        out.zero_()
        assert cu.lib().cm_gemm_bf16_tiled(a.data_ptr(), b.data_ptr(), out.data_ptr(), 1, 512, 64, 64, 64, ldc, 0, 0, 0, 0, pair, bn,
                                           cu.err_word(a.device).data_ptr(), cu.stream_ptr()) == 0, (pair, bn)
        cu.check_errors()
        assert _rel(out, (a.float() @ b.float().t())[0]) < 4e-3


@pytest.mark.parametrize("M,pair", [(96, 0), (288, 0), (288, 1)])
@pytest.mark.parametrize("out,accumulate", [(torch.bfloat16, False), (torch.float32, True)])
def test_mxfp8_gemm_result_in_an_unaligned_view(cu, M, pair, out, accumulate):
    """The same for the block-scaled GEMM, on one CTA and on a CTA pair."""
    from cppmega_b200.ops.cuda import mxfp8
    torch.manual_seed(M)
    N, K = 160, 96
    a, b = (mxfp8.quantize_rowwise(torch.randn(r, K, device="cuda").bfloat16()) for r in (M, N))
    for offset, pitch in ((1, 168), (0, 163)):
        buf = torch.randn(offset + M * pitch, device="cuda").to(out)
        before = buf.clone()
        C, C0 = (t[offset:].view(M, pitch)[:, :N] for t in (buf, before))
        assert mxfp8._lib().cm_mxfp8_gemm_tiled(a.payload.data_ptr(), a.swizzled().data_ptr(), b.payload.data_ptr(), b.swizzled().data_ptr(),
                                                C.data_ptr(), M, N, K, K, K, pitch, int(out == torch.float32), int(accumulate), pair,
                                                cu.err_word(C.device).data_ptr(), cu.stream_ptr()) == 0
        cu.check_errors()
        ref = mxfp8.dequantize(a).double() @ mxfp8.dequantize(b).double().t() + (C0.double() if accumulate else 0)
        assert ((C.double() - ref).norm() / ref.norm()).item() < (1e-5 if out == torch.float32 else 4e-3)
        C.copy_(C0)
        assert torch.equal(buf, before)


def _expert_layout(tiles, spare):
    """Expert segments of the given numbers of 128-row tiles, then ``spare`` unused ones: (tile_expert, seg_offsets, rows)."""
    te = [e for e, n in enumerate(tiles) for _ in range(n)] + [-1] * spare
    off = [0]
    for n in tiles:
        off.append(off[-1] + 128 * n)
    return (torch.tensor(te, dtype=torch.int32, device="cuda"), torch.tensor(off, dtype=torch.int32, device="cuda"), 128 * len(te))


PAIRS = 1 << 24       # rows in use that send any of these shapes to the CTA-pair kernel; the layout stays what the tensors say


@pytest.mark.parametrize("tiles,spare", [([7, 0, 5, 1, 8, 3], 3), ([1] * 23, 0), ([0, 0, 31, 0, 2], 6), ([12, 12], 0)])
@pytest.mark.parametrize("b_mn", [0, 1])
@pytest.mark.parametrize("N,K", [(4104, 136), (4544, 64)])
def test_expert_products_on_pairs_over_several_waves(cu, tiles, spare, b_mn, N, K):
    """More than three times as many row-pair tiles as CTA pairs, so that accumulators and stages come round while tiles that two experts share are
    worked on twice and unused ones are passed over: odd segments, empty experts first, in the middle and last."""
    torch.manual_seed(sum(tiles) + N)
    te, off, rows = _expert_layout(tiles, spare)
    E = len(tiles)
    assert cu.lib().cm_grouped_rows_plan(148, PAIRS, E, N, K, b_mn) == 1
    x = torch.randn(rows, K, device="cuda").bfloat16()
    x[int(off[-1]):] = float("nan")                                      # unused rows hold anything
    w = torch.randn(E, K, N, device="cuda").bfloat16() if b_mn else torch.randn(E, N, K, device="cuda").bfloat16()
    y = torch.full((rows, N), 3.0, device="cuda").bfloat16()
    assert cu.lib().cm_grouped_gemm_rows_bf16(x.data_ptr(), w.data_ptr(), y.data_ptr(), rows, N, K, E, b_mn, te.data_ptr(), PAIRS,
                                              cu.err_word(x.device).data_ptr(), cu.stream_ptr()) == 0
    cu.check_errors()
    for e in range(E):
        s = slice(int(off[e]), int(off[e + 1]))
        if s.start < s.stop:
            ref = x[s].double() @ (w[e].double() if b_mn else w[e].double().t())
            assert ((y[s].double() - ref).norm() / ref.norm()).item() < 4e-3, e
    assert (y[int(off[-1]):] == 3.0).all()


@pytest.mark.parametrize("tiles", [[3, 0, 1, 5, 0, 2, 1, 4], [0, 2, 0, 0, 1, 0, 6, 0]])
@pytest.mark.parametrize("out,accumulate", [(torch.bfloat16, 0), (torch.float32, 0), (torch.bfloat16, 1), (torch.float32, 1)])
def test_expert_weight_gradients_on_pairs_over_several_waves(cu, tiles, out, accumulate):
    """The same for the weight gradients: 240 tiles for 74 pairs, experts without rows in between (zeros, or left alone)."""
    torch.manual_seed(len(tiles))
    M, N, E = 1032, 1288, len(tiles)
    _, off, rows = _expert_layout(tiles, 2)
    assert cu.lib().cm_grouped_k_plan(PAIRS, E, M, accumulate) == 1
    a, b = torch.randn(rows, M, device="cuda").bfloat16(), torch.randn(rows, N, device="cuda").bfloat16()
    c = torch.randn(E, M, N, device="cuda").to(out)
    before = c.clone()
    assert cu.lib().cm_grouped_gemm_k_bf16(a.data_ptr(), b.data_ptr(), c.data_ptr(), rows, M, N, E, off.data_ptr(), PAIRS,
                                           int(out == torch.float32), accumulate, cu.err_word(a.device).data_ptr(), cu.stream_ptr()) == 0
    cu.check_errors()
    for e in range(E):
        s = slice(int(off[e]), int(off[e + 1]))
        ref = a[s].double().t() @ b[s].double() + (before[e].double() if accumulate else 0)
        if s.start == s.stop:
            assert torch.equal(c[e].double(), ref if accumulate else torch.zeros_like(ref))
        else:
            assert ((c[e].double() - ref).norm() / ref.norm()).item() < (1e-5 if out == torch.float32 else 4e-3), e
