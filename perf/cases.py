"""The calls of this framework whose speed is followed, with the work each one cannot do without and its 64-bit result.

Every case is one operator of the hybrid model (forward and backward), called the way a training program calls it: through
``cppmega_b200.ops.functional`` or, for the routed experts, through the dispatcher that ``parallel.fused_moe.attach`` installs.
Sizes are those of the presets in ``config/model.py`` (full, quarter, slice), of ``bench.py`` and of ``tools/kernel_bench.py``.
"""
from __future__ import annotations

import math
import types

import torch

from cppmega_b200.ops import functional as F_


def listed():
    return [
        # a projection of the smallest production-shaped model at its smallest micro-batch: launches and host time
        dict(name="linear_small", kind="linear", tokens=512, k=1024, n=2048),
        # the dense MLP of the quarter model on a batch that fills no tile
        dict(name="linear_ragged", kind="linear", tokens=4095, k=3584, n=18944),
        # the largest projection of the full model (Mamba in_proj) at the benchmark's micro-batch, 4 x 4096 tokens
        dict(name="linear_in_proj", kind="linear", tokens=16384, k=4096, n=24960),
        # the Mamba out_proj under the MXFP8 recipe
        dict(name="mxfp8_out_proj", kind="mxfp8", tokens=8192, k=8192, n=4096),
        # the routed experts of one MoE layer: 16 experts, top-4, uneven routing
        dict(name="experts", kind="experts", tokens=8192, hidden=4096, ffn=896, experts=16, topk=4),
        # the scan at the small shape of the scan micro-benchmark (state 64): launches and host time
        dict(name="scan_small", kind="scan", batch=2, seq=256, heads=8, groups=1, state=64),
        # the scan of one full-model layer on one sequence
        dict(name="scan_layer", kind="scan", batch=1, seq=4096, heads=128, groups=8, state=128),
        # the dense latent-attention layers of the full model
        dict(name="attention", kind="attention", batch=2, seq=4096, heads=32),
        # the sparse-attention layers: 256 selected keys per query
        dict(name="sparse_attention", kind="sparse", batch=2, seq=4096),
        # the matrix-state recurrence of the full model
        dict(name="m2rnn", kind="m2rnn", batch=2, seq=4096, heads=51),
        # vocabulary head and loss of the full model on half a micro-batch
        dict(name="head_loss", kind="loss", tokens=8192, hidden=4096, vocab=131072),
        # a layer norm of the full model at the benchmark's micro-batch
        dict(name="norm", kind="norm", rows=16384, width=4096),
    ]


def _log(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "mxfp8", "experts", "scan", "scan", "attention", "sparse", "m2rnn", "loss", "norm"])
    if kind == "linear":
        return dict(kind=kind, tokens=_log(rng, 256, 16384), k=_log(rng, 512, 8192, 8), n=_log(rng, 512, 24960, 8))
    if kind == "mxfp8":
        return dict(kind=kind, tokens=_log(rng, 512, 16384, 32), k=_log(rng, 1024, 8192, 32), n=_log(rng, 1024, 8192, 32))
    if kind == "experts":
        return dict(kind=kind, tokens=_log(rng, 256, 8192), hidden=rng.choice([1024, 2048, 3584, 4096]), ffn=rng.choice([512, 896]),
                    experts=16, topk=4)
    if kind == "scan":
        heads, groups = rng.choice([(8, 1), (16, 8), (32, 8), (32, 2), (56, 8), (64, 8), (112, 8), (128, 8)])
        return dict(kind=kind, batch=rng.choice([1, 2]), seq=_log(rng, 256, 2048, 32), heads=heads, groups=groups,
                    state=rng.choice([64, 128]))
    if kind == "attention":
        return dict(kind=kind, batch=rng.choice([1, 2]), seq=_log(rng, 256, 4096, 128), heads=rng.choice([8, 16, 28, 32]))
    if kind == "sparse":
        return dict(kind=kind, batch=rng.choice([1, 2]), seq=_log(rng, 300, 4096))
    if kind == "m2rnn":
        return dict(kind=kind, batch=rng.choice([1, 2]), seq=_log(rng, 256, 4096), heads=rng.choice([12, 44, 51]))
    if kind == "loss":
        return dict(kind=kind, tokens=_log(rng, 512, 8192), hidden=rng.choice([1024, 3584, 4096]), vocab=rng.choice([8192, 65536, 131072]))
    return dict(kind=kind, rows=_log(rng, 512, 32768), width=rng.choice([64, 128, 816, 1024, 3584, 4096]))


# ---- inputs --------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(*shape, std=1.0, dtype=torch.bfloat16, grad=False):
        t = torch.empty(shape, device="cuda").normal_(0, std, generator=g).to(dtype)
        return t.requires_grad_() if grad else t

    def uniform(*shape, lo=0.0, hi=1.0):
        return torch.empty(shape, device="cuda").uniform_(lo, hi, generator=g)

    c, kind = types.SimpleNamespace(**case), case["kind"]
    if kind in ("linear", "mxfp8"):
        return dict(kind=kind, x=normal(c.tokens, c.k, grad=True), w=normal(c.n, c.k, std=0.02, grad=True), dy=normal(c.tokens, c.n, std=0.1))
    if kind == "experts":
        from cppmega_b200.parallel import state
        from cppmega_b200.parallel.fused_moe import FusedMoEDispatcher, LocalMoEBuffers
        # sigmoid scores with a per-expert offset: some experts get a few times the rows of others
        score = torch.sigmoid(normal(c.tokens, c.experts, dtype=torch.float32) + normal(c.experts, std=0.5, dtype=torch.float32))
        top, ids = torch.topk(score, c.topk, dim=-1)
        buffers = LocalMoEBuffers(state.single_process_context(), c.hidden, c.experts, torch.device("cuda", torch.cuda.current_device()))
        experts = types.SimpleNamespace(weight1=normal(c.experts, 2 * c.ffn, c.hidden, std=0.02, grad=True),
                                        weight2=normal(c.experts, c.hidden, c.ffn, std=0.02, grad=True))
        return dict(kind=kind, x=normal(c.tokens, c.hidden, grad=True), p=(top / top.sum(-1, keepdim=True)).requires_grad_(), ids=ids,
                    experts=experts, dispatch=FusedMoEDispatcher(buffers, 0), dy=normal(c.tokens, c.hidden, std=0.1))
    if kind == "scan":
        B, S, H, G, N, R, P = c.batch, c.seq, c.heads, c.groups, c.state, 4, 64
        f32 = torch.float32
        # step sizes, decays and rotary angles as the mixer makes them: softplus step in about [0.001, 0.1], angles summed over steps
        dt = torch.exp(uniform(1, H, 1, lo=math.log(1e-3), hi=math.log(0.1)) + 0.3 * normal(B, H, S, dtype=f32))
        adt = -dt * torch.nn.functional.softplus(normal(B, H, S, dtype=f32))
        angles = torch.cumsum(normal(B, S, 1, N // 4, std=0.6, dtype=f32) * dt.permute(0, 2, 1).unsqueeze(-1), dim=1)
        norm = lambda t: (t.float() * torch.rsqrt(t.float().square().mean(-1, keepdim=True))).to(torch.bfloat16)  # noqa: E731
        ins = dict(q=norm(normal(B, S, G, R, N)).permute(0, 1, 3, 2, 4), k=norm(normal(B, S, G, R, N)).permute(0, 1, 3, 2, 4),
                   v=normal(B, S, H, P), adt=adt, dt=dt, trap=normal(B, H, S, dtype=f32), qb=1 + normal(H, R, N, std=0.1, dtype=f32),
                   kb=1 + normal(H, R, N, std=0.1, dtype=f32), psi=0.25 + normal(H, R, P, std=0.05, dtype=f32),
                   zeta=1 + normal(H, R, P, std=0.1, dtype=f32), phi=0.25 + normal(H, R, P, std=0.05, dtype=f32), angles=angles,
                   d=1 + normal(H, std=0.1, dtype=f32), z=normal(B, S, H, P))
        return dict(kind=kind, ins={n: t.requires_grad_() for n, t in ins.items()}, dy=normal(B, S, H, P, std=0.1))
    if kind == "attention":
        q, k = (normal(c.batch, c.seq, c.heads, 128, grad=True) for _ in range(2))
        return dict(kind=kind, q=q, k=k, v=normal(c.batch, c.seq, c.heads, 64, grad=True), dy=normal(c.batch, c.seq, c.heads, 64, std=0.1))
    if kind == "sparse":
        B, S, top = c.batch, c.seq, 256
        idx = torch.empty(B, S, top, dtype=torch.int32, device="cuda")
        for s in range(0, S, 1024):                 # distinct earlier positions, in no order; -1 where a query has fewer than 256
            e = min(s + 1024, S)
            score = uniform(B, e - s, S)
            score.masked_fill_(torch.arange(S, device="cuda")[None, :] > torch.arange(s, e, device="cuda")[:, None], -1.0)
            val, pos = torch.topk(score, top, dim=-1)
            idx[:, s:e] = torch.where(val >= 0, pos, -1).to(torch.int32)
        return dict(kind=kind, q=normal(B, S, 32, 128, grad=True), kv=normal(B, S, 128, grad=True), idx=idx, dy=normal(B, S, 32, 64, std=0.1))
    if kind == "m2rnn":
        B, S, H = c.batch, c.seq, c.heads
        silu = lambda t: torch.nn.functional.silu(t.float()).to(torch.bfloat16).requires_grad_()  # noqa: E731
        decay = uniform(H, lo=math.log(0.01), hi=math.log(16.0)).exp()
        f = torch.exp(-decay * torch.nn.functional.softplus(normal(B, S, H, dtype=torch.float32) - 4.0))
        w = (torch.eye(16, device="cuda").expand(H, 16, 16) + normal(H, 16, 16, std=0.02, dtype=torch.float32)).to(torch.bfloat16)
        return dict(kind=kind, q=silu(normal(B, S, 1, 64)), k=silu(normal(B, S, 1, 64)), v=silu(normal(B, S, H, 16)), w=w.requires_grad_(),
                    f=f.requires_grad_(), dy=normal(B, S, H, 16, std=0.1))
    if kind == "loss":
        labels = torch.randint(0, c.vocab, (c.tokens,), device="cuda", generator=g)
        labels[uniform(c.tokens) < 0.02] = -100
        return dict(kind=kind, x=normal(c.tokens, c.hidden, grad=True), w=normal(c.vocab, c.hidden, std=0.02, grad=True), labels=labels,
                    weights=(labels >= 0).float() / c.tokens)
    return dict(kind=kind, x=normal(c.rows, c.width, std=2.0, grad=True), w=(1 + normal(c.width, std=0.1, dtype=torch.float32)).to(torch.bfloat16).requires_grad_(),
                dy=normal(c.rows, c.width, std=0.1))


# ---- one pass -------------------------------------------------------------------------------------------------------

def _with_grads(y, dy, ins):
    out = {"d" + n: g for n, g in zip(ins, torch.autograd.grad(y, list(ins.values()), dy))}
    out["y"] = y.detach()
    return out


SCAN_ARGS = ("q", "k", "v", "adt", "dt", "trap", "qb", "kb", "psi", "zeta", "phi", "angles", "d", "z")


def run(s):
    kind = s["kind"]
    if kind == "linear":
        return _with_grads(F_.linear(s["x"], s["w"]), s["dy"], {"x": s["x"], "w": s["w"]})
    if kind == "mxfp8":
        with F_.precision_scope("mxfp8"):
            y = F_.linear(s["x"], s["w"])
        return _with_grads(y, s["dy"], {"x": s["x"], "w": s["w"]})
    if kind == "experts":
        e = s["experts"]
        y = s["dispatch"](s["x"], s["p"], s["ids"], e)
        return _with_grads(y, s["dy"], {"x": s["x"], "p": s["p"], "w1": e.weight1, "w2": e.weight2})
    if kind == "scan":
        y = F_.mimo_scan(*[s["ins"][n] for n in SCAN_ARGS], 4, 16)
        return _with_grads(y, s["dy"], s["ins"])
    if kind == "attention":
        return _with_grads(F_.causal_attention(s["q"], s["k"], s["v"], 128 ** -0.5), s["dy"], {n: s[n] for n in "qkv"})
    if kind == "sparse":
        return _with_grads(F_.sparse_mla(s["q"], s["kv"], s["idx"], 128 ** -0.5, 64), s["dy"], {"q": s["q"], "kv": s["kv"]})
    if kind == "m2rnn":
        return _with_grads(F_.m2rnn_scan(s["q"], s["k"], s["v"], s["w"], s["f"]), s["dy"], {n: s[n] for n in "qkvwf"})
    if kind == "loss":
        total, per_token = F_.linear_cross_entropy_weighted(s["x"], s["w"], s["labels"], s["weights"])
        dx, dw = torch.autograd.grad(total, [s["x"], s["w"]])
        return dict(y=total.detach(), per_token=per_token, dx=dx, dw=dw)
    return _with_grads(F_.rmsnorm(s["x"], s["w"], 1e-5), s["dy"], {"x": s["x"], "w": s["w"]})


# ---- what a pass cannot do without ------------------------------------------------------------------------------------

def work(case):
    c, kind = types.SimpleNamespace(**case), case["kind"]
    if kind in ("linear", "mxfp8"):
        return dict(bytes=2 * 2 * (c.tokens * c.k + c.tokens * c.n + c.n * c.k), flops=6.0 * c.tokens * c.k * c.n)
    if kind == "experts":
        weights, act = c.experts * 3 * c.ffn * c.hidden, c.tokens * c.hidden
        return dict(bytes=2 * (2 * weights + 4 * act) + 16 * c.tokens * c.topk, flops=18.0 * c.tokens * c.topk * c.hidden * c.ffn)
    if kind == "scan":
        tok = c.batch * c.seq
        qk, vz, ang, head = tok * c.groups * 4 * c.state, tok * c.heads * 64, tok * c.heads * c.state // 4, tok * c.heads
        # per token and head: state read-out and update, both twice more in the backward, and the rank-4 products
        return dict(bytes=2 * 2 * 2 * qk + 2 * 6 * vz + 4 * 2 * ang + 4 * 6 * head, flops=tok * c.heads * 4 * c.state * 64 * 12.0)
    if kind == "attention":
        n = c.batch * c.seq * c.heads
        return dict(bytes=2 * (4 * n * 128 + 4 * n * 64), flops=n * c.seq / 2 * 2.0 * (128 + 64 + 3 * 128 + 2 * 64))
    if kind == "sparse":
        n = c.batch * c.seq
        return dict(bytes=2 * n * (2 * 32 * 128 + 2 * 32 * 64 + 2 * 128) + 4 * n * 256, flops=n * 256 * 32 * 2.0 * (128 + 64 + 3 * 128 + 2 * 64))
    if kind == "m2rnn":
        n = c.batch * c.seq
        # per step and head the product of the 64 x 16 state with the 16 x 16 matrix, once forward and twice back, and the rank-1 terms
        return dict(bytes=2 * n * (4 * 64 + 4 * c.heads * 16) + 8 * n * c.heads, flops=n * c.heads * 64 * 16 * (2.0 * 16 * 3 + 20))
    if kind == "loss":
        return dict(bytes=4 * (c.tokens + c.vocab) * c.hidden, flops=6.0 * c.tokens * c.hidden * c.vocab)
    return dict(bytes=2 * 4 * c.rows * c.width, flops=12.0 * c.rows * c.width)


def tolerance(case):
    return TOLERANCE[case["kind"]]


# About four times the largest error of an output against its 64-bit value: one bf16 rounding of each result is 1.7e-3; the experts round
# the hidden activations and every expert's output as well, the attention and scan kernels their probabilities, scores and states.
TOLERANCE = {
    "linear": {"rel": 7e-3},
    "mxfp8": {"rel": 7e-3},
    "experts": {"rel": 1.6e-2},
    "scan": {"rel": 1.4e-2},
    "attention": {"rel": 1e-2},
    "sparse": {"rel": 1e-2},
    "m2rnn": {"rel": 7e-3},
    "loss": {"rel": 7e-3},
    "norm": {"rel": 7e-3},
}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------

def _d(t):
    return t.detach().double()


def exact(case, seed):
    s = prepare(case, seed)
    return globals()["_exact_" + case["kind"]](s)


def _exact_linear(s):
    x, w, dy = _d(s["x"]), _d(s["w"]), _d(s["dy"])
    return dict(y=x @ w.t(), dx=dy @ w, dw=dy.t() @ x)


def _mx(t, axis):
    """The MXFP8 rounding of a tensor along ``axis``: E4M3 values with one power of two per 32 of them."""
    u = t.detach().float().movedim(axis, -1)
    blk = u.reshape(*u.shape[:-1], -1, 32)
    amax = blk.abs().amax(-1, keepdim=True).double()
    e = torch.where(amax > 0, torch.ceil(torch.log2(amax.clamp_min(1e-38) / 448.0)), torch.zeros_like(amax)).clamp(-126, 127)
    q = (blk.double() * torch.exp2(-e)).clamp(-448, 448).float().to(torch.float8_e4m3fn).double() * torch.exp2(e)
    return q.reshape(u.shape).movedim(-1, axis)


def _exact_mxfp8(s):
    x, w, dy = s["x"], s["w"], s["dy"]
    return dict(y=_mx(x, 1) @ _mx(w, 1).t(), dx=_mx(dy, 1) @ _mx(w, 0), dw=_mx(dy, 0).t() @ _mx(x, 0))


def _exact_experts(s):
    x, p, dy, ids = _d(s["x"]), _d(s["p"]), _d(s["dy"]), s["ids"]
    y, dx, dp = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(p)
    dw1, dw2 = [], []
    for e in range(s["experts"].weight1.shape[0]):
        w1, w2 = _d(s["experts"].weight1[e]), _d(s["experts"].weight2[e])
        tok, slot = torch.nonzero(ids == e, as_tuple=True)
        xe, pe, ge = x[tok], p[tok, slot].unsqueeze(1), dy[tok]
        h = xe @ w1.t()
        a, b = h.chunk(2, dim=1)
        sg = torch.sigmoid(a)
        act = a * sg * b
        o = act @ w2.t()
        y.index_add_(0, tok, pe * o)
        dp[tok, slot] = (ge * o).sum(1)
        go = pe * ge
        dact = go @ w2
        dh = torch.cat([dact * b * sg * (1 + a * (1 - sg)), dact * a * sg], dim=1)
        dw2.append(go.t() @ act)
        dw1.append(dh.t() @ xe)
        dx.index_add_(0, tok, dh @ w1)
    return dict(y=y, dx=dx, dp=dp, dw1=torch.stack(dw1), dw2=torch.stack(dw2))


def _scan_heads(q, k, v, adt, dt, trap, qb, kb, psi, zeta, phi, angles, d, z, L=32):
    """One head group: q, k [B,S,R,N]; v, z [B,S,h,P]; adt, dt, trap [B,h,S]; angles [B,S,h,N/4].  Blocks of ``L`` tokens."""
    B, S, R, N = q.shape
    h, P, C = v.shape[2], v.shape[3], S // L

    def turned(t, bias):
        t = t.unsqueeze(2) + bias                                               # [B,S,h,R,N]
        n, half = N // 4, N // 2
        cs, sn = torch.cos(angles).unsqueeze(3), torch.sin(angles).unsqueeze(3)
        a, b = t[..., :n], t[..., half:half + n]
        return torch.cat([cs * a - sn * b, t[..., n:half], sn * a + cs * b, t[..., half + n:]], dim=-1)

    def blocks(t):                                                              # [B,S,h,R,*] -> [B,h,C,L,R,*]
        return t.reshape(B, C, L, h, R, -1).permute(0, 3, 1, 2, 4, 5)

    qq, kk, vv = blocks(turned(q, qb)), blocks(turned(k, kb)), blocks(v.unsqueeze(3) * psi)
    gamma = dt * torch.sigmoid(trap)
    after = dt * torch.sigmoid(-trap)
    ts = (gamma + torch.cat([after[..., 1:], torch.zeros_like(after[..., :1])], dim=-1)).reshape(B, h, C, L)
    gamma = gamma.reshape(B, h, C, L)
    cs = torch.cumsum(adt.reshape(B, h, C, L), dim=-1)
    low = torch.ones(L, L, dtype=torch.bool, device=q.device).tril(-1)
    fall = torch.exp((cs.unsqueeze(-1) - cs.unsqueeze(-2)).masked_fill(~low, -math.inf)) * ts.unsqueeze(-2)
    fall = fall + torch.diag_embed(gamma)                                       # [B,h,C,i,j]: weight of token j in the output of token i
    rows = lambda t: t.reshape(B, h, C, L * R, -1)  # noqa: E731
    score = rows(qq) @ rows(kk).transpose(-1, -2)
    score = score.reshape(B, h, C, L, R, L, R) * fall.reshape(B, h, C, L, 1, L, 1)
    o = score.reshape(B, h, C, L * R, L * R) @ rows(vv)
    carry = (ts * torch.exp(cs[..., -1:] - cs)).reshape(B, h, C, L, 1, 1)
    local = rows(kk * carry).transpose(-1, -2) @ rows(vv)                       # [B,h,C,N,P]
    state, starts = torch.zeros_like(local[:, :, 0]), []
    for c in range(C):
        starts.append(state)
        state = state * torch.exp(cs[:, :, c, -1])[..., None, None] + local[:, :, c]
    o = o + rows(qq * torch.exp(cs).reshape(B, h, C, L, 1, 1)) @ torch.stack(starts, dim=2)
    o = o.reshape(B, h, C, L, R, P).permute(0, 2, 3, 1, 4, 5).reshape(B, S, h, R, P) + d.reshape(h, 1, 1) * (v.unsqueeze(3) * psi)
    zz = z.unsqueeze(3) * zeta
    return (o * zz * torch.sigmoid(zz) * phi).sum(3)


def _exact_scan(s):
    ins = {n: _d(t) for n, t in s["ins"].items()}
    dy = _d(s["dy"])
    G, H = ins["q"].shape[3], ins["v"].shape[2]
    axis = dict(v=2, adt=1, dt=1, trap=1, qb=0, kb=0, psi=0, zeta=0, phi=0, angles=2, d=0, z=2)
    parts = []
    for g in range(G):
        part = {}
        for n in SCAN_ARGS:
            t = ins[n].select(3, g) if n in "qk" else ins[n].narrow(axis[n], g * (H // G), H // G)
            part[n] = t.clone().requires_grad_()
        y = _scan_heads(*[part[n] for n in SCAN_ARGS])
        grads = torch.autograd.grad(y, [part[n] for n in SCAN_ARGS], dy.narrow(2, g * (H // G), H // G))
        parts.append((y.detach(), grads))
    out = dict(y=torch.cat([y for y, _ in parts], dim=2))
    for i, n in enumerate(SCAN_ARGS):
        grads = [p[i] for _, p in parts]
        out["d" + n] = torch.stack(grads, dim=3) if n in "qk" else torch.cat(grads, dim=axis[n])
    return out


def _exact_attention(s):
    q, k, v, dy = (_d(s[n]) for n in ("q", "k", "v", "dy"))
    y, dq, dk, dv = torch.empty_like(v), torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    S, scale = q.shape[1], 128 ** -0.5
    future = torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1)
    for b in range(q.shape[0]):
        for h in range(q.shape[2]):
            qh, kh, vh, gh = q[b, :, h], k[b, :, h], v[b, :, h], dy[b, :, h]
            p = torch.softmax((qh @ kh.t() * scale).masked_fill_(future, -math.inf), dim=-1)
            o = p @ vh
            ds = p * (gh @ vh.t() - (gh * o).sum(1, keepdim=True)) * scale
            y[b, :, h], dv[b, :, h], dq[b, :, h], dk[b, :, h] = o, p.t() @ gh, ds @ kh, ds.t() @ qh
    return dict(y=y, dq=dq, dk=dk, dv=dv)


def _exact_sparse(s):
    q, kv, dy, idx = _d(s["q"]), _d(s["kv"]), _d(s["dy"]), s["idx"].long()
    y, dq, dkv, scale = torch.empty_like(dy), torch.empty_like(q), torch.zeros_like(kv), 128 ** -0.5
    for b in range(q.shape[0]):
        for i in range(0, q.shape[1], 512):
            at = slice(i, min(i + 512, q.shape[1]))
            sel = idx[b, at]
            rows = kv[b][sel.clamp_min(0)]                                      # [n,256,128]
            p = torch.softmax((q[b, at] @ rows.transpose(1, 2) * scale).masked_fill((sel < 0).unsqueeze(1), -math.inf), dim=-1)
            o = p @ rows[..., :64]
            ds = p * (dy[b, at] @ rows[..., :64].transpose(1, 2) - (dy[b, at] * o).sum(-1, keepdim=True)) * scale
            y[b, at], dq[b, at] = o, ds @ rows
            drows = ds.transpose(1, 2) @ q[b, at]
            drows[..., :64] += p.transpose(1, 2) @ dy[b, at]
            dkv[b].index_add_(0, sel.clamp_min(0).reshape(-1), drows.masked_fill((sel < 0).unsqueeze(-1), 0.0).reshape(-1, 128))
    return dict(y=y, dq=dq, dkv=dkv)


def _exact_m2rnn(s):
    ins = {n: _d(s[n]).requires_grad_() for n in "qkvwf"}
    q, k, v, w, f = (ins[n] for n in "qkvwf")
    B, S, H = f.shape
    h, ys = torch.zeros(B, H, 64, 16, dtype=torch.float64, device=q.device), []
    qt, kt, vt, ft = q.unbind(1), k.unbind(1), v.unbind(1), f.unbind(1)
    for t in range(S):
        new = torch.tanh(h @ w + kt[t].unsqueeze(-1) * vt[t].unsqueeze(-2))
        h = new + ft[t][..., None, None] * (h - new)
        ys.append((qt[t].unsqueeze(2) @ h).squeeze(2))
    return _with_grads(torch.stack(ys, dim=1), _d(s["dy"]), ins)


def _exact_loss(s):
    w, labels, weights = _d(s["w"]), s["labels"], _d(s["weights"])
    per_token, dx, dw = torch.zeros_like(weights), [], torch.zeros_like(w)
    for i in range(0, labels.numel(), 1024):
        x, lab = _d(s["x"][i:i + 1024]), labels[i:i + 1024]
        p = torch.log_softmax(x @ w.t(), dim=-1)
        at = torch.arange(lab.numel(), device=w.device)
        per_token[i:i + 1024] = -p[at, lab.clamp_min(0)] * (lab >= 0)
        p.exp_()
        p[at, lab.clamp_min(0)] -= 1
        p *= (weights[i:i + 1024] * (lab >= 0)).unsqueeze(1)
        dx.append(p @ w)
        dw.addmm_(p.t(), x)
    return dict(y=(per_token * weights).sum(), per_token=per_token, dx=torch.cat(dx), dw=dw)


def _exact_norm(s):
    ins = {n: _d(s[n]).requires_grad_() for n in "xw"}
    x, w = ins["x"], ins["w"]
    return _with_grads(x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w, _d(s["dy"]), ins)
