"""Python side of the fused Mamba3 MIMO scan backward: allocates and launches the kernels (a head count per group without a
reduction kernel is reduced by the tensor library)."""
from __future__ import annotations

import torch

from .. import functional as F_
from .kernels3 import LT, _as_bsgrn, token_strided


def mimo_bwd(saved, dy, states, tot):
    from . import lib, err_word, stream_ptr, _check
    Q, K, V, ADT, DT, Trap, Qb, Kb, Psi, Zeta, Phi, angles, D, Z = saved
    B, S, R, G, N = Q.shape
    H, P = V.shape[2], V.shape[3]
    C = S // LT
    dev = V.device
    hpg = H // G
    Qn, Kn = _as_bsgrn(Q), _as_bsgrn(K)
    f32 = lambda t: t.float().contiguous()
    ADTf, DTf, Trapf = f32(ADT), f32(DT), f32(Trap)
    dyc = dy.to(torch.bfloat16).contiguous()
    gbuf = torch.empty(B, H, C, N, P, dtype=torch.float32, device=dev)
    dend = torch.empty(B, H, C, N, P, dtype=torch.bfloat16, device=dev)
    dQh = torch.empty(B, S, H, R, N, dtype=torch.bfloat16, device=dev)
    dKh = torch.empty(B, S, H, R, N, dtype=torch.bfloat16, device=dev)
    dV = torch.empty(B, S, H, P, dtype=torch.bfloat16, device=dev)
    dZ = torch.empty(B, S, H, P, dtype=torch.bfloat16, device=dev)
    dAng = torch.empty(B, S, H, N // 4, dtype=torch.float32, device=dev)
    dADT = torch.empty(B, H, S, dtype=torch.float32, device=dev)
    dTs = torch.empty(B, H, S, dtype=torch.float32, device=dev)
    dGam = torch.empty(B, H, S, dtype=torch.float32, device=dev)
    alloc = torch.empty if B * S else torch.zeros                                  # nothing is launched for an empty batch
    e32 = lambda *shape: alloc(*shape, dtype=torch.float32, device=dev)
    dPsi, dZeta, dPhi, dD = e32(H, R, P), e32(H, R, P), e32(H, R, P), e32(H)      # zeroed by the first kernel
    dDT, dTrap = e32(B, H, S), e32(B, H, S)
    grouped = hpg in (1, 2, 4, 8, 16)
    if grouped:     # heads -> groups (Q/K are shared by the heads of a group) and per-head biases, one pass per tensor
        dQg, dKg = (torch.empty(B, S, G, R, N, dtype=torch.bfloat16, device=dev) for _ in range(2))
        dQb, dKb = e32(H, R, N), e32(H, R, N)
    Vs, ldV = token_strided(V)
    Zs, ldZ = token_strided(Z)
    ins = [Qn, Kn, Vs, Zs, dyc, ADTf, DTf, Trapf, f32(Qb), f32(Kb), f32(Psi), f32(Zeta), f32(Phi),
           f32(angles), f32(D), states, tot]
    outs = [gbuf, dend, dQh, dKh, dV, dZ, dAng, dADT, dTs, dGam, dPsi, dZeta, dPhi, dD, dDT, dTrap]
    reduced = [t.data_ptr() for t in (dQg, dKg, dQb, dKb)] if grouped else [None] * 4
    _check(lib().cm_mimo_scan_bwd(*[t.data_ptr() for t in ins], *[t.data_ptr() for t in outs], *reduced, B, S, H, G, N, ldV, ldZ,
                                  err_word(dev).data_ptr(), stream_ptr()), "cm_mimo_scan_bwd")
    F_.count_launch("mimo_scan_bwd", 3)
    del gbuf, dend
    if grouped:
        F_.count_launch("head_reduce", 2)
        dQ, dK = dQg.permute(0, 1, 3, 2, 4), dKg.permute(0, 1, 3, 2, 4)
    else:
        dQ = dQh.view(B, S, G, hpg, R, N).sum(3, dtype=torch.float32).permute(0, 1, 3, 2, 4)
        dK = dKh.view(B, S, G, hpg, R, N).sum(3, dtype=torch.float32).permute(0, 1, 3, 2, 4)
        dQb = dQh.sum((0, 1), dtype=torch.float32)
        dKb = dKh.sum((0, 1), dtype=torch.float32)
    del dQh, dKh
    return (dQ.to(Q.dtype), dK.to(K.dtype), dV.to(V.dtype), dADT.to(ADT.dtype), dDT.to(DT.dtype), dTrap.to(Trap.dtype),
            dQb.to(Qb.dtype), dKb.to(Kb.dtype), dPsi.to(Psi.dtype), dZeta.to(Zeta.dtype), dPhi.to(Phi.dtype),
            dAng.to(angles.dtype), dD.to(D.dtype), dZ.to(Z.dtype))
