"""Decaying linear attention with decays per channel, long prompts in pieces by matrix products: sizes off the tiles, partial pieces, several sequences, a state to
start from, rows that are not 16-byte aligned, numbers that are not finite, and a workspace that only the walk fits into."""

import pytest
import torch

from lit_gpt_b200 import _cabi as C
from lit_gpt_b200 import kernels as K

pytestmark = pytest.mark.gpu


def _exact(q, k, v, z, b, state, seqs, H, dk, dv, tau, scale, act):
    d = lambda t: t.detach().cpu().double()
    f = torch.nn.functional.silu if act else (lambda t: t)
    n = q.size(0)
    g = torch.exp(torch.nn.functional.logsigmoid(d(z) + d(b)) / tau).view(n, H, dk)
    qq, kk, vv = f(d(q)).view(n, H, dk) * scale, f(d(k)).view(n, H, dk), f(d(v)).view(n, H, dv)
    out, states = torch.zeros(n, H, dv, dtype=torch.float64), d(state).view(-1, H, dk, dv).clone()
    for first, rows, start, slot in seqs:
        S = states[slot] if start else torch.zeros(H, dk, dv, dtype=torch.float64)
        for t in range(first, first + rows):
            S = S * g[t][:, :, None] + kk[t][:, :, None] * vv[t][:, None]
            out[t] = torch.einsum("hij,hi->hj", S, qq[t])
        states[slot] = S
    return out.view(n, -1), states.view(states.size(0), -1)


def _inputs(lens, H, dk, dv, dtype, pad=0, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = sum(lens)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    w = H * (2 * dk + dv) + pad   # (the projections' columns of one row, as a layer slices them)
    p = r(n, w).to(dtype)
    q, k, v = p[:, pad : pad + H * dk], p[:, pad + H * dk : pad + 2 * H * dk], p[:, pad + 2 * H * dk :]
    z, b = r(n, H * dk), (torch.rand(H * dk, device="cuda", generator=gen) * 3).to(dtype)
    seqs, at = [], 0
    for i, m in enumerate(lens):
        seqs.append((at, m, 64 if i % 2 else 0, i))
        at += m
    return q, k, v, z, b, r(len(lens), H * dk * dv), seqs


CASES = [  # (lens, heads, dk, dv, dtype, act, pad); all but the last two are within the rule for pieces
    ((128,), 64, 128, 128, torch.bfloat16, False, 0),
    ((1025,), 8, 128, 128, torch.bfloat16, True, 0),
    ((1151, 1, 200), 8, 128, 128, torch.float32, False, 0),
    ((2048,), 4, 100, 200, torch.bfloat16, False, 3),
    ((1400,), 10, 97, 101, torch.float32, True, 1),
    ((1024,), 4, 64, 64, torch.bfloat16, False, 0),
    ((65, 700, 64), 8, 50, 97, torch.bfloat16, True, 0),
    ((1023,), 8, 128, 128, torch.bfloat16, False, 0),   # the walk: one row too few
    ((4800,), 4, 64, 64, torch.bfloat16, False, 0),     # the walk: half empty tiles in more than one wave
]


@pytest.mark.parametrize("lens,H,dk,dv,dtype,act,pad", CASES)
def test_linear_pieces(lens, H, dk, dv, dtype, act, pad):
    q, k, v, z, b, state, seqs = _inputs(lens, H, dk, dv, dtype, pad)
    want, want_s = _exact(q, k, v, z, b, state, seqs, H, dk, dv, 16.0, dk**-0.5, act)
    out = K.linear_attn(q, k, v, state, torch.tensor(seqs, dtype=torch.int32, device="cuda"), max(lens), H, dk, dv, silu=act, q_scale=dk**-0.5,
                        decay_in=z.clone(), decay_bias=b, tau=16.0)
    # fp32 products and sums: the decays' product over the ~1 / (1 - g) <= 2^6 tokens that count rounds by 2^-24 each, and as much again in the sums;
    # an activation of 16-bit numbers is good to 2^-21 of each factor, three of them in a product
    tol = 2**-17 + (3 * 2**-21 if act and dtype != torch.float32 else 0.0)
    for got, exact in ((out, want), (state, want_s)):
        assert ((got.cpu().double() - exact).norm() / exact.norm()).item() <= tol


def test_linear_pieces_nothing_of_later_tokens():
    H, D, n, at = 8, 128, 1100, 700
    q, k, v, z, b, state, seqs = _inputs((n,), H, D, D, torch.bfloat16)
    seqs_t = torch.tensor(seqs, dtype=torch.int32, device="cuda")
    run = lambda: K.linear_attn(q, k, v, torch.zeros_like(state), seqs_t, n, H, D, D, q_scale=1.0, decay_in=z.clone(), decay_bias=b, tau=16.0)
    clean = run()
    v[at, 5], k[at + 1, D + 7], q[at + 2, 3] = float("inf"), float("nan"), float("nan")
    got = run()
    assert torch.isfinite(got[:at]).all()
    # (a piece with such a number sums B v in order; the others as before)
    assert (got[:at] - clean[:at]).abs().max().item() <= 2**-17 * clean.abs().max().item()
    assert not torch.isfinite(got[at:, 5]).any() and torch.isnan(got[at + 1 :, D : 2 * D]).all()
    assert torch.isnan(got[at + 2, :D]).all()
    other = torch.ones(D, dtype=torch.bool, device="cuda")
    other[5] = False
    assert torch.isfinite(got[at + 3 :, :D][:, other]).all() and torch.isfinite(got[:, 2 * D :]).all()


def test_linear_pieces_workspace(monkeypatch):
    """Pieces by products are only taken where the workspace holds them; what the walk needs is enough."""
    need = lambda rows, heads, dk, dv: C.load_core().b200_linear_attn_workspace_bytes(rows, rows, 1, heads, dk, dv)
    pieces = lambda rows, heads, dk, dv: 4 * ((((rows + 63) // 64) * heads * dk * (dv + 1) + 3) // 4 * 4 + rows * heads * dk)
    assert need(2048, 8, 128, 128) == pieces(2048, 8, 128, 128)
    assert need(1023, 8, 128, 128) != pieces(1023, 8, 128, 128) and need(2048, 8, 32, 32) != pieces(2048, 8, 32, 32)
    q, k, v, z, b, state, seqs = _inputs((2048,), 8, 128, 128, torch.bfloat16)
    seqs_t, size = torch.tensor(seqs, dtype=torch.int32, device="cuda"), []
    run = lambda: K.linear_attn(q, k, v, torch.zeros_like(state), seqs_t, 2048, 8, 128, 128, decay_in=z.clone(), decay_bias=b, tau=16.0)
    old = K.linear_attn_tune(48)   # (the walk, in the pieces that it takes for this size on 148 SMs)
    try:
        walked = run()
    finally:
        K.linear_attn_tune(old)
    monkeypatch.setattr(K, "_ws", lambda tag, device, nbytes: size.append(nbytes) or torch.empty(nbytes // 4 - 64, dtype=torch.float32, device=device))
    assert torch.equal(run(), walked) and size == [pieces(2048, 8, 128, 128)]
