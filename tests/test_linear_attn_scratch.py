"""Scratch of decaying linear attention (csrc/linear_attn.cu): bounded for long prompts and steps of many sequences, and what the kind of decay needs."""
import pytest
import torch

from lit_gpt_b200 import _cabi as C

MB = 1 << 20


def _bytes(lens, heads, dk, dv, channel):
    return C.load_core().b200_linear_attn_workspace_bytes_ex(sum(lens), max(lens), len(lens), heads, dk, dv, channel)


@pytest.mark.parametrize("lens", [[2048], [32768], [131072], [8192] + [1] * 63, [1000] * 20, [4000] + [1] * 500])
@pytest.mark.parametrize("heads,dk,dv", [(8, 128, 128), (4, 64, 64), (64, 128, 256)])
def test_scratch_bounded(lens, heads, dk, dv):
    assert 0 < _bytes(lens, heads, dk, dv, 1) <= max(256 * MB, _bytes(lens, heads, dk, dv, 0))
    if heads * dk * dv >= 8 * 128 * 128 and max(lens) >= 2048:   # pieces on the tensor cores: those of the rows there are, not the longest sequence's for every one
        rows = sum((n + 63) // 64 for n in lens)
        assert _bytes(lens, heads, dk, dv, 1) <= min(256 * MB, 4 * heads * dk * (dv + 1 + 64) * (rows + len(lens)) + 16)


def test_fixed_decays_need_the_walk_only():
    for lens in ([2048], [32768], [131072]):
        assert _bytes(lens, 8, 128, 128, 0) <= 32 * MB
    lib = C.load_core()
    assert lib.b200_linear_attn_workspace_bytes(2048, 2048, 1, 8, 128, 128) == max(_bytes([2048], 8, 128, 128, 0), _bytes([2048], 8, 128, 128, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("lens,heads,dk,dv", [([3000], 64, 128, 128), ([1500, 70, 1, 1400], 64, 128, 128), ([2690, 2700], 60, 120, 136)])
def test_several_launches_pass_the_state_on(lens, heads, dk, dv):
    """More pieces than one launch's scratch holds: the next launch starts from the states that the one before left in the slots."""
    from lit_gpt_b200 import kernels as K

    n, g = sum(lens), torch.Generator(device="cuda").manual_seed(heads)
    assert sum((m + 63) // 64 for m in lens) * heads * dk * (dv + 1 + 64) * 4 > 256 * MB
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)   # noqa: E731
    q, k, v, z, b = r(n, heads * dk), r(n, heads * dk), r(n, heads * dv), r(n, heads * dk), r(heads * dk) + 2
    state = r(len(lens), heads * dk * dv)
    seqs, at = [], 0
    for i, m in enumerate(lens):
        seqs.append((at, m, 5 * (i % 2), len(lens) - 1 - i))
        at += m
    seqs = torch.tensor(seqs, dtype=torch.int32, device="cuda")

    def run():
        S = state.clone()
        return K.linear_attn(q, k, v, S, seqs, max(lens), heads, dk, dv, q_scale=dk**-0.5, decay_in=z.clone(), decay_bias=b, tau=16.0), S

    got = run()
    old = K.linear_attn_tune(64)   # token by token in pieces of 64
    try:
        want = run()
    finally:
        K.linear_attn_tune(old)
    for x, y in zip(got, want):
        assert ((x.double() - y.double()).norm() / y.double().norm()).item() <= 2**-18   # fp32 on either side: see test_gpu_linear_pieces.py
