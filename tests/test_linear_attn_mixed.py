"""Steps of decaying linear attention with decays per channel that mix prompts with single rows and short portions (csrc/linear_attn.cu: la_chunks): which way they go,
and that short sequences in a launch of their own come out as in the walk of all of them."""
import pytest
import torch

from lit_gpt_b200 import _cabi as C


def _pieces(lens, heads, dk, dv):
    """Whether a step goes in pieces on the tensor cores: its scratch then is not the walk's."""
    size = lambda channel: C.load_core().b200_linear_attn_workspace_bytes_ex(sum(lens), max(lens), len(lens), heads, dk, dv, channel)   # noqa: E731
    return size(1) != size(0)


def test_single_rows_make_no_prompt_longer():
    for singles in (0, 4, 24, 128):
        assert not _pieces([1000] + [1] * singles, 8, 128, 128)   # (the walk alone; 1024 rows are not)
        assert _pieces([2048] + [1] * singles, 8, 128, 128)
    assert _pieces([1024], 8, 128, 128) and not _pieces([1] * 2000, 8, 128, 128)
    assert not _pieces([1300], 4, 64, 64) and _pieces([2048], 4, 64, 64) and _pieces([2048] + [1] * 4, 4, 64, 64) and not _pieces([2048] + [1] * 24, 4, 64, 64)


@pytest.mark.gpu
@pytest.mark.parametrize("lens,heads,dk,dv", [
    ([1300] + [1] * 24, 8, 128, 128),              # single rows by the walk, in a launch of their own
    ([1] * 9 + [15, 16, 17, 900, 2, 64, 1, 700, 3] + [1] * 12, 8, 128, 128),
    ([2048] + [1] * 3, 8, 128, 128),               # in tiles, in the last wave
    ([1900] + [1] * 70, 4, 64, 64),
    ([1800], 4, 64, 64),
    ([5, 1500] + [1, 7] * 20, 10, 96, 104),
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_mixed_steps(lens, heads, dk, dv, dtype):
    from lit_gpt_b200 import kernels as K

    assert _pieces(lens, heads, dk, dv)
    n, g = sum(lens), torch.Generator(device="cuda").manual_seed(len(lens))
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)   # noqa: E731
    q, k, v, z, b = r(n, heads * dk).to(dtype), r(n, heads * dk).to(dtype), r(n, heads * dv).to(dtype), r(n, heads * dk), (r(heads * dk) + 2).to(dtype)
    state = r(len(lens) + 1, heads * dk * dv)
    seqs, at = [], 0
    for i, m in enumerate(lens):
        seqs.append((at, m, 0 if i % 3 == 1 else 7 * i, len(lens) - i))
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
    for first, m, _, slot in seqs.tolist():   # no sequence's rows or state far off for the others' sake
        assert ((got[0][first : first + m] - want[0][first : first + m]).norm() <= 2**-16 * want[0][first : first + m].norm()).item()
        assert ((got[1][slot] - want[1][slot]).norm() <= 2**-16 * want[1][slot].norm()).item()
    assert torch.equal(got[1][0], state[0])
