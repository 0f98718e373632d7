"""Long prompts of decaying linear attention in pieces by matrix products (csrc/linear_chunk.cuh): infinities and NaN come out where the walk has them, and as what they
are, and nowhere else."""
import pytest
import torch

from lit_gpt_b200 import kernels as K

pytestmark = pytest.mark.gpu

H, DK, DV, N, HEAD = 8, 128, 128, 1100, 3
INF, NAN = float("inf"), float("nan")


@pytest.mark.parametrize("dtype,silu", [(torch.bfloat16, False), (torch.float32, False), (torch.bfloat16, True)])
@pytest.mark.parametrize("what,at,value", [("k", 0, INF), ("k", 77, -INF), ("k", 1099, INF), ("q", 300, INF), ("q", 65, NAN), ("v", 130, INF), ("v", 639, -INF), ("z", 200, NAN),
                                           ("state", 0, INF), ("state", 0, NAN), ("k+q", 511, INF)])
def test_infinities_as_the_walk_has_them(what, at, value, dtype, silu):
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)   # noqa: E731
    p, z, b, state = r(N, H * (2 * DK + DV)).to(dtype), r(N, H * DK), (r(H * DK) + 2).to(dtype), r(1, H * DK * DV)
    q, k, v = p[:, : H * DK], p[:, H * DK : 2 * H * DK], p[:, 2 * H * DK :]
    col = HEAD * DK + 17
    for name in what.split("+"):
        if name == "state":
            state.view(H, DK, DV)[HEAD, 17, 40] = value
        else:
            {"q": q, "k": k, "v": v, "z": z}[name][at, col] = value
    seqs = torch.tensor([(0, N, 9, 0)], dtype=torch.int32, device="cuda")

    def run():
        S = state.clone()
        return K.linear_attn(q, k, v, S, seqs, N, H, DK, DV, silu=silu, q_scale=DK**-0.5, decay_in=z.clone(), decay_bias=b, tau=16.0), S

    got = run()
    old = K.linear_attn_tune(64)   # token by token in pieces of the same tokens
    try:
        want = run()
    finally:
        K.linear_attn_tune(old)
    for x, y in zip(got, want):
        fine = torch.isfinite(y)
        assert torch.equal(torch.isfinite(x), fine) and torch.equal(torch.isnan(x), torch.isnan(y)) and torch.equal(torch.sign(x[~fine].nan_to_num(0.0)), torch.sign(y[~fine].nan_to_num(0.0)))
        d = (x - y)[fine].double()
        assert (d.norm() / y[fine].double().norm()).item() <= 2**-17   # fp32 on either side: see test_gpu_linear_pieces.py
