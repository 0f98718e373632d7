"""Gated norm per head (csrc/delta.cu): heads on both sides of what a lane, part of a warp and a warp hold, rows that allow wide accesses and rows that do not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dv", [1, 4, 6, 12, 60, 64, 68, 100, 128, 132, 252, 255, 256])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shift", [0, 1])
def test_gated_rms_heads(dv, dtype, shift):
    from lit_gpt_b200 import kernels as K

    n, H, g = 37, 5, torch.Generator().manual_seed(dv)
    o = torch.randn(n, H * dv + 8, generator=g)
    z = torch.randn(n, H * dv + 8, generator=g).to(dtype)
    w = torch.rand(dv, generator=g).to(dtype)
    at = slice(4 + shift, 4 + shift + H * dv)   # (a shift of one number: no 16-byte boundary)
    for gate, weight in ((K.GATE_SILU, w), (K.GATE_SIGMOID, None)):
        out = torch.full((n, H * dv + 8), 7.0, dtype=dtype, device="cuda")
        K.gated_rms_heads(o.cuda()[:, at], z.cuda()[:, at], None if weight is None else weight.cuda(), H, dv, gate, 1e-5, out_scale=-1.25, out=out[:, at])
        od, zd = o[:, at].double().view(n, H, dv), z[:, at].double().view(n, H, dv)
        want = od / torch.sqrt((od * od).mean(-1, keepdim=True) + 1e-5) * (1.0 if weight is None else weight.double()) * -1.25
        want = want * torch.sigmoid(zd) * (zd if gate == K.GATE_SILU else 1.0)
        got = out.cpu()
        # a dozen fp32 roundings, then the result's own
        tol = (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) + 16 * 2.0 ** -24
        assert ((got[:, at].double().view(n, H, dv) - want).abs() <= tol * want.abs() + 1e-37).all()
        assert (got[:, : at.start] == 7).all() and (got[:, at.stop :] == 7).all()
