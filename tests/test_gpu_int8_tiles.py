"""LLM.int8() prompts: the widths of tile that the plan picks (csrc/int8.cu: i8_features), their edges, and the list of outlier columns that the row
quantisation's first CTA makes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one row tile and two, features that end inside a tile, tiles of 64 to 256 features; more outlier columns than one and two groups of eight
@pytest.mark.parametrize("M,N,Kd,n_out", [(129, 4104, 128, 0), (300, 4096, 192, 3), (777, 1104, 64, 64), (513, 11008, 128, 6), (260, 6152, 256, 17), (129, 12288, 64, 0),
                                          (1030, 5632, 128, 9), (17, 264, 1088, 11), (16, 40, 8256, 5)])
def test_linear_int8_tile_widths(M, N, Kd, n_out):
    from lit_gpt_b200 import kernels as K

    g = torch.Generator().manual_seed(M + N)
    w, x = (torch.randn(N, Kd, generator=g) * 0.05).half(), torch.randn(M, Kd, generator=g).clamp_(-5.5, 5.5).half()
    cols = torch.randperm(Kd, generator=g)[:n_out]
    x[:, cols] *= 12
    x[torch.arange(n_out) % M, cols] = 7.0      # each of them an outlier column for certain
    b = torch.randn(N, generator=g).half()
    cb, scb = K.quantize_int8(w.cuda())
    y = K.linear_int8(x.cuda(), cb, scb, b.cuda()).double().cpu()
    xd, cbd = x.double(), cb.cpu().double()
    out = (x.abs() >= 6).any(0)
    xr = torch.where(out, torch.zeros((), dtype=torch.float64), xd)
    sca = xr.abs().amax(1, keepdim=True)
    ca = (xr.float() * (127 / sca).float()).nan_to_num(0.0).double().round()      # as the kernel: fp32 factor, fp32 product, nearest even
    scb_d = scb.cpu().double()
    main = (ca @ cbd.T) * (sca * scb_d / 127 ** 2)
    side = xd[:, out] @ (cbd[:, out] * (scb_d / 127)[:, None]).half().double().T
    ref = main + b.double() + side
    # integer products are exact; then three roundings to fp16 of numbers no larger than the parts, and the fp32 side product
    part = main.abs() + b.double().abs() + side.abs() + (xd[:, out].abs() @ cbd[:, out].abs().T) * (scb_d / 127) * 2.0 ** -12
    assert ((y - ref).abs() <= 4 * 2.0 ** -11 * part + 2.0 ** -14).all(), ((y - ref).abs() / part).max()
