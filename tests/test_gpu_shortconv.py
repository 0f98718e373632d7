"""Short convolution with four taps on heads that lie on 16-byte boundaries (csrc/shortconv.cu: short_conv8_kernel) against the same sums in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TAPS = 4


def _reference(x, w, tail, seqs, col0, heads, dim, act, post, fr, rot, mscale, scale, eps):
    """(rows, heads, dim) in 64 bits, and what an element's rounding errors are measured by: its row's largest sum of magnitudes"""
    cols = slice(col0, col0 + heads * dim)
    out, mag = [], []
    for first, n, start, slot in seqs:
        before = torch.cat([torch.zeros(TAPS - 1, heads * dim, dtype=torch.float64), tail[slot][:, cols].double()])[-(TAPS - 1):]
        before[: max(0, TAPS - 1 - start)] = 0
        u = torch.cat([before, x[first : first + n, cols].double()])
        terms = torch.stack([u[j : j + n] * w[:, j].double() for j in range(TAPS)])
        y, m = terms.sum(0).view(n, heads, dim), terms.abs().sum(0).view(n, heads, dim).amax(-1, keepdim=True)
        if act:
            y = y * torch.sigmoid(y)
        if post == 1:
            ang = torch.arange(start, start + n, dtype=torch.float64)[:, None, None] * fr[: rot // 2]
            a, b = y[..., 0:rot:2], y[..., 1:rot:2]
            c, s = torch.cos(ang) * mscale, torch.sin(ang) * mscale
            y = torch.cat([torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2), y[..., rot:]], -1)
        mul = torch.full_like(m, scale)
        if post:
            mul = scale * (y.square().sum(-1, keepdim=True) / (dim if post == 1 else 1) + eps).rsqrt()
        out.append(y * mul)
        mag.append(m * mul)
    return torch.cat(out), torch.cat(mag)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("dim,hq,hk,rows", [(64, 8, 2, 1), (128, 16, 4, 37), (128, 5, 1, 403), (72, 8, 4, 1900), (256, 6, 3, 130), (200, 4, 12, 700), (8, 3, 3, 50)])
def test_short_conv_eight_channels(dtype, dim, hq, hk, rows):
    """Sequences that end anywhere in a strip of rows, begun before the step by fewer rows than there are taps, by more, or not at all; head counts that
    fill a CTA, divide it, or leave one head per CTA; groups of different activation, norm and output type."""
    from lit_gpt_b200 import kernels as K

    g = torch.Generator().manual_seed(rows + dim)
    cols = (hq + 2 * hk) * dim
    cuts = sorted({c for c in (0, 1, 2, 5, 11, 12, 30, rows // 3, rows // 2 + 3, rows - 2, rows) if 0 <= c <= rows})
    slots = torch.randperm(len(cuts) - 1, generator=g).tolist()
    seqs = [(a, b - a, (0, 700, 1, 2)[i % 4], slots[i]) for i, (a, b) in enumerate(zip(cuts, cuts[1:]))]
    x = torch.randn(rows, cols + 16, generator=g).to(dtype)
    w = (0.5 * torch.randn(cols, TAPS, generator=g)).to(dtype)
    tail = torch.randn(len(seqs), TAPS - 1, cols, generator=g).to(dtype)
    rot = min(dim, 64) // 2 * 2
    fr = 10000.0 ** (-torch.arange(0, rot // 2, dtype=torch.float64) / (rot // 2))
    q, k, v = (torch.empty(rows, h * dim, dtype=d, device="cuda") for h, d in ((hq, dtype), (hk, torch.float32), (hk, dtype)))
    wc, fc, c1, c2 = w.cuda(), fr.cuda(), hq * dim, (hq + hk) * dim
    groups = [K.conv_group(wc[:c1], q, 0, hq, dim, post=1, rot_dims=rot, inv_freq=fc, rot_mscale=1.1, eps=1e-5),
              K.conv_group(wc[c1:c2], k, c1, hk, dim, act=1, post=2, post_scale=0.25, eps=1e-6),
              K.conv_group(wc[c2:], v, c2, hk, dim, act=1)]
    row_seq = torch.cat([torch.full((n,), i, dtype=torch.int32) for i, (_, n, _, _) in enumerate(seqs)]).cuda()
    new_tail = tail.cuda()
    K.short_conv(x.cuda(), groups, TAPS, new_tail, torch.tensor(seqs, dtype=torch.int32).cuda(), row_seq)
    for got, col0, h, kw in ((q, 0, hq, (0, 1, fr, rot, 1.1, 1.0, 1e-5)), (k, c1, hk, (1, 2, fr, 0, 1.0, 0.25, 1e-6)), (v, c2, hk, (1, 0, fr, 0, 1.0, 1.0, 0.0))):
        ref, mag = _reference(x, w[col0 : col0 + h * dim], tail, seqs, col0, h, dim, *kw)
        # four products and their sums, the activation and the rotation: a few units of 2^-24 of the row's largest sum each; the norm's sum of `dim`
        # squares and its root act on the whole row; then the rounding to the output type
        half = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -24   # 8 and 24 significant bits
        err = (got.double().cpu().view(rows, h, dim) - ref).abs()
        assert (err <= 2.0 ** -19 * mag + 1.01 * half * ref.abs()).all(), float((err / mag).max())


def test_short_conv_extremes_of_silu():
    """Values whose exponential overflows or vanishes, infinities and NaN, as by x / (1 + exp(-x))."""
    from lit_gpt_b200 import kernels as K

    vals = torch.tensor([0.0, -0.0, 79.9, 80.1, -79.9, -80.1, -87.5, -88.8, -104.0, 1e30, -1e30, 3e38, float("inf"), float("-inf"), float("nan"), 1e-30])
    x = vals.repeat(8).view(1, 128).cuda()
    w = torch.zeros(128, 4)
    w[:, 3] = 1.0
    w, out = w.cuda(), torch.empty(1, 128, device="cuda")
    K.short_conv(x, [K.conv_group(w, out, 0, 2, 64, act=1)], 4, torch.zeros(1, 3, 128, device="cuda"),
                 torch.tensor([[0, 1, 0, 0]], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32, device="cuda"))
    want = (vals / (1 + torch.exp(-vals))).repeat(8)
    assert torch.equal(out.cpu()[0].isnan(), want.isnan())
    ok = ~want.isnan()
    assert torch.allclose(out.cpu()[0][ok], want[ok], rtol=4e-7, atol=1e-31)
