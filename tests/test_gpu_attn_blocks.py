"""Prompt attention on tensor memory (csrc/attn_tc05.cu): launches whose blocks of rows have two tiles, one, or the first ones two and the late ones one."""
import pytest
import torch

from tests.test_gpu_kernels import K, _attn_exact  # noqa: F401

pytestmark = pytest.mark.gpu


# tiles of 128 rows per head x heads, against 148 SMs: one each; a pair and ones; as many pairs as go; all pairs and a last one alone; several rounds
@pytest.mark.parametrize("H,G,T,start", [(40, 40, 300, 0), (40, 10, 500, 33), (32, 8, 613, 130), (32, 8, 640, 5), (74, 2, 385, 64), (50, 50, 641, 0), (149, 1, 257, 1)])
@pytest.mark.parametrize("hs", [64, 128])
def test_blocks_of_rows(K, H, G, T, start, hs):  # noqa: F811
    g = torch.Generator().manual_seed(T + H)
    S = start + T
    q = torch.randn(1, H, T, hs, generator=g).to(torch.bfloat16)
    k, v = (torch.randn(1, G, S, hs, generator=g).to(torch.bfloat16) for _ in range(2))
    pos = torch.arange(start, S)
    y = K.attn_prefill(q.cuda(), k.cuda(), v.cuda(), pos.cuda()).cpu().view(T, H, hs)
    of = [h // (H // G) for h in range(H)]   # every head, so that no block of rows can stand in for another's
    want = _attn_exact(q[0].transpose(0, 1), k[0, of].transpose(0, 1), v[0, of].transpose(0, 1), pos, torch.zeros(T), hs ** -0.5).view(T, H, hs)
    # weights and result rounded to bf16: two halves of a unit, the weights' as their root mean square over the keys at most; of a head, whichever
    err = ((y.double() - want).norm(dim=(0, 2)) / want.norm(dim=(0, 2))).max()
    assert err <= 2.0 ** -8, err
