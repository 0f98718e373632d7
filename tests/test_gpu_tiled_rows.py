"""``qgemv_tiled_rows``, the short wrapper of a plain 4-bit Linear: the same call as ``qgemv_tiled`` makes, and the same refusals."""
import pytest
import torch

from lit_gpt_b200 import _cabi as C
from lit_gpt_b200 import kernels as K
from tests.test_gpu_kernels import _gemv_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qt", ["nf4", "fp4", "int4"])
@pytest.mark.parametrize("N,Kdim,B,fold", [(512, 4096, 1, 1), (1024, 5120, 3, 1), (2048, 4096, 16, 1), (4096, 1376, 4, 2), (64, 48, 2, 4)])
def test_same_call_as_the_general_wrapper(qt, N, Kdim, B, fold):
    if fold > 1 and qt == "int4":
        pytest.skip("int4 groups end with a row: nothing to fold")
    _, x, packed, scale, bs, _ = _gemv_case(K, N, Kdim, B, qt, seed=N + B)
    tiled, x = K.tile_4bit(packed, scale, N // fold, Kdim * fold, qt, bs), x.cuda().bfloat16()
    bias = torch.randn(N, generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
    for b in (None, bias) if fold == 1 else (None,):
        want = K.qgemv_tiled(x, tiled, N, Kdim, qt, bs, bias=b, fold=fold)
        assert torch.equal(K.qgemv_tiled_rows(x, tiled, N, Kdim, qt, bs, b, fold), want)
        wide = torch.zeros(B, 2 * Kdim + 8, dtype=torch.bfloat16, device="cuda")
        wide[:, 8 : 8 + Kdim] = x
        assert torch.equal(K.qgemv_tiled_rows(wide[:, 8 : 8 + Kdim], tiled, N, Kdim, qt, bs, b, fold), want)   # rows further apart
        turned = x.t().contiguous().t()
        assert torch.equal(K.qgemv_tiled_rows(turned, tiled, N, Kdim, qt, bs, b, fold), want)                    # and columns
        assert K.qgemv_tiled_rows(x.view(1, B, Kdim), tiled, N, Kdim, qt, bs, b, fold).shape == (1, B, N)
    if fold == 1:
        strided = torch.stack((bias, torch.zeros_like(bias)), 1)[:, 0]
        assert torch.equal(K.qgemv_tiled_rows(x, tiled, N, Kdim, qt, bs, strided, 1), K.qgemv_tiled(x, tiled, N, Kdim, qt, bs, bias=bias))


def test_refusals():
    _, x, packed, scale, bs, _ = _gemv_case(K, 512, 4096, 2, "nf4", seed=1)
    tiled, x = K.tile_4bit(packed, scale, 512, 4096, "nf4", bs), x.cuda().bfloat16()
    bias = torch.zeros(512, device="cuda", dtype=torch.bfloat16)
    bad = [(x.cpu(), tiled, None, 1), (x, tiled.cpu(), None, 1), (x.float(), tiled, None, 1), (x[:, :4032], tiled, None, 1), (x, tiled, bias.float(), 1),
           (x.repeat(10, 1), tiled, None, 1)]
    for xx, tt, b, fold in bad:
        for call in (lambda: K.qgemv_tiled_rows(xx, tt, 512, 4096, "nf4", bs, b, fold), lambda: K.qgemv_tiled(xx, tt, 512, 4096, "nf4", bs, bias=b, fold=fold)):   # noqa: B023
            with pytest.raises((C.B200Error, NotImplementedError)):
                call()
