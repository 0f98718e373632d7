"""Prompt GEMM (csrc/qgemm.cu): tiles of fewer features than a CTA's 128, the packed weights' buffers of two k-blocks, and k ranges that start at odd ones."""
import pytest
import torch

from tests.test_gpu_kernels import K, _gemv_case  # noqa: F401

pytestmark = pytest.mark.gpu


# rows up to 128, 256 and more; an odd number of k-blocks (a buffer's second half past the row), ranges of an odd number of them, features that end inside a
# tile of 64, 80, 96, 160, 192, 224 and 256, several tiles a CTA
@pytest.mark.parametrize("M,N,Kdim", [(17, 11008, 192), (64, 9480, 320), (128, 12296, 64), (40, 2056, 1216), (150, 2048, 2112), (203, 11016, 448), (256, 14344, 128),
                                      (300, 12296, 192), (613, 4104, 576), (400, 14336, 64), (1030, 9480, 128), (203, 4136, 1088)])
@pytest.mark.parametrize("qt", ["nf4", "fp4", "int4"])
def test_qgemm_tile_widths(K, qt, M, N, Kdim):  # noqa: F811
    if qt == "int4" and Kdim % 128:
        Kdim += 64
    _, _, packed, scale, bs, deq = _gemv_case(K, N, Kdim, 1, qt, seed=M + N)
    # a single one per row: every product but one is zero, so whatever the order of the sums the result is the weight itself
    hot = torch.randint(0, Kdim, (M,), generator=torch.Generator().manual_seed(N))
    hot[: min(M, Kdim)] = torch.arange(Kdim)[: min(M, Kdim)]
    x = torch.nn.functional.one_hot(hot, Kdim).to(torch.bfloat16)
    assert torch.equal(K.qgemm(x.cuda(), packed, scale, N, Kdim, qt, bs).cpu(), deq.to(torch.bfloat16).T[hot])


@pytest.mark.parametrize("zero", [7.53, 0.0, 15.0, -2.25])
def test_qgemm_int4_scales(K, zero):  # noqa: F811
    """Scales and zero points that need all eleven bits of a half: bf16_rn(scale * (q - zero)) with an exact product, as the dequantise kernel has it."""
    N, Kdim, M = 264, 256, 64
    g = torch.Generator().manual_seed(3)
    packed = torch.randint(0, 256, (N * Kdim // 2,), dtype=torch.uint8, generator=g)
    scale = torch.stack([(torch.rand(N * 2, generator=g) * 0.1 + 1e-3).half(), torch.full((N * 2,), zero).half()], 1).contiguous()
    q = torch.stack([packed & 15, packed >> 4], 1).view(N, Kdim).double()   # element e of a word in bits 4 e
    w = (scale[:, 0].double().view(N, 2, 1) * (q.view(N, 2, 128) - scale[:, 1].double().view(N, 2, 1))).view(N, Kdim)
    hot = torch.randint(0, Kdim, (M,), generator=g)
    x = torch.nn.functional.one_hot(hot, Kdim).to(torch.bfloat16)
    y = K.qgemm(x.cuda(), packed.cuda(), scale.cuda().view(torch.int32).view(-1), N, Kdim, "int4", 128)
    assert torch.equal(y.cpu(), w.T[hot].to(torch.float32).to(torch.bfloat16))
