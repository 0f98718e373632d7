"""Prompt GEMM of up to 256 rows with the weights in tensor memory (csrc/qgemm_short.cu): edges of its tiles, of its stages of rows and of the ranges of k."""
import ctypes

import pytest
import torch

from lit_gpt_b200 import _cabi as C
from tests.test_gpu_kernels import K, _gemv_case  # noqa: F401

pytestmark = pytest.mark.gpu


def _off_boundary(scale):
    """The same scales four bytes past a 16-byte boundary, where the library keeps to its other GEMM (csrc/qgemm.cu)."""
    n = 4 // scale.element_size()
    view = torch.empty(scale.numel() + n, dtype=scale.dtype, device=scale.device)[n:].view(scale.shape)
    assert view.copy_(scale).data_ptr() % 16 == 4
    return view


# rows on both sides of what a stage of rows holds (64, 128) and of a multiple of 16; features that end inside a tile of 128; one unit of 256 k, an odd number of them,
# fewer and more than SMs (ranges of several tiles, tiles of several ranges), each shape as whole tiles, as ranges of k and as the library picks
@pytest.mark.parametrize("M", [1, 16, 17, 64, 65, 128, 129, 241, 256])
@pytest.mark.parametrize("N,Kdim", [(136, 256), (264, 1280), (1000, 768), (4104, 2304), (19208, 256), (38408, 512)])
@pytest.mark.parametrize("qt", ["nf4", "fp4", "int4"])
def test_one_hot_rows_read_the_weights(K, qt, M, N, Kdim):  # noqa: F811
    _, _, packed, scale, bs, deq = _gemv_case(K, N, Kdim, 1, qt, seed=M + N)
    hot = torch.randint(0, Kdim, (M,), generator=torch.Generator().manual_seed(N))
    x = torch.nn.functional.one_hot(hot, Kdim).to(torch.bfloat16).cuda()
    bias = torch.randn(N, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
    want = deq.to(torch.bfloat16).T[hot]
    plus = (want.float() + bias.float()).to(torch.bfloat16)
    assert torch.equal(K.qgemm(x, packed, scale, N, Kdim, qt, bs).cpu(), want)
    assert torch.equal(K.qgemm(x, packed, scale, N, Kdim, qt, bs, bias=bias.cuda()).cpu(), plus)
    for ranges in (False, True):
        assert torch.equal(K.qgemm_short(x, packed, scale, N, Kdim, qt, bs, ranges=ranges).cpu(), want)
        assert torch.equal(K.qgemm_short(x, packed, scale, N, Kdim, qt, bs, ranges=ranges, bias=bias.cuda()).cpu(), plus)


@pytest.mark.parametrize("M", [1, 17, 64, 65, 128, 129, 160, 176, 192, 203, 208])
@pytest.mark.parametrize("N,Kdim", [(136, 256), (1000, 1280), (11008, 4096), (19208, 512), (18952, 1280)])
@pytest.mark.parametrize("qt", ["nf4", "fp4", "int4"])
def test_pair_is_the_separate_launches(K, qt, M, N, Kdim):  # noqa: F811
    """Both projections and their product in one launch, as whole tiles and as ranges of k, and either projection alone, against the other GEMM: sums in another order
    of k, so some bf16 roundings of either projection go the other way by one unit, 2^-8 of the number at most."""
    _, _, p1, s1, bs, _ = _gemv_case(K, N, Kdim, 1, qt, seed=M)
    _, _, p2, s2, _, _ = _gemv_case(K, N, Kdim, 1, qt, seed=N)
    x = torch.randn(M, Kdim, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).cuda()
    gate, up = (K.qgemm(x, p, _off_boundary(s), N, Kdim, qt, bs) for p, s in ((p1, s1), (p2, s2)))
    ref = K.swiglu(gate, up)
    takes = K.qgemm_pair_workspace(M, N, Kdim, qt, bs) >= 0
    assert takes or M > 128   # beyond, another launch may be the shorter way
    calls = [(lambda r=r: K.qgemm_short(x, p1, s1, N, Kdim, qt, bs, ranges=r, up=(p2, s2)), ref) for r in (False, True)]
    calls += [(lambda r=r: K.qgemm_short(x, p1, s1, N, Kdim, qt, bs, ranges=r), gate) for r in (False, True)]
    calls += [(lambda: K.qgemm_pair(x, p1, s1, p2, s2, N, Kdim, qt, bs), ref)] if takes else []
    for call, want in calls:
        y = call()
        assert (y.double() - want.double()).norm() <= 2.0 ** -8 * want.double().norm()
        assert torch.equal(y, call())


@pytest.mark.parametrize("room", [None, "too little", "off a boundary"])
@pytest.mark.parametrize("M,N,Kdim", [(17, 4096, 4096), (100, 4096, 4096), (203, 4096, 11008)])
@pytest.mark.parametrize("qt", ["nf4", "int4"])
def test_less_scratch_than_asked_for(K, qt, M, N, Kdim, room):  # noqa: F811
    """Both C entries where the plan is ranges of k but the scratch for them is missing: whole tiles, the scratch untouched, the same result but for the sums' order."""
    _, _, p1, s1, bs, _ = _gemv_case(K, N, Kdim, 1, qt, seed=1)
    _, _, p2, s2, _, _ = _gemv_case(K, N, Kdim, 1, qt, seed=2)
    x = torch.randn(M, Kdim, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).cuda()
    for pair in (False, True):
        need = K.qgemm_pair_workspace(M, N, Kdim, qt, bs) if pair else C.load().b200_qgemm_workspace_bytes(M, N, Kdim)
        if need < 0:
            assert M > 128
            continue
        assert need > 0
        want = K.qgemm_pair(x, p1, s1, p2, s2, N, Kdim, qt, bs) if pair else K.qgemm(x, p1, s1, N, Kdim, qt, bs)
        ws = None if room is None else torch.full((need + 16,), 77, dtype=torch.uint8, device="cuda")[(8 if room == "off a boundary" else 0):]
        # (too little: a byte less for the pair; the single entry's other GEMM may do with less than was asked for, but not with that)
        size = 0 if room is None else need if room == "off a boundary" else need - 1 if pair else 15
        y = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        args = C.QGemmArgs(packed=p1.data_ptr(), scale=s1.data_ptr(), qtype=K.QTYPES[qt], blocksize=bs, M=M, N=N, K=Kdim, x=x.data_ptr(), y=y.data_ptr(),
                           workspace=C.ptr(ws), workspace_bytes=size)
        st = C.stream_ptr(x.device)
        C.check(C.load().b200_qgemm_pair(ctypes.byref(args), p2.data_ptr(), s2.data_ptr(), st) if pair else C.load().b200_qgemm(ctypes.byref(args), st), "qgemm")
        assert (y.double() - want.double()).norm() <= 2.0 ** -8 * want.double().norm()
        assert ws is None or ws.eq(77).all()


@pytest.mark.parametrize("M,N,Kdim", [(513, 11008, 4096), (700, 5632, 4096), (1281, 11008, 1024)])
@pytest.mark.parametrize("qt", ["nf4", "fp4", "int4"])
def test_pair_takes_long_prompts_that_swiglu_refuses(K, qt, M, N, Kdim):  # noqa: F811
    """The same sums in the same order as two GEMMs without k ranges: the same bits."""
    _, _, p1, s1, bs, _ = _gemv_case(K, N, Kdim, 1, qt, seed=M)
    _, _, p2, s2, _, _ = _gemv_case(K, N, Kdim, 1, qt, seed=N)
    x = torch.randn(M, Kdim, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).cuda()
    assert (K.qgemm_pair_workspace(M, N, Kdim, qt, bs) == 0) != K.qgemm_swiglu_supported(M, N, Kdim, qt, bs)
    one = K.qgemm_swiglu if K.qgemm_swiglu_supported(M, N, Kdim, qt, bs) else K.qgemm_pair
    assert torch.equal(one(x, p1, s1, p2, s2, N, Kdim, qt, bs), K.swiglu(K.qgemm(x, p1, s1, N, Kdim, qt, bs), K.qgemm(x, p2, s2, N, Kdim, qt, bs)))


def test_pair_refuses(K):  # noqa: F811
    for M, N, Kdim in ((209, 512, 512), (512, 512, 512), (32, 512, 320), (32, 500, 512), (1000, 500, 512)):
        assert K.qgemm_pair_workspace(M, N, Kdim, "nf4", 64) < 0
        x, w = torch.zeros(M, Kdim, dtype=torch.bfloat16, device="cuda"), torch.zeros(N * Kdim // 2, dtype=torch.uint8, device="cuda")
        s = torch.zeros(N * Kdim // 64, dtype=torch.float32, device="cuda")
        with pytest.raises(NotImplementedError):
            K.qgemm_pair(x, w, s, w, s, N, Kdim, "nf4", 64)


@pytest.mark.parametrize("zero", [7.53, 0.0, 16.0, 17.0, -2.25])
def test_int4_scales(K, zero):  # noqa: F811
    """Scales and zero points that need all eleven bits of a half, whole zero points up to 16 and others: bf16_rn(scale * (q - zero)) with an exact product."""
    N, Kdim, M = 264, 512, 40
    g = torch.Generator().manual_seed(3)
    packed = torch.randint(0, 256, (N * Kdim // 2,), dtype=torch.uint8, generator=g)
    scale = torch.stack([(torch.rand(N * 4, generator=g) * 0.1 + 1e-3).half(), torch.full((N * 4,), zero).half()], 1).contiguous()
    q = torch.stack([packed & 15, packed >> 4], 1).view(N, Kdim).double()   # element e of a word in bits 4 e
    w = (scale[:, 0].double().view(N, 4, 1) * (q.view(N, 4, 128) - scale[:, 1].double().view(N, 4, 1))).view(N, Kdim)
    hot = torch.randint(0, Kdim, (M,), generator=g)
    x = torch.nn.functional.one_hot(hot, Kdim).to(torch.bfloat16)
    y = K.qgemm(x.cuda(), packed.cuda(), scale.cuda().view(torch.int32).view(-1), N, Kdim, "int4", 128)
    assert torch.equal(y.cpu(), w.T[hot].to(torch.float32).to(torch.bfloat16))
