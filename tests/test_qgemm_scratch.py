"""Scratch of the prompt GEMM of up to 256 rows: a place for each part of a tile that a range of k can cut, and no more (asked of the library; nothing is launched)."""
import pytest

from lit_gpt_b200 import kernels as K
from lit_gpt_b200 import _cabi as C

SMS = 148


def _parts(N, Kdim):
    """CTAs and tiles, in the order of k, step on by a CTA, a tile or both from one part to the next."""
    tiles = -(-N // 128)
    ctas = min(SMS, tiles * (Kdim // 256))
    return min(ctas + tiles - 1, 2 * ctas)


@pytest.mark.parametrize("N,Kdim", [(4096, 14336), (4096, 4096), (12288, 4096), (5632, 2048), (136, 512), (18944, 4096), (24576, 1280)])
@pytest.mark.parametrize("M", [17, 64, 100, 128])
@pytest.mark.parametrize("qt,bs", [("nf4", 64), ("int4", 128)])
def test_pair(qt, bs, M, N, Kdim):
    assert 0 <= K.qgemm_pair_workspace(M, N, Kdim, qt, bs) <= 2 * M * 128 * 4 * _parts(N, Kdim)


@pytest.mark.parametrize("M,N,Kdim", [(256, 4096, 14336), (256, 4096, 11008), (203, 4096, 11008), (64, 11008, 4096)])
def test_one_matrix(M, N, Kdim):
    assert 0 < C.load().b200_qgemm_workspace_bytes(M, N, Kdim) <= M * 128 * 4 * _parts(N, Kdim)
