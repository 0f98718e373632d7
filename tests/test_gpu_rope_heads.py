"""Rotation and append of a prompt's heads (csrc/attn_decode.cu), whose threads take two or three heads at a time: batches that are not full, one past
full, and several.  Bit-equal to the rotation in torch."""

import pytest
import torch

from tests import test_gpu_kernels as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,hs,n", [(1, 1, 128, 128), (32, 32, 128, 128), (62, 1, 128, 64), (63, 1, 128, 128), (94, 1, 128, 128), (95, 1, 128, 32), (40, 40, 256, 64)])
def test_rope_kv_append_heads(H, G, hs, n, table):
    from lit_gpt_b200 import kernels

    base.test_rope_kv_append_units(kernels, 2, 3, H, G, hs, n, 9, table, torch.int64, False)


# launches of more than 6 CTAs per SM take no more threads than the heads need: one lane of heads, an odd number of units, part of a warp at the end
@pytest.mark.parametrize("table", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,T,H,G,hs,n", [(1, 1200, 1, 1, 128, 128), (2, 600, 32, 8, 128, 128), (1, 1000, 40, 40, 64, 32), (3, 400, 5, 1, 80, 48)])
def test_rope_kv_append_long_launches(B, T, H, G, hs, n, table):
    from lit_gpt_b200 import kernels

    base.test_rope_kv_append_units(kernels, B, T, H, G, hs, n, T + 7, table, torch.int64, True)
