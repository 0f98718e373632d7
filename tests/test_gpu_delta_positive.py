"""The chunked delta rule's products of tf32 halves (csrc/delta_chunk.cu) on inputs of one sign, as a silu leaves them, where whatever the tensor core cuts off adds up:
no further from 64 bits than fp32 multiply-adds are, in chunks and token by token."""
import pytest
import torch

from lit_gpt_b200 import kernels as K
from tests.test_gpu_delta_chunk import _exact, _stored

pytestmark = pytest.mark.gpu


# bounds: errors relative to the walk's of the same chunks with every product as fp32 multiply-adds (read-out up to 1.46, state up to 1.15 of it on these inputs), the
# mean of three seeds spreading by some 3 %
@pytest.mark.parametrize("mean,n,H,dk", [(1.0, 96, 16, 128), (1.0, 300, 8, 128), (0.0, 300, 8, 128), (1.0, 200, 8, 64)])
@pytest.mark.parametrize("channel", [False, True])
def test_delta_positive_inputs(monkeypatch, mean, n, H, dk, channel):
    errors = []
    for chunks in (True, False):
        monkeypatch.setattr(K, "DELTA_CHUNKED", chunks)
        sums = [0.0, 0.0]
        for seed in range(3):
            g = torch.Generator().manual_seed(seed + n)
            x = torch.nn.functional.silu(torch.randn(n, 3, H, dk, generator=g) + mean)
            unit = lambda t: (t / t.norm(dim=-1, keepdim=True)).reshape(n, -1)   # noqa: E731
            q, k, v = unit(x[:, 0]) * dk**-0.5, unit(x[:, 1]), x[:, 2].reshape(n, -1)
            cols = H * (dk if channel else 1)
            beta, dec = torch.randn(n, H, generator=g).bfloat16(), torch.randn(n, cols, generator=g).bfloat16()
            a_log, bias = (torch.rand(H, generator=g) * 2.5 - 1).bfloat16(), (torch.rand(cols, generator=g) * 4 - 5).bfloat16()
            seqs = torch.tensor([(0, n, 0, 0)], dtype=torch.int32)
            ref, S = _exact(q, k, v, beta, dec, a_log, bias, torch.zeros(1, H, dk, dk), seqs, H, H, dk, dk, channel)
            S = _stored(S, dk, 4 if dk <= 64 else 8)
            state = torch.zeros(S.shape, device="cuda")
            o = K.delta_rule(*(t.contiguous().cuda() for t in (q, k, v, beta, dec, a_log, bias)), state, seqs.cuda(), H, H, dk, dk, channel, max_rows=n)
            for i, (got, exact) in enumerate(((o, ref), (state, S))):
                sums[i] += ((got.cpu().double() - exact).norm() / exact.norm()).item() / 3
        errors.append(sums)
    (o, s), (ow, sw) = errors
    assert o <= 1.5 * ow and s <= 1.18 * sw, (errors, o / ow, s / sw)
