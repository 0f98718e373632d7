"""The chunked delta rule's products of tf32 halves (csrc/delta_chunk.cu): every width of the chain's CTAs against the recurrence in 64 bits, and numbers that
are not finite, which may reach no earlier token."""
import pytest
import torch

from tests.test_gpu_delta_chunk import _exact, _inputs, _stored

pytestmark = pytest.mark.gpu


@pytest.fixture()
def K(monkeypatch):
    from lit_gpt_b200 import kernels

    monkeypatch.setattr(kernels, "DELTA_CHUNKED", True)
    return kernels


def _run(K, data, lens, H, G, dk, dv, channel):
    q, k, v, beta, dec, a_log, bias, S0, seqs = (t.contiguous().cuda() for t in data)
    state = _stored(data[7], dk, 4 if dk <= 64 else 8).float().cuda()
    o = K.delta_rule(q, k, v, beta, dec, a_log, bias, state, seqs, H, G, dk, dv, channel, max_rows=max(lens))
    return o.cpu().double(), state.cpu().double()


# heads x value columns: eight columns a CTA where they fit the SMs at once, sixteen, then two groups of sixteen; the last two with columns past the values
@pytest.mark.parametrize("lens,H,dk,dv", [((96,), 8, 128, 128), ((96,), 17, 128, 120), ((96, 65), 20, 128, 128), ((70,), 24, 64, 100), ((64, 33), 40, 64, 68)])
@pytest.mark.parametrize("channel", [False, True])
def test_delta_split_products(K, lens, H, dk, dv, channel):
    data = _inputs(lens, (3,) * len(lens), H, H, dk, dv, channel, torch.float32, H, 0)
    o, s = _run(K, data, lens, H, H, dk, dv, channel)
    ref, S = _exact(*data, H, H, dk, dv, channel)
    for got, exact in ((o, ref), (s, _stored(S, dk, 4 if dk <= 64 else 8))):
        # each product is good to 2^-22; a sum of n of them and of the chunk's corrections (n <= 128, at random signs) to a few times that of its norm
        assert (got - exact).norm() <= 2.0 ** -20 * exact.norm()


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("what", ["v", "k", "beta", "decay"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_delta_not_finite(K, channel, what, bad):
    """One head's token 45 (of the second chunk) holds an infinity or NaN: its own and later read-outs may not be finite, earlier ones and the other heads' are
    as without it."""
    H, dk, dv, lens = 3, 128, 40, (90,)
    data = list(_inputs(lens, (0,), H, H, dk, dv, channel, torch.float32, 9, 0))
    want, S = _exact(*data, H, H, dk, dv, channel)
    i, at = {"v": (2, dv + 7), "k": (1, dk + 5), "beta": (3, 1), "decay": (4, dk + 9 if channel else 1)}[what]
    data[i] = data[i].clone().contiguous()
    data[i][45, at] = bad
    o, s = _run(K, data, lens, H, H, dk, dv, channel)
    o, want = o.view(90, H, dv), want.view(90, H, dv)
    for got, exact in ((o[:45], want[:45]), (o[:, ::2], want[:, ::2])):
        assert (got - exact).norm() <= 2.0 ** -20 * exact.norm()
    if bad != bad:
        assert not o[45:, 1].isfinite().all()
