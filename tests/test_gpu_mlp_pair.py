"""Gated MLP of 4-bit modules: which launch a number of rows takes through the module, and that every route gives the separate launches' result."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mlp(mode, d=512, ff=1024):
    from lit_gpt_b200.config import Config
    from lit_gpt_b200.model import LLaMAMLP
    from lit_gpt_b200.quant import QLinear

    g = torch.Generator().manual_seed(d + ff)
    with torch.device("meta"):
        mlp = LLaMAMLP(Config(n_embd=d, n_head=4, intermediate_size=ff, bias=False, _mlp_class="LLaMAMLP", vocab_size=64, padded_vocab_size=64, n_layer=1, block_size=64))
    for name, (o, i) in (("fc_1", (ff, d)), ("fc_2", (ff, d)), ("proj", (d, ff))):
        lin = torch.nn.Linear(i, o, bias=False, device="meta")
        lin.weight = torch.nn.Parameter((torch.randn(o, i, generator=g) * i ** -0.5).to(torch.bfloat16).cuda(), requires_grad=False)
        setattr(mlp, name, QLinear.from_linear(lin, mode, torch.bfloat16))
    return mlp


def _apart(mlp, x):
    from lit_gpt_b200 import kernels as K

    return mlp.proj(K.swiglu(mlp.fc_1(x), mlp.fc_2(x)))


def _off_boundary(t):
    """The same numbers four bytes past a 16-byte boundary."""
    n = 4 // t.element_size()
    view = torch.empty(t.numel() + n, dtype=t.dtype, device=t.device)[n:].view(t.shape)
    assert view.copy_(t).data_ptr() % 16 == 4
    return view


def _check(mlp, x):
    # one launch sums k in other ranges: its products may be rounded the other way, by a unit of 2^-8, and so may the result
    y, want = mlp(x), _apart(mlp, x)
    assert (y.double() - want.double()).norm() <= 2.0 ** -7 * want.double().norm()


@pytest.fixture
def routes(monkeypatch):
    from lit_gpt_b200 import kernels as K

    seen = []
    for name in ("qgemm_pair", "qgemm_swiglu"):
        monkeypatch.setattr(K, name, lambda *a, _f=getattr(K, name), _n=name: (seen.append(_n), _f(*a))[1])
    return seen


@pytest.mark.parametrize("rows", [17, 64, 128, 129, 203, 208, 209, 300, 512, 513, 700])
@pytest.mark.parametrize("mode", ["nf4", "int4"])
def test_routes(routes, mode, rows):
    from lit_gpt_b200 import kernels as K

    mlp = _mlp(mode)
    x = torch.randn(rows, 512, generator=torch.Generator().manual_seed(rows)).to(torch.bfloat16).cuda()
    bs = 128 if mode == "int4" else 64
    swiglu, pair = K.qgemm_swiglu_supported(rows, 1024, 512, mode, bs), K.qgemm_pair_workspace(rows, 1024, 512, mode, bs) >= 0
    _check(mlp, x)
    assert routes == (["qgemm_pair"] if pair else ["qgemm_swiglu"] if swiglu else [])
    assert routes or 128 < rows <= 512   # up to 128 rows and beyond 512 there is one launch at every size


@pytest.mark.parametrize("rows", [17, 128, 203, 600])
@pytest.mark.parametrize("mode", ["nf4", "int4"])
def test_scales_off_a_16_byte_boundary(routes, mode, rows):
    """Scales inside a larger buffer: up to 208 rows the launch that copies 16 bytes of them at a time is not taken, and the call runs all the same."""
    mlp = _mlp(mode)
    for m in (mlp.fc_1, mlp.fc_2):
        name = "sz" if mode == "int4" else "absmax"
        setattr(m, name, _off_boundary(getattr(m, name)))
    _check(mlp, torch.randn(rows, 512, generator=torch.Generator().manual_seed(rows)).to(torch.bfloat16).cuda())
    assert "qgemm_pair" not in routes or rows > 208


@pytest.mark.parametrize("rows", [40, 203, 600])
def test_hooks_and_released_layouts_keep_the_separate_launches(routes, rows):
    x = torch.randn(rows, 512, generator=torch.Generator().manual_seed(rows)).to(torch.bfloat16).cuda()
    mlp, outs = _mlp("nf4"), []
    handle = mlp.fc_2.register_forward_hook(lambda m, a, y: outs.append(y))
    mlp(x)
    assert not routes and outs[0].shape == (rows, 1024)
    handle.remove()
    want = mlp(x)
    assert routes
    del routes[:]
    assert all(m.release_reference_layout() for m in (mlp.fc_1, mlp.fc_2))
    y = mlp(x)
    assert not routes
    assert (y.double() - want.double()).norm() <= 2.0 ** -7 * want.double().norm()
