"""When the two projections of a gated MLP may run as one launch: only when nothing but QLinear.forward would have run for either."""
import pytest
import torch
import torch.nn as nn

from lit_gpt_b200 import _cabi as C
from lit_gpt_b200 import kernels as K
from lit_gpt_b200 import quant


@pytest.fixture
def pair(monkeypatch):
    monkeypatch.setattr(K, "qgemm_swiglu_supported", lambda *a: True)
    mods = [quant.QLinear(128, 256, bias=False, mode="nf4", device="meta", compute_dtype=torch.bfloat16) for _ in range(2)]
    monkeypatch.setattr(quant.QLinear, "is_quantized", True)
    return mods


def test_plain_modules(pair):
    assert quant.prefill_pair(*pair, 300)


@pytest.mark.parametrize("which", [0, 1])
def test_forward_of_an_instance(pair, which):
    pair[which].forward = lambda x: x
    assert not quant.prefill_pair(*pair, 300)


@pytest.mark.parametrize("register", [lambda m: m.register_forward_hook(lambda *a: None), lambda m: m.register_forward_pre_hook(lambda *a: None),
                                      lambda m: m.register_full_backward_hook(lambda *a: None)])
def test_hooks_of_a_module(pair, register):
    handle = register(pair[1])
    assert not quant.prefill_pair(*pair, 300)
    handle.remove()
    assert quant.prefill_pair(*pair, 300)


@pytest.mark.parametrize("register", [nn.modules.module.register_module_forward_hook, nn.modules.module.register_module_forward_pre_hook,
                                      nn.modules.module.register_module_full_backward_hook])
def test_hooks_of_all_modules(pair, register):
    handle = register(lambda *a: None)
    try:
        assert not quant.prefill_pair(*pair, 300)
    finally:
        handle.remove()
    assert quant.prefill_pair(*pair, 300)


@pytest.mark.parametrize("offsets,rows,taken", [((0, 0), 17, True), ((4, 0), 17, False), ((0, 4), 208, False), ((4, 4), 64, False), ((4, 4), 600, True)])
def test_scales_inside_a_larger_buffer(pair, monkeypatch, offsets, rows, taken):
    """The launch for up to 208 rows copies scales 16 bytes at a time: scales elsewhere keep to the launches that read them one by one."""
    monkeypatch.setattr(K, "qgemm_pair_workspace", lambda *a: 0)
    buffer = torch.zeros(64)
    first = -buffer.data_ptr() % 16 // 4   # the first number on a 16-byte boundary
    for m, bytes_on in zip(pair, offsets):
        monkeypatch.setattr(m, "packed", lambda scale=buffer[first + bytes_on // 4:]: (None, scale))
    assert quant.short_pair(*pair, rows) == taken


class _Cuda(torch.Tensor):
    """a CPU tensor that passes for a CUDA one: the checks come before anything reads it"""

    is_cuda = True


@pytest.mark.parametrize("call", ["qgemm", "qgemm_swiglu", "qgemm_pair"])
@pytest.mark.parametrize("shape", [(4, 256), (4, 64), (2, 2, 64)])
def test_rows_of_another_length_are_refused(call, shape):
    """Elements enough for whole rows are not enough: the output has a row per row of x."""
    t = lambda *s, dtype=torch.bfloat16: torch.zeros(*s, dtype=dtype).as_subclass(_Cuda)   # noqa: E731
    w = [t(128, 64, dtype=torch.uint8), t(128 * 2, dtype=torch.float32)]
    with pytest.raises(C.B200Error, match="rows of"):
        getattr(K, call)(t(*shape), *(w if call == "qgemm" else w * 2), 128, 128)
