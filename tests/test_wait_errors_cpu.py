"""Waits that gave up are reported: the error words of every loaded library, read at the end of generate() and wherever a loop reads a step's
tokens back.  The libraries are stand-ins here; tests/test_gpu_kernels.py lets a real wait run out."""
import pytest
import torch

import lit_gpt_b200.generate.base as generate_base
import lit_gpt_b200.generate.serve as serve
from lit_gpt_b200 import GPT, Config
from lit_gpt_b200 import _cabi as C
from lit_gpt_b200 import kernels as K
from lit_gpt_b200.chat import base as chat


class Words:
    def __init__(self, raised=0):
        self.raised = raised

    def b200_wait_errors_take(self, devices):
        got, self.raised = self.raised & devices, self.raised & ~devices
        return got


@pytest.mark.parametrize("full,core", [(Words(1), None), (None, Words(4)), (Words(), Words(1)), (Words(2), Words(2))])
def test_words_of_every_loaded_library(monkeypatch, full, core):
    monkeypatch.setattr(C, "_lib", full)
    monkeypatch.setattr(C, "_core", core)
    with pytest.raises(C.B200Error, match="gave up a bounded wait"):
        K.raise_wait_errors()
    K.raise_wait_errors()   # reported once
    assert not any(lib.raised for lib in (full, core) if lib)


def test_no_library_is_loaded_to_ask(monkeypatch):
    monkeypatch.setattr(C, "_lib", None)
    monkeypatch.setattr(C, "_core", None)
    monkeypatch.setattr(C, "load", lambda *a: pytest.fail("loaded"))
    K.raise_wait_errors()
    K.check_gemv_errors(torch.device("cpu"))


def _model():
    torch.manual_seed(1)
    model = GPT(Config(block_size=32, vocab_size=16, padded_vocab_size=16, n_layer=1, n_head=2, n_embd=8)).eval()
    model.max_seq_length = 32
    model.set_kv_cache(batch_size=1)
    return model


def test_generate_reads_them_on_one_gpu(monkeypatch):
    asked = []
    monkeypatch.setattr(K, "check_gemv_errors", asked.append)
    generate_base.generate(_model(), torch.tensor([1, 2, 3]), 8, temperature=0.0)
    assert asked == [torch.device("cpu")]
    list(chat.generate(_model(), torch.tensor([1, 2, 3]), 8, temperature=0.0))
    assert len(asked) == 2


def test_loops_that_read_tokens_back_raise(monkeypatch):
    monkeypatch.setattr(C, "_lib", Words(1))
    with pytest.raises(C.B200Error, match="bounded wait"):
        list(chat.generate(_model(), torch.tensor([1, 2, 3]), 8, temperature=0.0, stop_tokens=([15, 15],)))

    class Served:
        device = torch.device("cpu")

        def set_kv_cache(self, batch_size):
            pass

    session = serve.Session(Served(), slots=1)
    assert session.step([]) is None
    C._lib.raised = 1
    with pytest.raises(C.B200Error, match="bounded wait"):
        session.step([])
