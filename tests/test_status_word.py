"""The device's status word: one that a tracer or a transform hands out in place of memory is not kept for the calls after it."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

import lightop_b200 as lo
from lightop_b200 import _lib

DEV = torch.device("cuda", 0)


def _fake(fn):
    with FakeTensorMode():
        fn()


def _grad(fn):
    torch.func.grad(lambda x: (fn(), x.sum())[1])(torch.ones(2))


def _functionalize(fn):
    torch.func.functionalize(lambda x: (fn(), x)[1])(torch.ones(2))


@pytest.mark.parametrize("under", [_fake, pytest.param(_grad, marks=pytest.mark.gpu), pytest.param(_functionalize, marks=pytest.mark.gpu)])
def test_a_word_without_memory_is_not_kept(under, monkeypatch):
    monkeypatch.setattr(lo, "_status_words", {})
    under(lambda: lo.device_status_word(DEV))
    assert lo._status_words == {}


@pytest.mark.gpu
def test_a_first_call_that_a_transform_refuses_leaves_the_native_host_step(monkeypatch):
    monkeypatch.setattr(lo, "_status_words", {})
    x, w, s = torch.ones(1, 128, dtype=torch.bfloat16, device=DEV), torch.ones(128, 128, dtype=torch.int8, device=DEV), torch.ones(1, 1, device=DEV)
    with pytest.raises(RuntimeError, match="data pointer"):
        torch.func.grad(lambda v: lo.gemm_ops.apply_w8a8_block_int8_linear(v, w, [128, 128], s).float().sum())(x)
    word = lo.device_status_word(DEV)
    assert word.data_ptr() != 0 and lo.device_status_word(DEV) is word
    assert _lib.host.linear(x, w, [128, 128], s, word) is not None
    lo.check_device_status()
