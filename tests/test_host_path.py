"""The native host side of small calls (csrc/host.cpp): it takes the usual form of a call with the results of the general path, and answers
None, without an error, for every other one."""
import itertools
import threading

import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

import lightop_b200 as lo
from lightop_b200 import _lib, synthetic

DEV = "cuda"


class _Refuses:
    """The host module as it answers a form that it does not take."""

    def __getattr__(self, name):
        return lambda *a: None


class _FunctionMode(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _DispatchMode(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _Sub(torch.Tensor):
    pass


@pytest.mark.parametrize("value", [None, 3, "x", torch.zeros(2, 2), torch.zeros(2, 2, dtype=torch.int8), [128, 128]])
def test_other_arguments_are_refused_without_an_error(value):
    for fn, n in ((_lib.host.topk_softmax, 4), (_lib.host.fused_experts, 17), (_lib.host.linear, 5)):
        for count in (0, n - 1, n, n + 1):
            assert fn(*([value] * count)) is None


def _layer(channel, E=8, M=24, H=256, I=256, k=2, ids=torch.int32):
    w1, w2, s1, s2 = synthetic.make_weights(E, H, I, seed=1, device=DEV)
    if channel:
        s1, s2 = synthetic.make_channel_scales(E, H, I, seed=1, device=DEV)
    x, logits = synthetic.make_activations(M, H, E, seed=2, device=DEV)
    w, i = torch.empty(M, k, device=DEV), torch.empty(M, k, dtype=ids, device=DEV)
    lo.moe.topk_softmax(w, i, None, logits, True)
    kw = dict(use_int8_w8a8=True, per_channel_quant=channel, block_shape=None if channel else [128, 128], w1_scale=s1, w2_scale=s2)
    return (x, w1, w2, w, i), kw


@pytest.mark.gpu
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("ids", [torch.int32, torch.int64])
def test_layer_has_the_bits_of_the_general_path(channel, ids, monkeypatch):
    (x, w1, w2, w, i), kw = _layer(channel, ids=ids)
    emap = torch.tensor([0, -1, 1, 2, -1, 3, 4, 5], dtype=torch.int32, device=DEV)
    shared = torch.randn_like(x)
    cache = torch.empty(x.shape[0] * 2 * x.shape[1], dtype=torch.bfloat16, device=DEV)
    for m, sh, c, inplace, factor in itertools.product((None, emap), (None, shared), (None, cache), (False, True), (None, 1.0, 2.5)):
        extra = dict(kw, expert_map=m, global_num_experts=8 if m is not None else -1, shared_output=sh, inplace=inplace, routed_scaling_factor=factor)
        xa, xb = x.clone(), x.clone()
        a = lo.moe.fused_experts_impl_int8(xa, w1, w2, w, i, c, **extra)
        assert (a is xa) == inplace
        with monkeypatch.context() as mp:
            mp.setattr(_lib, "host", _Refuses())
            b = lo.moe.fused_experts_impl_int8(xb, w1, w2, w, i, c, **extra)
        assert torch.equal(a, b) and a.dtype == b.dtype and a.stride() == b.stride()
    lo.check_device_status()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 7168), (3, 256), (2, 5, 512), (300, 896), (256,)])
def test_linear_and_gate_have_the_bits_of_the_general_path(shape, monkeypatch):
    K = shape[-1]
    x = torch.randn(*shape, device=DEV).to(torch.bfloat16)
    w = torch.randint(-127, 128, (576, K), device=DEV, dtype=torch.int8)
    s = torch.rand(5, K // 128, device=DEV) * 9e-3 + 1e-3
    bias = torch.randn(576, device=DEV).to(torch.bfloat16)
    logits = torch.randn(37, 64, device=DEV)
    assert _lib.host.linear(x, w, [128, 128], s, lo.device_status_word(x.device)) is not None

    def run():
        out = [lo.gemm_ops.apply_w8a8_block_int8_linear(x, w, [128, 128], s), lo.gemm_ops.apply_w8a8_block_int8_linear(x, w, (128, 128), s, bias=bias)]
        for g, t in itertools.product((logits, logits.half(), logits.bfloat16()), (torch.int32, torch.int64)):
            out += [torch.empty(37, 6, device=DEV), torch.empty(37, 6, dtype=t, device=DEV)]
            lo.moe.topk_softmax(out[-2], out[-1], None, g, True)
        return out
    a = run()
    monkeypatch.setattr(_lib, "host", _Refuses())
    for p, q in zip(a, run()):
        assert torch.equal(p, q) and p.shape == q.shape and p.dtype == q.dtype


@pytest.mark.gpu
def test_other_forms_are_left_to_the_general_path(monkeypatch):
    (x, w1, w2, w, i), kw = _layer(False)
    status = lo.device_status_word(x.device)
    s1, s2 = kw["w1_scale"], kw["w2_scale"]

    def host(**change):
        a = dict(x=x, w1=w1, w2=w2, w=w, i=i, cache=None, s1=s1, s2=s2, emap=None, shared=None, block=[128, 128], channel=False, experts=-1, on_input=False,
                 factor=1.0, inplace=False, status=status)
        a.update(change)
        return _lib.host.fused_experts(*a.values())
    assert host() is not None
    wide = torch.empty(x.shape[0], 2 * x.shape[1], dtype=x.dtype, device=DEV)[:, ::2]
    for change in (dict(x=x.float()), dict(x=wide), dict(x=x[:, :128]), dict(x=x[:0]), dict(x=x.as_subclass(_Sub)), dict(w1=w1[:, :384]), dict(w1=w1.cpu()),
                   dict(w2=w2[:4]), dict(w=w.half()), dict(w=w[:-1]), dict(i=i.to(torch.int16)), dict(i=i[:-1]), dict(i=i.t().contiguous().t()),
                   dict(cache=torch.empty(5, dtype=torch.bfloat16, device=DEV)), dict(s1=s1.half()), dict(s1=s1[:, :1]), dict(s2=s2[:1]),
                   dict(emap=torch.zeros(8, dtype=torch.int64, device=DEV)), dict(shared=torch.zeros_like(x)[:1]), dict(block=[64, 128]), dict(block=None),
                   dict(channel=True), dict(experts=None), dict(experts=1 << 40), dict(on_input=True), dict(factor="1"), dict(factor=2), dict(inplace=None),
                   dict(status=None)):
        assert host(**change) is None, change
    for mode in (_FunctionMode(), _DispatchMode()):
        with mode:
            assert host() is None
    ref = lo.moe.fused_experts_impl_int8(x, w1, w2, w, i, None, **kw)
    for n in ("23", "0x20", "", "7 8"):
        monkeypatch.setenv("LMSLIM_FUSED_MOE_CHUNK_SIZE", n)
        assert host() is None, n
    monkeypatch.setenv("LMSLIM_FUSED_MOE_CHUNK_SIZE", "7")
    assert torch.equal(lo.moe.fused_experts_impl_int8(x, w1, w2, w, i, None, **kw), ref)
    monkeypatch.setenv("LMSLIM_FUSED_MOE_CHUNK_SIZE", "24")
    assert torch.equal(host(), ref)
    # errors are those of the general path
    with pytest.raises(AssertionError):
        lo.moe.fused_experts_impl_int8(wide, w1, w2, w, i, None, **kw)
    with pytest.raises(RuntimeError, match="cache13"):
        lo.moe.fused_experts_impl_int8(x, w1, w2, w, i, torch.empty(5, dtype=torch.bfloat16, device=DEV), **kw)
    with pytest.raises(_lib.LightopError):      # more (token, slot) experts than there are: refused by the C ABI, raised by its message
        lo.moe.topk_softmax(torch.empty(2, 65, device=DEV), torch.empty(2, 65, dtype=torch.int32, device=DEV), None, torch.randn(2, 64, device=DEV), True)
    xs = torch.randn(3, 2, 256, device=DEV).to(torch.bfloat16)
    wl, sl = torch.randint(-127, 128, (128, 256), device=DEV, dtype=torch.int8), torch.rand(1, 2, device=DEV)
    seen = []
    torch.vmap(lambda r: (seen.append(_lib.host.linear(r, wl, [128, 128], sl, status)), r)[1])(xs)
    assert seen == [None]


@pytest.mark.gpu
def test_threads_on_their_own_streams():
    (x, w1, w2, w, i), kw = _layer(False, M=32)
    ref = lo.moe.fused_experts_impl_int8(x, w1, w2, w, i, None, **kw)
    torch.cuda.synchronize()
    bad = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(200):
                if not torch.equal(lo.moe.fused_experts_impl_int8(x, w1, w2, w, i, None, **kw), ref):
                    bad.append(1)
    threads = [threading.Thread(target=work) for _ in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad
