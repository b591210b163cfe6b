"""GPU test of the SiLU at every finite bf16 gate, in both of its forms, with an up value that is a power of two: one gate decides a row's scale, so
that one unit of bf16 in its SiLU is seen for certain."""
import pytest
import torch

from oracle import moe_block_int8 as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gates():
    """Every finite gate, its SiLU with CUDA's exponential and an fp32 division, a power of two that brings it near 1 (within 2^-120 .. 2^120)."""
    g = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    g = g[g.isfinite()].to(DEV)
    f = g.float()
    silu = (f / (1.0 + torch.exp(-f))).to(torch.bfloat16)
    exponent = torch.frexp(f.double() / (1.0 + torch.exp(-f.double())))[1]
    up = torch.ldexp(torch.ones_like(f, dtype=torch.float64), (1 - exponent).clamp(-120, 120)).to(torch.bfloat16)
    return g, silu, up


def test_the_library_form_rounds_as_the_exact_value():
    # (what the two forms are compared with; from -89 on the fp32 exponential's sum is infinite and the quotient -0)
    g, silu, _ = _gates()
    x = g.double() / (1.0 + torch.exp(-g.double()))
    e = torch.frexp(x)[1].clamp(min=-125)      # eight bits of mantissa, half to even; bf16's subnormals end at 2^-133
    exact = torch.ldexp(torch.round(torch.ldexp(x, 8 - e)), e - 8)
    differ = g[exact != silu.double()]
    assert bool((differ <= -89).all()) and bool((silu[g <= -89] == 0).all())


def test_quantiser():
    import lightop_b200 as lo
    g, silu, up = _gates()
    x = torch.zeros(len(g), 16, dtype=torch.bfloat16, device=DEV)
    x[:, 0], x[:, 8] = g, up
    q, s = lo.activation.fuse_silu_mul_quant(x)
    act = (silu.float() * up.float()).to(torch.bfloat16).float()
    assert torch.equal(s.view(-1), act.abs() / torch.full_like(act, 127.0))
    assert torch.equal(q[:, 0].int(), 127 * torch.sign(act).int()) and not q[:, 1:].any()


def test_epilogue():
    # K block 0 makes the gate (1 x the token's first scale), K block 1 the up value; the down weights pick one channel
    import lightop_b200 as lo
    from lightop_b200 import _lib
    lib = _lib.load()
    g, silu, up = _gates()
    T, H, I = len(g), 256, 128
    w1, w2 = torch.zeros(1, 2 * I, H, dtype=torch.int8, device=DEV), torch.zeros(1, H, I, dtype=torch.int8, device=DEV)
    w1[:, :I, 0], w1[:, I:, 128], w2[:, :, 5] = 1, 1, 1
    s1, s2 = torch.ones(1, 2, 2, device=DEV), torch.ones(1, 2, 1, device=DEV)
    xq = torch.zeros(T, H, dtype=torch.int8, device=DEV)
    xq[:, 0], xq[:, 128] = 1, 1
    xs = torch.stack([g.float(), up.float()], 1).contiguous()
    expert = torch.zeros(T, dtype=torch.int32, device=DEV)
    out = torch.empty(T, H, dtype=torch.bfloat16, device=DEV)
    ws = torch.empty(lib.lo_fused_moe_workspace_bytes(T, 1, 1, 1, H, I), dtype=torch.uint8, device=DEV)
    st = lib.lo_expert_rows_block_int8(_lib.ptr(xq), _lib.ptr(xs), _lib.ptr(expert), 0, _lib.ptr(w1), _lib.ptr(w2), _lib.ptr(s1), _lib.ptr(s2), T, 1, H, I,
                                       _lib.ptr(out), _lib.ptr(ws), ws.numel(), _lib.ptr(lo.device_status_word(out.device)), _lib.current_stream(out.device))
    _lib.check(st, "expert rows")
    lo.check_device_status()
    # denominators beyond 2^126 have no normal reciprocal: those gates give zero
    silu = torch.where((g <= -87.5) & (g > -89), torch.zeros_like(silu), silu)
    act = (silu.float() * up.float()).to(torch.bfloat16)
    q, s = O.group_quant_int8(act.cpu().view(-1, 1).expand(-1, 128).contiguous(), 128)
    want = (q[:, 0].float() * s[:, 0]).to(torch.bfloat16)
    assert torch.equal(out.cpu().float(), want.float().view(-1, 1).expand(-1, H))
