"""CPU tests of the C-ABI boundary: the library loads, exports what the header declares,
and rejects bad arguments before touching a device."""
import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "lightop_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(lo_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported():
    from lightop_b200 import _lib
    lib = ctypes.CDLL(_lib.LIB_PATH)
    names = _declared_symbols()
    assert len(names) >= 13
    for n in names:
        assert hasattr(lib, n), f"{n} declared in the header but not exported"


def test_binding_covers_header():
    from lightop_b200 import _lib
    assert sorted(_lib.PROTOTYPES) == _declared_symbols()


def test_version_and_error_string():
    from lightop_b200 import _lib
    lib = _lib.load()
    assert lib.lo_version() == 1
    assert isinstance(lib.lo_last_error(), bytes)


def test_argument_validation_needs_no_device():
    from lightop_b200 import _lib
    lib = _lib.load()
    # null pointers
    assert lib.lo_group_quant_int8(0, _lib.LO_BF16, 4, 128, 1e-10, 0, 0, 0) == 1
    assert b"null" in lib.lo_last_error()
    # zero work is a no-op that succeeds
    assert lib.lo_group_quant_int8(0, _lib.LO_BF16, 0, 128, 1e-10, 0, 0, 0) == 0
    assert lib.lo_topk_softmax(0, _lib.LO_F32, 0, 8, 2, 1, 0, 0, _lib.LO_I32, 0, 0) == 0
    # expert count outside the supported range
    assert lib.lo_topk_softmax(16, _lib.LO_F32, 4, 4096, 2, 1, 16, 16, _lib.LO_I32, 0, 0) == 1
    assert lib.lo_moe_sum(16, 16, 0, _lib.LO_BF16, 4, 2, 12, 1.0, 0, 0, 0) == 1   # H not a multiple of 8
    assert lib.lo_fused_moe_workspace_bytes(32, 8, 8, 2, 256, 512) > 32 * 256
    with pytest.raises(_lib.LightopError):
        _lib.check(1, "probe")


def test_python_api_refuses_cpu_tensors():
    from lightop_b200 import moe, quant
    x = torch.zeros(4, 256, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="CUDA"):
        quant.per_token_group_quant_int8(x, 128)
    with pytest.raises(AssertionError):
        quant.per_token_group_quant_int8(torch.zeros(4, 100, dtype=torch.bfloat16), 128)
    with pytest.raises(RuntimeError, match="CUDA"):
        moe.moe_align_block_size(torch.zeros(4, 2, dtype=torch.int32), 16, 8)


def test_fused_experts_contract_checks():
    from lightop_b200 import moe
    x = torch.zeros(4, 256, dtype=torch.bfloat16)
    w1 = torch.zeros(2, 512, 256, dtype=torch.int8)
    w2 = torch.zeros(2, 256, 256, dtype=torch.int8)
    tw = torch.zeros(4, 2)
    ti = torch.zeros(4, 2, dtype=torch.int32)
    with pytest.raises(AssertionError):            # neither int8 nor fp8 requested
        moe.fused_experts_impl_int8(x, w1, w2, tw, ti, None)
    with pytest.raises(AssertionError, match="Hidden size"):
        moe.fused_experts_impl_int8(x[:, :128], w1, w2, tw, ti, None, use_int8_w8a8=True, block_shape=[128, 128])
    with pytest.raises(NotImplementedError):       # per-channel flag together with a block shape
        moe.fused_experts_impl_int8(x, w1, w2, tw, ti, None, use_int8_w8a8=True, per_channel_quant=True,
                                    block_shape=[128, 128])
    with pytest.raises(AssertionError, match="block or channel-wise"):      # the reference's own rule
        moe.fused_experts_impl_int8(x, w1, w2, tw, ti, None, use_int8_w8a8=True)
    with pytest.raises(RuntimeError):              # CPU tensors never reach a kernel
        moe.fused_experts_impl_int8(x, w1, w2, tw, ti, None, use_int8_w8a8=True, per_channel_quant=True,
                                    w1_scale=torch.zeros(2, 512, 1), w2_scale=torch.zeros(2, 256, 1))
    with pytest.raises(ValueError, match="activation"):
        moe.fused_experts_impl_int8(x, w1, w2, tw, ti, None, use_int8_w8a8=True, block_shape=[128, 128],
                                    activation="gelu", w1_scale=tw, w2_scale=tw)


def test_api_names_present():
    import lightop_b200
    for name in ["topk_softmax", "moe_align_block_size", "moe_align_block_size_out", "moe_sum", "moe_gemm_w8a8",
                 "fused_experts_impl_int8", "fused_experts_impl_int8_marlin", "ep_scatter", "ep_gather",
                 "ep_build_m_indices", "moe_fused_gate", "kimi_k2_moe_fused_gate", "moe_fused_gate_sqrtsoftplus",
                 "moe_fused_gate_sqrtsoftplus_v41_hcu", "moe_fused_gate_sqrtsoftplus_v41_hcu_fused",
                 "moe_fused_gate_sqrtsoftplus_v41_hcu_deepep", "topk_ids_postprocess"]:
        assert hasattr(lightop_b200.moe, name)
    assert hasattr(lightop_b200.quant, "per_token_group_quant_int8")
    assert hasattr(lightop_b200.quant, "per_token_quant_int8")
    assert hasattr(lightop_b200.activation, "fuse_silu_mul_quant")


def test_noalloc_size_check_boundary_without_a_gpu():
    """The scratch-free entry point refuses a shape by its workspace need before anything else happens: at the
    DeepSeek-V3 shape 402 tokens fit its 64 MiB array and 403 do not (the size check needs no device)."""
    from lightop_b200 import _lib
    lib = _lib.load()
    args = dict(E=256, k=8, H=7168, I=2048)
    assert lib.lo_fused_moe_workspace_bytes(402, args["E"], args["E"], args["k"], args["H"], args["I"]) <= 64 << 20
    assert lib.lo_fused_moe_workspace_bytes(403, args["E"], args["E"], args["k"], args["H"], args["I"]) > 64 << 20

    def call(M):
        st = lib.lo_fused_moe_block_int8_noalloc(0, 0, 0, 0, 0, 0, 0, _lib.LO_I32, 0, args["E"], M, args["E"], args["k"],
                                                 args["H"], args["I"], 0, 0, 0, 0, 1.0, 0, 0)
        return st, lib.lo_last_error()
    st, msg = call(403)
    assert st == 1 and b"built-in array" in msg
    st, msg = call(402)           # passes the size check; what stops it afterwards is the missing device or the null pointers
    assert st != 0 and b"built-in array" not in msg


def _entries_with_vector_access(lib):
    """(entry, arguments with `None` at the pointer under test, positions of such pointers) of every entry whose kernels read or
    write caller memory 16 bytes at a time.  The addresses are never used: each call has to be refused on the host."""
    from lightop_b200 import _lib
    P, E, M, k, H, I = 4096, 2, 4, 2, 128, 128
    big = 1 << 30
    fused = [P] * 7 + [_lib.LO_I32, 0, E, M, E, k, H, I, P, P, P, 0, 1.0, P, big, 0, 0]
    channel = [P, _lib.LO_BF16] + [P] * 6 + [_lib.LO_I32, 0, E, M, E, k, H, I, P, P, P, 0, 1.0, P, big, 0, 0]
    gemm = [P, P, M, P, P, E, 128, H, P, P, 0, P, 64, P, P, M * k, k, 16, P, big, 0]
    return [(lib.lo_fused_moe_block_int8, fused, (0, 15, 16, 17)),
            (lib.lo_fused_moe_channel_int8, channel, (0, 16, 17, 18)),
            (lib.lo_moe_grouped_gemm_i8_block, gemm, (0,)),
            (lib.lo_moe_grouped_gemm_i8_channel, gemm, (0,)),
            (lib.lo_expert_rows_block_int8, [P] * 8 + [M, E, H, I, P, P, big, 0, 0], (0,)),
            (lib.lo_moe_sum, [P, P, P, _lib.LO_BF16, M, k, H, 1.0, 0, 0, 0], (0, 1, 2)),
            (lib.lo_ep_scatter, [P, P, 1, P, _lib.LO_I32, 0, 0, P, P, P, P, M, k, H, 64, E, 16, 0], (0, 7)),
            (lib.lo_ep_dispatch_pack, [P, P, P, _lib.LO_I32, P, P, M, k, H, E, 2, P, P, P, P, 0], (0, 11)),
            (lib.lo_ep_dispatch_put, [P, P, P, _lib.LO_I32, P, P, P, M, k, H, E, 2, P, P, 0], (0,)),
            (lib.lo_ep_gather, [P, P, _lib.LO_I32, P, P, 0, P, M, k, H, 0], (0, 6))]


def test_misaligned_caller_memory_is_refused_on_the_host():
    from lightop_b200 import _lib
    lib = _lib.load()
    for entry, args, positions in _entries_with_vector_access(lib):
        for i in positions:
            for off in (2, 8):
                bad = list(args)
                bad[i] += off
                assert entry(*bad) == 1, (entry.__name__, i, off)
                assert b"16-byte aligned" in lib.lo_last_error(), (entry.__name__, i, lib.lo_last_error())


def test_alignment_does_not_matter_without_work():
    from lightop_b200 import _lib
    lib = _lib.load()
    assert lib.lo_moe_sum(18, 18, 0, _lib.LO_BF16, 0, 2, 128, 1.0, 0, 0, 0) == 0
    assert lib.lo_ep_gather(18, 16, _lib.LO_I32, 16, 16, 0, 18, 0, 2, 128, 0) == 0
    assert lib.lo_ep_dispatch_put(18, 16, 16, _lib.LO_I32, 16, 16, 16, 0, 2, 128, 2, 2, 16, 16, 0) == 0
