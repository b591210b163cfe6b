"""ctypes binding of ``liblightop_b200.so`` (the C ABI declared in include/lightop_b200.h).

There is no fallback: if the library is missing or a call fails, an exception is raised.  (``host``, the native host side of small calls, is
an addition to this layer: what it does not take, this layer does.)
"""
from __future__ import annotations

import ctypes
import os
import sysconfig
import warnings
from ctypes import c_char_p, c_float, c_int, c_int32, c_int64, c_size_t, c_void_p

import torch


class _NoHost:
    """In the place of the native host step where it cannot be used: it takes no call, so that the general path has them all."""

    @staticmethod
    def _nothing(*args):
        return None

    bind = topk_softmax = fused_experts = linear = _nothing


def _import_host():
    """csrc/host.cpp as it was built for this torch and Python, or a stand-in.  The kernels and their results are the same without it, small calls take
    up to 20 us more on the host; a torch without CUDA has no use for it."""
    if torch.version.cuda is None:
        return _NoHost()
    here = f"[built for torch {torch.__version__}, Python {sysconfig.get_config_var('SOABI')}]"
    try:
        from . import _host
        built_for = getattr(_host, "built_for", "[built for a torch that it does not name]")
        if built_for == here:
            return _host
        why = f"it is {built_for[1:-1]}, this is {here[len('[built for '):-1]}"
    except ImportError as e:
        why = str(e)
    warnings.warn(f"lightop_b200/_host.so is not used, small calls take longer on the host: {why}; `python lightop_b200/build.py` builds it", RuntimeWarning)
    return _NoHost()


host = _import_host()

_HERE = os.path.dirname(os.path.abspath(__file__))
# LIGHTOP_B200_LIB overrides the location of the shared library (e.g. an instrumented build)
LIB_PATH = os.environ.get("LIGHTOP_B200_LIB") or os.path.join(_HERE, "liblightop_b200.so")

LO_F32, LO_F16, LO_BF16, LO_I32, LO_I64, LO_U32 = 0, 1, 2, 3, 4, 5
LO_GATE_SIGMOID, LO_GATE_SQRT_SOFTPLUS, LO_GATE_SQRT_SOFTPLUS_SAFE = 0, 1, 2
LO_WEIGHT_NONE, LO_WEIGHT_FP32, LO_WEIGHT_BF16_PRODUCT = 0, 1, 2

_DTYPE_CODE = {
    torch.float32: LO_F32, torch.float16: LO_F16, torch.bfloat16: LO_BF16,
    torch.int32: LO_I32, torch.int64: LO_I64,
}
if hasattr(torch, "uint32"):
    _DTYPE_CODE[torch.uint32] = LO_U32

# name -> (restype, argtypes); mirrors include/lightop_b200.h one to one
PROTOTYPES = {
    "lo_version": (c_int, []),
    "lo_last_error": (c_char_p, []),
    "lo_sm_count": (c_int, []),
    "lo_launch_count": (ctypes.c_longlong, []),
    "lo_pair_launch_count": (ctypes.c_longlong, []),
    "lo_topk_softmax": (c_int, [c_void_p, c_int, c_int64, c_int, c_int, c_int, c_void_p, c_void_p, c_int,
                                c_void_p, c_void_p]),
    "lo_moe_align_block_size": (c_int, [c_void_p, c_int, c_int64, c_int, c_int, c_void_p, c_int, c_void_p,
                                        c_int64, c_void_p, c_int64, c_void_p, c_void_p]),
    "lo_group_quant_int8": (c_int, [c_void_p, c_int, c_int64, c_int, c_float, c_void_p, c_void_p, c_void_p]),
    "lo_moe_sum": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_int64, c_int, c_int64, c_float, c_void_p,
                           c_void_p, c_void_p]),
    "lo_grouped_gemm_workspace_bytes": (c_size_t, [c_int64, c_int, c_int64]),
    "lo_moe_grouped_gemm_i8_block": (c_int, [c_void_p, c_void_p, c_int64, c_void_p, c_void_p, c_int, c_int64,
                                             c_int64, c_void_p, c_void_p, c_int, c_void_p, c_int64, c_void_p,
                                             c_void_p, c_int64, c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "lo_fused_moe_workspace_bytes": (c_size_t, [c_int64, c_int, c_int, c_int, c_int64, c_int64]),
    "lo_fused_moe_workspace_layout": (c_int, [c_int64, c_int, c_int, c_int, c_int64, c_int64, c_void_p]),
    "lo_fused_moe_block_int8": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                        c_int, c_void_p, c_int, c_int64, c_int, c_int, c_int64, c_int64,
                                        c_void_p, c_void_p, c_void_p, c_int, c_float, c_void_p, c_size_t,
                                        c_void_p, c_void_p]),
    "lo_fused_moe_block_int8_noalloc": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                                c_int, c_void_p, c_int, c_int64, c_int, c_int, c_int64, c_int64,
                                                c_void_p, c_void_p, c_void_p, c_int, c_float, c_void_p, c_void_p]),
    "lo_ep_dispatch_row_bytes": (c_int64, [c_int64]),
    "lo_ep_dispatch_pack": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_int64, c_int, c_int64,
                                    c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p]),
    "lo_ep_dispatch_plan": (c_int, [c_void_p, c_int, c_void_p, c_int64, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p]),
    "lo_ep_dispatch_put": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_int64, c_int,
                                   c_int64, c_int, c_int, c_void_p, c_void_p, c_void_p]),
    "lo_expert_rows_block_int8_packed_put": (c_int, [c_void_p, c_int64, c_void_p, c_void_p, c_void_p, c_void_p, c_int,
                                                     c_int64, c_int64, c_void_p, c_void_p, c_int, c_void_p, c_size_t,
                                                     c_void_p, c_void_p]),
    "lo_peer_alloc": (c_int, [c_size_t, c_void_p]),
    "lo_words_to_host": (c_int, [c_void_p, c_void_p, c_int64, c_void_p]),
    "lo_peer_free": (c_int, [c_void_p]),
    "lo_peer_handle_bytes": (c_int, []),
    "lo_peer_export": (c_int, [c_void_p, c_void_p]),
    "lo_peer_open": (c_int, [c_void_p, c_void_p]),
    "lo_peer_close": (c_int, [c_void_p]),
    "lo_expert_rows_packed_workspace_bytes": (c_size_t, [c_int64, c_int, c_int64, c_int64]),
    "lo_expert_rows_block_int8_packed": (c_int, [c_void_p, c_int64, c_void_p, c_void_p, c_void_p, c_void_p, c_int,
                                                 c_int64, c_int64, c_void_p, c_void_p, c_size_t, c_void_p, c_void_p]),
    "lo_expert_rows_block_int8": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                          c_void_p, c_int64, c_int, c_int64, c_int64, c_void_p, c_void_p, c_size_t,
                                          c_void_p, c_void_p]),
    "lo_block_int8_linear_workspace_bytes": (c_size_t, [c_int64]),
    "lo_block_int8_linear": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_int64, c_void_p,
                                     c_void_p, c_size_t, c_void_p, c_void_p]),
    "lo_block_int8_linear_split_workspace_bytes": (c_size_t, [c_int64, c_int64, c_int64]),
    "lo_block_int8_linear_dynamic_workspace_bytes": (c_size_t, [c_int64, c_int64, c_int64]),
    "lo_block_int8_linear_dynamic_scratch_bytes": (c_size_t, [c_int64, c_int64, c_int64, c_int]),
    "lo_block_int8_linear_dynamic": (c_int, [c_void_p, c_int, c_void_p, c_void_p, c_int64, c_int64, c_int64, c_void_p,
                                             c_void_p, c_size_t, c_void_p, c_void_p]),
    "lo_moe_fused_gate": (c_int, [c_void_p, c_int, c_void_p, c_int, c_int64, c_int, c_int, c_int, c_int, c_int, c_float,
                                  c_int, c_void_p, c_void_p, c_int, c_void_p]),
    "lo_moe_gate_topk": (c_int, [c_void_p, c_int, c_void_p, c_int, c_int64, c_int64, c_int, c_int, c_int, c_int, c_int, c_int, c_int,
                                 c_float, c_float, c_float, c_void_p, c_int, c_int, c_void_p, c_void_p, c_int, c_void_p]),
    "lo_topk_ids_postprocess": (c_int, [c_void_p, c_int, c_int64, c_int64, c_void_p, c_int, c_int64, c_void_p, c_int,
                                        c_void_p]),
    "lo_per_token_quant_int8": (c_int, [c_void_p, c_int, c_int64, c_int64, c_void_p, c_void_p, c_void_p]),
    "lo_silu_mul_quant_int8": (c_int, [c_void_p, c_int64, c_int64, c_void_p, c_void_p, c_void_p]),
    "lo_moe_grouped_gemm_i8_channel": (c_int, [c_void_p, c_void_p, c_int64, c_void_p, c_void_p, c_int, c_int64,
                                               c_int64, c_void_p, c_void_p, c_int, c_void_p, c_int64, c_void_p,
                                               c_void_p, c_int64, c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "lo_fused_moe_channel_workspace_bytes": (c_size_t, [c_int64, c_int, c_int, c_int, c_int64, c_int64]),
    "lo_fused_moe_channel_int8": (c_int, [c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                          c_void_p, c_int, c_void_p, c_int, c_int64, c_int, c_int, c_int64, c_int64,
                                          c_void_p, c_void_p, c_void_p, c_int, c_float, c_void_p, c_size_t,
                                          c_void_p, c_void_p]),
    "lo_silu_mul_quant_int8_masked": (c_int, [c_void_p, c_int64, c_int64, c_int64, c_void_p, c_void_p, c_void_p, c_void_p]),
    "lo_m_grouped_gemm_workspace_bytes": (c_size_t, [c_int64, c_int]),
    "lo_m_grouped_w8a8_gemm_nt_contig": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int64,
                                                 c_int, c_int64, c_int64, c_void_p, c_size_t, c_void_p, c_void_p]),
    "lo_m_grouped_w8a8_gemm_nt_masked": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int,
                                                 c_int64, c_int64, c_int64, c_void_p, c_size_t, c_void_p, c_void_p]),
    "lo_m_grouped_w8a8_gemm_nt_masked_expected": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int,
                                                          c_int64, c_int64, c_int64, c_int64, c_void_p, c_size_t, c_void_p, c_void_p]),
    "lo_profile_enable": (c_int, [c_int]),
    "lo_profile_read": (c_int, [c_void_p]),
    "lo_ep_scatter": (c_int, [c_void_p, c_void_p, c_int, c_void_p, c_int, c_void_p, c_void_p, c_void_p,
                              c_void_p, c_void_p, c_void_p, c_int64, c_int, c_int64, c_int64, c_int, c_int,
                              c_void_p]),
    "lo_ep_build_m_indices": (c_int, [c_void_p, c_int, c_int64, c_void_p, c_int64, c_int, c_int, c_void_p]),
    "lo_ep_gather": (c_int, [c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_int64, c_int,
                             c_int64, c_void_p]),
}

_lib = None


class LightopError(RuntimeError):
    """A C-ABI call returned a non-zero status."""


def load() -> ctypes.CDLL:
    """Load the shared library (once) and attach the prototypes."""
    global _lib
    if _lib is not None:
        return _lib
    if not os.path.exists(LIB_PATH):
        raise ImportError(
            f"{LIB_PATH} is missing: build it with `python lightop_b200/build.py` "
            "(there is no CPU or eager fallback)")
    lib = ctypes.CDLL(LIB_PATH)
    for name, (res, args) in PROTOTYPES.items():
        fn = getattr(lib, name)
        fn.restype = res
        fn.argtypes = args
    host.bind({name: ctypes.cast(getattr(lib, name), c_void_p).value for name in PROTOTYPES}, check)
    _lib = lib
    return lib


def check(status: int, what: str) -> None:
    if status != 0:
        msg = load().lo_last_error()
        raise LightopError(f"{what}: status {status}: {msg.decode() if msg else ''}")


def dtype_code(dt: torch.dtype) -> int:
    try:
        return _DTYPE_CODE[dt]
    except KeyError:
        raise TypeError(f"unsupported dtype {dt}") from None


def ptr(t) -> int:
    """Device address of a tensor (None -> NULL)."""
    return 0 if t is None else t.data_ptr()


def require_cuda(*tensors) -> None:
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise RuntimeError("lightop_b200 runs on CUDA tensors only (no CPU fallback)")


class _NoSwitch:
    __slots__ = ()

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        return False


_NO_SWITCH = _NoSwitch()


def on_device(device: torch.device):
    """``torch.cuda.device(device)``, free of charge when that device is current already (the context manager proper costs
    several microseconds a call, more than the launch it encloses)."""
    index = device.index
    return _NO_SWITCH if index is None or index == torch.cuda.current_device() else torch.cuda.device(device)


def current_stream(device: torch.device) -> int:
    """Handle of the device's current stream, without building a ``torch.cuda.Stream`` around it."""
    index = device.index
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if index is None else index)


def f32(t: torch.Tensor) -> torch.Tensor:
    """``t`` as a contiguous fp32 tensor, itself where it is one."""
    return t if t.dtype is torch.float32 and t.is_contiguous() else t.to(torch.float32).contiguous()
