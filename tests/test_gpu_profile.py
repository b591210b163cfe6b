"""Stage times of the fused layers: five durations, and none for a stage that a call does not have."""
import ctypes

import pytest
import torch

from lightop_b200 import synthetic

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 32 x 2 pairs are aligned and quantised by one kernel, 200 x 2 and the per-channel layer by two; in an order in which an event of an
# earlier call would be found by a later one
@pytest.mark.parametrize("calls", [[(200, False), (32, False), (32, True), (32, False), (200, False)]])
def test_stage_times(calls):
    import lightop_b200 as lo
    from lightop_b200 import _lib
    lib = _lib.load()
    E, H, I, k = 8, 256, 512, 2
    w1, w2, s1, s2 = synthetic.make_weights(E, H, I, seed=0, device=DEV)
    c1, c2 = synthetic.make_channel_scales(E, H, I, device=DEV)
    for M, channel in calls:
        x = torch.randn(M, H, device=DEV).to(torch.bfloat16)
        ids = torch.stack([torch.randperm(E)[:k] for _ in range(M)]).to(torch.int32).to(DEV)
        w = torch.rand(M, k, device=DEV)
        kw = dict(per_channel_quant=True, block_shape=None, w1_scale=c1, w2_scale=c2) if channel else dict(block_shape=[128, 128], w1_scale=s1, w2_scale=s2)
        ms = (ctypes.c_float * 5)(*[-1.0] * 5)
        lib.lo_profile_enable(1)
        try:
            lo.moe.fused_experts_impl_int8(x, w1, w2, w, ids, None, use_int8_w8a8=True, **kw)
            assert lib.lo_profile_read(ms) == 0
        finally:
            lib.lo_profile_enable(0)
        joined = M * k <= 256 and not channel
        assert (ms[0] == 0) == joined and all(ms[i] > 0 for i in range(1, 5)), list(ms)
