"""Layers whose tokens name one expert several times (a batch of padding tokens carries the same id in every slot): an expert then gets more rows than
the call has tokens, and its chunks must still fit the GEMM instantiation that the number of tokens chooses."""
import pytest
import torch

from lightop_b200 import synthetic
from oracle import moe_block_int8 as O
from oracle import moe_channel_int8 as OC
from util import assert_out_close

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 8 x 8 and 5 x 7: more rows than the smallest instantiation holds; 40 x 8: than the second; 100 x 8: than the third, with an average that asks for the
# widest; 16 x 32: through the alignment kernel instead of the one-kernel form
@pytest.mark.parametrize("M,k,E,dtype", [(8, 8, 256, torch.int32), (5, 7, 9, torch.int64), (40, 8, 4, torch.int32), (100, 8, 4, torch.int32),
                                         (16, 32, 64, torch.int32), (1, 64, 3, torch.int32)])
@pytest.mark.parametrize("ids_of", ["zero", "two"])
@pytest.mark.parametrize("fmt", ["block", "channel"])
def test_layer_against_the_oracle(M, k, E, dtype, ids_of, fmt):
    import lightop_b200 as lo
    H, I = 256, 256
    g = torch.Generator().manual_seed(M * k + E)
    ids = torch.zeros(M, k, dtype=dtype) if ids_of == "zero" else torch.randint(0, 2, (M, k), generator=g).to(dtype) * (E - 1)
    x = torch.randn(M, H, generator=g).to(torch.bfloat16)
    w = torch.rand(M, k, generator=g)
    w1, w2, s1, s2 = synthetic.make_weights(E, H, I, seed=4)
    if fmt == "block":
        kw = dict(block_shape=[128, 128])
        ref = O.fused_moe_block_int8(x, w1, w2, s1, s2, w, ids)
    else:
        s1, s2 = synthetic.make_channel_scales(E, H, I, seed=4)
        kw = dict(block_shape=None, per_channel_quant=True)
        ref = OC.fused_moe_channel_int8(x, w1, w2, s1, s2, w, ids)
    y = lo.moe.fused_experts_impl_int8(x.to(DEV), w1.to(DEV), w2.to(DEV), w.to(DEV), ids.to(DEV), None, use_int8_w8a8=True,
                                       w1_scale=s1.to(DEV), w2_scale=s2.to(DEV), **kw)
    torch.cuda.synchronize()
    lo.check_device_status()
    assert_out_close(y, ref, f"{fmt} M={M} k={k} E={E}")
