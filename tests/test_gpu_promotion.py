"""GPU test of the block-scaled GEMM's promotion loop: every number of 16-column pieces a warp can own (0 to 5), at chunk widths
on both sides of each, in all four instantiations, with K-block counts that leave a remainder in a batch of four scale tables."""
import pytest
import torch

from lightop_b200 import synthetic
from oracle import moe_block_int8 as O
from util import assert_gemm_close, assert_out_close

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M", [1, 16, 17, 33, 48, 49, 64, 80, 81, 97, 112, 128, 129, 144, 145, 160])
@pytest.mark.parametrize("H,I", [(640, 384), (128, 256)])      # 5 and 3, 1 and 2 K blocks
def test_one_expert_every_chunk_width(M, H, I):
    # one expert that gets every token: one chunk of M rows in both GEMMs of the layer
    import lightop_b200 as lo
    w1, w2, w1_s, w2_s = synthetic.make_weights(1, H, I, seed=M)
    x, logits = synthetic.make_activations(M, H, 1, seed=M + 1)
    w, ids = O.route_topk_softmax(logits, 1, renormalize=True)
    ref = O.fused_moe_block_int8(x, w1, w2, w1_s, w2_s, w, ids)
    y = lo.moe.fused_experts_impl_int8(x.to(DEV), w1.to(DEV), w2.to(DEV), w.to(DEV), ids.to(DEV), None, use_int8_w8a8=True,
                                       block_shape=[128, 128], w1_scale=w1_s.to(DEV), w2_scale=w2_s.to(DEV))
    torch.cuda.synchronize()
    lo.check_device_status()
    assert_out_close(y, ref, f"M={M} H={H} I={I}")


@pytest.mark.parametrize("M,N,K", [(5, 128, 128), (31, 256, 384), (128, 200, 896), (131, 136, 1152), (257, 384, 512)])
def test_linear_remainders(M, N, K):
    # bit-level bar of the unfused GEMM (one bf16 step, on at most 1e-3 of the outputs)
    import lightop_b200 as lo
    g = torch.Generator().manual_seed(M + N + K)
    aq, a_s = O.group_quant_int8(torch.randn(M, K, generator=g).to(torch.bfloat16), 128)
    B = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8)
    b_s = torch.rand((N + 127) // 128, K // 128, generator=g) * 9e-3 + 1e-3
    ref = O.block_int8_matmul(aq, B, a_s, b_s, (128, 128), torch.bfloat16)
    out = lo.gemm_ops.matmul_block_int8(aq.to(DEV), B.to(DEV), a_s.to(DEV), b_s.to(DEV), [128, 128], torch.bfloat16)
    torch.cuda.synchronize()
    lo.check_device_status()
    assert_gemm_close(out, ref, f"linear {M}x{N}x{K}")
