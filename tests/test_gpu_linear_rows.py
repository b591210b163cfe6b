"""The one-kernel form of the dense linear (one to four rows) against the quantiser and the GEMM as two operators: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(M, N, K, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    x = (torch.randn(M, K, generator=g) * torch.exp(torch.randn(M, 1, generator=g))).to(dtype).to(DEV)
    B = torch.randint(-128, 128, (N, K), generator=g, dtype=torch.int8).to(DEV)
    return x, B, (torch.rand((N + 127) // 128, K // 128, generator=g) * 9e-3 + 1e-3).to(DEV)


def _both(x, B, b_s):
    import lightop_b200 as lo
    from lightop_b200 import _lib
    lib = _lib.load()
    before = lib.lo_launch_count()
    one = lo.gemm_ops.apply_w8a8_block_int8_linear(x, B, [128, 128], b_s)
    assert lib.lo_launch_count() - before == 1
    q, s = lo.quant.per_token_group_quant_int8(x, 128)
    two = lo.gemm_ops.matmul_block_int8(q, B, s, b_s, [128, 128], torch.bfloat16).to(x.dtype)
    torch.cuda.synchronize()
    lo.check_device_status()
    return one, two


# outputs: fewer than a CTA's, remainders of 4, 8, 16 and 32 outputs a CTA, across blocks of 128; K: one, five, eleven and 56 blocks (a warp
# takes four at a time, its loads run 64 units ahead), and many
@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(1, 128), (5, 640), (127, 1408), (129, 7168), (576, 7168), (1187, 384), (2373, 640), (4745, 128), (9001, 384), (9472, 128)])
def test_one_kernel_has_the_bits_of_the_two_operators(M, N, K):
    one, two = _both(*_inputs(M, N, K, torch.bfloat16, M + N + K))
    assert torch.equal(one, two), int((one != two).sum())


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(1, 300, 2048), (2, 4096, 1280), (2, 129, 512), (1, 40, 32768)])
def test_other_input_types(M, N, K, dtype):
    one, two = _both(*_inputs(M, N, K, dtype, M + N + K))
    assert torch.equal(one, two)


# three and four rows of fp16: up to one CTA a SM, and more
@pytest.mark.parametrize("M,N,K", [(3, 576, 1408), (4, 129, 7168), (3, 1187, 640), (4, 4745, 384), (4, 1, 128)])
def test_fp16_rows(M, N, K):
    one, two = _both(*_inputs(M, N, K, torch.float16, M + N + K))
    assert torch.equal(one, two)


def test_rows_with_nan_infinity_zeros_and_tiny_values():
    x, B, b_s = _inputs(4, 200, 1024, torch.bfloat16, 5)
    x[0, 130] = float("nan")
    x[1, 5], x[1, 700] = float("inf"), -float("inf")
    x[2] = 0.0
    x[3, 128:256] = 1e-38
    one, two = _both(x, B, b_s)
    assert torch.equal(one.isnan(), two.isnan()) and torch.equal(one.nan_to_num(), two.nan_to_num())


def test_larger_calls_keep_the_other_form():
    from lightop_b200 import _lib
    size = _lib.load().lo_block_int8_linear_dynamic_workspace_bytes
    assert size(5, 128, 128) > 0 and size(4, 1024, 7168) > 0 and size(1, 9473, 128) > 0 and size(1, 16384, 2048) > 0 and size(2, 128, 65536) > 0
    assert size(1, 4096, 7168) == 0 and size(2, 1024, 7168) == 0
