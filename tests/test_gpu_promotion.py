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


@pytest.mark.parametrize("M,N,K", [(1, 576, 7168), (3, 201, 4096), (33, 128, 4224), (64, 1000, 4096), (129, 136, 7168), (300, 576, 4224), (500, 520, 4096)])
def test_linear_with_a_split_k_extent(M, N, K):
    # 32, 33 and 56 K blocks in parts that end even and uneven, rows and columns that leave remainders (201 * 3 is odd: the scalar
    # form of the reduction), one to four chunks; the same call without room for the parts takes the undivided form
    import lightop_b200 as lo
    from lightop_b200 import _lib
    lib = _lib.load()
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    aq, a_s = O.group_quant_int8(x, 128)
    B = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8)
    b_s = torch.rand((N + 127) // 128, K // 128, generator=g) * 9e-3 + 1e-3
    ref = O.block_int8_matmul(aq, B, a_s, b_s, (128, 128), torch.bfloat16)
    d_aq, d_as, d_B, d_bs = aq.to(DEV), a_s.to(DEV), B.to(DEV), b_s.to(DEV)
    assert lib.lo_block_int8_linear_split_workspace_bytes(M, N, K) >= 4 * 2 * M * N      # at least two parts
    out = lo.gemm_ops.matmul_block_int8(d_aq, d_B, d_as, d_bs, [128, 128], torch.bfloat16)
    fused = lo.gemm_ops.apply_w8a8_block_int8_linear(x.to(DEV), d_B, [128, 128], d_bs)
    whole = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ws = torch.empty(256, dtype=torch.uint8, device=DEV)
    st = lib.lo_block_int8_linear(d_aq.data_ptr(), d_as.data_ptr(), d_B.data_ptr(), d_bs.data_ptr(), M, N, K, whole.data_ptr(),
                                  ws.data_ptr(), 256, 0, torch.cuda.current_stream().cuda_stream)
    assert st == 0
    torch.cuda.synchronize()
    lo.check_device_status()
    assert_gemm_close(out, ref, f"split linear {M}x{N}x{K}")
    assert_gemm_close(whole, ref, f"undivided linear {M}x{N}x{K}")
    assert torch.equal(out, fused)
    # the sum of the parts is no further from 64 bits than the undivided sum (before their rounding to bf16 both err by a few
    # ulps of fp32, so the bf16 results may differ by one step where they straddle a rounding)
    exact = sum((aq[:, i:i + 128].double() @ B[:, i:i + 128].double().T) * a_s[:, i // 128, None].double()
                * b_s[:, i // 128].double().repeat_interleave(128)[:N] for i in range(0, K, 128))
    err = [float((y.cpu().double() - exact).norm() / exact.norm()) for y in (out, whole)]
    assert err[0] <= err[1] * 1.001


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(5, 256), (2, 3, 4096), (256,)])
def test_linear_in_one_call_equals_its_two_operators(dtype, shape):
    import lightop_b200 as lo
    g = torch.Generator().manual_seed(len(shape))
    x = torch.randn(*shape, generator=g).to(dtype).to(DEV)
    K = shape[-1]
    B = torch.randint(-127, 128, (200, K), generator=g, dtype=torch.int8).to(DEV)
    b_s = (torch.rand(2, K // 128, generator=g) * 9e-3 + 1e-3).to(DEV)
    bias = torch.randn(200, generator=g).to(dtype).to(DEV)
    q, s = lo.quant.per_token_group_quant_int8(x.reshape(-1, K), 128)
    ref = lo.gemm_ops.matmul_block_int8(q, B, s, b_s, [128, 128], output_dtype=dtype)
    y = lo.gemm_ops.apply_w8a8_block_int8_linear(x, B, [128, 128], b_s)
    assert y.dtype == dtype and y.shape == x.shape[:-1] + (200,) and torch.equal(y.reshape(ref.shape), ref)
    yb = lo.gemm_ops.apply_w8a8_block_int8_linear(x, B, [128, 128], b_s, bias=bias)
    assert torch.equal(yb.reshape(ref.shape), (ref + bias).to(dtype))
    # a strided input takes the general path, with the same result
    wide = torch.zeros(*shape[:-1], 2 * K, dtype=dtype, device=DEV)
    wide[..., ::2] = x
    assert torch.equal(lo.gemm_ops.apply_w8a8_block_int8_linear(wide[..., ::2], B, [128, 128], b_s), y)


@pytest.mark.parametrize("offset", [1, 4])      # elements of bf16: 2 and 8 bytes off a 16-byte boundary
@pytest.mark.parametrize("M,N,K", [(5, 256, 384), (131, 136, 512), (1, 576, 7168)])
def test_linear_output_off_a_16_byte_boundary(M, N, K, offset):
    # a caller's C that begins anywhere in a buffer: the row stores take the scalar form, the elements around stay untouched
    import lightop_b200 as lo
    from lightop_b200 import _lib
    lib = _lib.load()
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    B = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8).to(DEV)
    b_s = (torch.rand((N + 127) // 128, K // 128, generator=g) * 9e-3 + 1e-3).to(DEV)
    q, s = lo.quant.per_token_group_quant_int8(x, 128)
    ref = lo.gemm_ops.matmul_block_int8(q, B, s, b_s, [128, 128], torch.bfloat16)
    stream = torch.cuda.current_stream().cuda_stream
    for form in ("undivided", "split", "dynamic"):
        buf = torch.full((M * N + 16,), 7.0, dtype=torch.bfloat16, device=DEV)
        c = buf[offset:offset + M * N]
        n = {"undivided": 256, "split": lib.lo_block_int8_linear_split_workspace_bytes(M, N, K),
             "dynamic": lib.lo_block_int8_linear_dynamic_workspace_bytes(M, N, K)}[form]
        ws = torch.empty(n, dtype=torch.uint8, device=DEV)
        if form == "dynamic":
            st = lib.lo_block_int8_linear_dynamic(x.data_ptr(), _lib.LO_BF16, B.data_ptr(), b_s.data_ptr(), M, N, K, c.data_ptr(), ws.data_ptr(), n, 0, stream)
        else:
            st = lib.lo_block_int8_linear(q.data_ptr(), s.data_ptr(), B.data_ptr(), b_s.data_ptr(), M, N, K, c.data_ptr(), ws.data_ptr(), n, 0, stream)
        assert st == 0, form
        assert_gemm_close(c.view(M, N), ref, f"{form} {M}x{N}x{K} at {offset}")
        assert bool((buf[:offset] == 7.0).all()) and bool((buf[offset + M * N:] == 7.0).all()), form


def test_moe_gemm_output_off_a_16_byte_boundary():
    import lightop_b200 as lo
    E, k, H, N, M, block = 8, 2, 256, 384, 33, 16
    g = torch.Generator().manual_seed(9)
    w = torch.randint(-127, 128, (E, N, H), generator=g, dtype=torch.int8).to(DEV)
    w_s = (torch.rand(E, N // 128, H // 128, generator=g) * 9e-3 + 1e-3).to(DEV)
    q, s = lo.quant.per_token_group_quant_int8(torch.randn(M, H, generator=g).to(torch.bfloat16).to(DEV), 128)
    ids = torch.randint(0, E, (M, k), generator=g, dtype=torch.int32).to(DEV)
    wgt = torch.rand(M, k, generator=g).to(DEV)
    sorted_ids, expert_ids, num_post = lo.moe.moe_align_block_size(ids, block, E)
    ref = torch.empty(M, k, N, dtype=torch.bfloat16, device=DEV)
    lo.moe.moe_gemm_w8a8(q, w, ref, s, w_s, wgt, sorted_ids, expert_ids, num_post, k, {"BLOCK_SIZE_M": block})
    buf = torch.full((M * k * N + 8,), 7.0, dtype=torch.bfloat16, device=DEV)
    out = buf[3:3 + M * k * N].view(M, k, N)
    lo.moe.moe_gemm_w8a8(q, w, out, s, w_s, wgt, sorted_ids, expert_ids, num_post, k, {"BLOCK_SIZE_M": block})
    assert torch.equal(out, ref) and bool((buf[:3] == 7.0).all()) and bool((buf[3 + M * k * N:] == 7.0).all())


@pytest.mark.parametrize("N,K", [(576, 7168), (201, 4096), (1024, 4224), (256, 640)])
def test_linear_rows_do_not_depend_on_the_batch(N, K):
    # the same row among 1 and among 700 others: chunks of other widths, the K extent split or not, the same bits
    import lightop_b200 as lo
    g = torch.Generator().manual_seed(N + K)
    x = torch.randn(700, K, generator=g).to(torch.bfloat16).to(DEV)
    B = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8).to(DEV)
    b_s = (torch.rand((N + 127) // 128, K // 128, generator=g) * 9e-3 + 1e-3).to(DEV)
    whole = lo.gemm_ops.apply_w8a8_block_int8_linear(x, B, [128, 128], b_s)
    for M in (1, 3, 17, 64, 128, 129, 300):
        part = lo.gemm_ops.apply_w8a8_block_int8_linear(x[:M].contiguous(), B, [128, 128], b_s)
        assert torch.equal(part, whole[:M]), f"{M} rows: {int((part != whole[:M]).sum())} outputs differ"
    torch.cuda.synchronize()
    lo.check_device_status()


@pytest.mark.parametrize("M,N,K", [(1, 576, 7168), (2, 129, 4096), (16, 2048, 7168), (65, 136, 4096), (128, 1024, 4096), (129, 576, 4224), (1, 1, 65536), (3, 256, 4352)])
def test_split_linear_has_the_bits_of_the_undivided_form(M, N, K):
    import lightop_b200 as lo
    from lightop_b200 import _lib
    lib = _lib.load()
    g = torch.Generator().manual_seed(M + N + K)
    A = torch.randint(-127, 128, (M, K), generator=g, dtype=torch.int8).to(DEV)
    a_s = (torch.rand(M, K // 128, generator=g) * 1e-2).to(DEV)
    B = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8).to(DEV)
    b_s = (torch.rand((N + 127) // 128, K // 128, generator=g) * 1e-2).to(DEV)
    out = []
    n = lib.lo_block_int8_linear_split_workspace_bytes(M, N, K)
    assert n >= 4 * (K // 128) * M * N          # the call is split
    for nbytes in (n, 256):
        c = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        ws = torch.empty(nbytes, dtype=torch.uint8, device=DEV)
        assert lib.lo_block_int8_linear(A.data_ptr(), a_s.data_ptr(), B.data_ptr(), b_s.data_ptr(), M, N, K, c.data_ptr(), ws.data_ptr(), nbytes, 0,
                                        torch.cuda.current_stream().cuda_stream) == 0
        out.append(c)
    torch.cuda.synchronize()
    lo.check_device_status()
    assert torch.equal(out[0], out[1])


def test_undivided_linear_keeps_no_scratch():
    import lightop_b200 as lo
    from lightop_b200 import _lib
    lib = _lib.load()
    M, N, K = 5, 256, 384
    g = torch.Generator().manual_seed(3)
    q, s = lo.quant.per_token_group_quant_int8(torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV), 128)
    B = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8).to(DEV)
    b_s = (torch.rand(2, 3, generator=g) * 9e-3 + 1e-3).to(DEV)
    assert lib.lo_block_int8_linear_split_workspace_bytes(M, N, K) == 0
    c = torch.zeros(M, N, dtype=torch.bfloat16, device=DEV)
    assert lib.lo_block_int8_linear(q.data_ptr(), s.data_ptr(), B.data_ptr(), b_s.data_ptr(), M, N, K, c.data_ptr(), 0, 0, 0,
                                    torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(c, lo.gemm_ops.matmul_block_int8(q, B, s, b_s, [128, 128], torch.bfloat16))
