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


# both sides of every limit, by the kernels that a call launches: K by the outputs a CTA (4 up to 1184 outputs, 8 up to 2368, 16 up to 4736, 32), the number of
# weights, of outputs and of rows, the shared memory
BF16, F16, F32 = torch.bfloat16, torch.float16, torch.float32


@pytest.mark.parametrize("M,N,inside,outside,dtypes", [
    (1, 2400, 10240, 10368, (BF16, F16)), (1, 4800, 3584, 3712, (BF16, F16)), (1, 2368, 12544, 12672, (BF16,)), (1, 9472, 128, None, (BF16, F16, F32)),
    (1, 9473, None, 128, (BF16, F16, F32)), (1, 128, 42496, 42624, (F16,)),
    (2, 1200, 10240, 10368, (BF16, F16)), (2, 2400, 7168, 7296, (BF16, F16)), (2, 4800, 2048, 2176, (BF16, F16)),
    (1, 1200, 20480, 20608, (F32,)), (1, 2400, 7168, 7296, (F32,)), (1, 4800, 2048, 2176, (F32,)),
    (2, 64, 8192, 8320, (F32,)), (2, 1200, 5120, 5248, (F32,)), (2, 2400, 3072, 3200, (F32,)), (2, 4800, 1536, 1664, (F32,)), (2, 9216, 1408, 1536, (F32,)),
    (3, 1024, 4352, 4480, (BF16, F16)), (4, 1024, 4352, 4480, (BF16, F16)), (4, 128, 10624, 10752, (BF16,)), (3, 128, None, 128, (F32,)), (5, 128, None, 128, (BF16, F16, F32))])
def test_both_sides_of_the_limits(M, N, inside, outside, dtypes):
    import lightop_b200 as lo
    from lightop_b200 import _lib
    lib = _lib.load()
    for dtype in dtypes:
        for K, one in ((inside, True), (outside, False)):
            if K is None:
                continue
            x, B, b_s = _inputs(M, N, K, dtype, M + N + K)
            before = lib.lo_launch_count()
            y = lo.gemm_ops.apply_w8a8_block_int8_linear(x, B, [128, 128], b_s)
            launches = lib.lo_launch_count() - before
            assert (launches == 1) == one, (dtype, K, launches)
            q, s = lo.quant.per_token_group_quant_int8(x, 128)
            assert torch.equal(y, lo.gemm_ops.matmul_block_int8(q, B, s, b_s, [128, 128], torch.bfloat16).to(dtype)), (dtype, K)
    lo.check_device_status()


@pytest.mark.parametrize("M,N,K,dtype,one", [(1, 576, 1408, BF16, True), (4, 576, 1408, F16, True), (4, 576, 1408, F32, False), (5, 128, 256, BF16, False)])
def test_workspace_asked_for_is_the_workspace_needed(M, N, K, dtype, one):
    # the query by type is 0 exactly where a null workspace is taken; a byte less than it is refused, and the size for all types serves every type
    from lightop_b200 import _lib
    lib = _lib.load()
    x, B, b_s = _inputs(M, N, K, dtype, 3)
    need = lib.lo_block_int8_linear_dynamic_scratch_bytes(M, N, K, _lib.dtype_code(dtype))
    every = lib.lo_block_int8_linear_dynamic_workspace_bytes(M, N, K)
    assert (need == 0) == one and every > 0 and need in (0, every)
    ws = torch.empty(every, dtype=torch.uint8, device=DEV)

    def call(ptr, size):
        c = torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV)
        st = lib.lo_block_int8_linear_dynamic(x.data_ptr(), _lib.dtype_code(dtype), B.data_ptr(), b_s.data_ptr(), M, N, K, c.data_ptr(), ptr, size, 0,
                                              torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return st, c

    want = call(ws.data_ptr(), every)
    assert want[0] == 0
    st, c = call(0, 0)
    assert (st == 0) == one and (st != 0 or torch.equal(c, want[1]))
    if not one:
        assert call(ws.data_ptr(), need - 1)[0] != 0


@pytest.mark.parametrize("M,K,at", [(1, 2048, 0), (4, 1024, 0), (2, 1024, 512), (2, 1024, -512)])
def test_output_over_the_input(M, K, at):
    # C on top of x (at elements off): the rows are read before anything is stored
    from lightop_b200 import _lib
    lib = _lib.load()
    x, B, b_s = _inputs(M, K, K, BF16, 9)
    every = lib.lo_block_int8_linear_dynamic_workspace_bytes(M, K, K)
    ws = torch.empty(every, dtype=torch.uint8, device=DEV)
    apart = torch.empty(M, K, dtype=torch.bfloat16, device=DEV)
    both = torch.empty(M * K + 1024, dtype=torch.bfloat16, device=DEV)
    mine = both[512:512 + M * K]
    stream = torch.cuda.current_stream().cuda_stream

    def call(src, dst, w, size):
        return lib.lo_block_int8_linear_dynamic(src, _lib.LO_BF16, B.data_ptr(), b_s.data_ptr(), M, K, K, dst, w, size, 0, stream)

    assert call(x.data_ptr(), apart.data_ptr(), 0, 0) == 0
    for _ in range(20):
        mine.copy_(x.view(-1))
        assert call(mine.data_ptr(), both.data_ptr() + (512 + at) * 2, ws.data_ptr(), every) == 0
        assert torch.equal(both[512 + at:512 + at + M * K], apart.view(-1))
    mine.copy_(x.view(-1))
    assert call(mine.data_ptr(), both.data_ptr() + (512 + at) * 2, 0, 0) != 0 and torch.equal(mine, x.view(-1))
    # side by side is apart
    side = torch.empty(2 * M * K, dtype=torch.bfloat16, device=DEV)
    side[:M * K].copy_(x.view(-1))
    assert call(side.data_ptr(), side.data_ptr() + 2 * M * K, 0, 0) == 0 and torch.equal(side[M * K:], apart.view(-1))
