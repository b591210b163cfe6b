"""GPU test of the grouped GEMM on pairs of CTAs against its form on single ones.  Calls large enough for pairs are computed again in a way
that takes the other form (an odd number of output tiles, or one expert at a time), and every output must have the same bits.  Chunk widths
on both sides of the MMA's 32-row granule and of the boxes that a half of a chunk is loaded with."""
import pytest
import torch

from lightop_b200 import synthetic

pytestmark = pytest.mark.gpu
DEV = "cuda"
# rows per expert: every edge of pieces, granules and boxes, a full chunk, more than one, none
COUNTS = [1, 16, 17, 31, 32, 33, 64, 65, 80, 96, 97, 112, 113, 128, 129, 144, 145, 160, 161, 200, 256, 257, 300, 0]


def _int8(g, *shape):
    return torch.randint(-127, 128, shape, generator=g, device=DEV, dtype=torch.int8)


@pytest.mark.parametrize("M,tiles,K", [(65, 256, 14336), (96, 256, 14336), (97, 256, 14336), (112, 256, 14336), (200, 130, 14336),
                                       (1000, 34, 7168), (3999, 10, 6272)])
def test_dense_linear(M, tiles, K):
    import lightop_b200 as lo
    g = torch.Generator(device=DEV).manual_seed(M + tiles + K)
    q, s = _int8(g, M, K), torch.rand(M, K // 128, generator=g, device=DEV) * 0.05 + 1e-3
    w, w_s = _int8(g, tiles * 128, K), torch.rand(tiles, K // 128, generator=g, device=DEV) * 9e-3 + 1e-3
    n = (tiles - 1) * 128
    pairs = lo.gemm_ops.matmul_block_int8(q, w, s, w_s, [128, 128], torch.bfloat16)
    for order in (torch.arange(tiles), torch.arange(tiles).flip(0)):      # (the second one has the last tile)
        order = order.to(DEV)
        single = lo.gemm_ops.matmul_block_int8(q, w.view(tiles, 128, K)[order].reshape(-1, K)[:n].contiguous(), s, w_s[order][:-1].contiguous(),
                                               [128, 128], torch.bfloat16)
        torch.cuda.synchronize()
        lo.check_device_status()
        assert torch.equal(pairs.view(M, tiles, 128)[:, order].reshape(M, -1)[:, :n], single)


@pytest.mark.parametrize("block,channel", [(128, False), (128, True), (256, True)])
def test_grouped_gemm(block, channel):
    import lightop_b200 as lo
    E, tiles, K = len(COUNTS), 16, 7168
    g = torch.Generator(device=DEV).manual_seed(block)
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32, device=DEV) for e, c in enumerate(COUNTS)])
    ids = ids[torch.randperm(len(ids), generator=g, device=DEV)].view(-1, 1)
    M = len(ids)
    q, w = _int8(g, M, K), _int8(g, E, tiles * 128, K)
    if channel:
        s, w_s = torch.rand(M, 1, generator=g, device=DEV) * 0.05 + 1e-3, torch.rand(E, tiles * 128, 1, generator=g, device=DEV) * 9e-4 + 1e-4
    else:
        s, w_s = torch.rand(M, K // 128, generator=g, device=DEV) * 0.05 + 1e-3, torch.rand(E, tiles, K // 128, generator=g, device=DEV) * 9e-3 + 1e-3
    wgt = torch.rand(M, 1, generator=g, device=DEV)
    order = lo.moe.moe_align_block_size(ids, block, E)

    def run(w, w_s):
        out = torch.full((M, 1, w.shape[1]), float("nan"), dtype=torch.bfloat16, device=DEV)
        lo.moe.moe_gemm_w8a8(q, w.contiguous(), out, s, w_s.contiguous(), wgt, *order, 1, {"BLOCK_SIZE_M": block})
        return out
    n = (tiles - 1) * 128
    pairs, single = run(w, w_s), run(w[:, :n], w_s[:, :n] if channel else w_s[:, :-1])
    torch.cuda.synchronize()
    lo.check_device_status()
    assert torch.equal(pairs[..., :n], single) and not torch.isnan(pairs.float()).any()


@pytest.mark.parametrize("counts", [COUNTS, [min(c, 160) for c in COUNTS], [c // 2 for c in COUNTS]])
@pytest.mark.parametrize("channel", [False, True])
def test_layer(counts, channel):
    import lightop_b200 as lo
    E, H, I = len(counts), 7168, 2048
    w1, w2, w1_s, w2_s = synthetic.make_weights(E, H, I, seed=1, device=DEV)
    if channel:
        w1_s, w2_s = synthetic.make_channel_scales(E, H, I, seed=1, device=DEV)
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32, device=DEV) for e, c in enumerate(counts)])
    ids = ids[torch.randperm(len(ids), device=DEV, generator=torch.Generator(device=DEV).manual_seed(2))]
    x, _ = synthetic.make_activations(len(ids), H, E, seed=3, device=DEV)
    w = torch.rand(len(ids), device=DEV) + 0.5

    def run(rows, first, last, **kw):
        return lo.moe.fused_experts_impl_int8(x[rows], w1[first:last], w2[first:last], w[rows].view(-1, 1), (ids[rows] - first).view(-1, 1), None,
                                              use_int8_w8a8=True, per_channel_quant=channel, block_shape=None if channel else [128, 128],
                                              w1_scale=w1_s[first:last], w2_scale=w2_s[first:last], **kw)
    y = run(torch.arange(len(ids), device=DEV), 0, E)
    for e in range(E):
        rows = torch.nonzero(ids == e).reshape(-1)
        if len(rows):
            assert torch.equal(y[rows], run(rows, e, e + 1)), counts[e]
    lo.check_device_status()


@pytest.mark.parametrize("max_m", [128, 160, 300])
def test_masked_layout_by_hint(max_m):
    # the hint decides on the form: none, too few rows for pairs, enough, more than there can be, and what is no number
    import lightop_b200 as lo
    E, N, K = 24, 2048, 7168
    g = torch.Generator(device=DEV).manual_seed(max_m)
    a, w = (_int8(g, E, max_m, K), torch.rand(E, max_m, 1, generator=g, device=DEV)), (_int8(g, E, N, K), torch.rand(E, N, 1, generator=g, device=DEV))
    rows = torch.tensor([min(c, max_m) for c in COUNTS], dtype=torch.int32, device=DEV)
    outs = []
    for hint in (0, 1, 100, 1 << 70, -5, None):
        d = torch.full((E, max_m, N), -5.0, dtype=torch.bfloat16, device=DEV)
        lo.gemm_ops.m_grouped_w8a8_gemm_nt_masked(a, w, d, rows, hint)
        outs.append(d)
    torch.cuda.synchronize()
    lo.check_device_status()
    assert all(torch.equal(outs[0], d) for d in outs[1:])
    for e in range(E):
        assert bool((outs[0][e, int(rows[e]):] == -5.0).all()) and not bool((outs[0][e, :int(rows[e])] == -5.0).all(1).any())


def test_pairs_in_a_graph():
    # captured with the kernels around them and replayed on other inputs at the same addresses
    import lightop_b200 as lo
    g = torch.Generator(device=DEV).manual_seed(5)
    x = torch.randn(1000, 7168, generator=g, device=DEV).to(torch.bfloat16)
    w, w_s = _int8(g, 34 * 128, 7168), torch.rand(34, 56, generator=g, device=DEV) * 9e-3 + 1e-3
    run = lambda: lo.gemm_ops.apply_w8a8_block_int8_linear(x, w, [128, 128], w_s)  # noqa: E731
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = run()
    for _ in range(3):
        x.copy_(torch.randn(1000, 7168, generator=g, device=DEV).to(torch.bfloat16))
        graph.replay()
        assert torch.equal(y, run())
    lo.check_device_status()
