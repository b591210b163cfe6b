"""GPU tests of the streaming kernels where their instruction-saving forms could differ from the plain ones: quotients from a
refined reciprocal against the library's division, and the top-k sum at the sizes where its split changes."""
import pytest
import torch

from oracle import moe_block_int8 as O

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.fixture(scope="module")
def lo():
    import lightop_b200
    return lightop_b200


@pytest.mark.parametrize("dtype,bits", [(torch.bfloat16, 7), (torch.float16, 10)])
@pytest.mark.parametrize("exponent", [0, -6, 9])
def test_group_quant_every_pair_of_maximum_and_element(lo, dtype, bits, exponent):
    """The code of an element depends on it and on its group's maximum only, and is the same for both times a power of two: every
    mantissa of the maximum with every element of the nine octaves below it (what is smaller has code 0)."""
    n = 1 << bits
    mant = 1.0 + torch.arange(n, dtype=torch.float64) / n
    elems = torch.cat([mant * 2.0 ** -e for e in range(9)])
    elems = torch.cat([elems, -elems])
    per = 127
    rows = -(-elems.numel() // per)
    body = torch.zeros(rows * per, dtype=torch.float64)
    body[:elems.numel()] = elems
    for top in mant.split(128):
        x = torch.empty(top.numel(), rows, 128, dtype=torch.float64)
        x[..., 0] = top[:, None]
        b = body.view(1, rows, per).expand(top.numel(), rows, per)
        x[..., 1:] = torch.where(b.abs() <= top[:, None, None], b, torch.zeros((), dtype=torch.float64))
        x = (x * 2.0 ** exponent).to(dtype).reshape(-1, 128)
        q_ref, s_ref = O.group_quant_int8(x, 128)
        q, s = lo.quant.per_token_group_quant_int8(x.to(DEV), 128)
        assert torch.equal(s.cpu(), s_ref) and torch.equal(q.cpu(), q_ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_group_quant_infinity_nan_and_the_ends_of_the_range(lo, dtype):
    big = torch.finfo(dtype).max
    x = torch.randn(8, 256, generator=torch.Generator().manual_seed(3)).to(dtype)
    x[0, 5] = float("inf")
    x[1, 130] = float("-inf")
    x[2, 7] = float("nan")
    x[3, :128] = 0
    x[4, :128] = torch.finfo(dtype).tiny
    x[5, 3], x[5, 4] = big, -big
    x[6, 129] = float("nan")
    x[6, 128] = float("inf")
    q, s = lo.quant.per_token_group_quant_int8(x.to(DEV), 128)
    # the kernel's rule: the maximum passes over NaN, the quotient is the IEEE one, NaN has the code -128
    v = x.float().view(8, 2, 128)
    eps = float(torch.tensor(1e-10).to(dtype))
    amax = torch.where(v.isnan(), torch.zeros(()), v.abs()).amax(-1).clamp(min=eps)
    scale = amax / 127.0
    r = v / scale[..., None]
    want = torch.where(r.isnan(), torch.full((), -128.0), r.clamp(-128, 127)).trunc().to(torch.int8)
    assert torch.equal(s.cpu(), scale) and torch.equal(q.cpu().view(8, 2, 128), want)


def test_group_quant_codes_that_begin_on_eight_bytes(lo):
    from lightop_b200 import _lib
    x = torch.randn(9, 256, generator=torch.Generator().manual_seed(4)).to(torch.bfloat16).to(DEV)
    q, s = lo.quant.per_token_group_quant_int8(x, 128)
    room = torch.zeros(9 * 256 + 16, dtype=torch.int8, device=DEV)
    s2 = torch.empty_like(s)
    assert _lib.load().lo_group_quant_int8(x.data_ptr(), _lib.LO_BF16, 18, 128, 1e-10, room.data_ptr() + 8, s2.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(room[8:8 + 9 * 256].view(9, 256), q) and torch.equal(s2, s)
    assert not room[:8].any() and not room[-8:].any()


@pytest.mark.parametrize("group", [64, 128, 256])
def test_group_quant_fp32_on_both_sides_of_the_wide_form(lo, group):
    """Eight elements a thread up to 2^24 elements, sixteen above: a large call has the bits of its parts."""
    K = 7168
    x = torch.randn(2341, K, generator=torch.Generator(device=DEV).manual_seed(group), device=DEV)
    x[5, :group] = 0
    assert x.numel() > 1 << 24 and x[:2340].numel() <= 1 << 24
    q, s = lo.quant.per_token_group_quant_int8(x, group)
    for part in (slice(0, 2340), slice(2333, 2341)):
        q2, s2 = lo.quant.per_token_group_quant_int8(x[part], group)
        assert torch.equal(q[part], q2) and torch.equal(s[part], s2)
    q_ref, s_ref = O.group_quant_int8(x[:9].cpu(), group)
    assert torch.equal(q[:9].cpu(), q_ref) and torch.equal(s[:9].cpu(), s_ref)


def test_silu_quant_every_gate(lo):
    """Every bf16 gate, with eight of one magnitude range to a row so that small results keep their codes."""
    gates = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).to(DEV)
    gates = gates[~gates.isnan()]
    gates = torch.cat([gates, gates[:-gates.numel() % 8]]).view(-1, 8)
    extra = torch.tensor([[float("inf"), 1, -1, 2, float("-inf"), 0, 5, float("nan")], [float("-inf")] * 8, [-3.0e38, -100, -90, -89, -88.5, -88, -87, -80]],
                         dtype=torch.bfloat16, device=DEV)
    gates = torch.cat([gates, extra])
    up = torch.randn(gates.shape, generator=torch.Generator().manual_seed(6)).to(torch.bfloat16).to(DEV)
    q, s = lo.activation.fuse_silu_mul_quant(torch.cat([gates, up], 1).contiguous())
    g = gates.float()
    act = ((g / (1.0 + torch.exp(-g))).to(torch.bfloat16).float() * up.float()).to(torch.bfloat16).float()
    amax = torch.where(act.isnan(), torch.zeros((), device=DEV), act.abs()).amax(-1, keepdim=True)
    r = act * torch.where(amax == 0, torch.zeros((), device=DEV), torch.full_like(amax, 127.0) / amax)
    want = torch.where(r.isnan(), torch.full((), -128.0, device=DEV), r.round().clamp(-128, 127)).to(torch.int8)
    assert torch.equal(s.view(-1, 1), amax / torch.full_like(amax, 127.0))
    assert torch.equal(q.view_as(want), want)


# both numbers of threads a row (by rows and by width), widths that fill the last vector a thread keeps in part, and rows too wide to
# be kept, which are read and evaluated twice
@pytest.mark.parametrize("rows,d", [(3, 8), (3, 1544), (700, 1544), (700, 4096), (5, 4104), (700, 4104), (5, 8192), (3, 8200), (310, 8200), (2, 18432)])
def test_silu_quant_widths(lo, rows, d):
    g = torch.Generator(device=DEV).manual_seed(rows + d)
    x = (torch.randn(rows, 2 * d, generator=g, device=DEV) * 4).to(torch.bfloat16)
    x[1] = 0
    q, s = lo.activation.fuse_silu_mul_quant(x)
    gate, up = x[:, :d].float(), x[:, d:].float()
    act = ((gate / (1.0 + torch.exp(-gate))).to(torch.bfloat16).float() * up).to(torch.bfloat16).float()
    amax = act.abs().amax(-1, keepdim=True)
    r = act * torch.where(amax == 0, torch.zeros((), device=DEV), torch.full_like(amax, 127.0) / amax)
    assert torch.equal(s.view(-1, 1), amax / torch.full_like(amax, 127.0))
    assert torch.equal(q, r.round().clamp(-128, 127).to(torch.int8))


# the forms' lines (two and twelve full blocks a SM) from both sides, columns that do not fill the last block, slots that are all, some or
# not there, more than 32 of them
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,k,H", [(1, 8, 7168), (296, 8, 7168), (297, 8, 7168), (1185, 3, 2056), (1300, 2, 256), (5, 37, 264), (1200, 40, 136), (400, 9, 8200)])
def test_moe_sum_split(lo, dtype, M, k, H):
    g = torch.Generator(device=DEV).manual_seed(M + k)
    a = torch.randn(M, k, H, generator=g, device=DEV).to(dtype)
    mask = torch.rand(M, k, generator=g, device=DEV) < 0.3
    mask[0] = False
    mask[-1] = True
    bias = torch.randn(M, H, generator=g, device=DEV).to(dtype)
    for m in (None, mask):
        for b, f in ((None, 1.0), (bias, 2.5)):
            out = torch.empty(M, H, dtype=dtype, device=DEV)
            lo.moe.moe_sum(a, out, bias=b, expert_mask=m, factor=f)
            acc = torch.zeros(M, H, device=DEV)
            for j in range(k):
                acc = acc + (a[:, j].float() if m is None else torch.where(m[:, j:j + 1], a[:, j].float(), torch.zeros((), device=DEV)))
            if b is None:
                assert torch.equal(out, (acc * f).to(dtype))
            else:      # one fused or two rounded operations: half a step of the product and of the sum, then of the result's type
                want = acc.double() * f + b.double()
                tol = 2.0 ** -23 * (acc.double() * f).abs() + 2.0 ** (-8 if dtype == torch.bfloat16 else -23) * want.abs() + 1e-30
                assert bool(((out.double() - want).abs() <= tol).all())


@pytest.mark.parametrize("M", [7, 600])
def test_layer_of_a_shard_passes_over_tokens_without_a_local_expert(lo, M):
    """One expert of eight is local: most tokens have no position in the sorted rows, some have several slots."""
    from lightop_b200 import synthetic
    E, k, H, I = 8, 2, 256, 256
    w1, w2, w1_s, w2_s = synthetic.make_weights(E, H, I, seed=1, device=DEV)
    x, logits = synthetic.make_activations(M, H, E, seed=2, device=DEV)
    weights = torch.empty(M, k, device=DEV)
    ids = torch.empty(M, k, dtype=torch.int32, device=DEV)
    lo.moe.topk_softmax(weights, ids, None, logits, True)
    total = torch.zeros(M, H, dtype=torch.float64, device=DEV)
    for e in range(E):
        emap = torch.full((E,), -1, dtype=torch.int32, device=DEV)
        emap[e] = 0
        y = lo.moe.fused_experts_impl_int8(x, w1[e:e + 1].contiguous(), w2[e:e + 1].contiguous(), weights, ids, torch.empty(M * k * H, dtype=torch.bfloat16, device=DEV),
                                           use_int8_w8a8=True, block_shape=[128, 128], w1_scale=w1_s[e:e + 1].contiguous(), w2_scale=w2_s[e:e + 1].contiguous(),
                                           global_num_experts=E, expert_map=emap)
        assert not y[~(ids == e).any(1)].any()
        total += y.double()
    y = lo.moe.fused_experts_impl_int8(x, w1, w2, weights, ids, torch.empty(M * k * H, dtype=torch.bfloat16, device=DEV), use_int8_w8a8=True,
                                       block_shape=[128, 128], w1_scale=w1_s, w2_scale=w2_s)
    # every row once in each: the parts are rounded to bf16 where the whole is rounded once
    assert float((total - y.double()).norm() / y.double().norm()) < 2 ** -8


# four warps copy a position's row up to eight positions a SM, one above: the same ids in front of more positions that do not exist
@pytest.mark.parametrize("K", [128, 1152, 8192, 16384])
@pytest.mark.parametrize("channel", [True, False])
def test_row_copy_on_both_sides_of_the_number_of_warps(lo, K, channel):
    M, E, k, N = 40, 4, 2, 128
    g = torch.Generator(device=DEV).manual_seed(K)
    ids = torch.rand(M, E, generator=g, device=DEV).topk(k, dim=1).indices.to(torch.int32)
    aq = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    w = torch.randint(-127, 128, (E, N, K), generator=g, device=DEV, dtype=torch.int8)
    a_s = torch.rand(M, 1 if channel else K // 128, generator=g, device=DEV) + 0.5
    w_s = torch.rand(E, N if channel else 1, 1 if channel else K // 128, generator=g, device=DEV) + 0.5
    sorted_ids, expert_ids, num_post = lo.moe.moe_align_block_size(ids, 16, E)
    outs = []
    for more in (0, 1600):
        s = torch.cat([sorted_ids, sorted_ids.new_full((more,), M * k)])
        e = torch.cat([expert_ids, expert_ids.new_zeros(more // 16)])
        out = torch.full((M, k, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        lo.moe.moe_gemm_w8a8(aq, w, out, a_s, w_s, None, s, e, num_post, k, {"BLOCK_SIZE_M": 16})
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    # the whole sum of a row, with the scales as they are in exact arithmetic
    want = torch.stack([(aq.double().view(M, -1, K // a_s.shape[1]) * a_s.double()[..., None]).view(M, K) @
                        (w[e].double().view(N, -1, K // w_s.shape[2]) * w_s[e].double()[..., None]).view(N, K).t() for e in range(E)], 1)
    want = torch.gather(want, 1, ids.long()[..., None].expand(M, k, N))
    # K / 128 fp32 products and sums, then one rounding to bf16
    assert float((outs[0].double() - want).norm() / want.norm()) < 2 ** -8


def test_layer_of_a_shard_reads_positions_or_rows_first(lo, monkeypatch):
    """One expert of eight is local and the absent tokens' rows are more than 8 MB: positions first.  The same tokens in smaller calls:
    rows first.  Every row has the same bits."""
    from lightop_b200 import synthetic
    M, E, k, H, I = 11003, 8, 2, 512, 128
    w1, w2, w1_s, w2_s = synthetic.make_weights(E, H, I, seed=3, device=DEV)
    x, logits = synthetic.make_activations(M, H, E, seed=4, device=DEV)
    weights = torch.empty(M, k, device=DEV)
    ids = torch.empty(M, k, dtype=torch.int32, device=DEV)
    lo.moe.topk_softmax(weights, ids, None, logits, True)
    emap = torch.full((E,), -1, dtype=torch.int32, device=DEV)
    emap[3] = 0

    def layer():
        return lo.moe.fused_experts_impl_int8(x, w1[3:4].contiguous(), w2[3:4].contiguous(), weights, ids, None, use_int8_w8a8=True, block_shape=[128, 128],
                                              w1_scale=w1_s[3:4].contiguous(), w2_scale=w2_s[3:4].contiguous(), global_num_experts=E, expert_map=emap)
    y = layer()
    assert not y[~(ids == 3).any(1)].any() and bool(y[(ids == 3).any(1)].any(1).all())
    monkeypatch.setenv("LMSLIM_FUSED_MOE_CHUNK_SIZE", "2999")
    assert torch.equal(layer(), y)


@pytest.mark.parametrize("H", [8, 2056])
def test_reductions_of_more_than_65535_tokens(lo, H):
    T, k = 65541, 2
    g = torch.Generator(device=DEV).manual_seed(H)
    a = torch.randn(T, k, H, generator=g, device=DEV).to(torch.bfloat16)
    mask = torch.rand(T, k, generator=g, device=DEV) < 0.5
    out = torch.empty(T, H, dtype=torch.bfloat16, device=DEV)
    lo.moe.moe_sum(a, out)
    assert torch.equal(out, (a[:, 0].float() + a[:, 1].float()).to(torch.bfloat16))
    lo.moe.moe_sum(a, out, expert_mask=mask)
    m = mask.float()[..., None]
    assert torch.equal(out, (a[:, 0].float() * m[:, 0] + a[:, 1].float() * m[:, 1]).to(torch.bfloat16))
    ids = torch.zeros(T, k, dtype=torch.int32, device=DEV)
    inv = torch.randperm(T * k, generator=g, device=DEV).to(torch.int32).view(T, k)
    w = torch.tensor([1.0, 2.0], device=DEV).expand(T, k).contiguous()      # (products by powers of two are exact: one rounding)
    lo.moe.ep_gather(a.view(T * k, H), ids, w, inv, None, out)
    rows = a.view(T * k, H)[inv.long()].float()
    assert torch.equal(out, (rows[:, 0] + 2.0 * rows[:, 1]).to(torch.bfloat16))


# several tokens a block and a last block that is not full, every form (up to two, up to twelve, more, and more than twenty full blocks
# a SM, fp32 up to six), columns that leave threads of a token's last warp or block without any
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M,k,H", [(1, 1, 8), (67, 8, 256), (301, 8, 1024), (607, 3, 1032), (299, 8, 5120), (9001, 5, 264), (9601, 2, 264), (15001, 2, 264), (5801, 2, 1056), (1700, 33, 4112)])
def test_moe_sum_forms(lo, dtype, M, k, H):
    g = torch.Generator(device=DEV).manual_seed(M + H)
    a = torch.randn(M, k, H, generator=g, device=DEV).to(dtype)
    mask = torch.rand(M, k, generator=g, device=DEV) < 0.4
    valid = torch.tensor([M - M // 3], dtype=torch.int32, device=DEV)
    for m in (None, mask):
        acc = torch.zeros(M, H, device=DEV)
        for j in range(k):
            acc = acc + (a[:, j].float() if m is None else torch.where(m[:, j:j + 1], a[:, j].float(), torch.zeros((), device=DEV)))
        out = torch.full((M, H), 7.0, dtype=dtype, device=DEV)
        lo.moe.moe_sum(a, out, expert_mask=m, num_local_tokens=valid, factor=0.5)
        n = int(valid)
        assert torch.equal(out[:n], (acc[:n] * 0.5).to(dtype)) and bool((out[n:] == 7.0).all())
        none = torch.full_like(out, 7.0)
        lo.moe.moe_sum(a, none, expert_mask=m, num_local_tokens=-valid)
        assert bool((none == 7.0).all())


@pytest.mark.parametrize("M,H", [(5501, 1152), (6003, 1024), (300, 1024), (9601, 512)])
def test_layer_sum_with_few_local_experts(lo, monkeypatch, M, H):
    """One expert of eight is local: the form of four vectors a thread above twenty full blocks a SM, the others below and for narrow
    rows.  The same tokens in smaller calls have the same bits."""
    from lightop_b200 import synthetic
    E, k, I = 8, 2, 128
    w1, w2, w1_s, w2_s = synthetic.make_weights(E, H, I, seed=5, device=DEV)
    x, logits = synthetic.make_activations(M, H, E, seed=6, device=DEV)
    weights = torch.empty(M, k, device=DEV)
    ids = torch.empty(M, k, dtype=torch.int32, device=DEV)
    lo.moe.topk_softmax(weights, ids, None, logits, True)
    emap = torch.full((E,), -1, dtype=torch.int32, device=DEV)
    emap[2] = 0
    shared = torch.randn(M, H, generator=torch.Generator(device=DEV).manual_seed(7), device=DEV).to(torch.bfloat16)

    def layer(ids):
        return lo.moe.fused_experts_impl_int8(x, w1[2:3].clone(), w2[2:3].clone(), weights, ids, None, use_int8_w8a8=True, block_shape=[128, 128],
                                              w1_scale=w1_s[2:3].clone(), w2_scale=w2_s[2:3].clone(), global_num_experts=E, expert_map=emap,
                                              routed_scaling_factor=2.5, shared_output=shared)
    y = layer(ids)
    assert torch.equal(y[~(ids == 2).any(1)], shared[~(ids == 2).any(1)])
    assert torch.equal(layer(ids.long()), y)
    monkeypatch.setenv("LMSLIM_FUSED_MOE_CHUNK_SIZE", "97")
    assert torch.equal(layer(ids), y)
