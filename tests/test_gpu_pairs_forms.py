"""GPU test of which form of the grouped GEMM, pairs of CTAs or single ones, each side of the comparisons in test_gpu_pairs.py takes, so that a rule
which sends both sides to one form fails; and the same comparisons for what that file leaves out: 160-row chunks of the block-scaled layer,
blocks without a local expert, a table of output row addresses, a partition of few SMs."""
import functools

import pytest
import test_gpu_ep_emulated
import test_gpu_pairs as pairs
import torch

from lightop_b200 import _lib, synthetic

pytestmark = pytest.mark.gpu
DEV = "cuda"
# with more experts of several chunks, 152 rows on average: the block-scaled layer's table is cut at 160 rows
COUNTS_WIDE = pairs.COUNTS + [320, 321, 480, 319, 337, 175]


def _on_pairs():
    return _lib.load().lo_pair_launch_count()


def _forms(monkeypatch, module, name):
    """From now on, for every call of module.name, the grouped GEMMs that it ran on pairs (and the call's arguments)."""
    call, forms = getattr(module, name), []

    def counted(*args, **kw):
        before = _on_pairs()
        out = call(*args, **kw)
        forms.append((_on_pairs() - before, args))
        return out
    monkeypatch.setattr(module, name, counted)
    return forms


def _cases(test, names):
    """The cases of a test there."""
    return next(m.args[1] for m in test.pytestmark if m.name == "parametrize" and m.args[0] == names)


@pytest.mark.parametrize("M,tiles,K", _cases(pairs.test_dense_linear, "M,tiles,K"))
def test_dense_linear(monkeypatch, M, tiles, K):
    import lightop_b200 as lo
    forms = _forms(monkeypatch, lo.gemm_ops, "matmul_block_int8")
    pairs.test_dense_linear(M, tiles, K)
    assert [n for n, _ in forms] == [1, 0, 0]


@pytest.mark.parametrize("block,channel", _cases(pairs.test_grouped_gemm, "block,channel"))
@pytest.mark.parametrize("absent", [False, True])
def test_grouped_gemm(monkeypatch, block, channel, absent):
    import lightop_b200 as lo
    E = len(pairs.COUNTS)
    local = torch.arange(E, dtype=torch.int32, device=DEV)
    if absent:      # every third expert is another rank's
        local[::3] = -1
    align, ids = lo.moe.moe_align_block_size, []

    def align_mapped(topk_ids, block_size, num_experts):
        ids.append(topk_ids)
        order = align(topk_ids, block_size, num_experts, local)
        assert bool((order[1][:int(order[2]) // block_size] == -1).any()) == absent
        return order
    monkeypatch.setattr(lo.moe, "moe_align_block_size", align_mapped)
    forms = _forms(monkeypatch, lo.moe, "moe_gemm_w8a8")
    pairs.test_grouped_gemm(block, channel)
    assert [n for n, _ in forms] == [1, 0]
    gone = local[ids[0].view(-1).long()] < 0
    out = forms[0][1][2]
    assert not bool(out[gone].any()) and bool((out[~gone] != 0).any(-1).all())


@pytest.mark.parametrize("counts", _cases(pairs.test_layer, "counts") + [COUNTS_WIDE])
@pytest.mark.parametrize("channel", [False, True])
def test_layer(monkeypatch, counts, channel):
    import lightop_b200 as lo
    forms = _forms(monkeypatch, lo.moe, "fused_experts_impl_int8")
    pairs.test_layer(counts, channel)
    # (with few rows an expert the block-scaled down GEMM stays below the line)
    assert forms[0][0] == (2 if channel or sum(counts) // len(counts) >= 83 else 1)
    assert len(forms) > 20 and all(n == 0 for n, _ in forms[1:])


@pytest.mark.parametrize("max_m", _cases(pairs.test_masked_layout_by_hint, "max_m"))
def test_masked_layout_by_hint(monkeypatch, max_m):
    import lightop_b200 as lo
    forms = _forms(monkeypatch, lo.gemm_ops, "m_grouped_w8a8_gemm_nt_masked")
    pairs.test_masked_layout_by_hint(max_m)
    assert {args[4]: n for n, args in forms} == {0: 0, 1: 0, 100: 1, 1 << 70: 1, -5: 0, None: 0}


def test_pairs_in_a_graph():
    before = _on_pairs()
    pairs.test_pairs_in_a_graph()
    assert _on_pairs() - before == 1 + 1 + 3      # once ahead, once captured, and after each replay


def test_expert_rows_into_addresses(monkeypatch):
    # the expert side of expert parallelism with a table of row addresses (two emulated ranks in this GPU's memory, which do not wait on one another), at
    # sizes that take pairs; compared with the layer of one GPU there
    import lightop_b200 as lo
    monkeypatch.setattr(synthetic, "make_weights", functools.partial(synthetic.make_weights, device=DEV))
    before = _on_pairs()
    test_gpu_ep_emulated.test_peer_transport_with_emulated_ranks(lo, 2, 32, 4, 7168, 2048, (760, 340))
    # both GEMMs of either rank's experts (137 rows each), and of the larger comparison (340 tokens: 64-row chunks, single CTAs)
    assert _on_pairs() - before == 4 + 2


@pytest.mark.parametrize("sms", [8, 64])
def test_pairs_in_a_partition(sms):
    # a green context of few SMs: the pairs of a call run after one another there
    import lightop_b200 as lo
    from torch.cuda import green_contexts
    if not green_contexts.SUPPORTED:
        pytest.skip("torch without green contexts")
    g = torch.Generator(device=DEV).manual_seed(6)
    x = torch.randn(1000, 7168, generator=g, device=DEV).to(torch.bfloat16)
    w, w_s = pairs._int8(g, 34 * 128, 7168), torch.rand(34, 56, generator=g, device=DEV) * 9e-3 + 1e-3
    want = lo.gemm_ops.apply_w8a8_block_int8_linear(x, w, [128, 128], w_s)
    torch.cuda.synchronize()
    part = green_contexts.GreenContext.create(sms, 0)
    part.set_context()
    try:
        before = _on_pairs()
        got = lo.gemm_ops.apply_w8a8_block_int8_linear(x, w, [128, 128], w_s)
        assert _on_pairs() - before == 1
        torch.cuda.synchronize()
    finally:
        part.pop_context()
    lo.check_device_status()
    assert torch.equal(got, want)
