"""Alignment as a cluster of sixteen CTAs with batches of ids: both sides of the number of ids from which it takes the call, a last batch and a
last segment that are short, segments of more than one batch, ids outside the experts (with the other forms beside it), and the positions and
chunks that a layer gets from it."""
import pytest
import torch

from oracle import moe_block_int8 as O
from test_gpu_kernels import _check_align
from test_gpu_route_small import _layer, check_tables

pytestmark = pytest.mark.gpu


# 6144 ids: the first call; 65536: a batch of 128 ids a warp exactly; 65537 and 70001: a second batch, of few ids; 131073: a third
@pytest.mark.parametrize("M,k", [(6143, 1), (768, 8), (6145, 1), (1024, 8), (8192, 8), (65537, 1), (10001, 7), (43691, 3)])
@pytest.mark.parametrize("E,dtype", [(8, torch.int64), (256, torch.int32)])
def test_order_and_tables(M, k, E, dtype):
    import lightop_b200 as lo
    g = torch.Generator().manual_seed(M + E)
    ids = torch.randint(0, E, (M, k), generator=g).to(dtype)
    _check_align(lo, ids, E, 16)
    emap = torch.full((E,), -1, dtype=torch.int32)
    emap[E // 4:E // 2] = torch.arange(E // 2 - E // 4, dtype=torch.int32)
    _check_align(lo, ids, E, 16, expert_map=emap, ignore=True)


@pytest.mark.parametrize("M,E", [(20000, 1024), (24576, 1024), (6144, 1), (30000, 3)])
def test_ends_of_the_number_of_experts(M, E):
    import lightop_b200 as lo
    ids = torch.randint(0, E, (M, 1), generator=torch.Generator().manual_seed(M), dtype=torch.int32)
    _check_align(lo, ids, E, 128)


def _with_ids_outside(ids, E, seed):
    """A tenth of the ids replaced by ones that name no expert: negative, E and beyond, numbers that a narrower type would take for an expert."""
    outside = [-1, E, E + 70000, 65536, 65536 + E // 2, -65536, 2 ** 31 - 1, -2 ** 31]
    if ids.dtype == torch.int64:
        outside += [2 ** 32, 2 ** 32 + E // 2, 2 ** 33, -2 ** 40, 2 ** 63 - 1, -2 ** 63]
    g = torch.Generator().manual_seed(seed)
    flat = ids.reshape(-1)
    at = torch.randperm(flat.numel(), generator=g)[:max(len(outside), flat.numel() // 10)]
    flat[at] = torch.tensor(outside, dtype=torch.int64)[torch.arange(at.numel()) % len(outside)].to(ids.dtype)
    return ids


# one CTA; the cluster of eight; of sixteen with one batch a warp, and with several
@pytest.mark.parametrize("numel", [97, 2047, 2048, 6143, 6144, 70001])
@pytest.mark.parametrize("E,dtype", [(8, torch.int64), (40, torch.int32), (256, torch.int64)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_ids_outside_the_experts(numel, E, dtype, mode):
    import lightop_b200 as lo
    g = torch.Generator().manual_seed(numel + E)
    ids = _with_ids_outside(torch.randint(0, E, (numel, 1), generator=g).to(dtype), E, numel)
    emap = torch.full((E,), -1, dtype=torch.int32)
    emap[E // 4:E // 2] = torch.arange(E // 2 - E // 4, dtype=torch.int32)
    inside = (ids >= 0) & (ids < E)
    local = torch.where(inside, ids.to(torch.int64), torch.tensor(-1))
    if mode == 1:
        local = torch.where(inside, emap[local.clamp(min=0)].to(torch.int64), torch.tensor(-1))
    s, e, n = lo.moe.moe_align_block_size(ids.cuda(), 16, E, emap.cuda() if mode else None, ignore_invalid_experts=mode == 1)
    s_ref, e_ref, n_ref = O.align_block_size(local, E, 16)
    if mode == 2:
        e_ref = emap[e_ref.long()]
    total = int(n.item())
    assert total == int(n_ref.item()) and torch.equal(s.cpu()[:total], s_ref) and torch.equal(e.cpu()[:total // 16], e_ref.to(torch.int32))
    assert bool((s.cpu()[total:] == numel).all()) and bool((e.cpu()[total // 16:] == -1).all())


# the positions (by the rows that the quantiser scattered with them) and the chunk table of a layer: 6144 ids and one less, several batches a
# warp, 128-row and 160-row chunks
@pytest.mark.parametrize("M,k,E,dtype", [(6143, 1, 16, torch.int32), (3072, 2, 16, torch.int32), (2100, 3, 100, torch.int64), (22000, 3, 8, torch.int32)])
@pytest.mark.parametrize("mapped", [False, True])
def test_positions_and_chunks_of_a_layer(M, k, E, dtype, mapped):
    import lightop_b200 as lo
    g = torch.Generator().manual_seed(M + E)
    ids = _with_ids_outside(torch.randint(0, E, (M, k), generator=g).to(dtype), E, M)
    x = torch.randn(M, 128, generator=g).to(torch.bfloat16).cuda()
    local, emap, E_local = torch.where((ids >= 0) & (ids < E), ids.to(torch.int64), torch.tensor(-1)), None, E
    if mapped:
        E_local = E // 4
        emap = torch.full((E,), -1, dtype=torch.int32)
        emap[torch.randperm(E, generator=g)[:E_local]] = torch.arange(E_local, dtype=torch.int32)
        local = torch.where(local >= 0, emap[local.clamp(min=0)].to(torch.int64), torch.tensor(-1))
    _, t, launches, _ = _layer(M, k, E, 128, 128, ids.cuda(), x, emap.cuda() if mapped else None, E_local)
    assert launches == 5
    check_tables(t, local, E, *lo.quant.per_token_group_quant_int8(x, 128))
