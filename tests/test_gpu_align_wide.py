"""Alignment as a cluster of sixteen CTAs with batches of ids: both sides of the number of ids from which it takes the call, a last batch and a
last segment that are short, segments of more than one batch, ids outside the experts."""
import pytest
import torch

from test_gpu_kernels import _check_align

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
