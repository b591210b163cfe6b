"""Alignment of many ids in a partition of the device (a green context) that has no room for the cluster of sixteen CTAs."""
import pytest
import torch

from test_gpu_kernels import _check_align

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,E", [(6144, 8), (24576, 1024)])          # two CTAs a SM by their shared memory, and one
def test_partition_without_room_for_the_wide_cluster(M, E):
    import lightop_b200 as lo
    from torch.cuda import green_contexts
    if not green_contexts.SUPPORTED:
        pytest.skip("torch without green contexts")
    ids = torch.randint(0, E, (M, 1), generator=torch.Generator().manual_seed(M), dtype=torch.int32)
    _check_align(lo, ids, E, 16)          # the whole device first: its answer must not serve the partition
    torch.cuda.synchronize()
    part = green_contexts.GreenContext.create(8, 0)
    part.set_context()
    try:
        _check_align(lo, ids, E, 16)
        torch.cuda.synchronize()
    finally:
        part.pop_context()
    _check_align(lo, ids, E, 16)
