"""Alignment and expert-parallel plans from two threads at once, with numbers of experts whose shared memory differs: what one call asks the runtime for
must not take from the other between its preparation and its launch."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("numel", [512, 4096, 30000])          # the single CTA, the clusters of eight and of sixteen
def test_many_and_few_experts_side_by_side(numel):
    from lightop_b200 import _lib
    lib = _lib.load()
    gate = threading.Barrier(2)
    failed, padded = [], {}

    def work(E):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            ids = (torch.arange(numel, device=DEV) % E).to(torch.int32)
            cap = numel + E * 15
            out = torch.empty(cap, dtype=torch.int32, device=DEV)
            blocks = torch.empty(-(-cap // 16), dtype=torch.int32, device=DEV)
            n = torch.empty(1, dtype=torch.int32, device=DEV)
            plan = torch.empty(numel, dtype=torch.int32, device=DEV)
            gate.wait()
            for _ in range(400):
                st = lib.lo_moe_align_block_size(ids.data_ptr(), _lib.LO_I32, numel, E, 16, 0, 0, out.data_ptr(), cap, blocks.data_ptr(), blocks.numel(),
                                                 n.data_ptr(), stream.cuda_stream)
                st2 = lib.lo_ep_build_m_indices(ids.data_ptr(), _lib.LO_I32, numel, plan.data_ptr(), numel, E, 1, stream.cuda_stream)
                if st or st2:
                    failed.append((E, st, st2))
        stream.synchronize()
        padded[E] = int(n.item())

    threads = [threading.Thread(target=work, args=(E,)) for E in (1024, 400)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[:4]
    assert padded == {E: sum(-(-(numel // E + (e < numel % E)) // 16) * 16 for e in range(E)) for E in (1024, 400)}
