"""Small block-scaled layers, whose alignment and quantisation are one kernel: its order, tables, codes and scales against the alignment
operator and the group quantiser, at the edges of its range; the layer against the oracle on both sides of the limit."""
import ctypes

import pytest
import torch

from oracle import moe_block_int8 as O
from util import assert_out_close

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(M, k, E, H, I, ids, x, expert_map=None, E_local=None):
    """One call of the C entry; (out, tables read back from the workspace, launches)."""
    import lightop_b200 as lo
    from lightop_b200 import _lib, synthetic
    lib = _lib.load()
    E_local = E_local or E
    w1, w2, s1, s2 = synthetic.make_weights(E_local, H, I, seed=3, device=DEV)
    wgt = torch.rand(M, k, generator=torch.Generator().manual_seed(1)).to(DEV)
    ws = torch.full((lib.lo_fused_moe_workspace_bytes(M, E_local, E, k, H, I),), 0x5a, dtype=torch.uint8, device=DEV)
    cache = torch.empty(M * k * H, dtype=torch.bfloat16, device=DEV)
    out = torch.empty(M, H, dtype=torch.bfloat16, device=DEV)
    before = lib.lo_launch_count()
    st = lib.lo_fused_moe_block_int8(x.data_ptr(), w1.data_ptr(), w2.data_ptr(), s1.data_ptr(), s2.data_ptr(), wgt.data_ptr(), ids.data_ptr(),
                                     _lib.LO_I64 if ids.dtype == torch.int64 else _lib.LO_I32, expert_map.data_ptr() if expert_map is not None else 0,
                                     E, M, E_local, k, H, I, cache.data_ptr(), 0, out.data_ptr(), 0, 1.0, ws.data_ptr(), ws.numel(), 0,
                                     torch.cuda.current_stream().cuda_stream)
    assert st == 0
    torch.cuda.synchronize()
    off = (ctypes.c_int64 * 8)()
    assert lib.lo_fused_moe_workspace_layout(M, E_local, E, k, H, I, off) == 0
    cap, raw = off[7], ws.cpu()
    i32 = lambda at, n: raw[at:at + 4 * n].view(torch.int32)
    n_pad, n_chunks = i32(off[0], 2).tolist()
    tables = {"n_pad": n_pad, "chunks": i32(off[4], 4 * n_chunks).view(-1, 4), "sorted": i32(off[3], cap),
              "xq": raw[off[1]:off[1] + cap * H].view(torch.int8).view(cap, H), "xs": raw[off[2]:off[2] + 4 * cap * (H // 128)].view(torch.float32).view(cap, -1)}
    return out, tables, lib.lo_launch_count() - before, (w1, w2, s1, s2, wgt)


def check_tables(t, local_ids, E, q, s):
    """Tables, rows and scales read back from a layer's workspace against the codes and scales of the tokens; ids outside [0, E) have no row."""
    M, k = local_ids.shape
    q, s, flat = q.cpu(), s.cpu(), local_ids.reshape(-1).tolist()
    by_expert = [[] for _ in range(E)]
    for i, v in enumerate(flat):
        if 0 <= v < E:
            by_expert[v].append(i)
    avg = M * k // E
    most = 160 if avg >= 120 else (64 if avg <= 48 else 128)
    want, chunks = [], []
    for e, mine in enumerate(by_expert):
        n = -(-len(mine) // most)
        per = -(-(-(-len(mine) // n)) // 16) * 16 if n else 0
        chunks += [[e, len(want) + r, min(per, len(mine) - r), (len(mine) - r - 1) // per] for r in range(0, len(mine), per or 1)]
        want += mine + [M * k] * (-len(mine) % 16)
    assert t["n_pad"] == len(want) and t["sorted"].tolist() == want + [M * k] * (t["sorted"].numel() - len(want))
    assert t["chunks"].tolist() == chunks
    rows = torch.tensor(want)
    real = rows < M * k
    token = rows[real] // k
    assert torch.equal(t["xq"][:len(want)][real], q[token]) and torch.equal(t["xs"][:len(want)][real], s[token])


# one id; many ids of one expert (more than a segment, more than a chunk); no multiple of anything; rows of one share and of several
# (256 lanes of sixteen elements); the largest call; ids outside the experts; as many experts as there can be
@pytest.mark.parametrize("M,k,E,H,same,dtype", [(1, 1, 1, 128, False, torch.int32), (1, 8, 256, 7168, False, torch.int32), (17, 3, 9, 640, False, torch.int64),
                                                (32, 8, 256, 4096, False, torch.int32), (128, 2, 4, 256, True, torch.int32), (128, 2, 1024, 128, False, torch.int32),
                                                (33, 7, 40, 4224, False, torch.int64), (100, 2, 3, 384, True, torch.int32)])
def test_tables_rows_and_scales(M, k, E, H, same, dtype):
    import lightop_b200 as lo
    g = torch.Generator().manual_seed(M + k + E)
    ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(M)]).to(dtype)
    if same:
        ids[:] = E - 1
    ids[M // 2, k - 1] = -1 if M > 1 else ids[0, k - 1]            # a slot without an expert
    x = torch.randn(M, H, generator=g).to(torch.bfloat16).to(DEV)
    _, t, launches, _ = _layer(M, k, E, H, 128, ids.to(DEV), x)
    assert launches == 4
    check_tables(t, ids, E, *lo.quant.per_token_group_quant_int8(x, 128))


@pytest.mark.parametrize("M", [32, 33])          # 256 ids are one kernel, 264 are two
@pytest.mark.parametrize("mapped", [False, True])
def test_layer_on_both_sides_of_the_limit(M, mapped):
    k, E, H, I = 8, 32, 512, 256
    g = torch.Generator().manual_seed(M)
    x = torch.randn(M, H, generator=g).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(M)]).to(torch.int32)
    emap, E_local = None, E
    if mapped:
        E_local = 8
        emap = torch.full((E,), -1, dtype=torch.int32)
        emap[torch.randperm(E, generator=g)[:E_local]] = torch.arange(E_local, dtype=torch.int32)
    out, _, launches, (w1, w2, s1, s2, wgt) = _layer(M, k, E, H, I, ids.to(DEV), x.to(DEV), emap.to(DEV) if mapped else None, E_local)
    assert launches == (4 if M * k <= 256 else 5)
    local = emap[ids.long()] if mapped else ids
    ref = O.fused_moe_block_int8(x, w1.cpu(), w2.cpu(), s1.cpu(), s2.cpu(), torch.where(local >= 0, wgt.cpu(), torch.zeros(())), local.clamp(min=0).to(torch.int32))
    assert_out_close(out, ref, f"M={M} mapped={mapped}")
