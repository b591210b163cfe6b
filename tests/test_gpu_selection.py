"""GPU tests of the selections by warp reductions (ties, signed zeros, infinities) and of the alignment on both sides of the number
of ids from which a cluster takes it."""
import pytest
import torch

from test_gpu_kernels import _check_align

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.fixture(scope="module")
def lo():
    import lightop_b200
    return lightop_b200


def _tied_rows(M, E, seed):
    """Rows of few distinct values: many ties, both zeros, experts masked with -inf."""
    g = torch.Generator().manual_seed(seed)
    values = torch.tensor([0.0, -0.0, 1.0, -1.0, 2.5, float("-inf"), 1e-40, -1e-40])
    x = values[torch.randint(0, values.numel(), (M, E), generator=g)]
    x[:, 0] = 3.0
    return x


@pytest.mark.parametrize("E,k", [(1, 1), (8, 2), (31, 5), (33, 8), (128, 8), (256, 8), (300, 32), (1024, 8)])
def test_topk_softmax_ties(lo, E, k):
    x = _tied_rows(65, E, E)
    weights = torch.empty(65, k, device=DEV)
    ids = torch.empty(65, k, dtype=torch.int32, device=DEV)
    lo.moe.topk_softmax(weights, ids, None, x.to(DEV), False)
    # equal logits: the lower expert first (-0 and 0 are equal); once only -inf is left its order does not matter, the weight is 0
    want = torch.sort(x + 0.0, dim=1, descending=True, stable=True).indices[:, :k]
    p = torch.softmax(x, 1)
    finite = torch.gather(x, 1, want) > float("-inf")
    assert torch.equal(ids.cpu().long()[finite], want[finite])
    torch.testing.assert_close(weights.cpu(), torch.where(finite, torch.gather(p, 1, want), torch.zeros(())), rtol=2e-5, atol=2e-6)


# groups of 32 experts are registers of the warp, other sizes are walked in shared memory
@pytest.mark.parametrize("E,groups,keep,k", [(256, 8, 4, 8), (64, 2, 1, 6), (1024, 32, 4, 8), (512, 16, 16, 8), (256, 16, 4, 8), (256, 4, 2, 8), (96, 3, 2, 4)])
def test_grouped_gate_with_ties(lo, E, groups, keep, k):
    g = torch.Generator().manual_seed(E + groups)
    x = torch.randint(-3, 4, (130, E), generator=g).float()       # scores in steps: ties inside and between groups
    x += torch.randint(0, 2, (130, E), generator=g) * 0.25
    bias = torch.zeros(E)
    w, ids = lo.moe.moe_fused_gate(x.to(DEV), bias.to(DEV), groups, keep, k, 0, 2.5, False)
    s = torch.sigmoid(x.to(DEV)).cpu()
    top2 = s.view(130, groups, -1).topk(min(2, E // groups), dim=2).values.sum(2)
    kept = torch.sort(top2, dim=1, descending=True, stable=True).indices[:, :keep]
    mask = torch.zeros(130, groups, dtype=torch.bool).scatter_(1, kept, True).repeat_interleave(E // groups, 1)
    order = torch.sort(torch.where(mask, s, torch.full((), float("-inf"))), dim=1, descending=True, stable=True).indices[:, :k]
    assert torch.equal(ids.cpu().long(), order)
    p = torch.gather(s, 1, order)
    torch.testing.assert_close(w.cpu(), p / p.sum(1, keepdim=True), rtol=2e-5, atol=2e-6)


@pytest.mark.parametrize("numel_rows,k", [(255, 8), (256, 8), (257, 8), (2047, 1), (2049, 1), (300, 8), (1023, 8)])
@pytest.mark.parametrize("E", [8, 256])
def test_align_around_the_cluster(lo, numel_rows, k, E):
    g = torch.Generator().manual_seed(numel_rows + E)
    _check_align(lo, torch.randint(0, E, (numel_rows, k), generator=g, dtype=torch.int32), E, 16)


@pytest.mark.parametrize("E,keep,k,shared", [(8, 2, 2, 0), (32, 8, 8, 0), (32, 32, 6, 0), (2, 1, 1, 0), (16, 5, 6, 1)])
def test_grouped_gate_with_groups_of_one_expert(lo, E, keep, k, shared):
    """The score of such a group is its expert's: the groups kept are the best experts."""
    x = torch.randn(130, E, generator=torch.Generator().manual_seed(E + keep))
    bias = torch.linspace(-0.5, 0.5, E)
    w, ids = lo.moe.moe_fused_gate(x.to(DEV), bias.to(DEV), E, keep, k, shared, 2.5, False)
    s = torch.sigmoid(x.to(DEV)).cpu()
    order = torch.sort(s + bias, dim=1, descending=True, stable=True).indices[:, :k - shared]
    assert torch.equal(ids.cpu().long()[:, :k - shared], order)
    p = torch.gather(s, 1, order)
    torch.testing.assert_close(w.cpu()[:, :k - shared], p / p.sum(1, keepdim=True), rtol=2e-5, atol=2e-6)
    assert bool((ids.cpu()[:, k - shared:] == E).all())


@pytest.mark.parametrize("E,groups,keep,k", [(256, 8, 4, 8), (256, 16, 4, 8), (256, 1, 1, 8), (64, 2, 1, 6)])
def test_gate_passes_over_nan(lo, E, groups, keep, k):
    """A NaN counts as -inf: it is taken only where nothing else is left, and the other experts' order and weights stay."""
    g = torch.Generator().manual_seed(E + groups)
    x = torch.randn(66, E, generator=g)
    x[torch.rand(66, E, generator=g) < 0.3] = float("nan")
    x[0] = float("nan")
    w, ids = lo.moe.moe_fused_gate(x.to(DEV), torch.zeros(E, device=DEV), groups, keep, k, 0, 2.5, False)
    w, ids = w.cpu(), ids.cpu().long()
    assert bool(((ids >= 0) & (ids < E)).all())
    s = torch.sigmoid(x.to(DEV)).cpu()
    s = torch.where(s.isnan(), torch.full((), float("-inf")), s)[1:]
    top2 = s.view(65, groups, -1).topk(2, dim=2).values.sum(2)
    kept = torch.sort(top2, dim=1, descending=True, stable=True).indices[:, :keep]
    mask = torch.zeros(65, groups, dtype=torch.bool).scatter_(1, kept, True).repeat_interleave(E // groups, 1)
    order = torch.sort(torch.where(mask, s, torch.full((), float("-inf"))), dim=1, descending=True, stable=True).indices[:, :k]
    assert torch.equal(ids[1:], order)
    p = torch.gather(s, 1, order)
    torch.testing.assert_close(w[1:], p / p.sum(1, keepdim=True), rtol=2e-5, atol=2e-6)


def test_topk_softmax_passes_over_nan(lo):
    g = torch.Generator().manual_seed(5)
    x = torch.randn(66, 256, generator=g)
    x[torch.rand(66, 256, generator=g) < 0.3] = float("nan")
    x[0] = float("nan")
    weights = torch.empty(66, 8, device=DEV)
    ids = torch.empty(66, 8, dtype=torch.int32, device=DEV)
    lo.moe.topk_softmax(weights, ids, None, x.to(DEV), False)
    ids = ids.cpu().long()
    assert bool(((ids >= 0) & (ids < 256)).all())
    s = torch.where(x.isnan(), torch.full((), float("-inf")), x)
    assert torch.equal(ids[1:], torch.sort(s, dim=1, descending=True, stable=True).indices[1:, :8])
    assert bool(weights.isnan().all())      # (a NaN is in the row's denominator)
