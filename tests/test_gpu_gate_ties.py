"""GPU test of the softmax gate's selection where keys are equal: the lower expert id comes first, in a lane's own keys and across lanes,
at every number of experts a lane has (1 to 32, whole and ragged)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("E", [5, 32, 33, 64, 100, 128, 200, 256, 300, 512, 777, 1024])
@pytest.mark.parametrize("values", [1, 2, 5])
def test_equal_logits(E, values):
    import lightop_b200 as lo
    M, k = 129, min(E, 10)
    g = torch.Generator().manual_seed(E + values)
    x = torch.randint(0, values, (M, E), generator=g).float()
    x[0], x[1, ::2] = 0.0, -float("inf")
    w, ids = torch.empty(M, k, device=DEV), torch.empty(M, k, dtype=torch.int32, device=DEV)
    lo.moe.topk_softmax(w, ids, None, x.to(DEV), True)
    # descending logits, ascending ids among equals
    order = torch.sort(x, dim=1, descending=True, stable=True).indices[:, :k]
    rows = torch.ones(M, dtype=torch.bool)
    rows[1] = int((x[1] > -float("inf")).sum()) >= k      # (erased keys and logits of -inf are alike)
    assert torch.equal(ids.cpu()[rows].long(), order[rows])
    p = torch.softmax(x.double(), dim=1).gather(1, order)
    # exponential and quotients within a few units in the last place each
    torch.testing.assert_close(w.cpu()[rows].double(), (p / p.sum(1, keepdim=True))[rows], rtol=2e-6, atol=0)
