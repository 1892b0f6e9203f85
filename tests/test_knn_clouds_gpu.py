"""Batches of small problems with few features against fp64 torch: chunk and group edges, ties, overflowing lists."""
import pytest
import torch

import flashlib_b200 as fl
from flashlib_b200 import _lib

pytestmark = pytest.mark.gpu


def _check(q, x, k, vals, idxs):
    dist = (q.double()[:, :, None] - x.double()[:, None]).square_().sum(-1)
    ref = dist.sort(dim=2, stable=True).values[..., :k]
    got = dist.gather(2, idxs.long())
    # an fp32 sum of d squares of rounded differences: within (d + 2) 2^-24 of its value
    eps = (q.shape[2] + 2) * 2.0 ** -24
    assert ((vals - got).abs() <= eps * got).all()
    assert ((got - ref).abs() <= 2 * eps * ref).all()
    assert (vals[..., 1:] >= vals[..., :-1]).all()
    assert all(len(set(r)) == k for r in idxs.reshape(-1, k)[:200].tolist())


@pytest.mark.parametrize("d", [1, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("B,nq,m,k", [(2, 1, 1, 1), (3, 33, 40, 16), (2, 129, 1025, 17), (5, 300, 257, 40), (2, 64, 2500, 16), (40, 500, 700, 5)])
def test_shapes(d, B, nq, m, k):
    g = torch.Generator().manual_seed(d * 1000 + m)
    q, x = torch.randn(B, nq, d, generator=g).cuda(), torch.randn(B, m, d, generator=g).cuda()
    _check(q, x, k, *fl.flash_knn(q, x, k))


def test_strided_rows():
    g = torch.Generator().manual_seed(1)
    wide = torch.randn(3, 400, 7, generator=g).cuda()
    _check(wide[:, :, 1:4], wide[:, :, 1:4], 16, *fl.flash_knn(wide[:, :, 1:4], wide[:, :, 1:4], 16))


@pytest.mark.parametrize("k", [16, 40])
def test_overflowing_lists(k):
    # all rows equal; few distinct rows; neighbours that all fall in one group of the first pass
    x = torch.zeros(2, 900, 3, device="cuda")
    vals, idxs = fl.flash_knn(x, x, k)
    assert (vals == 0).all() and (idxs == torch.arange(k, device="cuda")).all()
    x = torch.randn(2, 5, 3, device="cuda").repeat(1, 200, 1)
    vals, idxs = fl.flash_knn(x, x, k)
    assert (vals == 0).all()
    rows = torch.arange(1000, device="cuda")
    assert (idxs == (rows % 5)[None, :, None] + 5 * torch.arange(k, device="cuda")).all()
    x = torch.randn(2, 2048, 3, device="cuda") * 1e-3
    x[:, :, 0] += (torch.arange(2048, device="cuda") % 128).float()
    _check(x[:, :256], x, k, *fl.flash_knn(x[:, :256], x, k))


def test_rows_without_a_finite_distance():
    x = torch.randn(2, 60, 3, device="cuda")
    x[:, 10], x[:, 20], x[:, 30:50] = float("nan"), float("inf"), 1e30
    vals, idxs = fl.flash_knn(x[:, :4], x, 40)
    finite = 60 - 22
    assert torch.isfinite(vals[..., :finite]).all() and torch.isinf(vals[..., finite:]).all()
    assert (idxs != 10).all()
    assert (idxs[..., finite:] == torch.tensor([20, 30], device="cuda")).all()


@pytest.mark.parametrize("B,nq,m,d,k", [(2, 16, 65_536, 3, 16), (3, 1, 20_001, 16, 40), (2, 300, 40_000, 8, 10), (2, 1, 300_000, 3, 5)])
def test_few_queries_of_large_problems(B, nq, m, d, k):
    """Shapes that go to the tile kernel, which deals a problem's rows to many blocks."""
    assert _lib.load().fl_knn_batch_workspace_bytes(B, nq, m, d, k) > 1024
    g = torch.Generator().manual_seed(m)
    q, x = torch.randn(B, nq, d, generator=g).cuda(), torch.randn(B, m, d, generator=g).cuda()
    vals, idxs = fl.flash_knn(q, x, k)
    want = torch.cat([((q[:, i:i + 1].double() - x.double()) ** 2).sum(-1)[:, None].topk(k, dim=2, largest=False).values
                      for i in range(nq)], 1)
    own = ((q.double()[:, :, None] - x.double()[torch.arange(B, device="cuda")[:, None, None], idxs.long()]) ** 2).sum(-1)
    eps = (d + 2) * 2.0 ** -24
    assert ((vals - own).abs() <= eps * own).all() and ((own - want).abs() <= 2 * eps * want).all()
