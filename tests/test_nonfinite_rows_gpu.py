"""Rows with NaN or infinite values: they are nobody's neighbours, and the finite rows around them are found as if
they were not there.  Against fp64 brute force over the finite rows."""
import pytest
import torch

import flashlib_b200 as fl
from flashlib_b200 import _lib
from flashlib_b200.ivf_flat import index_from_centroids, ivf_fine_scan
from flashlib_b200.knn import knn_f32

pytestmark = pytest.mark.gpu

NAN, INF = float("nan"), float("inf")


def _check(q, db, k, d, i):
    finite = torch.isfinite(db).all(1)
    rows = finite.nonzero()[:, 0]
    kk = min(k, rows.numel())
    x = db[rows].double()
    near = torch.cat([((x * x).sum(1) - 2 * s @ x.T).topk(min(kk + 8, rows.numel()), dim=1, largest=False).indices
                      for s in q.double().split(1_000)])
    want = torch.cat([((s[:, None] - x[n]) ** 2).sum(-1).sort(1).values[:, :kk]
                      for s, n in zip(q.double().split(1_000), near.split(1_000))])
    assert finite[i[:, :kk].long()].all() and (i[:, :kk] >= 0).all()
    own = ((q.double()[:, None] - db[i[:, :kk].long()].double()) ** 2).sum(-1)
    # an fp32 sum of d squares of rounded differences: within (d + 2) 2^-24 of its value
    eps = (q.shape[1] + 2) * 2.0 ** -24
    assert ((d[:, :kk].double() - own).abs() <= eps * own).all()
    assert ((own - want).abs() <= 2 * eps * want).all()
    assert torch.isinf(d[:, kk:]).all()


@pytest.mark.parametrize("m,nq,k", [(20_000, 600, 10), (20_000, 1_000, 40), (3_000, 700, 16), (60_000, 130, 10), (40_000, 9_000, 10),
                                    (40_000, 9_000, 40)])
@pytest.mark.parametrize("bad", ["nan", "inf", "inf and a zero query", "overflowing norm"])
def test_tensor_core_plan_with_one_bad_row(m, nq, k, bad):
    g = torch.Generator().manual_seed(m + nq)
    db = torch.randn(m, 64, generator=g)
    q = torch.randn(nq, 64, generator=g)
    if bad == "nan":
        db[m // 3, 5] = NAN
    elif bad == "overflowing norm":
        db[m // 3] = 3e19
    else:
        db[m // 3, 5] = INF
    if "zero" in bad:
        q[7] = 0
    db, q = db.cuda(), q.cuda()
    d, i, info = knn_f32(q, db, k, mode=_lib.FL_KNN_BF16_RERANK)
    finite = db.clone()
    finite[m // 3] = INF                     # (a row of 3e19 has no finite fp32 distance)
    _check(q, finite, k, d, i)


@pytest.mark.parametrize("nq", [1, 4, 7])
@pytest.mark.parametrize("k", [1, 10, 40])
@pytest.mark.parametrize("n_bad", [1, 12, 130, 250])
def test_few_query_scan_with_bad_rows_in_front(nq, k, n_bad):
    """NaN among the first 256 rows of a block, from which its starting threshold is taken."""
    g = torch.Generator().manual_seed(n_bad)
    db = torch.randn(400, 24, generator=g)
    db[:n_bad:2], db[1:n_bad:2] = NAN, INF
    q = torch.randn(nq, 24, generator=g)
    for sign in (1.0, -1.0):                 # (a NaN keeps its sign through some operations)
        x = (db * sign).cuda()
        d, i, _ = knn_f32(q.cuda(), x, k, mode=_lib.FL_KNN_EXACT_SIMT)
        _check(q.cuda(), x, k, d, i)


@pytest.mark.parametrize("n_bad", [1, 40, 200])
def test_inverted_lists_with_bad_rows(n_bad):
    g = torch.Generator().manual_seed(n_bad)
    X = torch.randn(3_000, 32, generator=g)
    centroids = torch.randn(4, 32, generator=g).cuda()
    index = index_from_centroids(X.cuda(), centroids, D=32, nprobe=4)
    for c in range(4):                       # the first rows of every list
        s = int(index.list_offsets[c])
        index.data[s:s + n_bad:2] = NAN
        index.data[s + 1:s + n_bad:2] = INF
    Q = torch.randn(20, 32, generator=g).cuda()
    probed = torch.arange(4, dtype=torch.int32, device="cuda").expand(20, 4).contiguous()
    for k, mode in ((1, "exact"), (10, "exact"), (50, "exact"), (10, "bf16"), (16, "bf16")):
        vals, pos = ivf_fine_scan(Q, index, probed, k, mode=mode)
        _check(Q, index.data, k, vals, pos)
