"""The paths that calls of few queries take, at the edges of their ranges: the CUDA-core scan for few
queries (kNN and inverted lists), the tensor-core plan with pools in global memory as pairs and a
seeding sample dealt to several CTAs, and the streamed query tile for rows of more than 512 features.
All against fp64 brute force on the values as stored."""
import pytest
import torch

import flashlib_b200 as fl
from flashlib_b200 import _lib
from flashlib_b200.ivf_flat import ivf_fine_scan
from flashlib_b200.knn import knn_f32
from tests import parity

pytestmark = pytest.mark.gpu


def _fp64_neighbours(q, db, k):
    qd, dbd = q.double(), db.double()
    d64 = (qd * qd).sum(-1, keepdim=True) + (dbd * dbd).sum(-1)[None, :] - 2.0 * qd @ dbd.T
    return d64.topk(k, dim=1, largest=False).indices.cpu().numpy()


def _check(q, db, k, d, i):
    res = parity.knn_parity(q.float().cpu().numpy(), db.float().cpu().numpy(), d.cpu().numpy(), i.cpu().numpy(),
                            _fp64_neighbours(q, db, k))
    assert res["ok"], res


# queries: 1 to 4 share a row read (5: a second, ragged group); rows: below one pass of a block (256), one more
# than a pass, many ranges; k: the pool classes 32 / 128; features: 16-byte loads and their tails
@pytest.mark.parametrize("nq,m,d,k,dtype", [
    (1, 1, 1, 1, torch.float32), (1, 255, 4, 32, torch.float32), (4, 257, 36, 33, torch.float32),
    (5, 40_001, 130, 128, torch.float32), (3, 300_000, 128, 10, torch.float32), (2, 70_000, 37, 100, torch.float32),
    (7, 5_000, 1000, 5, torch.float32), (1, 100_000, 64, 10, torch.bfloat16), (4, 20_000, 129, 16, torch.float16),
    (512, 600, 24, 8, torch.float32)])
def test_few_query_scan(nq, m, d, k, dtype):
    g = torch.Generator().manual_seed(nq + m + d)
    db = torch.randn(m, d, generator=g).to(dtype).cuda()
    q = torch.randn(nq, d, generator=g).to(dtype).cuda()
    d_, i_, info = knn_f32(q, db, k, mode=_lib.FL_KNN_EXACT_SIMT)
    _check(q, db, k, d_, i_)


def test_few_query_scan_orders_ties_by_row():
    """Every row is there 50 times over: more ties at the k-th distance than a pool holds."""
    g = torch.Generator().manual_seed(3)
    base = torch.randn(200, 16, generator=g)
    db = base.repeat(50, 1).cuda()
    for k in (10, 32, 100):
        d_, i_, _ = knn_f32(base[:3].cuda(), db, k, mode=_lib.FL_KNN_EXACT_SIMT)
        assert torch.all(d_[:, :min(k, 50)] == 0)
        want = torch.arange(3)[:, None] + 200 * torch.arange(min(k, 50))[None, :]
        assert torch.equal(i_[:, :min(k, 50)].cpu().long(), want)


@pytest.mark.parametrize("nq,nprobe,k,nlist", [(1, 1, 1, 3), (1, 40, 100, 40), (9, 5, 10, 64), (130, 16, 33, 300)])
def test_few_query_scan_of_inverted_lists(nq, nprobe, k, nlist):
    g = torch.Generator().manual_seed(nq + nlist)
    X = torch.randn(6_000, 48, generator=g).cuda()
    Q = torch.randn(nq, 48, generator=g).cuda()
    index = fl.flash_ivf_flat_build(X, nlist, nprobe=nprobe, niter=2)
    probed = fl.flash_knn(Q, index.centroids, nprobe, return_distances=False)
    vals, pos = ivf_fine_scan(Q, index, probed, k, mode="exact")
    offs = index.list_offsets.cpu()
    for qi in range(0, nq, max(1, nq // 8)):
        rows = torch.cat([torch.arange(offs[c], offs[c + 1]) for c in probed[qi].tolist()])
        kk = min(k, rows.numel())
        d64 = ((index.data[rows.cuda()].double() - Q[qi].double()) ** 2).sum(-1)
        ref = rows[d64.topk(kk, largest=False).indices.cpu()]
        res = parity.knn_parity(Q[qi:qi + 1].cpu().numpy(), index.data.cpu().numpy(), vals[qi:qi + 1, :kk].cpu().numpy(),
                                pos[qi:qi + 1, :kk].cpu().numpy(), ref[None].numpy())
        assert res["ok"], (qi, res)
        assert torch.all(pos[qi, kk:] == -1) and torch.all(torch.isinf(vals[qi, kk:]))


# query tiles: one row, a full tile, one more; databases of one tile (no seeding), two, a ragged last tile, many ranges;
# k on both sides of the pool classes (16 / 17) and the largest; clustered rows, whose pools fill
@pytest.mark.parametrize("spread", [1.0, 0.05])
@pytest.mark.parametrize("nq,m,d,k", [(1, 256, 64, 10), (128, 257, 64, 16), (129, 512, 100, 17), (1, 300_001, 128, 16),
                                      (300, 40_000, 256, 112), (1000, 20_000, 64, 10), (900, 5_000, 33, 50)])
def test_pair_pool_plan(nq, m, d, k, spread):
    g = torch.Generator().manual_seed(nq + m)
    centres = torch.randn(20, d, generator=g) * (1.0 if spread < 1 else 0.0)
    db = (centres[torch.randint(0, 20, (m,), generator=g)] + spread * torch.randn(m, d, generator=g)).cuda()
    q = (centres[torch.randint(0, 20, (nq,), generator=g)] + spread * torch.randn(nq, d, generator=g)).cuda()
    d_, i_, info = knn_f32(q, db, k, mode=_lib.FL_KNN_BF16_RERANK)
    assert info["status"][_lib.FL_STATUS_ERROR].item() == 0
    _check(q, db, k, d_, i_)
    if spread == 1.0:
        assert info["fallback_rows"] <= nq // 10, info


@pytest.mark.parametrize("nq,m,d,k,dtype", [(600, 3_000, 513, 10, torch.float32), (300, 9_000, 576, 16, torch.bfloat16),
                                            (200, 20_000, 1000, 40, torch.float16), (2_000, 30_000, 768, 5, torch.bfloat16)])
def test_rows_of_more_than_512_features(nq, m, d, k, dtype):
    """Automatic mode streams the query tile beside the database chunks; the explicit tensor-core mode
    stays with the shapes it had."""
    g = torch.Generator().manual_seed(nq + d)
    db = torch.randn(m, d, generator=g).to(dtype).cuda()
    q = torch.randn(nq, d, generator=g).to(dtype).cuda()
    assert _lib.load().fl_knn_wants_plane(nq, m, d, k)
    d_, i_, info = knn_f32(q, db, k)
    assert info["mode"] == _lib.FL_KNN_BF16_RERANK and info["fallback_rows"] <= nq // 10, info
    _check(q, db, k, d_, i_)
    d_x, i_x, _ = knn_f32(q, db, k, mode=_lib.FL_KNN_EXACT_SIMT)
    assert torch.equal(d_x, d_) and (i_x == i_).float().mean().item() > 0.999


def test_deferred_status_of_many_calls():
    """Status words of deferred calls arrive in pinned host memory: more calls than slots, then none left."""
    from flashlib_b200 import knn as knn_mod
    g = torch.Generator().manual_seed(1)
    db = torch.randn(30_000, 32, generator=g).cuda()
    q = torch.randn(600, 32, generator=g).cuda()
    for _ in range(150):
        fl.flash_knn(q, db, 5)
    assert len(knn_mod._PENDING_STATUS) <= 64
    fl.check_pending()
    assert len(knn_mod._PENDING_STATUS) == 0


# few pairs: two launches, a block per pair; many that share their lists: grouped by list (lists of 1 562 rows)
@pytest.mark.parametrize("nq,nprobe,k,few", [(8, 4, 10, True), (4, 16, 50, True), (400, 16, 50, False), (120, 60, 10, False),
                                             (500, 16, 100, False)])
def test_inverted_list_scan_by_pairs_and_sharing(nq, nprobe, k, few):
    g = torch.Generator().manual_seed(nq)
    X = torch.randn(100_000, 32, generator=g).cuda()
    Q = torch.randn(nq, 32, generator=g).cuda()
    from flashlib_b200.ivf_flat import index_from_centroids
    index = index_from_centroids(X, X[:64].clone(), D=32, nprobe=nprobe)
    probed = torch.rand(nq, 64, generator=g).argsort(1)[:, :nprobe].int().cuda()
    index.half_norms()
    before = _lib.load().fl_launch_count()
    vals, pos = ivf_fine_scan(Q, index, probed, k, mode="exact")
    assert (_lib.load().fl_launch_count() - before == 2) == few
    offs = index.list_offsets.cpu()
    for qi in range(0, nq, max(1, nq // 8)):
        rows = torch.cat([torch.arange(offs[c], offs[c + 1]) for c in probed[qi].tolist()])
        d64 = ((index.data[rows.cuda()].double() - Q[qi].double()) ** 2).sum(-1)
        ref = rows[d64.topk(k, largest=False).indices.cpu()]
        res = parity.knn_parity(Q[qi:qi + 1].cpu().numpy(), index.data.cpu().numpy(), vals[qi:qi + 1].cpu().numpy(),
                                pos[qi:qi + 1].cpu().numpy(), ref[None].numpy())
        assert res["ok"], (qi, res)


# sizes on both sides of the rule: two launches are the scan, the tile kernel takes more
@pytest.mark.parametrize("nq,m,d,k,dtype,few", [(300, 20_000, 64, 10, torch.float32, True), (512, 60_000, 1024, 10, torch.float32, False),
                                                (256, 20_000, 64, 100, torch.float32, False), (32, 20_000, 64, 100, torch.float32, True),
                                                (512, 20_000, 100, 10, torch.bfloat16, False), (512, 20_000, 128, 10, torch.bfloat16, True),
                                                (8, 20_000, 333, 10, torch.float16, True)])
def test_exact_mode_by_queries_k_and_row_reads(nq, m, d, k, dtype, few):
    g = torch.Generator().manual_seed(nq + d)
    db, q = torch.randn(m, d, generator=g).to(dtype).cuda(), torch.randn(nq, d, generator=g).to(dtype).cuda()
    before = _lib.load().fl_launch_count()
    d_, i_, _ = knn_f32(q, db, k, mode=_lib.FL_KNN_EXACT_SIMT)
    assert (_lib.load().fl_launch_count() - before == 2) == few
    _check(q, db, k, d_, i_)


@pytest.mark.parametrize("nq,m,d", [(600, 3_000, 700), (1_000, 20_000, 64)])
def test_automatic_mode_without_room_for_a_plane(monkeypatch, nq, m, d):
    from flashlib_b200 import knn as knn_mod
    g = torch.Generator().manual_seed(d)
    db, q = torch.randn(m, d, generator=g).cuda(), torch.randn(nq, d, generator=g).cuda()

    def full(self, db):
        raise torch.OutOfMemoryError("no room")

    monkeypatch.setattr(knn_mod.DbPlane, "__init__", full)
    d_, i_, info = knn_f32(q, db, 10)
    assert info["mode"] == _lib.FL_KNN_EXACT_SIMT
    _check(q, db, 10, d_, i_)
    with pytest.raises(torch.OutOfMemoryError):
        knn_f32(q, db, 10, mode=_lib.FL_KNN_BF16_RERANK)


def test_no_second_stage_without_room_for_its_plane(monkeypatch):
    from flashlib_b200 import knn as knn_mod
    g = torch.Generator().manual_seed(1)
    db, q = torch.randn(20_000, 64, generator=g).cuda(), torch.randn(1_000, 64, generator=g).cuda()

    def full(self, db):
        raise torch.OutOfMemoryError("no room")

    monkeypatch.setattr(knn_mod.DbPlane, "split_ptr", full)
    d_, i_, info = knn_f32(q, db, 10)
    assert info["mode"] == _lib.FL_KNN_BF16_RERANK and not info["second_stage"]
    _check(q, db, 10, d_, i_)
