"""Operand planes and other kept buffers that one stream fills and another reads at once, and those met under capture."""
import copy
import pickle

import pytest
import torch

import flashlib_b200 as fl
from flashlib_b200 import _lib
from flashlib_b200 import kmeans as kmeans_mod
from flashlib_b200 import knn as knn_mod
from flashlib_b200.ivf_flat import flash_ivf_flat_search, index_from_centroids, ivf_fine_scan
from flashlib_b200.knn import DbPlane, get_plane, knn_f32

pytestmark = pytest.mark.gpu

LAG = 200_000_000               # clock cycles that the filling stream is kept busy before it fills


def _data(m=20_000, d=64, nq=700, seed=0):
    g = torch.Generator().manual_seed(seed)
    db, q = torch.randn(m, d, generator=g).cuda(), torch.randn(nq, d, generator=g).cuda()
    torch.cuda.synchronize()
    return db, q


def _late(fill):
    """Runs ``fill`` on a stream that is busy, and returns another stream."""
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        torch.cuda._sleep(LAG)
        fill()
    return b


@pytest.mark.parametrize("stage2", [False, True])
def test_plane_filled_on_another_stream(stage2):
    db, q = _data()
    want = knn_f32(q, db.clone(), 10, mode=_lib.FL_KNN_BF16_RERANK, second_stage=stage2)[:2]
    torch.cuda.synchronize()

    def fill():
        plane = get_plane(db)
        if stage2:
            plane.split_ptr(db)

    with torch.cuda.stream(_late(fill)):
        got = knn_f32(q, db, 10, mode=_lib.FL_KNN_BF16_RERANK, second_stage=stage2)[:2]
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_plane_dropped_while_another_stream_reads_it():
    db, q = _data()
    want = knn_f32(q, db, 10, mode=_lib.FL_KNN_BF16_RERANK, second_stage=False)[:2]
    torch.cuda.synchronize()
    plane = DbPlane(db)
    torch.cuda.synchronize()
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        torch.cuda._sleep(LAG)
        got = knn_f32(q, db, 10, mode=_lib.FL_KNN_BF16_RERANK, plane=plane, second_stage=False, check_status=False)[:2]
    nbytes = plane.buf.numel()
    del plane
    for _ in range(4):           # would be given the plane's memory
        torch.empty(nbytes, dtype=torch.uint8, device="cuda").fill_(255)
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_cast_rows_filled_on_another_stream():
    db, q = _data()
    want = fl.flash_knn(q, db.clone(), 5, tol=1e-2)
    torch.cuda.synchronize()
    with torch.cuda.stream(_late(lambda: knn_mod._cast_rows_cached(db, torch.float16))):
        qh = q.to(torch.float16)
        got = knn_f32(qh, knn_mod._cast_rows_cached(db, torch.float16), 5)[:2]
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_sample_plane_filled_on_another_stream():
    x, c = _data(m=70_000, nq=300)
    want = fl.euclid_assign_triton(x[None].clone(), c[None], mode="bf16")
    torch.cuda.synchronize()
    with torch.cuda.stream(_late(lambda: kmeans_mod._x_plane(x))):
        got = fl.euclid_assign_triton(x[None], c[None], mode="bf16")
    torch.cuda.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("mode", ["exact", "bf16"])
def test_inverted_file_plane_filled_on_another_stream(mode):
    db, q = _data(m=30_000, nq=4_000)
    index = index_from_centroids(db, db[:32].clone(), D=64, nprobe=8)
    probed = torch.arange(8, dtype=torch.int32, device="cuda").expand(4_000, 8).contiguous()
    torch.cuda.synchronize()
    ref = copy.deepcopy(index)
    want = ivf_fine_scan(q, ref, probed, 10, mode=mode)
    torch.cuda.synchronize()
    with torch.cuda.stream(_late(lambda: ivf_fine_scan(q[:300], index, probed[:300], 10, mode=mode))):
        got = ivf_fine_scan(q, index, probed, 10, mode=mode)
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_index_with_planes_can_be_copied():
    db, q = _data(m=30_000, nq=500)
    index = fl.flash_ivf_flat_build(db, 16, nprobe=8, niter=2)
    want = flash_ivf_flat_search(index, q, 5)
    for other in (copy.deepcopy(index), pickle.loads(pickle.dumps(index))):
        got = flash_ivf_flat_search(other, q, 5)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_plane_filled_under_capture_is_not_met_outside():
    db, q = _data()
    fresh = db.clone()
    want = knn_f32(q, db, 10, mode=_lib.FL_KNN_BF16_RERANK, check_status=False)[:2]
    fl.check_pending()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):            # (the graph has not run: what it builds is not there yet)
        in_graph = knn_f32(q, fresh, 10, mode=_lib.FL_KNN_BF16_RERANK, check_status="deferred")[:2]
    eager = knn_f32(q, fresh, 10, mode=_lib.FL_KNN_BF16_RERANK, check_status=False)[:2]
    graph.replay()
    torch.cuda.synchronize()
    for got in (eager, in_graph):
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_plane_of_a_graph_outlives_its_cache():
    db, q = _data()
    want = knn_f32(q, db, 10, mode=_lib.FL_KNN_BF16_RERANK, check_status=False)[:2]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = knn_f32(q, db, 10, mode=_lib.FL_KNN_BF16_RERANK, check_status="deferred")[:2]
    others = [torch.randn(20_000, 64, device="cuda") for _ in range(6)]
    for o in others:
        knn_f32(q, o, 10, mode=_lib.FL_KNN_BF16_RERANK, check_status=False)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
