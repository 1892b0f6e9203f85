"""The one-row-per-thread k-means kernels against fp64 torch, at the edges of their feature blocks and chunks."""
import pytest
import torch

import flashlib_b200 as fl
from flashlib_b200 import kmeans as km

pytestmark = pytest.mark.gpu


def _problem(B, n, d, K, seed):
    g = torch.Generator().manual_seed(seed)
    means = 2.0 * torch.randn(B, K, d, generator=g)
    comp = torch.randint(0, K, (B, n), generator=g)
    x = torch.gather(means, 1, comp[..., None].expand(-1, -1, d)) + torch.randn(B, n, d, generator=g)
    return x.cuda(), x[:, torch.randperm(n, generator=g)[:K]].contiguous().cuda()


def _check_labels(x, c, lab):
    dist = (x.double()[:, :, None] - c.double()[:, None]).square_().sum(-1)
    got = dist.gather(2, lab.long()[..., None])[..., 0]
    best = dist.min(2).values
    # an fp32 sum of d squares of rounded differences: each within (d + 2) 2^-24 of its value
    assert (got - best <= 2 * (x.shape[2] + 2) * 2.0 ** -24 * got).all()


@pytest.mark.parametrize("d", [1, 2, 4, 5, 8, 15, 16, 17, 24, 31, 33, 40, 48, 63, 64, 65, 96, 127, 128])
@pytest.mark.parametrize("B,n,K", [(1, 1, 1), (1, 129, 3), (3, 515, 70), (1, 1000, 300), (1, 20000, 9)])
def test_assign_rows(B, n, d, K):
    K = min(K, n)
    x, c = _problem(B, n, d, K, seed=d)
    _check_labels(x, c, fl.euclid_assign_triton(x, c, mode="exact"))


@pytest.mark.parametrize("d,n,K", [(3, 303_500, 64), (8, 303_104, 300), (16, 310_001, 40)])
def test_assign_four_rows_a_thread(d, n, K):
    x, c = _problem(1, n, d, K, seed=7)
    lab = fl.euclid_assign_triton(x, c, mode="exact")
    for s in (slice(0, 3000), slice(n - 3000, n)):
        _check_labels(x[:, s], c, lab[:, s])


def test_assign_strided_and_unaligned_rows():
    x, c = _problem(1, 700, 16, 20, seed=1)
    for off in (0, 1):
        wide = torch.full((1, 700, 21), float("nan"), device="cuda")
        wide[:, :, off:off + 16] = x
        _check_labels(x, c, fl.euclid_assign_triton(wide[:, :, off:off + 16], c, mode="exact"))


def test_assign_rows_without_a_finite_distance():
    x, c = _problem(1, 64, 8, 5, seed=2)
    big = c[0, [3, 1]] * 1e20                       # distances overflow, inner products do not
    x[0, 0], x[0, 1], x[0, 2, 0], x[0, 3, 0] = big[0], big[1], float("inf"), float("nan")
    lab = fl.euclid_assign_triton(x, c, mode="exact")[0].cpu()
    score = (x[0, :2].double() @ c[0].double().T).cpu()       # the half norms vanish beside the products
    top2 = score.topk(2, dim=1).indices
    assert all(int(lab[i]) == int(top2[i].min()) for i in range(2))
    assert 0 <= int(lab[2]) < 5 and int(lab[3]) == 2 ** 31 - 1
    _check_labels(x[:, 4:], c, lab[None, 4:].cuda())


@pytest.mark.parametrize("B,n,d,K,iters", [(1, 3001, 33, 20, 20), (1, 5000, 8, 16, 18), (4, 1500, 4, 16, 6), (2, 700, 70, 9, 5), (1, 9, 3, 9, 2)])
def test_lloyd_loop_matches_single_steps(B, n, d, K, iters):
    x, init = _problem(B, n, d, K, seed=3)
    ids, cents, n_iter = km.batch_kmeans_Euclid(x, K, max_iters=iters, init_centroids=init)
    assert n_iter == iters
    cur = init.clone()
    for _ in range(iters):
        lab = fl.euclid_assign_triton(x, cur, mode="exact")
        cur, _, _ = fl.triton_lloyd_centroid_step_euclid(x, lab, cur)
    # sums in another order: a row at a boundary may change sides and move two centroids by 1 / (rows of a cluster)
    assert (ids != lab).float().mean() <= 2e-3
    assert (cents - cur).norm() <= 2e-3 * cur.norm()


@pytest.mark.parametrize("B,n,d,K", [(1, 4000, 12, 8), (1, 3000, 100, 12), (3, 800, 6, 4)])
def test_lloyd_loop_stops_when_no_centroid_moves(B, n, d, K):
    x, init = _problem(B, n, d, K, seed=5)
    tol = 1e-8 if B == 1 else 1e-3           # full sums have no fixed order: they move in the last bits
    ids, cents, n_iter = km.batch_kmeans_Euclid(x, K, max_iters=200, tol=tol, init_centroids=init)
    assert 1 < n_iter < 200
    again, moved, more = km.batch_kmeans_Euclid(x, K, max_iters=1, init_centroids=cents)
    assert more == 1 and (again == ids).float().mean() >= 0.999
    assert (moved - cents).abs().max() <= 1e-3
    # one iteration fewer has not converged yet
    assert km.batch_kmeans_Euclid(x, K, max_iters=n_iter - 1, tol=tol, init_centroids=init)[2] == n_iter - 1


def test_lloyd_loop_keeps_empty_clusters():
    x, init = _problem(1, 500, 8, 6, seed=6)
    init[0, 5] = 1e6
    _, cents, _ = km.batch_kmeans_Euclid(x, 6, max_iters=4, init_centroids=init)
    assert torch.equal(cents[0, 5], init[0, 5])


@pytest.mark.parametrize("n,d,K,dup", [(3000, 128, 200, 0), (3000, 33, 70, 0), (5000, 64, 130, 8), (1500, 250, 65, 1500)])
def test_tensor_core_assignment_of_unprovable_points(n, d, K, dup):
    # centroids in near-equal and equal pairs: no scoring bound decides between the two; with `dup` points (a few, or
    # more than the direct pass takes) on the bisector of two equal centroids the lower index wins
    x, c = _problem(1, n, d, K, seed=11)
    c[0, K // 2:2 * (K // 2)] = c[0, :K // 2] * (1 + 1e-6)
    c[0, K - 1] = c[0, 0]
    if dup:
        x[0, :dup] = c[0, 0]
    lab = fl.euclid_assign_triton(x, c, mode="bf16")
    _check_labels(x, c, lab)
    assert (lab[0, :dup] == 0).all()
    x[0, 7, 0] = float("nan")
    lab = fl.euclid_assign_triton(x, c, mode="bf16")
    _check_labels(x[:, 8:], c, lab[:, 8:])


# clusters around the number of labels a warp folds (16); rows in the order of their clusters, in runs that
# end inside a warp, or in none; features that fill their block or not, staged rows (d > 16) among them
@pytest.mark.parametrize("order", ["sorted", "runs", "random"])
@pytest.mark.parametrize("K", [1, 2, 16, 17, 40])
@pytest.mark.parametrize("B,n,d", [(1, 1_001, 1), (2, 5_003, 3), (3, 2_000, 4), (1, 9_999, 8), (2, 4_100, 13), (4, 3_333, 16),
                                   (2, 310_000, 16), (1, 4_097, 17), (2, 3_000, 33), (1, 5_000, 128)])
def test_sums_of_rows_that_share_a_cluster(B, n, d, K, order):
    x, _ = _problem(B, n, d, K, seed=K)
    c0 = x[:, torch.linspace(0, n - 1, K).long()].contiguous()
    lab = fl.euclid_assign_triton(x, c0, mode="exact")
    if order != "random":
        key = lab if order == "sorted" else (torch.arange(n, device="cuda") // 37) % 7 * K + lab
        at = key.long().argsort(dim=1, stable=True)
        x = torch.gather(x, 1, at[..., None].expand(-1, -1, d)).contiguous()
    lab, cent, _ = fl.flash_kmeans(x, K, max_iters=1, init_centroids=c0)
    one = torch.nn.functional.one_hot(lab.long(), K).double()
    cnt = one.sum(1)
    want = torch.where(cnt[..., None] > 0, one.transpose(1, 2) @ x.double() / cnt.clamp_min(1)[..., None], c0.double())
    size = one.transpose(1, 2) @ x.double().abs() / cnt.clamp_min(1)[..., None]
    # a sum of n fp32 terms in any order: within n 2^-24 of the sum of their sizes; one more rounding for the division
    assert ((cent.double() - want).abs() <= (cnt[..., None] + 2) * 2.0 ** -24 * (size + c0.abs())).all()
