"""Lloyd loops on the tensor cores: an iteration scores only the points whose distance bounds no longer prove
their label, so every label is checked against all centroids in fp64."""
import pytest
import torch

from flashlib_b200 import kmeans

pytestmark = pytest.mark.gpu


def data(kind, n, d, K, g):
    x = torch.randn(n, d, generator=g)
    if kind == "blobs":
        x += 2.0 * torch.randn(K, d, generator=g)[torch.randint(0, K, (n,), generator=g)]
    elif kind == "far":                       # a common offset: wide error bands, few points proven
        x = 0.1 * x + 30.0
    elif kind == "large":                     # beyond fp16's range: operands stay bf16
        x = 1e6 * x
    elif kind == "outlier":                   # one row beyond fp16's range among rows inside it
        x[n // 3] *= 1e6
    elif kind == "duplicates":
        x = x[torch.randint(0, max(2, K // 2), (n,), generator=g)]
    return x


# sizes around the tiles of 128 points, 256 centroids and 64 features
CASES = [("blobs", 60_001, 128, 300), ("blobs", 129_000, 33, 256), ("randn", 70_000, 64, 257), ("far", 66_000, 20, 260),
         ("large", 70_000, 16, 256), ("outlier", 65_700, 40, 256), ("duplicates", 66_000, 24, 256), ("blobs", 200_000, 96, 64),
         ("blobs", 127, 8, 5), ("blobs", 300, 8, 1)]


def loop(x, K, iters, tol=0.0):
    """The tensor-core loop whatever kernel the size rules would take."""
    cur = x[:K].clone()
    nxt = torch.empty_like(cur)
    sums, cnts = torch.empty_like(cur), torch.empty(K, dtype=torch.int32, device="cuda")
    labels = torch.empty(len(x), dtype=torch.int32, device="cuda")
    ran = kmeans._lloyd_tc(x, K, cur, nxt, sums, cnts, labels, iters, tol, kmeans.DELTA_REFRESH)
    return labels, (nxt if ran % 2 else cur), (cur if ran % 2 else nxt), ran


def check_nearest(x, labels, old):
    d = x.shape[1]
    for part, lab in zip(x.double().split(20_000), labels.long().split(20_000)):
        d2 = torch.cdist(part, old.double(), compute_mode="donot_use_mm_for_euclid_dist").square()
        # fp32 sums of d squares: 2^-23 a term (two roundings each) at most
        assert torch.all(d2.gather(1, lab[:, None])[:, 0] <= d2.min(1).values * (1 + (d + 8) * 2.0 ** -22))


@pytest.mark.parametrize("kind,n,d,K", CASES)
@pytest.mark.parametrize("iters", [2, 9, 18])
def test_labels_and_centroids(kind, n, d, K, iters):
    x = data(kind, n, d, K, torch.Generator().manual_seed(n + d)).cuda()
    labels, new, old, ran = loop(x, K, iters)
    assert ran == iters
    check_nearest(x, labels, old)
    # the centroids are the means of the rows that carry their labels, from fp32 sums that met up to n rows on the way:
    # each addition errs by 2^-24 of a partial sum, at most the most rows a cluster held times the largest value
    sums = torch.zeros(K, d, dtype=torch.float64, device="cuda").index_add_(0, labels.long(), x.double())
    cnt = torch.bincount(labels.long(), minlength=K)
    want = torch.where(cnt[:, None] > 0, sums / cnt.clamp_min(1)[:, None], old.double())
    most = max(int(cnt.max()), n // 4) * x.abs().max().double()
    slack = (2.0 ** -24 * n ** 0.5 * 4 * most / cnt.clamp_min(1))[:, None]       # (roundings of n additions, either way)
    assert torch.all((new.double() - want).abs() <= slack)


def test_convergence_ends_the_loop():
    x = data("blobs", 70_000, 32, 300, torch.Generator().manual_seed(5)).cuda()
    labels, new, old, ran = loop(x, 300, 90, tol=1e-3)
    assert 1 < ran < 90
    assert (new - old).norm(dim=1).max().item() < 1e-3
    check_nearest(x, labels, old)


def test_rows_that_are_no_numbers():
    """They are listed in every iteration and harm no other row of the first."""
    x = data("blobs", 66_000, 32, 256, torch.Generator().manual_seed(6)).cuda()
    x[700] = float("nan")
    labels, _, old, _ = loop(x, 256, 1)
    ok = torch.arange(len(x), device="cuda") != 700
    check_nearest(x[ok], labels[ok], old)
    loop(x, 256, 6)
    torch.cuda.synchronize()
