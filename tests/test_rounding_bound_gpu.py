"""Operands whose bf16 roundings all go one way, so that the errors of a score add up in place of averaging out:
the scoring error bound has to cover them, or a pass accepts a list that misses the nearest row.

bf16 keeps 8 significant bits: rounding moves a value by up to 2^-8 of itself, so a product of two rounded
vectors may be off by nearly 2^-7 ||q|| ||x||.  The data below come within 0.0068 to 0.0078 of it."""
import pytest
import torch

import flashlib_b200 as fl
from flashlib_b200 import _lib
from flashlib_b200.ivf_flat import index_from_centroids, ivf_fine_scan
from flashlib_b200.knn import knn_f32

pytestmark = pytest.mark.gpu

DOWN = 1 + 2.0 ** -8 - 2.0 ** -16       # rounds down to 1, by nearly 2^-8
UP = 1 + 2.0 ** -8 + 2.0 ** -16         # rounds up to 1 + 2^-7


def _rows(m, d=64, n_near=20, n_mid=600, seed=0):
    """Row 0 equals the query (DOWN, ..., DOWN) and loses 2^-8 on both sides of the product.  The others lie on a
    bf16 grid and lose it on the query's side only: 20 rows at a squared distance of about 0.15, 600 at
    0.38 and the rest far away, so row 0 scores like a row at 1.0 where the error allowed for is the
    difference between 0.15 and 0.9."""
    g = torch.Generator().manual_seed(seed)

    def shell(n, dist):
        # `dist * 64^2` coordinates (with repetition) moved by one step of 1/64 from 1, both ways alike
        x = torch.ones(n, d, dtype=torch.float64)
        steps = int(round(dist * 4096))
        base = steps // d
        amp = int(max(1, round(base ** 0.5)))
        moved = min(d, max(2, steps // (amp * amp)) // 2 * 2)
        for r in range(n):
            p = torch.randperm(d, generator=g)[:moved]
            x[r, p[: moved // 2]] += amp / 64
            x[r, p[moved // 2:]] -= amp / 64
        return x

    far = 1.0 + torch.randint(-24, 25, (m - 1 - n_near - n_mid, d), generator=g).double() / 64
    x = torch.cat([torch.full((1, d), DOWN, dtype=torch.float64), shell(n_near, 0.15), shell(n_mid, 0.38), far]).float()
    order = torch.randperm(m, generator=g)
    at = int((order == 0).nonzero())
    return x[order].contiguous(), at


@pytest.mark.parametrize("m,nq,mode,stage2", [(100_000, 1, _lib.FL_KNN_BF16_RERANK, False), (100_000, 600, _lib.FL_KNN_AUTO, True),
                                              (20_000, 2_000, _lib.FL_KNN_BF16_RERANK, False), (400_000, 20_000, _lib.FL_KNN_AUTO, False)])
@pytest.mark.parametrize("k", [1, 10, 40])
def test_knn_finds_the_row_at_distance_zero(m, nq, mode, stage2, k):
    x, at = _rows(m)
    q = torch.full((nq, 64), DOWN)
    d, i, _ = knn_f32(q.cuda(), x.cuda(), k, mode=mode, second_stage=stage2)
    want = ((x.double() - DOWN) ** 2).sum(1).topk(k, largest=False).values.cuda()
    assert (i[:, 0] == at).all() and (d[:, 0] == 0).all()
    # fp32 sums of 64 squares of exact differences against fp64: (64 + 2) 2^-24
    assert ((d.double() - want).abs() <= 66 * 2.0 ** -24 * want).all()


def test_inverted_lists_find_the_row_at_distance_zero():
    x, at = _rows(60_000)
    x, at = x.cuda(), at
    centroids = torch.stack([torch.full((64,), 1.0), torch.full((64,), -3.0)]).cuda()
    index = index_from_centroids(x, centroids, D=64, nprobe=2)
    q = torch.full((1_200, 64), DOWN).cuda()
    probed = torch.tensor([[0, 1]], dtype=torch.int32, device="cuda").expand(1_200, 2).contiguous()
    vals, pos = ivf_fine_scan(q, index, probed, 10, mode="bf16")
    assert (vals[:, 0] == 0).all() and (index.ids[pos[:, 0].long()] == at).all()


@pytest.mark.parametrize("d", [64, 160])
def test_labels_of_a_point_between_two_opposite_centroids(d):
    """x = (DOWN, UP, 1), c = (DOWN, -UP, s): <x, c> is a small positive number whose rounded form is
    2 n 2^-7 below it, and -c mirrors that."""
    n = (d - 4) // 2
    x = torch.ones(d, dtype=torch.float64)
    x[:n], x[n:2 * n] = DOWN, UP
    c = torch.zeros(d, dtype=torch.float64)
    c[:n], c[n:2 * n] = DOWN, -UP
    gap = n * (UP * UP - DOWN * DOWN) + 0.01 * n / 30
    hi = torch.tensor(gap).bfloat16().double()
    mid = (torch.tensor(gap) - hi).bfloat16().double()
    c[2 * n], c[2 * n + 1] = hi, mid
    X = x.float()[None].repeat(4_096, 1).cuda()
    C = torch.cat([c[None], -c[None], -0.9 * x[None].repeat(254, 1)]).float()
    lead = (X[0].double().cpu() @ C[0].double()).item()
    assert 0 < lead < 0.02 * d
    got = fl.euclid_assign_triton(X[None], C.cuda()[None], mode="bf16")[0]
    assert (got == 0).all()


@pytest.mark.parametrize("entry", ["norms", "row norm alone"])
def test_shards_find_the_row_at_distance_zero(entry):
    from flashlib_b200 import sharded
    from tests.test_sharded_gpu import run_shards
    x, at = _rows(160_000)
    q = torch.full((400, 64), DOWN).cuda()
    if entry == "norms":
        kern, outs, msgs = run_shards(x.cuda(), q, 10, 2)
    else:
        class OneNorm(sharded.DeviceKnnKernels):
            def seeded(self, q, db, k, row_offset, plane, cls, gmax, ctx):
                lib = _lib.load()
                ws, ws_bytes, status = ctx
                d, i = torch.empty(q.shape[0], k, device="cuda"), torch.empty(q.shape[0], k, dtype=torch.int32, device="cuda")
                one = gmax[:1].clone()
                _lib.check(lib.fl_knn_seeded_f32(q.data_ptr(), q.shape[0], q.stride(0), db.data_ptr(), db.shape[0],
                                                 db.stride(0), q.shape[1], k, plane.ptr, row_offset, cls.data_ptr(),
                                                 one.data_ptr(), d.data_ptr(), i.data_ptr(), ws.data_ptr(), ws_bytes,
                                                 status.data_ptr(), torch.cuda.current_stream().cuda_stream))
                return d, i, status
        plain, sharded.DeviceKnnKernels = sharded.DeviceKnnKernels, OneNorm
        try:
            kern, outs, msgs = run_shards(x.cuda(), q, 10, 2)
        finally:
            sharded.DeviceKnnKernels = plain
    d, i, _ = kern.merge(torch.cat(msgs), 400, 10, 2)
    assert (i[:, 0] == at).all() and (d[:, 0] == 0).all()


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("spread", [0.0, 4.0])
def test_accumulation_stays_within_its_part_of_the_bound(d, spread):
    """Operands that bf16 holds exactly leave the accumulation alone: one sign, so that truncations add up, and
    magnitudes over several binades.  Allowed: one 2^-23 per product (score_acc); the norm columns add the rounding of
    ||x||^2 and three more additions, 1e-6 ||x||^2."""
    from tests.test_knn_tc_gpu import tc_scores
    g = torch.Generator().manual_seed(d)
    q = ((1 + torch.rand(128, d, generator=g)) * torch.exp2(spread * torch.rand(128, d, generator=g))).bfloat16().float().cuda()
    x = ((1 + torch.rand(2_000, d, generator=g)) * torch.exp2(spread * torch.rand(2_000, d, generator=g))).bfloat16().float().cuda()
    got = tc_scores(q, x)[:, :2_000].double()
    qd, xd = q.double(), x.double()
    err = (got - (qd @ xd.T - 0.5 * (xd * xd).sum(1)[None])).abs()
    prod = qd.norm(dim=1)[:, None] * xd.norm(dim=1)[None]
    assert (err <= 1.25e-7 * (d + 16) * prod + 1e-6 * (xd * xd).sum(1)[None]).all()
    print("largest accumulation error: %.3f of its bound" % (err / (1.25e-7 * (d + 16) * prod)).max().item())
