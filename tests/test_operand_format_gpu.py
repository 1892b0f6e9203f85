"""Operand planes of the tensor-core assignment and of the inverted file: fp16 or bf16 by what rounding takes from a
sample of the rows.  The results do not depend on the choice."""
import pytest
import torch

import flashlib_b200 as fl
from flashlib_b200 import kmeans

pytestmark = pytest.mark.gpu


def rows(kind, n, d, g):
    x = torch.randn(n, d, generator=g)
    if kind == "tiny":                # below fp16's smallest normal number: bf16
        x *= 1e-7
    elif kind == "large":             # beyond fp16's range: bf16
        x *= 1e6
    elif kind == "outlier":           # rows the sample does not meet lie beyond fp16's range
        x[n // 3] *= 1e6
    elif kind == "bf16":              # bf16 takes nothing from these
        x = x.bfloat16().float()
    elif kind == "edge":              # around fp16's largest number
        x = 65_504.0 * x
    return x


KINDS = ["plain", "tiny", "large", "outlier", "bf16", "edge"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("d", [3, 64, 129])
def test_labels(kind, d):
    g = torch.Generator().manual_seed(d)
    x = rows(kind, 5_001, d, g).cuda()
    c = rows(kind, 300, d, g).cuda()
    got = kmeans.euclid_assign_triton(x[None], c[None], mode="tc")[0].long()
    dist = torch.cdist(x.double(), c.double(), compute_mode="donot_use_mm_for_euclid_dist").square()
    mine, least = dist.gather(1, got[:, None])[:, 0], dist.min(1).values
    # fp32 sums of d squares: 2^-23 a term (two roundings each) at most
    assert torch.all(mine <= least * (1 + (d + 8) * 2.0 ** -22)), ((mine - least) / least).max()


@pytest.mark.parametrize("kind", KINDS)
def test_inverted_file(kind):
    d, k = 33, 7
    g = torch.Generator().manual_seed(8)
    x, q = rows(kind, 20_000, d, g).cuda(), rows(kind, 1_000, d, g).cuda()
    torch.manual_seed(0)
    ivf = fl.IVFFlat(nlist=16, nprobe=16, n_neighbors=k, niter=3).fit(x)          # every list probed: exact search
    dist = ivf.kneighbors(q)[0].double()
    want = torch.cdist(q.double(), x.double(), compute_mode="donot_use_mm_for_euclid_dist").square().topk(k, largest=False).values
    assert torch.allclose(dist, want, rtol=(d + 8) * 2.0 ** -22)
