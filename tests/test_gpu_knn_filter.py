"""Neighbour distances on either side of the counts from which the query is set up beside the gathering (four blocks of 256 queries on each
of 148 SMs) and from which it passes points by eight at a time (`-m gpu`): against brute force in float64 for a part of the points, with
clusters, duplicates and far points among them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4 * 148 * 256, 4 * 148 * 256 + 1, 32 * 9472, 32 * 9472 + 1, 500_009])
def test_large_clouds_are_exact(n):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from simple_knn._C import distCUDA2
    g = torch.Generator().manual_seed(n)
    pts = torch.randn(n, 3, generator=g)
    pts[: n // 4] *= 0.01                                   # a dense middle
    pts[n // 4: n // 4 + 4000] = pts[:4000]                 # points twice
    pts[n // 4: n // 4 + 500] = pts[7]                      # one of them five hundred times
    pts[-300:] *= 50.0
    pts = pts[torch.randperm(n, generator=g)].cuda()
    got = distCUDA2(pts).double()
    p = pts.double()
    pick = torch.randperm(n, generator=g)[:1536].cuda()
    pick[:64] = (p.norm(dim=1).topk(64).indices)            # the farthest too
    want = torch.empty(len(pick), device="cuda", dtype=torch.float64)
    for lo in range(0, len(pick), 128):
        who = pick[lo:lo + 128]
        d = torch.zeros(len(who), n, device="cuda", dtype=torch.float64)
        for a in range(3):
            d += (p[who, a][:, None] - p[None, :, a]) ** 2
        d[torch.arange(len(who), device="cuda"), who] = float("inf")
        want[lo:lo + 128] = d.topk(3, dim=1, largest=False).values.mean(dim=1)
    assert torch.allclose(got[pick], want, rtol=1e-5, atol=0)
