"""Neighbour distances at the sizes where a leaf, a node of a level or the width of the sort keys changes (`-m gpu`)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 32, 1023, 1025, 32769, 65535, 65537])
def test_every_tree_shape_is_exact(n):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from simple_knn._C import distCUDA2
    g = torch.Generator().manual_seed(n)
    pts = torch.randn(n, 3, generator=g)
    pts[: n // 8] *= 40.0                     # far points set the extent, most points share few cells of it
    pts = pts.cuda()
    got = distCUDA2(pts).double()
    want = torch.empty_like(got)
    p = pts.double()
    for lo in range(0, n, 2048):              # brute force, in slices
        d = torch.cdist(p[lo:lo + 2048], p, compute_mode="donot_use_mm_for_euclid_dist") ** 2
        i = torch.arange(d.shape[0], device="cuda")
        d[i, lo + i] = float("inf")
        want[lo:lo + 2048] = d.topk(3, dim=1, largest=False).values.mean(dim=1)
    assert torch.allclose(got, want, rtol=1e-5, atol=0)
