"""Neighbour distances of clouds in which some points are no numbers (`-m gpu`): the others' are those of the cloud without them."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 1025, 5000, 66_000])
def test_points_that_are_no_numbers_are_passed_by(n):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from simple_knn._C import distCUDA2
    g = torch.Generator().manual_seed(n)
    pts = torch.randn(n, 3, generator=g)
    bad = torch.zeros(n, dtype=torch.bool)
    bad[torch.randperm(n, generator=g)[:max(2, n // 200)]] = True
    pts[bad, torch.randint(0, 3, (int(bad.sum()),), generator=g)] = math.nan
    got = distCUDA2(pts.cuda()).cpu()
    assert torch.equal(got[~bad], distCUDA2(pts[~bad].cuda()).cpu())       # exact either way, whatever the order of the points
    assert torch.isinf(got[bad]).all()
