"""Tile lists on the GPU (`-m gpu`): one tile's list of a chosen length, spread in depth or all at one distance, on either side of
every line at which the way it is sorted changes, against the per-ray search."""
import math

import pytest
import torch

from raygaussx_b200 import _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", ["spread", "plane"])
@pytest.mark.parametrize("n", [1, 31, 33, 2048, 2049, 5000, 16384, 16385])
def test_list_of_any_length_matches_the_per_ray_search(n, depth):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from raygaussx_b200 import render_optix as ro
    dev = torch.device("cuda")
    sc = scenes.tiny_scene(n=n, width=4, height=4, log_scale_mean=-7.0, density_scale=30.0, seed=n)
    cam = scenes.SimpleCamera((4.0, 0.0, 0.0), fovx=math.radians(2), fovy=math.radians(2), width=4, height=4)      # one tile
    g = torch.Generator().manual_seed(n)
    side = (torch.rand(n, 2, generator=g) - 0.5) * (1.6 * math.tan(math.radians(1)))
    t = 2 + 4 * torch.rand(n, 1, generator=g)
    if depth == "plane":                           # one distance for all but one: a bucket holds the whole list
        t = torch.full((n, 1), 4.0)
        t[0] = 1.5
        sc.scales = torch.full_like(sc.scales, math.exp(-7.0))
        sc.quaternions = torch.tensor([[1.0, 0.0, 0.0, 0.0]]).repeat(n, 1)
    sc.positions = torch.cat([4 - t, side * t], 1)
    tens = [x.to(dev).contiguous() for x in sc.tensors()]
    cam.to(dev)
    cs = ro.camera_struct(cam)
    r = ro.get_renderer()
    r.build(*tens[:4])
    got = {}
    for label, flags in (("lists", 0), ("per_ray", _lib.FLAG_PER_RAY_SEARCH)):
        r.reset_counters()
        rgb, alpha, dist = r.forward(*tens, cs, r._march(0.0025, False, 2048, False, 1e-3, None, 4, flags | _lib.FLAG_COUNT_WORK),
                                     want_alpha=True, want_depth=True)
        got[label] = (rgb.clone(), alpha.clone(), dist.clone(), r.read_counters())
    for k in ("rays", "slabs", "slabs_hit", "closest_queries", "hits", "hits_hash", "overflow_slabs"):
        assert got["lists"][3][k] == got["per_ray"][3][k], k
    assert n < 100 or got["lists"][3]["hits"] > n // 40
    for a, b, tol in zip(got["lists"][:3], got["per_ray"][:3], (1e-5, 1e-5, 1e-4)):
        assert (a - b).abs().max().item() < tol
