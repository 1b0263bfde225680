"""What the march by patches leaves untested on the GPU (`-m gpu`): Gaussians that no ray of a patch meets inside the rays' windows, and
pairs whose Gaussian lies behind every ray of a tile.  Hits, counted and hashed, against the per-ray search, from outside and from
among the Gaussians, at fields of view from a hundredth of a degree to 150 degrees, with needles, discs and balls."""
import math

import pytest
import torch

from raygaussx_b200 import _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["needles", "discs", "balls"])
@pytest.mark.parametrize("fov,width,height", [(0.01, 17, 9), (2.0, 205, 203), (60.0, 6, 5), (60.0, 150, 131), (60.0, 200, 200), (60.0, 201, 200), (60.0, 258, 250),
                                              (150.0, 13, 11),
                                              (150.0, 210, 199)])
@pytest.mark.parametrize("inside", [False, True])
def test_nothing_that_is_met_is_left_out(shape, fov, width, height, inside):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from raygaussx_b200 import render_optix as ro
    dev = torch.device("cuda")
    sc = scenes.tiny_scene(n=1200, width=width, height=height, log_scale_mean=-2.2 if inside else -3.0, density_scale=3.0, seed=width)
    thin = {"needles": [1.0, 0.01, 0.01], "discs": [1.0, 1.0, 0.005], "balls": [1.0, 1.0, 1.0]}[shape]
    sc.scales = sc.scales * torch.tensor(thin) * (3.0 if shape != "balls" else 1.0)
    if fov < 1:                                    # on the axis of the view, or nothing is met
        sc.positions = sc.positions * torch.tensor([1.0, 1e-4, 1e-4])
    eye = (0.05, -0.03, 0.02) if inside else (4.0, 0.0, 0.0)
    cam = scenes.SimpleCamera(eye, target=(-1.0, 0.0, 0.0), fovx=math.radians(fov), fovy=math.radians(fov * 0.9), width=width, height=height)
    tens = [t.to(dev).contiguous() for t in sc.tensors()]
    cam.to(dev)
    cs = ro.camera_struct(cam)
    r = ro.get_renderer()
    r.build(*tens[:4])
    got = {}
    for label, flags in (("lists", 0), ("per_ray", _lib.FLAG_PER_RAY_SEARCH)):
        r.reset_counters()
        rgb, alpha, dist = r.forward(*tens, cs, r._march(0.01, True, 1200, False, 1e-3, None, height, flags | _lib.FLAG_COUNT_WORK),
                                     want_alpha=True, want_depth=True)
        got[label] = (rgb.clone(), alpha.clone(), dist.clone(), r.read_counters())
    for k in ("rays", "slabs", "slabs_hit", "closest_queries", "hits", "hits_hash", "overflow_slabs"):
        assert got["lists"][3][k] == got["per_ray"][3][k], k
    assert got["lists"][3]["hits"] > 0
    # Hits are met in another order: the sums' last bits differ, T with them, and the spacing of the next samples.  A sample at the rim may
    # then fall on the other side: there the density is the threshold that truncates a Gaussian, so the pixel moves by no more than that
    # times the largest spacing, 4 dt (the distance by that times the ray's length, below 10); a handful of rays in a hundred thousand.
    rim = 0.1 * 4 * 0.01
    for a, b, tol, most in zip(got["lists"][:3], got["per_ray"][:3], (1e-5, 1e-5, 1e-4), (rim, rim, 10 * rim)):
        d = (a - b).abs()
        assert d.max().item() < most and (d > tol).float().mean().item() < 1e-3


@pytest.mark.parametrize("thin", [[1.0, 1e-3, 1e-3], [1.0, 1.0, 1e-3], [1.0, 0.1, 3e-4]])
def test_gaussians_nearest_at_the_eye_are_not_taken_to_lie_behind_it(thin):
    """Needles and discs of a thousand to one that hold the eye and are closest to the ray right there: whether that is in front or behind is
    decided by rounding, and has to be decided by the march, not by the lists."""
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from raygaussx_b200 import render_optix as ro
    dev = torch.device("cuda")
    n = 1500
    sc = scenes.tiny_scene(n=n, width=1, height=1, seed=11)
    g = torch.Generator().manual_seed(5)
    q = torch.randn(n, 4, generator=g)
    sc.quaternions = q / q.norm(dim=1, keepdim=True)
    sc.scales = torch.tensor(thin).repeat(n, 1) * torch.exp(0.3 * torch.randn(n, 1, generator=g))
    sc.densities = torch.full((n,), 0.3)
    w, x, y, z = sc.quaternions.double().unbind(1)
    rows = [1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
            2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]
    turn, s = torch.stack(rows, 1).reshape(n, 3, 3), sc.scales.double()
    along = turn[:, 0, :] / s                                  # the ray's direction (1, 0, 0), in the frame of the Gaussian
    off = torch.randn(n, 3, generator=g).double()
    off = off - (off * along).sum(1, keepdim=True) / (along * along).sum(1, keepdim=True) * along
    off = 0.9 * off / off.norm(dim=1, keepdim=True)            # the eye there: at right angles to the ray
    sc.positions = -(turn @ (off * s)[:, :, None])[:, :, 0].float()
    cam = scenes.SimpleCamera((0.0, 0.0, 0.0), target=(1.0, 0.0, 0.0), width=1, height=1).to(dev)
    cs = ro.camera_struct(cam)
    tens = [t.to(dev).contiguous() for t in sc.tensors()]
    r = ro.Renderer(dev)
    r.build(*tens[:4])
    got = []
    for flags in (0, _lib.FLAG_PER_RAY_SEARCH):
        r.reset_counters()
        r.forward(*tens, cs, r._march(0.01, False, 4096, False, 1e-3, None, 1, flags | _lib.FLAG_COUNT_WORK))
        got.append(r.read_counters())
    assert got[0]["hits"] > n // 4
    for k in ("rays", "slabs", "slabs_hit", "closest_queries", "hits", "hits_hash", "overflow_slabs"):
        assert got[0][k] == got[1][k], k
